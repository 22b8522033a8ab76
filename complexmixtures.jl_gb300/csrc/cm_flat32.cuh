// cm_flat32.cuh -- FP32 real pass of the PAIRS layout with one lane per
// solvent atom.
//
// One warp per (frame, solute molecule) work item.  The warp walks the cell
// stencil row by row; in self mode only the forward half (the own cell with
// v > s, then the cells whose offset is positive in (z, y, x) order), so every
// unordered molecule pair is met once.  The cells of a stencil row are
// consecutive in the cell-sorted molecule table, so a row is one or two
// contiguous ranges of it; a lane finds the x offset of its molecule's cell by
// comparing its position with the row's cell starts.  A solvent molecule is a
// candidate if its bounding sphere reaches the solute's.
//
// Each batch of up to 32 candidates is expanded into its atoms; an atom
// farther than cutoff + solute radius from the solute centroid cannot hold a
// pair within the cutoff and is dropped.  The remaining atoms are evaluated 32
// at a time, one per lane, against the solute atoms in shared memory (two
// solute atoms per instruction), and the lanes fold their rows into
// per-candidate slots with shared-memory atomics:
//   k1  the smallest row (d^2 bits, the solvent atom in the lowest five),
//   m2  the second-smallest row (by displacement: old = atomicMin(k1, key);
//       atomicMin(m2, max(old, key))),
//   r1  d^2 of the solvent molecule's reference atom to the closest solute atom,
//   r2  (self) d^2 of the solute molecule's reference atom to the closest atom
//       of the solvent molecule.
// Lane c then goes through candidate c's winning row again for the solute
// atom and the second-smallest distance, and decides: records inside the
// guard band of the cutoff, of a bin edge or of dbulk, or with a
// second-closest pair within 2 delta of the closest, go to the guard queue
// for the exact FP64 rules.
//
// On 10,000 14-atom molecules (cutoff 10 A, 64 frames) the tiled real pass
// took 10,220 us with 64-bit keys that carried the solute atom through every
// row (eleven operations a pair), 8,000 us so; its counters: 61 % issue, 74 %
// of the L1 port (gathers of the candidates' atoms and the shared-memory
// traffic of the queues).
#pragma once
#include "cm_kernels.cuh"

namespace cmk {

// Two CTAs of 12 warps per SM at 80 registers.  At 64 registers (one CTA of 32
// warps) the batch spills 170 bytes: 174 us instead of 130 on 181 14-atom
// molecules in 19,338 waters, 20 frames; three CTAs of 8 warps 132.
#ifndef CM_FLAT_WARPS
#define CM_FLAT_WARPS 12
#endif
#ifndef CM_FLAT_MIN_CTAS
#define CM_FLAT_MIN_CTAS 2
#endif
constexpr int kFlatWarps = CM_FLAT_WARPS;  // warps per CTA
constexpr int kAtomQueue = 64;   // per-warp atom queue (float4: t, tag)

// The 32 candidates' fold slots, one array per field: the lanes of a flush
// hold different candidates, and their atomics then fall on distinct banks.
struct CandSlots {
    unsigned int k1[32], m2[32], r1[32], r2[32];
};

constexpr unsigned kNoRow = 0xffffffffu;
constexpr unsigned kRowBits = 31u;  // the low bits of a row's key hold the solvent atom (kMaxSmallMol = 32)

// Shared memory of one warp after the histograms.
struct FlatWarpSmem {
    float4 oxy[kMaxSmallMol / 2];  // solute atom offsets, negated, two atoms (a, a + 1): -x, -x', -y, -y'
    float2 oz[kMaxSmallMol / 2];   // -z, -z'
    float4 oref;                   // the reference atom's offset, negated
    float4 aq[kAtomQueue];         // atom queue (circular): t = position relative to the solute centroid, w = tag c << 8 | b
    float4 cq[kQueue];             // candidate queue: D = centroid displacement, w = molecule index
    int cc[kQueue];                // candidate queue: packed cell offset | 1 << 31: may be sampled
    CandSlots cand;
};

__host__ __device__ constexpr size_t flat_warp_smem() { return sizeof(FlatWarpSmem); }

// Two FP32 operations per instruction (each IEEE round to nearest, as the
// scalar ones).
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// The solute molecule's offsets into the warp's shared memory (negated pairs;
// the odd atom's partner lies beyond every cutoff).
__device__ __forceinline__ void load_solute(FlatWarpSmem &W, const float4 *so, int aps, int iref, int lane) {
    for (int i = lane; 2 * i < aps; i += 32) {
        const float4 u = so[2 * i];
        const float4 v = 2 * i + 1 < aps ? so[2 * i + 1] : make_float4(-1e18f, -1e18f, -1e18f, 0.f);
        W.oxy[i] = make_float4(-u.x, -v.x, -u.y, -v.y);
        W.oz[i] = make_float2(-u.z, -v.z);
        if (iref >> 1 == i) W.oref = iref & 1 ? make_float4(-v.x, -v.y, -v.z, 0.f) : make_float4(-u.x, -u.y, -u.z, 0.f);
    }
}

// Squared distances of t to the two solute atoms of pair i.
struct T2 {
    unsigned long long x, y, z;
};
__device__ __forceinline__ unsigned long long d2_pair(const FlatWarpSmem &W, const T2 &t, int i) {
    const float4 xy = W.oxy[i];
    const float2 z = W.oz[i];
    const unsigned long long ex = add2(t.x, pack2(xy.x, xy.y)), ey = add2(t.y, pack2(xy.z, xy.w)),
                             ez = add2(t.z, pack2(z.x, z.y));
    return fma2(ez, ez, fma2(ey, ey, mul2(ex, ex)));
}

// Evaluate n queued atoms from `head` on (one per lane): each lane's smallest
// squared distance to the solute atoms, its row, is folded into its
// candidate's slots.  k1 keeps the smallest row and m2 the second-smallest, as
// the row's bits with the solvent atom in the five lowest: a lower bound of
// the row, 2^-18 below it at most.  Which solute atom it was, and the
// second-smallest distance inside the row, is left to the candidate's winning
// row (flat_decide), so the loop is three packed operations and a minimum per
// atom pair.  APS > 0 is the compile-time solute molecule size.
template <bool SELF, int APS, bool IMAGES>
__device__ __forceinline__ void flat_flush(const DevSys &S, FlatWarpSmem &W, int head, int n, int lane, LocalStats &st) {
    if (lane < n) {
        const float4 e = W.aq[(head + lane) & (kAtomQueue - 1)];
        const int tag = __float_as_int(e.w);
        const int c = tag >> 8, b = tag & 0xff;
        const T2 t{pack2(e.x, e.x), pack2(e.y, e.y), pack2(e.z, e.z)};
        float ma = INFINITY, mb = INFINITY;
        const int aps = APS > 0 ? APS : S.aps;
        if (APS > 0) {
#pragma unroll
            for (int i = 0; i < (APS + 1) / 2; ++i) {
                float lo, hi;
                unpack2(d2_pair(W, t, i), lo, hi);
                ma = fminf(ma, lo);
                mb = fminf(mb, hi);
            }
        } else {
#pragma unroll 2
            for (int i = 0; 2 * i < aps; ++i) {
                float lo, hi;
                unpack2(d2_pair(W, t, i), lo, hi);
                ma = fminf(ma, lo);
                mb = fminf(mb, hi);
            }
        }
        const unsigned row = __float_as_uint(fminf(ma, mb));
        st.atompairs += (unsigned long long)aps;
        CandSlots &C = W.cand;
        const unsigned key = (row & ~kRowBits) | (unsigned)b;
        const unsigned old = atomicMin(&C.k1[c], key);
        atomicMin(&C.m2[c], max(old, key));
        if (b == S.iref) {
            if (IMAGES) atomicMin(&C.r1[c], row);  // a row per image
            else C.r1[c] = row;
        }
        if (SELF) {
            const float4 o = W.oref;
            const float dx = e.x + o.x, dy = e.y + o.y, dz = e.z + o.z;
            atomicMin(&C.r2[c], __float_as_uint(fmaf(dz, dz, fmaf(dy, dy, dx * dx))));
        }
    }
    __syncwarp();
}

// The record of a molecule pair from its FP32 pass: the smallest squared
// distance m1 and its atoms (a1, b1), the second-smallest m2, the solvent
// reference atom's row r1 and (self) the solute reference atom's column r2.
// sslot: the solute molecule's row of the bulk flags, -1 if it is not sampled;
// vsampled: (self) the solvent molecule may be sampled.
template <bool SELF>
__device__ __forceinline__ void decide_pair(const DevSys &S, const Bufs &B, const SHist &h, const PairsFrame &Pf,
                                            const Guard &g, int f, int s, int sslot, bool vsampled, int v, int code, float m1, float m2,
                                            int a1, int b1, float r1, float r2, LocalStats &st) {
    if (m1 > g.cutp2) return;  // no atom pair within the cutoff
    const float dmin = sqrtf(m1);
    // hard: the closest pair, or the cutoff or dbulk decision, needs the full
    // FP64 rules (guard queue)
    const float d2nd = __fadd_ru(dmin, g.two_delta);
    bool hard = m1 >= g.cutm2 || m2 <= __fmul_ru(d2nd, d2nd);
    if (S.usecutoff) hard = hard || (dmin >= g.dbulk_lo && dmin <= g.dbulk_hi);
    if (hard) {
        // past the capacity the record is dropped and k_queue_check has the
        // chunk redone without queues
        const int slot = atomicAdd(B.counters + 0, 1);
        if (slot < B.gq_cap) B.gq[slot] = make_int4(s, v, code, f);
        return;
    }
    // otherwise each of the md bin, the solvent reference-atom row and (self)
    // the solute reference-atom column is decided here, or marked -2 when it
    // lies within the guard band of a bin edge or of the cutoff: the edge
    // kernel then computes it from FP64 pair distances
    int bin = bin32(g, dmin);
    if (bin < 0) bin = -2;
    int rb1 = -1, rb2 = -1;
    if (r1 <= g.cutp2) {
        rb1 = r1 < g.cutm2 ? bin32(g, sqrtf(r1)) : -1;
        if (rb1 < 0) rb1 = -2;
    }
    if (SELF && r2 <= g.cutp2) {
        rb2 = r2 < g.cutm2 ? bin32(g, sqrtf(r2)) : -1;
        if (rb2 < 0) rb2 = -2;
    }
    if (bin == -2 || rb1 == -2 || rb2 == -2) {
        const int slot = atomicAdd(B.counters + 3, 1);
        if (slot < B.eq_cap) {
            B.eq[3 * slot] = make_int4(s, v, code, f);
            B.eq[3 * slot + 1] = make_int4(a1 | b1 << 8, rb1, rb2, bin);
            B.eq[3 * slot + 2] = make_int4(__float_as_int(dmin), 0, 0, 0);
        }
        return;
    }
    const int bulk = S.usecutoff ? (dmin > g.dbulk_hi) : 0;
    if (SELF) {
        apply_pair_self(S, h, bin, a1, (int64_t)s * S.aps + a1, b1, (int64_t)v * S.apv + b1, rb1 >= 0, rb1, rb2 >= 0, rb2);
        st.hits += 2;
    } else {
        apply_hit_local(S, h, false, bin, a1, (int64_t)v * S.apv + b1, b1, rb1 >= 0, rb1);
        st.hits++;
    }
    if (Pf.slot) {
        const unsigned char code1 = (unsigned char)(1 + bulk);
        if (sslot >= 0) Pf.flags[(int64_t)sslot * S.mv + v] = code1;
        if (SELF && vsampled) {
            const int vs = Pf.slot[v];
            if (vs >= 0) Pf.flags[(int64_t)vs * S.mv + s] = code1;
        }
    }
}

__device__ __forceinline__ void cand_slots_clear(CandSlots &C, int lane) {
    C.k1[lane] = kNoRow;
    C.m2[lane] = kNoRow;
    C.r1[lane] = 0x7f800000u;
    C.r2[lane] = 0x7f800000u;
}

// The atoms of the first nc (<= 32) entries of the warp's candidate queue
// against the solute.  An entry folds into the slot of its place in the queue
// or (IMAGES) into the slot W.cc names.  The expansion takes two adjacent
// atoms of every entry at a time: one 32-byte sector per load and entry (the
// gathers through the SM's L1 port weigh most), and the lanes of one flush
// hold at most two atoms of an entry, so their shared-memory atomics rarely
// meet on one slot.
template <bool SELF, int APS, bool IMAGES>
__device__ __forceinline__ void flat_expand(const DevSys &S, FlatWarpSmem &W, const PairsFrame &Pf, float rs2, int lane, int nc,
                                            LocalStats &st) {
    const int apv = S.apv;
    // 2^sh lanes per entry: two in a full batch, whose entries go in two halves
    // (the lanes of entry i, then of 16 + i), more in a short one
    const bool two = nc > 16;
    const int sh = two ? 1 : max(1, min(5, __clz(nc - 1) - 27));
    const int ci = lane >> sh, sub = lane & ((1 << sh) - 1);
    const int i0 = ci < nc ? ci : 0, i1 = two && 16 + ci < nc ? 16 + ci : 0;
    const float4 D0 = W.cq[i0], D1 = W.cq[i1];
    const int s0 = IMAGES ? W.cc[i0] : ci, s1 = IMAGES ? W.cc[i1] : 16 + ci;
    const float4 *o0 = Pf.vo32 + (int64_t)__float_as_int(D0.w) * apv, *o1 = Pf.vo32 + (int64_t)__float_as_int(D1.w) * apv;
    int head = 0, nq = 0;
    auto queue = [&](const float4 &t, bool keep) {
        const unsigned mask = __ballot_sync(0xffffffffu, keep);
        if (keep) W.aq[(head + nq + __popc(mask & ((1u << lane) - 1u))) & (kAtomQueue - 1)] = t;
        nq += __popc(mask);
        if (nq >= 32) {
            __syncwarp();
            flat_flush<SELF, APS, IMAGES>(S, W, head, 32, lane, st);
            head += 32;
            nq -= 32;
        }
    };
    for (int b0 = 0; b0 < apv; b0 += 1 << sh) {
        const int b = b0 + sub;
        const int bl = b < apv ? b : b0;
        const float4 oa = o0[bl];
        float4 ob = make_float4(0.f, 0.f, 0.f, 0.f);
        if (two) ob = o1[bl];
        const float4 t0 = make_float4(D0.x + oa.x, D0.y + oa.y, D0.z + oa.z, __int_as_float(s0 << 8 | b));
        queue(t0, ci < nc && b < apv && fmaf(t0.z, t0.z, fmaf(t0.y, t0.y, t0.x * t0.x)) <= rs2);
        if (two) {
            const float4 t1 = make_float4(D1.x + ob.x, D1.y + ob.y, D1.z + ob.z, __int_as_float(s1 << 8 | b));
            queue(t1, 16 + ci < nc && b < apv && fmaf(t1.z, t1.z, fmaf(t1.y, t1.y, t1.x * t1.x)) <= rs2);
        }
    }
    __syncwarp();
    if (nq > 0) flat_flush<SELF, APS, IMAGES>(S, W, head, nq, lane, st);
}

// The winning row of a slot again, against every solute atom: the smallest
// distance of t with its atom, and the second-smallest.
template <int APS>
__device__ __forceinline__ void winning_row(const DevSys &S, const FlatWarpSmem &W, float tx, float ty, float tz, float &m1,
                                            float &m2, int &a1) {
    const T2 t{pack2(tx, tx), pack2(ty, ty), pack2(tz, tz)};
    const int aps = APS > 0 ? APS : S.aps;
#pragma unroll 2
    for (int i = 0; 2 * i < aps; ++i) {
        float lo, hi;
        unpack2(d2_pair(W, t, i), lo, hi);
        m2 = fminf(m2, fmaxf(m1, lo));
        a1 = lo < m1 ? 2 * i : a1;
        m1 = fminf(m1, lo);
        m2 = fminf(m2, fmaxf(m1, hi));
        a1 = hi < m1 ? 2 * i + 1 : a1;
        m1 = fminf(m1, hi);
    }
}

// One batch: the first nc (<= 32) entries of the warp's candidate queue, lane
// c candidate c.  After the expansion lane c goes through its candidate's
// winning row again, for the solute atom and the second-smallest distance in
// it, and decides.  A row whose key is not the smallest although its distance
// is (keys are truncated) leaves m2 at most its distance, which makes the
// record hard, so the winning row is the right one wherever it is used.
template <bool SELF, int APS>
__device__ __forceinline__ void flat_batch(const DevSys &S, const Bufs &B, const SHist &h, FlatWarpSmem &W,
                                           const PairsFrame &Pf, const Guard &g, int f, int s, int sslot, float rs2,
                                           int lane, int nc, LocalStats &st) {
    CandSlots &C = W.cand;
    cand_slots_clear(C, lane);
    __syncwarp();
    flat_expand<SELF, APS, false>(S, W, Pf, rs2, lane, nc, st);
    if (lane >= nc) return;
    st.molpairs++;
    const unsigned k1 = C.k1[lane];
    // no row, or (the key is a lower bound) no atom pair within the cutoff
    if (k1 == kNoRow || __uint_as_float(k1 & ~kRowBits) > g.cutp2) return;
    const int b1 = (int)(k1 & kRowBits);
    const float4 D = W.cq[lane];
    const int v = __float_as_int(D.w);
    const float4 ob = Pf.vo32[(int64_t)v * S.apv + b1];
    float m1 = INFINITY, m2 = C.m2[lane] == kNoRow ? INFINITY : __uint_as_float(C.m2[lane] & ~kRowBits);
    int a1 = 0;
    winning_row<APS>(S, W, D.x + ob.x, D.y + ob.y, D.z + ob.z, m1, m2, a1);
    const int cc = W.cc[lane];
    decide_pair<SELF>(S, B, h, Pf, g, f, s, sslot, cc < 0, v, cc & 0x7fffffff, m1, m2, a1, b1, __uint_as_float(C.r1[lane]),
                      __uint_as_float(C.r2[lane]), st);
}

__device__ __forceinline__ void image_at(const Images &im, int img, int &dx, int &dy, int &dz) {
    const int ix = img % im.cnt[0], iy = (img / im.cnt[0]) % im.cnt[1], iz = img / (im.cnt[0] * im.cnt[1]);
    dx = im.base[0] + ix * im.step[0];
    dy = im.base[1] + iy * im.step[1];
    dz = im.base[2] + iz * im.step[2];
}

// One solute molecule of a frame that needs several images per molecule pair
// (a box of less than three search cells along an axis): 32 molecules of a
// cell at a time, lane c molecule c.  An image whose molecule's bounding sphere
// reaches the solute's is an entry of the queue and folds into its molecule's
// slot, so the slots end with the values over all images.  (The generic
// kernel evaluates every atom pair of every image, one lane per molecule: 300
// 9-atom molecules in a 30 A box, cutoff 9 A, 16 frames: 5,473 us a pass with the
// generic kernel, 1,048 with this one, which spills 76 to 160 bytes at the 80
// registers of two CTAs per SM.)
template <bool SELF, int APS>
__device__ __forceinline__ void flat_images(const DevSys &S, const Bufs &B, const SHist &h, FlatWarpSmem &W,
                                            const PairsFrame &Pf, const Guard &g, int f, int s, int sslot, const float4 qs,
                                            int sc, float rsc, int part, int parts, int lane, LocalStats &st) {
    const FrameGeom &G = *Pf.G;
    const FrameScratch &F = *Pf.F;
    CandSlots &C = W.cand;
    const unsigned below = (1u << lane) - 1u;
    const int n0 = G.n[0], n1 = G.n[1], n2 = G.n[2];
    const bool m0 = F.multi & 1, m1 = F.multi & 2, m2 = F.multi & 4;
    const int e0 = m0 ? n0 : 2 * F.L[0] + 1, e1 = m1 ? n1 : 2 * F.L[1] + 1, e2 = m2 ? n2 : 2 * F.L[2] + 1;
    const int cx = sc % n0, cy = (sc / n0) % n1, cz = sc / (n0 * n1);
    const float rs2 = rsc * rsc;
    const float4 *cq32 = B.cq32 + (int64_t)f * B.mv;
    for (int ic = part; ic < e0 * e1 * e2; ic += parts) {
        const int ix = ic % e0, iy = (ic / e0) % e1, iz = ic / (e0 * e1);
        const int dx = m0 ? ix - cx : ix - F.L[0], dy = m1 ? iy - cy : iy - F.L[1], dz = m2 ? iz - cz : iz - F.L[2];
        const int xc = m0 ? ix : wrap_cell(cx + dx, n0), yc = m1 ? iy : wrap_cell(cy + dy, n1),
                  zc = m2 ? iz : wrap_cell(cz + dz, n2);
        const int cell = (zc * n1 + yc) * n0 + xc;
        const int beg = Pf.cstart[cell], end = Pf.cstart[cell + 1];
        const int code = pack_delta(dx, dy, dz);
        const Images im = images_of(G, F, code);
        const int ni = image_count(im);
        for (int p0 = beg; p0 < end; p0 += 32) {
            const int p = min(p0 + lane, end - 1);
            const float4 q = cq32[p];
            const int v = Pf.cmol[p];
            const bool valid = p0 + lane < end && (!SELF || v > s);
            const float R = rsc + q.w;
            const float bx = q.x - qs.x, by = q.y - qs.y, bz = q.z - qs.z;
            cand_slots_clear(C, lane);
            __syncwarp();
            int cnt = 0;
            unsigned mine = 0;  // the lane's images in reach, of the first 32
            for (int i = 0; i < ni; ++i) {
                int jx, jy, jz;
                image_at(im, i, jx, jy, jz);
                const float4 o = Pf.off32[off_index(jx, jy, jz)];
                const float Dx = bx + o.x, Dy = by + o.y, Dz = bz + o.z;
                const bool in = valid && fmaf(Dz, Dz, fmaf(Dy, Dy, Dx * Dx)) <= R * R;
                const unsigned mask = __ballot_sync(0xffffffffu, in);
                if (in) {
                    const int pos = cnt + __popc(mask & below);
                    W.cq[pos] = make_float4(Dx, Dy, Dz, __int_as_float(v));
                    W.cc[pos] = lane;
                    if (i < 32) mine |= 1u << i;
                }
                cnt += __popc(mask);
                if (cnt >= 32) {
                    __syncwarp();
                    flat_expand<SELF, APS, true>(S, W, Pf, rs2, lane, 32, st);
                    __syncwarp();
                    cnt -= 32;
                    float4 rq = make_float4(0.f, 0.f, 0.f, 0.f);
                    int rc = 0;
                    if (lane < cnt) {
                        rq = W.cq[32 + lane];
                        rc = W.cc[32 + lane];
                    }
                    __syncwarp();
                    if (lane < cnt) {
                        W.cq[lane] = rq;
                        W.cc[lane] = rc;
                    }
                    __syncwarp();
                }
            }
            __syncwarp();
            if (cnt > 0) flat_expand<SELF, APS, true>(S, W, Pf, rs2, lane, cnt, st);
            __syncwarp();
            if (valid) st.molpairs++;
            const unsigned k1 = C.k1[lane];
            if (valid && k1 != kNoRow && !(__uint_as_float(k1 & ~kRowBits) > g.cutp2)) {
                const int b1 = (int)(k1 & kRowBits);
                const float4 ob = Pf.vo32[(int64_t)v * S.apv + b1];
                float d1 = INFINITY, d2 = C.m2[lane] == kNoRow ? INFINITY : __uint_as_float(C.m2[lane] & ~kRowBits);
                int a1 = 0;
                // the winning atom's row in every image it was evaluated in: m2 already holds all but the smallest,
                // truncated, and those found here again only confirm it
                float e1 = INFINITY, e2 = INFINITY;
                unsigned left = ni > 32 ? 1u : mine;
                for (int i = 0; left; i += ni > 32) {
                    const int j = ni > 32 ? i : __ffs(left) - 1;
                    if (ni > 32) left = i + 1 < ni;
                    else left &= left - 1;
                    int jx, jy, jz;
                    image_at(im, j, jx, jy, jz);
                    const float4 o = Pf.off32[off_index(jx, jy, jz)];
                    const float tx = (bx + o.x) + ob.x, ty = (by + o.y) + ob.y, tz = (bz + o.z) + ob.z;
                    if (!(fmaf(tz, tz, fmaf(ty, ty, tx * tx)) <= rs2)) continue;
                    winning_row<APS>(S, W, tx, ty, tz, e1, e2, a1);
                }
                d1 = e1;
                d2 = fminf(d2, e2);
                decide_pair<SELF>(S, B, h, Pf, g, f, s, sslot, true, v, code, d1, d2, a1, b1, __uint_as_float(C.r1[lane]),
                                  __uint_as_float(C.r2[lane]), st);
            }
            __syncwarp();
        }
    }
}

// skip_tile: the frames the tiled kernel took (FrameScratch::tile) are
// skipped, and the kernel returns at once when that is every frame.
template <bool SELF, int APS>
__global__ void __launch_bounds__(kFlatWarps * 32, CM_FLAT_MIN_CTAS) k_pairs_flat32(DevSys S, Bufs B, int skip_tile) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned int *hbase = (unsigned int *)smem_raw;
    const int hw = hist_words(S);
    FlatWarpSmem *wsm = (FlatWarpSmem *)(smem_raw + (((size_t)hw * 4 + 15) & ~(size_t)15));
    if (skip_tile) {
        int any = 0;
        for (int f = threadIdx.x; f < B.nf; f += blockDim.x) any |= (B.FS[f].tile == 0);
        if (!__syncthreads_or(any)) return;
    }
    shist_zero(S, hbase);
    __syncthreads();
    SHist h = shist_bind(S, hbase);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    FlatWarpSmem &W = wsm[warp];
    LocalStats st;
    const int aps = S.aps;
    const int64_t items = (int64_t)B.nf * B.ms;
    for (int64_t t = (int64_t)blockIdx.x * kFlatWarps + warp; t < items; t += (int64_t)gridDim.x * kFlatWarps) {
        const int f = (int)(t / B.ms), s = (int)(t - (int64_t)f * B.ms);
        const PairsFrame Pf = pairs_frame(B, f, SELF);
        const FrameScratch &F = *Pf.F;
        if (!F.ok) {
            if (lane == 0) raise_err(S, ERR_STENCIL);
            continue;
        }
        if (F.multi) continue;  // several images per pair: k_pairs_images32 takes the frame
        if (skip_tile && F.tile) continue;
        const FrameGeom &G = *Pf.G;
        const Guard g = F.g;
        const float4 qs = Pf.sq32[s];
        const int sc = Pf.scell[s];
        const int sslot = Pf.slot ? Pf.slot[s] : -1;
        __syncwarp();
        load_solute(W, Pf.so32 + (int64_t)s * aps, aps, S.iref, lane);
        __syncwarp();
        const float rsc = g.cut_pre + qs.w;     // candidate molecules: centroid within rsc + r_v
        const float rs2 = rsc * rsc;            // candidate atoms: within rsc of the solute centroid
        const float4 *cq32 = B.cq32 + (int64_t)f * B.mv;
        const int *cmol = Pf.cmol;
        const int *cstart = Pf.cstart;
        const int n0 = G.n[0], n1 = G.n[1], n2 = G.n[2];
        const int cx = sc % n0, cyz = sc / n0, cy = cyz % n1, cz = cyz / n1;
        const int L0 = F.L[0], L1 = F.L[1], L2 = F.L[2];
        int cnt = 0;
        for (int dz = SELF ? 0 : -L2; dz <= L2; ++dz) {
            int zc = cz + dz;
            zc = zc < 0 ? zc + n2 : (zc >= n2 ? zc - n2 : zc);
            for (int dy = (SELF && dz == 0) ? 0 : -L1; dy <= L1; ++dy) {
                int yc = cy + dy;
                yc = yc < 0 ? yc + n1 : (yc >= n1 ? yc - n1 : yc);
                const int row = (zc * n1 + yc) * n0;
                const bool own_row = SELF && dz == 0 && dy == 0;
                // the row's stencil offsets, lane j holding dx = j - L0
                float4 rowoff = make_float4(0.f, 0.f, 0.f, 0.f);
                if (lane <= 2 * L0) rowoff = Pf.off32[off_index(lane - L0, dy, dz)];
                // unwrapped x range of the row, split at the box edges into
                // contiguous pieces of the cell-sorted table
                const int ulo = cx + (own_row ? 0 : -L0), uhi = cx + L0;
                for (int piece = 0; piece < 3; ++piece) {
                    const int plo = piece == 0 ? ulo : (piece == 1 ? max(ulo, 0) : max(ulo, n0));
                    const int phi = piece == 0 ? min(uhi, -1) : (piece == 1 ? min(uhi, n0 - 1) : uhi);
                    if (plo > phi) continue;
                    const int shift = piece == 0 ? n0 : (piece == 1 ? 0 : -n0);
                    const int first = row + plo + shift;          // first cell of the piece
                    const int ncell = phi - plo + 1;
                    const int beg = cstart[first], end = cstart[first + ncell];
                    if (beg == end) continue;
                    // cell starts inside the piece, one per lane
                    const int bnd = lane + 1 < ncell ? cstart[first + lane + 1] : 0x7fffffff;
                    for (int p0 = beg; p0 < end; p0 += 32) {
                        const int p = p0 + lane;
                        const bool in = p < end;
                        const int pc = in ? p : end - 1;
                        const float4 q = cq32[pc];
                        const int v = cmol[pc];
                        int k = 0;  // cells of the piece that start at or before p
                        for (int j = 0; j + 1 < ncell; ++j) k += p >= __shfl_sync(0xffffffffu, bnd, j) ? 1 : 0;
                        const int dx = plo + k - cx;
                        const int src = dx + L0;
                        const float ox = __shfl_sync(0xffffffffu, rowoff.x, src);
                        const float oy = __shfl_sync(0xffffffffu, rowoff.y, src);
                        const float oz = __shfl_sync(0xffffffffu, rowoff.z, src);
                        float4 Dv;
                        Dv.x = (q.x - qs.x) + ox;
                        Dv.y = (q.y - qs.y) + oy;
                        Dv.z = (q.z - qs.z) + oz;
                        Dv.w = __int_as_float(v);
                        const float rr = rsc + q.w;
                        const bool cand = in && fmaf(Dv.z, Dv.z, fmaf(Dv.y, Dv.y, Dv.x * Dv.x)) <= rr * rr &&
                                          !(own_row && dx == 0 && v <= s);
                        const unsigned mask = __ballot_sync(0xffffffffu, cand);
                        const int pos = cnt + __popc(mask & ((1u << lane) - 1u));
                        if (cand) {
                            W.cq[pos] = Dv;
                            W.cc[pos] = pack_delta(dx, dy, dz) | 0x80000000;
                        }
                        cnt += __popc(mask);
                        if (cnt >= 32) {
                            __syncwarp();
                            flat_batch<SELF, APS>(S, B, h, W, Pf, g, f, s, sslot, rs2, lane, 32, st);
                            __syncwarp();
                            float4 rq = make_float4(0.f, 0.f, 0.f, 0.f);
                            int rc = 0;
                            if (lane < cnt - 32) {
                                rq = W.cq[32 + lane];
                                rc = W.cc[32 + lane];
                            }
                            __syncwarp();
                            if (lane < cnt - 32) {
                                W.cq[lane] = rq;
                                W.cc[lane] = rc;
                            }
                            cnt -= 32;
                            __syncwarp();
                        }
                    }
                }
            }
        }
        __syncwarp();
        if (cnt > 0) flat_batch<SELF, APS>(S, B, h, W, Pf, g, f, s, sslot, rs2, lane, cnt, st);
        __syncwarp();
    }
    stats_flush(S, st, false);
    __syncthreads();
    shist_flush(S, h, false);
}

// The frames that need several images per molecule pair, `parts` warps per
// (frame, solute molecule), each on every parts-th cell; returns at once when
// the chunk has none.
template <bool SELF, int APS>
__global__ void __launch_bounds__(kFlatWarps * 32, CM_FLAT_MIN_CTAS) k_pairs_images32(DevSys S, Bufs B, int parts) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned int *hbase = (unsigned int *)smem_raw;
    FlatWarpSmem *wsm = (FlatWarpSmem *)(smem_raw + (((size_t)hist_words(S) * 4 + 15) & ~(size_t)15));
    int any = 0;
    for (int f = threadIdx.x; f < B.nf; f += blockDim.x) any |= B.FS[f].multi;
    if (!__syncthreads_or(any)) return;
    shist_zero(S, hbase);
    __syncthreads();
    const SHist h = shist_bind(S, hbase);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    FlatWarpSmem &W = wsm[warp];
    LocalStats st;
    const int64_t items = (int64_t)B.nf * B.ms * parts;
    for (int64_t t = (int64_t)blockIdx.x * kFlatWarps + warp; t < items; t += (int64_t)gridDim.x * kFlatWarps) {
        const int part = (int)(t % parts);
        const int f = (int)(t / parts / B.ms), s = (int)(t / parts - (int64_t)f * B.ms);
        const PairsFrame Pf = pairs_frame(B, f, SELF);
        const FrameScratch &F = *Pf.F;
        if (!F.ok || !F.multi) continue;
        const Guard g = F.g;
        const float4 qs = Pf.sq32[s];
        __syncwarp();
        load_solute(W, Pf.so32 + (int64_t)s * S.aps, S.aps, S.iref, lane);
        __syncwarp();
        flat_images<SELF, APS>(S, B, h, W, Pf, g, f, s, Pf.slot ? Pf.slot[s] : -1, qs, Pf.scell[s], g.cut_pre + qs.w, part,
                               parts, lane, st);
    }
    stats_flush(S, st, false);
    __syncthreads();
    shist_flush(S, h, false);
}

// ------------------------------------------------------------ tiled real pass
// Self mode.  The stencil walk of k_pairs_flat32 gathers each neighbour
// cell's molecule table from L2 once per solute molecule, one warp per
// molecule, and was most of that kernel's time.  Here a CTA takes one home
// cell: it stages the molecules of the cell's half stencil (the home cell,
// its row forward, the rest of its plane forward, the planes above) in
// shared memory once -- each as its cell-relative centroid plus the cell's
// stencil offset, with its radius and, packed with its index, the staged
// cell -- and its warps then claim the home cell's molecules one by one and
// test each against the whole staged table, 32 candidates per round.  The
// candidates then go through flat_batch exactly as in k_pairs_flat32 (the
// displacement is formed as (q_v + off) - q_s, an order the guard band
// covers), so the records, and the guard and edge queues, are the same.
#ifndef CM_TILE_WARPS
#define CM_TILE_WARPS 12
#endif
#ifndef CM_TILE_MIN_CTAS
#define CM_TILE_MIN_CTAS 2
#endif
constexpr int kTileWarps = CM_TILE_WARPS;
constexpr int kTileStage = 1024;  // staged neighbour molecules per pass

// The half-stencil cells of a home cell.
struct TileCellTab {
    int nbeg[kTileCells + 1];   // first staged position of each cell (prefix of the cells' molecule counts)
    int cbeg[kTileCells];       // the cell's first position in the cell-sorted molecule table
    int code[kTileCells];       // the cell's packed stencil offset
};

struct TileSmem {
    float4 w[kTileStage];       // staged molecule: centroid + stencil offset (x, y, z), half its square
    int v[kTileStage];          // molecule index | staged cell << 24 | sampled << 31
    TileCellTab c;
    int next;                   // next home molecule to claim
    int item;                   // the CTA's current (frame, home cell) item
};

__host__ __device__ constexpr size_t tile_smem_extra() { return sizeof(TileSmem) + 16; }

// Stencil offset of half-stencil cell k: the home cell's row forward
// (k <= L0), the rest of its plane forward, then the planes above.
__device__ __forceinline__ void half_stencil_cell(int k, const int *L, int &dx, int &dy, int &dz) {
    const int wx = 2 * L[0] + 1;
    if (k <= L[0]) {
        dx = k; dy = 0; dz = 0;
        return;
    }
    k -= L[0] + 1;
    if (k < wx * L[1]) {
        dy = 1 + k / wx; dx = k % wx - L[0]; dz = 0;
        return;
    }
    k -= wx * L[1];
    const int wxy = wx * (2 * L[1] + 1);
    dz = 1 + k / wxy;
    const int r = k % wxy;
    dy = r / wx - L[1];
    dx = r % wx - L[0];
}

// Fill the cell table of home cell (cx, cy, cz), K <= kTileCells cells; every
// thread of the CTA calls it (two barriers).
__device__ __forceinline__ void tile_cells(const FrameGeom &G, const FrameScratch &F, const int *cstart, int cx, int cy,
                                           int cz, int K, TileCellTab &T) {
    const int tid = threadIdx.x, lane = tid & 31;
    const int n0 = G.n[0], n1 = G.n[1], n2 = G.n[2];
    if (tid < K) {
        int dx, dy, dz;
        half_stencil_cell(tid, F.L, dx, dy, dz);
        const int c = (wrap_cell(cz + dz, n2) * n1 + wrap_cell(cy + dy, n1)) * n0 + wrap_cell(cx + dx, n0);
        T.cbeg[tid] = cstart[c];
        T.nbeg[tid + 1] = cstart[c + 1] - cstart[c];
        T.code[tid] = pack_delta(dx, dy, dz);
    }
    if (tid == 0) T.nbeg[0] = 0;
    __syncthreads();
    if (tid < 32) {
        // inclusive prefix of the K <= kTileCells counts, four per lane
        int c[4], sum = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = 4 * lane + j;
            c[j] = k < K ? T.nbeg[k + 1] : 0;
            sum += c[j];
        }
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        int run = incl - sum;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = 4 * lane + j;
            run += c[j];
            if (k < K) T.nbeg[k + 1] = run;
        }
    }
    __syncthreads();
}

// Staged molecule m of the table: its cell k and its position in the
// cell-sorted molecule table.
__device__ __forceinline__ int tile_molecule(const TileCellTab &T, int K, int m, int &k) {
    int lo = 0, hi = K;  // the cell with nbeg[k] <= m < nbeg[k + 1]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (T.nbeg[mid] <= m) lo = mid;
        else hi = mid;
    }
    k = lo;
    return T.cbeg[lo] + (m - T.nbeg[lo]);
}

// Stage n molecules of the half stencil from position m0 on, up to the next
// multiple of 32 with entries that are no candidates; the CTA's threads share them.
template <typename TILE>
__device__ __forceinline__ void tile_stage(TILE &T, const PairsFrame &Pf, const FrameScratch &F, const float4 *cq32, int K, int m0,
                                           int n) {
    for (int i = threadIdx.x; i < ((n + 31) & ~31); i += blockDim.x) {
        if (i >= n) {
            T.w[i] = make_float4(0.f, 0.f, 0.f, INFINITY);
            continue;
        }
        int k, dx, dy, dz;
        const int p = tile_molecule(T.c, K, m0 + i, k);
        half_stencil_cell(k, F.L, dx, dy, dz);
        const float4 of = Pf.off32[off_index(dx, dy, dz)];
        const float4 q = cq32[p];
        const float x = q.x + of.x, y = q.y + of.y, z = q.z + of.z;
        T.w[i] = make_float4(x, y, z, 0.5f * fmaf(z, z, fmaf(y, y, x * x)));
        const int v = Pf.cmol[p];
        T.v[i] = v | (k << 24) | (Pf.slot && Pf.slot[v] >= 0 ? 0x80000000 : 0);
    }
}

template <int APS>
__global__ void __launch_bounds__(kTileWarps * 32, CM_TILE_MIN_CTAS) k_pairs_tile32(DevSys S, Bufs B) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned int *hbase = (unsigned int *)smem_raw;
    const int hw = hist_words(S);
    FlatWarpSmem *wsm = (FlatWarpSmem *)(smem_raw + (((size_t)hw * 4 + 15) & ~(size_t)15));
    TileSmem &T = *(TileSmem *)(((uintptr_t)(wsm + kTileWarps) + 15) & ~(uintptr_t)15);
    shist_zero(S, hbase);
    __syncthreads();
    SHist h = shist_bind(S, hbase);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
    const unsigned below = (1u << lane) - 1u;
    FlatWarpSmem &W = wsm[warp];
    LocalStats st;
    const int aps = S.aps;
    const int64_t ncap = B.cs - 1;
    const int64_t items = (int64_t)B.nf * ncap;
    // CTAs claim (frame, home cell) items from counters[6] (zeroed with the
    // chunk's counters): the items' costs vary with the cells' occupancy
    for (;;) {
        __syncthreads();  // the previous item's staged table and claim are no longer read
        if (tid == 0) T.item = atomicAdd(B.counters + 6, 1);
        __syncthreads();
        const int64_t t = T.item;
        if (t >= items) break;
        const int f = (int)(t / ncap), H = (int)(t - (int64_t)f * ncap);
        const PairsFrame Pf = pairs_frame(B, f, true);
        const FrameScratch &F = *Pf.F;
        const FrameGeom &G = *Pf.G;
        // every thread takes the same branches: the conditions depend on the item only
        if (!F.ok || !F.tile || H >= G.ncell) continue;
        const int hbeg = Pf.cstart[H], nH = Pf.cstart[H + 1] - hbeg;
        if (nH == 0) continue;
        const int n0 = G.n[0], n1 = G.n[1];
        const int cx = H % n0, cy = (H / n0) % n1, cz = H / (n0 * n1);
        const int K = (F.L[0] + 1) + (2 * F.L[0] + 1) * F.L[1] + (2 * F.L[0] + 1) * (2 * F.L[1] + 1) * F.L[2];
        const Guard g = F.g;
        const float4 *cq32 = B.cq32 + (int64_t)f * B.mv;
        tile_cells(G, F, Pf.cstart, cx, cy, cz, K, T.c);
        const int M = T.c.nbeg[K];
        for (int m0 = 0; m0 < M; m0 += kTileStage) {
            const int n = min(kTileStage, M - m0), nr = (n + 31) & ~31;
            if (m0 > 0) __syncthreads();  // the previous pass's table is no longer read
            tile_stage(T, Pf, F, cq32, K, m0, n);
            if (tid == 0) T.next = 0;
            __syncthreads();
            // the home molecules, claimed one at a time
            for (;;) {
                int sl = 0;
                if (lane == 0) sl = atomicAdd(&T.next, 1);
                sl = __shfl_sync(0xffffffffu, sl, 0);
                if (sl >= nH) break;
                const int s = Pf.cmol[hbeg + sl];
                const float4 qs = Pf.sq32[s];
                const int sslot = Pf.slot ? Pf.slot[s] : -1;
                __syncwarp();
                load_solute(W, Pf.so32 + (int64_t)s * aps, aps, S.iref, lane);
                __syncwarp();
                const float rsc = g.cut_pre + qs.w;
                const float rs2 = rsc * rsc;
                const float R = rsc + F.rmax_s;
                const float thr = 0.5f * (R * R - fmaf(qs.z, qs.z, fmaf(qs.y, qs.y, qs.x * qs.x)));
                // within the home cell (the first staged positions) only the molecules after this one
                const int lo = max(0, sl + 1 - m0);
                int cnt = 0;
                for (int base = lo & ~31; base < nr; base += 1024) {
                    const int nj = min(32, (nr - base) >> 5);
                    unsigned bits = 0;
#pragma unroll 4
                    for (int j = 0; j < nj; ++j) {
                        const float4 w = T.w[base + 32 * j + lane];
                        if (fmaf(-w.x, qs.x, fmaf(-w.y, qs.y, fmaf(-w.z, qs.z, w.w))) <= thr) bits |= 1u << j;
                    }
                    if (base + lane < lo) bits &= ~1u;
                    for (;;) {
                        const unsigned mask = __ballot_sync(0xffffffffu, bits != 0);
                        if (mask == 0) break;
                        if (bits) {
                            const int p = base + 32 * (__ffs(bits) - 1) + lane;
                            const int pos = cnt + __popc(mask & below);
                            const float4 w = T.w[p];
                            const int vk = T.v[p];
                            W.cq[pos] = make_float4(w.x - qs.x, w.y - qs.y, w.z - qs.z, __int_as_float(vk & 0xffffff));
                            W.cc[pos] = T.c.code[(vk >> 24) & 127] | (vk & 0x80000000);
                            bits &= bits - 1;
                        }
                        cnt += __popc(mask);
                        if (cnt >= 32) {
                            __syncwarp();
                            flat_batch<true, APS>(S, B, h, W, Pf, g, f, s, sslot, rs2, lane, 32, st);
                            __syncwarp();
                            cnt -= 32;
                            float4 rq = make_float4(0.f, 0.f, 0.f, 0.f);
                            int rc = 0;
                            if (lane < cnt) {
                                rq = W.cq[32 + lane];
                                rc = W.cc[32 + lane];
                            }
                            __syncwarp();
                            if (lane < cnt) {
                                W.cq[lane] = rq;
                                W.cc[lane] = rc;
                            }
                            __syncwarp();
                        }
                    }
                }
                __syncwarp();
                if (cnt > 0) flat_batch<true, APS>(S, B, h, W, Pf, g, f, s, sslot, rs2, lane, cnt, st);
                __syncwarp();
            }
        }
    }
    stats_flush(S, st, false);
    __syncthreads();
    shist_flush(S, h, false);
}

// ----------------------------------------------- tiled real pass, small molecules
// Self mode, molecules of up to kDirectMax atoms (water).  k_pairs_tile32
// spends most of its instructions per candidate on expanding it into atoms,
// on the shared-memory folds and on batches that end with every home molecule
// (53 candidates of a water at cutoff 10: batches of 32 and 21).  A small
// molecule's few atom pairs fit one lane's registers, so here a lane takes a
// whole candidate pair, and the warp's queue holds (home molecule, staged
// molecule) pairs of any home molecules, so that its batches are full until the
// staged table changes.  The test of a home molecule against the staged
// table is |w - q|^2 <= R^2 as |w|^2 / 2 - w q <= (R^2 - |q|^2) / 2, three
// multiply-adds on a staged (w, |w|^2 / 2), R the reach of the largest
// molecule of the frame; its rounding (under 2e-3 A^2 for cells of 25 A) is far
// inside the margin of cut_pre (R times 1e-3 (1 + range), 0.15 A^2 for water),
// and a frame of much wider cells is left to k_pairs_flat32 (FrameScratch::tile).  A lane keeps its hits of up to 32 rounds in a
// bit mask; the masks are compacted into the queue afterwards.  The distances
// are formed as in flat_flush, so the records and the queues are the same.
// 19,338 waters, cutoff 10 A, 16 frames: 1,979 us in k_pairs_tile32, 746 here
// (12 or 20 warps per CTA: 801, 825); the candidates' decisions and the gathers
// of their atoms bound it (73 % issue, 69 % of the L1 port).  At 64 registers
// molecules of 3, 4 and 5 atoms spill 32, 96 and 180 bytes.
#ifndef CM_DIRECT_WARPS
#define CM_DIRECT_WARPS 16
#endif
constexpr int kDirectWarps = CM_DIRECT_WARPS;
constexpr int kDirectMax = 5;       // atoms per molecule
constexpr int kDirectStage = 1536;  // staged molecules per pass (a multiple of 32; positions take 11 bits of a queue entry)
constexpr int kDirectHome = 256;    // home molecules per pass

struct DirectSmem {
    float4 w[kDirectStage];   // staged molecule: centroid + stencil offset, half its square
    int v[kDirectStage];      // molecule index | staged cell << 24 | sampled << 31
    float4 hq[kDirectHome];   // home molecule: centroid, test threshold
    int hs[kDirectHome];      // its index | sampled << 31
    int q[kDirectWarps][64];  // the warps' pair queues: staged position | home molecule << 11
    TileCellTab c;
    int next;
    int item;
};

__host__ __device__ constexpr size_t direct_smem_extra() { return sizeof(DirectSmem) + 16; }

template <int APM>
__global__ void __launch_bounds__(kDirectWarps * 32, 2) k_pairs_direct32(DevSys S, Bufs B) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned int *hbase = (unsigned int *)smem_raw;
    DirectSmem &T = *(DirectSmem *)(smem_raw + (((size_t)hist_words(S) * 4 + 15) & ~(size_t)15));
    shist_zero(S, hbase);
    __syncthreads();
    const SHist h = shist_bind(S, hbase);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
    const unsigned below = (1u << lane) - 1u;
    int *Q = T.q[warp];
    LocalStats st;
    const int64_t ncap = B.cs - 1;
    const int64_t items = (int64_t)B.nf * ncap;
    // CTAs claim (frame, home cell) items from counters[6], as k_pairs_tile32
    for (;;) {
        __syncthreads();  // the previous item's table and claim are no longer read
        if (tid == 0) T.item = atomicAdd(B.counters + 6, 1);
        __syncthreads();
        const int64_t t = T.item;
        if (t >= items) break;
        const int f = (int)(t / ncap), H = (int)(t - (int64_t)f * ncap);
        const PairsFrame Pf = pairs_frame(B, f, true);
        const FrameScratch &F = *Pf.F;
        const FrameGeom &G = *Pf.G;
        if (!F.ok || !F.tile || H >= G.ncell) continue;
        const int hbeg = Pf.cstart[H], nH = Pf.cstart[H + 1] - hbeg;
        if (nH == 0) continue;
        const int n0 = G.n[0], n1 = G.n[1];
        const int cx = H % n0, cy = (H / n0) % n1, cz = H / (n0 * n1);
        const int K = (F.L[0] + 1) + (2 * F.L[0] + 1) * F.L[1] + (2 * F.L[0] + 1) * (2 * F.L[1] + 1) * F.L[2];
        const Guard g = F.g;
        const float rmax = F.rmax_s;
        const float4 *cq32 = B.cq32 + (int64_t)f * B.mv;
        tile_cells(G, F, Pf.cstart, cx, cy, cz, K, T.c);
        const int M = T.c.nbeg[K];
        // one pair per lane: the first n entries of the warp's queue
        auto evaluate = [&](int n) {
            __syncwarp();
            if (lane < n) {
                const int e = Q[lane];
                const int p = e & 2047, sl = e >> 11;
                const float4 w = T.w[p], q = T.hq[sl];
                const int vk = T.v[p], hs = T.hs[sl];
                const int v = vk & 0xffffff, s = hs & 0x7fffffff;
                const float Dx = w.x - q.x, Dy = w.y - q.y, Dz = w.z - q.z;
                float4 oa[APM];
#pragma unroll
                for (int a = 0; a < APM; ++a) oa[a] = Pf.so32[(int64_t)s * APM + a];
                float m1 = INFINITY, m2 = INFINITY, r1 = INFINITY, r2 = INFINITY;
                int k1 = 0;
#pragma unroll
                for (int b = 0; b < APM; ++b) {
                    const float4 ob = Pf.so32[(int64_t)v * APM + b];
                    const float tx = Dx + ob.x, ty = Dy + ob.y, tz = Dz + ob.z;
                    float row = INFINITY;
#pragma unroll
                    for (int a = 0; a < APM; ++a) {
                        const float ex = tx - oa[a].x, ey = ty - oa[a].y, ez = tz - oa[a].z;
                        const float d2 = fmaf(ez, ez, fmaf(ey, ey, ex * ex));
                        m2 = fminf(m2, fmaxf(m1, d2));
                        k1 = d2 < m1 ? (a << 8 | b) : k1;
                        m1 = fminf(m1, d2);
                        row = fminf(row, d2);
                        if (a == S.iref) r2 = fminf(r2, d2);
                    }
                    if (b == S.iref) r1 = row;
                }
                st.molpairs++;
                st.atompairs += (unsigned long long)(APM * APM);
                decide_pair<true>(S, B, h, Pf, g, f, s, hs < 0 ? Pf.slot[s] : -1, vk < 0, v, T.c.code[(vk >> 24) & 127], m1,
                                  m2, k1 >> 8, k1 & 0xff, r1, r2, st);
            }
            __syncwarp();
        };
        for (int h0 = 0; h0 < nH; h0 += kDirectHome)
            for (int m0 = 0; m0 < M; m0 += kDirectStage) {
                const int nh = min(kDirectHome, nH - h0), n = min(kDirectStage, M - m0);
                const int nr = (n + 31) & ~31;
                __syncthreads();  // the previous pass's tables are no longer read
                tile_stage(T, Pf, F, cq32, K, m0, n);
                for (int i = tid; i < nh; i += blockDim.x) {
                    const float4 q = cq32[hbeg + h0 + i];
                    const float R = (g.cut_pre + q.w) + rmax;
                    T.hq[i] = make_float4(q.x, q.y, q.z, 0.5f * (R * R - fmaf(q.z, q.z, fmaf(q.y, q.y, q.x * q.x))));
                    const int s = Pf.cmol[hbeg + h0 + i];
                    T.hs[i] = s | (Pf.slot && Pf.slot[s] >= 0 ? 0x80000000 : 0);
                }
                if (tid == 0) T.next = 0;
                __syncthreads();
                int cnt = 0;
                // the lanes' hits (bit j: staged position base + 32 j + lane) with home molecule sl into the queue
                auto push = [&](unsigned bits, int base, int sl) {
                    for (;;) {
                        const unsigned mask = __ballot_sync(0xffffffffu, bits != 0);
                        if (mask == 0) break;
                        if (bits) {
                            Q[cnt + __popc(mask & below)] = (base + 32 * (__ffs(bits) - 1) + lane) | sl << 11;
                            bits &= bits - 1;
                        }
                        cnt += __popc(mask);
                        if (cnt >= 32) {
                            evaluate(32);
                            cnt -= 32;
                            const int rest = lane < cnt ? Q[32 + lane] : 0;
                            __syncwarp();
                            if (lane < cnt) Q[lane] = rest;
                            __syncwarp();
                        }
                    }
                };
                // two home molecules at a time share the loads of the staged table
                for (;;) {
                    int sl = 0;
                    if (lane == 0) sl = atomicAdd(&T.next, 2);
                    sl = __shfl_sync(0xffffffffu, sl, 0);
                    if (sl >= nh) break;
                    const float4 q = T.hq[sl], r = T.hq[min(sl + 1, nh - 1)];
                    const float rthr = sl + 1 < nh ? r.w : -INFINITY;
                    // within the home cell (the first staged positions) only the molecules after this one
                    const int lo = max(0, h0 + sl + 1 - m0), lo2 = max(0, h0 + sl + 2 - m0);
                    for (int base = lo & ~31; base < nr; base += 1024) {
                        const int nj = min(32, (nr - base) >> 5);
                        unsigned bits = 0, bits2 = 0;
#pragma unroll 4
                        for (int j = 0; j < nj; ++j) {
                            const float4 w = T.w[base + 32 * j + lane];
                            const float u = fmaf(-w.x, q.x, fmaf(-w.y, q.y, fmaf(-w.z, q.z, w.w)));
                            const float u2 = fmaf(-w.x, r.x, fmaf(-w.y, r.y, fmaf(-w.z, r.z, w.w)));
                            if (u <= q.w) bits |= 1u << j;
                            if (u2 <= rthr) bits2 |= 1u << j;
                        }
                        if (base + lane < lo) bits &= ~1u;
                        if (base + lane < lo2) bits2 &= ~1u;
                        if (base + 32 + lane < lo2) bits2 &= ~2u;
                        push(bits, base, sl);
                        push(bits2, base, sl + 1);
                    }
                }
                if (cnt > 0) evaluate(cnt);
            }
    }
    stats_flush(S, st, false);
    __syncthreads();
    shist_flush(S, h, false);
}

// ------------------------------------------------------------ guard kernel
// Exact processing of the candidates deferred by the FP32 real pass, one warp
// per queued molecule pair: the lanes split the pair's atom pairs (over its
// images), for the FP32 pass and for the filtered FP64 scan, and the lanes'
// results are merged.  The FP64 minimum is merged by the reference's tie rule
// (distance, then the larger (solute atom, solvent atom) pair; in self mode the
// second direction's key is (solvent atom, solute atom)), which does not
// depend on the order in which pairs are visited, so the records are those of
// pairs_decide.

// Atom pair i of a molecule pair: image i / (aps apv), then solvent atom b and
// solute atom a; the quotients from FP32 reciprocals are exact for every pair
// of up to 32 atoms a side and up to 16^3 images.
struct PairIndex {
    float inv_pi, inv_aps;
    int per_img, aps;
    __device__ __forceinline__ void at(int i, int &img, int &b, int &a) const {
        img = (int)((float(i) + 0.5f) * inv_pi);
        const int r = i - img * per_img;
        b = (int)((float(r) + 0.5f) * inv_aps);
        a = r - b * aps;
    }
};

// FP32 pass of pairs_pass32 with the pairs split over the lanes; every lane
// ends with the merged result (second-smallest over the union: the smaller of
// the larger minimum and the smaller second minima).
template <bool SELF>
__device__ __forceinline__ void pass32_warp(const DevSys &S, const float4 *__restrict__ off32, const Images &im, float4 qs,
                                            float4 qv, const float4 *os, const float4 *ov, const PairIndex &pi, int total,
                                            int lane, Pass32 &P) {
    constexpr unsigned kFull = 0xffffffffu;
    P.m1 = P.m2 = P.r1 = P.r2 = INFINITY;
    P.k1 = 0x7fffffff;
    const int apv = S.apv, iref = S.iref;
    int cur = -1;
    float Dx = 0.f, Dy = 0.f, Dz = 0.f;
    for (int i = lane; i < total; i += 32) {
        int img, b, a;
        pi.at(i, img, b, a);
        if (img != cur) {
            int dx, dy, dz;
            image_at(im, img, dx, dy, dz);
            const float4 o = off32[off_index(dx, dy, dz)];
            Dx = (qv.x - qs.x) + o.x;
            Dy = (qv.y - qs.y) + o.y;
            Dz = (qv.z - qs.z) + o.z;
            cur = img;
        }
        const float4 ob = ov[b], oa = os[a];
        const float tx = Dx + ob.x, ty = Dy + ob.y, tz = Dz + ob.z;
        const float ex = tx - oa.x, ey = ty - oa.y, ez = tz - oa.z;
        const float d2 = fmaf(ez, ez, fmaf(ey, ey, ex * ex));
        const int k = a * apv + b;
        P.m2 = fminf(P.m2, fmaxf(P.m1, d2));
        P.k1 = d2 < P.m1 ? k : P.k1;
        P.m1 = fminf(P.m1, d2);
        if (b == iref) P.r1 = fminf(P.r1, d2);
        if (SELF && a == iref) P.r2 = fminf(P.r2, d2);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float m1 = __shfl_xor_sync(kFull, P.m1, o), m2 = __shfl_xor_sync(kFull, P.m2, o);
        const int k1 = __shfl_xor_sync(kFull, P.k1, o);
        P.m2 = fminf(fmaxf(P.m1, m1), fminf(P.m2, m2));
        if (m1 < P.m1 || (m1 == P.m1 && k1 < P.k1)) {
            P.m1 = m1;
            P.k1 = k1;
        }
        P.r1 = fminf(P.r1, __shfl_xor_sync(kFull, P.r1, o));
        if (SELF) P.r2 = fminf(P.r2, __shfl_xor_sync(kFull, P.r2, o));
    }
}

// pairs_exact with the pairs split over the lanes (FP32 filter), merged over
// the warp; every lane ends with the result.
template <bool SELF>
__device__ void exact_warp(const DevSys &S, const FrameGeom &G, const Bufs &B, ExactMol &X,
                           const float4 *__restrict__ off32, const Images &im, float4 qs32, float4 qv32,
                           const float4 *os32, const float4 *ov32, float thr_arg, float thr_r1, float thr_r2,
                           const PairIndex &pi, int total, int lane, Exact64 &E) {
    constexpr unsigned kFull = 0xffffffffu;
    best_init(E.B);
    E.rr1 = INFINITY;
    E.rr2 = INFINITY;
    E.evals = 0;
    const int iref = S.iref;
    const double cut2 = S.cut2;
    int cur = -1;
    float Fx = 0.f, Fy = 0.f, Fz = 0.f;
    for (int i = lane; i < total; i += 32) {
        int img, b, a;
        pi.at(i, img, b, a);
        if (img != cur) {
            int dx, dy, dz;
            image_at(im, img, dx, dy, dz);
            const float4 of = off32[off_index(dx, dy, dz)];
            Fx = (qv32.x - qs32.x) + of.x;
            Fy = (qv32.y - qs32.y) + of.y;
            Fz = (qv32.z - qs32.z) + of.z;
            cur = img;
        }
        const float4 ob32 = ov32[b], oa32 = os32[a];
        const float ex = (Fx + ob32.x) - oa32.x, ey = (Fy + ob32.y) - oa32.y, ez = (Fz + ob32.z) - oa32.z;
        const float d2f = fmaf(ez, ez, fmaf(ey, ey, ex * ex));
        if (!(d2f <= thr_arg || (b == iref && d2f <= thr_r1) || (SELF && a == iref && d2f <= thr_r2))) continue;
        const double d2 = exact_pair_d2(B, G, X, a, b);
        E.evals++;
        if (d2 <= cut2) {
            if (b == iref) E.rr1 = fmin(E.rr1, d2);
            if (SELF && a == iref) E.rr2 = fmin(E.rr2, d2);
            best_update<SELF>(E.B, d2, a, b);
        }
    }
    // merge: smallest d = sqrt(d2); among equal d the larger (a, b), and in
    // self mode separately the larger (b, a)
    double d = E.B.d2 <= cut2 ? best_d(E.B) : INFINITY;
    double d2 = E.B.d2;
    int a1 = E.B.a, b1 = E.B.b, a2 = E.B.a2, b2 = E.B.b2;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double od = __shfl_xor_sync(kFull, d, o), od2 = __shfl_xor_sync(kFull, d2, o);
        const int oa1 = __shfl_xor_sync(kFull, a1, o), ob1 = __shfl_xor_sync(kFull, b1, o);
        const int oa2 = __shfl_xor_sync(kFull, a2, o), ob2 = __shfl_xor_sync(kFull, b2, o);
        if (od < d) {
            d = od;
            d2 = od2;
            a1 = oa1; b1 = ob1; a2 = oa2; b2 = ob2;
        } else if (od == d) {
            if (oa1 > a1 || (oa1 == a1 && ob1 > b1)) { a1 = oa1; b1 = ob1; }
            if (SELF && (ob2 > b2 || (ob2 == b2 && oa2 > a2))) { a2 = oa2; b2 = ob2; }
        }
        E.rr1 = fmin(E.rr1, __shfl_xor_sync(kFull, E.rr1, o));
        if (SELF) E.rr2 = fmin(E.rr2, __shfl_xor_sync(kFull, E.rr2, o));
        E.evals += __shfl_xor_sync(kFull, E.evals, o);
    }
    E.B.d2 = d2;
    E.B.d = d <= 1e300 ? d : -1.0;
    E.B.a = a1; E.B.b = b1; E.B.a2 = a2; E.B.b2 = b2;
}

// pairs_decide with the warp-parallel pass and scans; the statistics are
// counted on lane 0.
template <bool SELF>
__device__ void decide_warp(const DevSys &S, const FrameGeom &G, const Bufs &B, ExactMol &X, const Guard &g,
                            const Pass32 &P, const float4 *__restrict__ off32, const Images &im, float4 qs32, float4 qv32,
                            const float4 *os32, const float4 *ov32, int s, int64_t v, const PairIndex &pi, int total,
                            int lane, DirRec &r1, DirRec &r2, LocalStats &st) {
    r1 = dir_none(S);
    r2 = dir_none(S);
    if (P.m1 > g.cutp2) return;
    const float d1 = sqrtf(P.m1);
    const bool amb = P.m1 >= g.cutm2 || (sqrtf(P.m2) - d1) <= g.two_delta;
    if (amb) {
        const float t = d1 + g.two_delta;
        const float thr = __fmul_ru(t, t);
        float thr1 = -1.f, thr2 = -1.f;
        if (P.r1 <= g.cutp2) { const float u = sqrtf(P.r1) + g.two_delta; thr1 = __fmul_ru(u, u); }
        if (SELF && P.r2 <= g.cutp2) { const float u = sqrtf(P.r2) + g.two_delta; thr2 = __fmul_ru(u, u); }
        if (!SELF) thr2 = INFINITY;
        Exact64 E;
        exact_warp<SELF>(S, G, B, X, off32, im, qs32, qv32, os32, ov32, thr, thr1, thr2, pi, total, lane, E);
        records_from_exact<SELF>(S, E, s, v, r1, r2);
        if (lane == 0) {
            st.guard++;
            st.guard_pairs += E.evals;
            if (E.B.d2 <= S.cut2) st.maxerr = fmax(st.maxerr, fabs((double)d1 - best_d(E.B)));
        }
        return;
    }
    // unambiguous: the FP32 minimum pair is the exact minimum pair, within cutoff
    const int a = P.k1 / S.apv, b = P.k1 - a * S.apv;
    int bin = bin32(g, d1);
    double d64 = -1.0;
    if (bin < 0 || (S.usecutoff && d1 >= g.dbulk_lo && d1 <= g.dbulk_hi)) {
        d64 = sqrt(exact_pair_d2(B, G, X, a, b));
        bin = setbin0(d64, S.binstep);
        if (lane == 0) {
            st.guard++;
            st.guard_pairs += 1;
            st.maxerr = fmax(st.maxerr, fabs((double)d1 - d64));
        }
    }
    const int bulk = S.usecutoff ? (d64 >= 0.0 ? (d64 > S.dbulk) : (d1 > g.dbulk_hi)) : 0;
    r1.within = 1;
    r1.i_local = a;
    r1.j = v * S.apv + b;
    r1.bin = bin;
    r1.bulk = bulk;
    if (SELF) {
        r2.within = 1;
        r2.i_local = b;
        r2.j = (int64_t)s * S.aps + a;
        r2.bin = bin;
        r2.bulk = bulk;
    }
    // reference-atom rows (and columns in self mode)
    for (int dir = 0; dir < (SELF ? 2 : 1); ++dir) {
        const float rm = dir == 0 ? P.r1 : P.r2;
        DirRec &r = dir == 0 ? r1 : r2;
        if (rm > g.cutp2) continue;
        const int rb = rm < g.cutm2 ? bin32(g, sqrtf(rm)) : -1;
        if (rb >= 0) {
            r.ref = 1;
            r.rbin = rb;
            continue;
        }
        const float u = sqrtf(rm) + g.two_delta;
        const float thr = __fmul_ru(u, u);
        Exact64 E;
        exact_warp<SELF>(S, G, B, X, off32, im, qs32, qv32, os32, ov32, -1.f, dir == 0 ? thr : -1.f, dir == 1 ? thr : -1.f,
                         pi, total, lane, E);
        const double rr = dir == 0 ? E.rr1 : E.rr2;
        if (lane == 0) {
            st.guard++;
            st.guard_pairs += E.evals;
        }
        if (rr <= S.cut2) {
            r.ref = 1;
            r.rbin = setbin0(sqrt(rr), S.binstep);
        }
    }
}

constexpr int kGuardWarps = 4;  // warps per CTA of k_pairs_guard

template <bool SELF>
__global__ void __launch_bounds__(kGuardWarps * 32) k_pairs_guard(DevSys S, Bufs B) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ float4 s_os[kGuardWarps][kMaxSmallMol], s_ov[kGuardWarps][kMaxSmallMol];
    unsigned int *hbase = (unsigned int *)smem_raw;
    shist_zero(S, hbase);
    __syncthreads();
    SHist h = shist_bind(S, hbase);
    LocalStats st;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int aps = S.aps, apv = S.apv;
    PairIndex pi;
    pi.per_img = aps * apv;
    pi.aps = aps;
    pi.inv_pi = 1.0f / (float)pi.per_img;
    pi.inv_aps = 1.0f / (float)aps;
    const int n = min(B.counters[0], B.gq_cap);
    // warps claim records from counters[7] (zeroed with the chunk's
    // counters): a record's cost varies with its exact scan
    for (;;) {
        int i = 0;
        if (lane == 0) i = atomicAdd(B.counters + 7, 1);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= n) break;
        const int4 it = B.gq[i];
        const int s = it.x, v = it.y, f = it.w;
        const PairsFrame Pf = pairs_frame(B, f, SELF);
        const FrameScratch &F = *Pf.F;
        const Images im = images_of(*Pf.G, F, it.z);
        const int total = pi.per_img * image_count(im);
        const float4 qs32 = Pf.sq32[s], qv32 = Pf.vq32[v];
        __syncwarp();
        if (lane < aps) s_os[warp][lane] = Pf.so32[(int64_t)s * aps + lane];
        if (lane < apv) s_ov[warp][lane] = Pf.vo32[(int64_t)v * apv + lane];
        __syncwarp();
        Pass32 P;
        pass32_warp<SELF>(S, Pf.off32, im, qs32, qv32, s_os[warp], s_ov[warp], pi, total, lane, P);
        DirRec r1, r2;
        ExactMol X = exact_mol(S, f, s, v);
        decide_warp<SELF>(S, *Pf.G, B, X, F.g, P, Pf.off32, im, qs32, qv32, s_os[warp], s_ov[warp], s, v, pi, total, lane, r1,
                          r2, st);
        if (lane == 0) emit<SELF>(S, h, r1, r2, s, v, Pf.slot, Pf.flags, st);
    }
    stats_flush(S, st, false);
    __syncthreads();
    shist_flush(S, h, false);
}

// The random-insertion slots inside k_random_fast's band (rq2), one warp per
// slot: placed in FP64 from the FP32 offsets (the narrow band gp), the pairs and the molecule's atoms split over the lanes, and
// decided by decide_warp.  One thread per slot waited 360 us for its chain of
// FP64 operations (14-atom molecules), whatever the number of slots.
__global__ void __launch_bounds__(kGuardWarps * 32) k_random_records(DevSys S, Bufs B) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ float4 s_os[kGuardWarps][kMaxSmallMol], s_ov[kGuardWarps][kMaxSmallMol];
    __shared__ double s_u[kGuardWarps][3][kMaxSmallMol];
    unsigned int *hbase = (unsigned int *)smem_raw;
    const int n = B.counters[10];
    if ((int64_t)blockIdx.x * kGuardWarps >= n) return;
    shist_zero(S, hbase);
    __syncthreads();
    const SHist h = shist_bind(S, hbase);
    LocalStats st;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int aps = S.aps, apv = S.apv;
    PairIndex pi;
    pi.per_img = aps * apv;
    pi.aps = aps;
    pi.inv_pi = 1.0f / (float)pi.per_img;
    pi.inv_aps = 1.0f / (float)aps;
    for (int i = blockIdx.x * kGuardWarps + warp; i < n; i += gridDim.x * kGuardWarps) {
        const int2 e = B.rq2[i];
        const Sample sm = B.samples[e.x];
        const int s = sm.s, k = e.y, f = sm.pad;
        const PairsFrame Pf = pairs_frame(B, f, S.self);
        const FrameGeom &G = *Pf.G;
        const FrameScratch &F = *Pf.F;
        int jmol, c0[3];
        uint64_t fk[3];
        float q0[3];
        uint64_t rs = draw_slot_bits(S, G.frame_id, sm, k, Pf.bulk, Pf.nbulk, jmol, fk);
        centre32(G, F.fx, fk, c0, q0);
        const Images im = centre_images(G, F, Pf.scell[s], c0);
        double A[9], fc[3];
        for (int q = 0; q < 3; ++q) fc[q] = (double)fk[q] * 0x1.0p-53;
        draw_rotation(rs, A);
        ExactMol X = exact_mol_placed(S, G, f, s, jmol, fc, A);
        raw_atom(B, true, f, X.vbase + S.iref, X.xr);
        __syncwarp();
        if (lane < aps) s_os[warp][lane] = Pf.so32[(int64_t)s * aps + lane];
        if (lane < apv) {
            const float4 w = Pf.vo32[(int64_t)jmol * apv + lane];
            double r[3], x[3], u[3];
            matvec_rm(A, w.x, w.y, w.z, r);
            s_ov[warp][lane] = make_float4((float)r[0], (float)r[1], (float)r[2], 0.f);
            raw_atom(B, true, f, X.vbase + lane, x);
            exact_unwrapped(G, x, X.xr, u);
            for (int q = 0; q < 3; ++q) s_u[warp][q][lane] = u[q];
        }
        __syncwarp();
        // the mean in the order of exact_mol_ready
        double cm = 0.0;
        if (lane < 3) {
            for (int b = 0; b < apv; ++b) cm = add(cm, s_u[warp][lane][b]);
            cm = div(cm, (double)apv);
        }
        for (int q = 0; q < 3; ++q) X.cm[q] = __shfl_sync(0xffffffffu, cm, q);
        X.ready = 1;
        const float4 qs32 = Pf.sq32[s], qv32 = make_float4(q0[0], q0[1], q0[2], 0.f);
        const int total = pi.per_img * image_count(im);
        Pass32 P;
        pass32_warp<false>(S, Pf.off32, im, qs32, qv32, s_os[warp], s_ov[warp], pi, total, lane, P);
        DirRec r1, r2;
        decide_warp<false>(S, G, B, X, F.gp, P, Pf.off32, im, qs32, qv32, s_os[warp], s_ov[warp], s, k, pi, total, lane, r1, r2,
                           st);
        if (lane == 0 && r1.within) {
            apply_hit_local(S, h, true, r1.bin, r1.i_local, r1.j, (int)(r1.j - (int64_t)k * apv), r1.ref, r1.rbin);
            st.hits++;
        }
    }
    stats_flush(S, st, true);
    __syncthreads();
    shist_flush(S, h, true);
}

// setbin0 without its FP64 division where the quotient is not near an integer
// (the product is within 4 u64 of it).
__device__ __forceinline__ int setbin0_fast(double d, double step, double inv) {
    const double k = d * inv, r = rint(k);
    if (fabs(k - r) <= 1e-9 * (k + 1.0)) return setbin0(d, step);
    const int b = (int)ceil(k);
    return (b < 1 ? 1 : b) - 1;
}

// Edge kernel: records whose closest atom pair is known from the FP32 pass
// (second-closest pair beyond 2 delta, cutoff and dbulk clear) but whose md
// bin, solvent reference-atom row or solute reference-atom column (marked -2)
// lies within the guard band of a bin edge or of the cutoff.  Each marked
// value comes from exact pair distances (exact_d2): the closest pair for the
// md bin; for the row the pairs of the solvent molecule's reference atom whose
// FP32 distance is within 2 delta of their smallest (nearly always one), for
// the column those of the solute molecule's.
//
// One thread per record, one marked value per lane and round: a record has
// nearly always one, and a round takes the warp's lanes through the same FP64
// chain whichever value theirs is.  FP64 instructions hold a quarter of an SM
// for 64 cycles each and bound the kernel; with the three kinds of value in
// separate branches and a division per bin it ran 7.5 lanes wide, 927 us on 64
// frames of 10,000 14-atom molecules, 300 so.
template <bool SELF>
__global__ void __launch_bounds__(128) k_pairs_edge(DevSys S, Bufs B) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned int *hbase = (unsigned int *)smem_raw;
    const int n = min(B.counters[3], B.eq_cap);
    if ((int64_t)blockIdx.x * blockDim.x >= n) return;
    shist_zero(S, hbase);
    __syncthreads();
    SHist h = shist_bind(S, hbase);
    LocalStats st;
    const double inv = 1.0 / S.binstep;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int4 e = B.eq[3 * i], x = B.eq[3 * i + 1], y = B.eq[3 * i + 2];
        const int s = e.x, v = e.y, f = e.w;
        const int a1 = x.x & 0xff, b1 = (x.x >> 8) & 0xff;
        int rb1 = x.y, rb2 = x.z, bin = x.w;
        const float d32 = __int_as_float(y.x);
        const PairsFrame Pf = pairs_frame(B, f, SELF);
        const Images im = images_of(*Pf.G, *Pf.F, e.z);
        const FrameGeom &G = *Pf.G;
        const Guard &g = Pf.F->g;
        const float4 qs = Pf.sq32[s], qv = Pf.vq32[v];
        const float4 *os32 = Pf.so32 + (int64_t)s * S.aps, *ov32 = Pf.vo32 + (int64_t)v * S.apv;
        ExactMol X = exact_mol(S, f, s, v);
        st.guard++;
        int bulk = S.usecutoff ? (d32 > g.dbulk_hi) : 0;
        // FP32 squared distance of atoms a and b, the smallest over the images, formed as in the FP32 passes
        auto d2_of = [&](int a, int b) {
            const float4 oa = os32[a], ob = ov32[b];
            float best = INFINITY;
            CM_FOR_IMAGES(im, dx, dy, dz) {
                const float4 o = Pf.off32[off_index(dx, dy, dz)];
                const float ex = (((qv.x - qs.x) + o.x) + ob.x) - oa.x;
                const float ey = (((qv.y - qs.y) + o.y) + ob.y) - oa.y;
                const float ez = (((qv.z - qs.z) + o.z) + ob.z) - oa.z;
                best = fminf(best, fmaf(ez, ez, fmaf(ey, ey, ex * ex)));
            }
            return best;
        };
        unsigned need = (bin == -2 ? 1u : 0u) | (rb1 == -2 ? 2u : 0u) | (SELF && rb2 == -2 ? 4u : 0u);
        while (need) {
            const int which = __ffs(need) - 1;
            need &= need - 1;
            const bool row = which == 1;
            int a = a1, b = b1, at = 0, cnt = 0;
            float thr = 0.f, m2 = INFINITY;
            if (which != 0) {
                cnt = row ? S.aps : S.apv;
                float m = INFINITY;
                for (int j = 0; j < cnt; ++j) {
                    const float d2 = d2_of(row ? j : S.iref, row ? S.iref : j);
                    m2 = fminf(m2, fmaxf(m, d2));
                    at = d2 < m ? j : at;
                    m = fminf(m, d2);
                }
                const float t = sqrtf(m) + g.two_delta;
                thr = __fmul_ru(t, t);
                a = row ? at : S.iref;
                b = row ? S.iref : at;
            }
            double rr = exact_pair_d2(B, G, X, a, b);
            st.guard_pairs += 1;
            if (which != 0 && m2 <= thr)
                for (int j = 0; j < cnt; ++j) {
                    if (j == at || !(d2_of(row ? j : S.iref, row ? S.iref : j) <= thr)) continue;
                    rr = fmin(rr, exact_pair_d2(B, G, X, row ? j : S.iref, row ? S.iref : j));
                    st.guard_pairs += 1;
                }
            const double d64 = sqrt(rr);
            const int k = setbin0_fast(d64, S.binstep, inv);
            if (which == 0) {
                bin = k;
                bulk = S.usecutoff ? (d64 > S.dbulk) : 0;
                st.maxerr = fmax(st.maxerr, fabs((double)d32 - d64));
            } else {
                const int r = rr <= S.cut2 ? k : -1;
                if (row) rb1 = r;
                else rb2 = r;
            }
        }
        apply_hit_local(S, h, false, bin, a1, (int64_t)v * S.apv + b1, b1, rb1 >= 0, rb1);
        st.hits++;
        if (SELF) {
            apply_hit_local(S, h, false, bin, b1, (int64_t)s * S.aps + a1, a1, rb2 >= 0, rb2);
            st.hits++;
        }
        if (Pf.slot) {
            const unsigned char code1 = (unsigned char)(1 + bulk);
            const int sl = Pf.slot[s];
            if (sl >= 0) Pf.flags[(int64_t)sl * S.mv + v] = code1;
            if (SELF) {
                const int vs = Pf.slot[v];
                if (vs >= 0) Pf.flags[(int64_t)vs * S.mv + s] = code1;
            }
        }
    }
    stats_flush(S, st, false);
    __syncthreads();
    shist_flush(S, h, false);
}

}  // namespace cmk
