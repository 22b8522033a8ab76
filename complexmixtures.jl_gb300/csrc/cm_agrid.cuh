// cm_agrid.cuh -- candidate grid of the ATOMS layout for a single solute
// molecule (a protein or a long chain: configs 1, 2 and 4), FP32 search.
//
// The question the ATOMS search answers per solvent molecule is, site by
// site, "which solute atom is closest, how close is the second, and how close
// is the closest atom to the reference site" (src/minimum_distances.jl:30-39,
// 107-120).  With one solute molecule that is a nearest-neighbour query
// against one fixed point set per frame, asked once per real solvent molecule
// and n_random_samples times per slot of the random insertion
// (src/mddf.jl:65-88, 403-423).  So per frame each search cell is split into
// K^3 fine cells, and each fine cell g gets the list of solute atoms a with
//
//     dmin(a, g) <= min( min_a' dmax(a', g), cutoff ) + margin,
//
// dmin / dmax the smallest / largest distance from a to a point of g (exact
// box distances for orthogonal cells, the fine cell's bounding sphere
// otherwise) and margin = 2 delta + 1e-3 (1 + cutoff).  For a point y of g the
// nearest atom is within min_a' dmax(a', g), so the list holds every atom
// within (nearest distance + 2 delta) of y, and every atom within the cutoff
// when nothing is closer.  A query (one site) reads its fine cell's list and
// evaluates only those atoms: the smallest FP32 distance, its atom, the
// second-smallest value (exact whenever it is within 2 delta of the smallest;
// the guard test only asks that) and the reference site's smallest distance
// are then the values a walk over every stencil cell gives, and every decision
// follows the FP32 + guard rules of atoms_decide.  A query whose record lies
// inside the guard band is listed for k_agrid_records, which decides it from
// exact distances (agrid_record), its exact scans reading the same lists, so
// the counts stay the oracle's.
//
// A list entry is the atom's FP32 position from the fine cell's search-cell
// origin, q_a + off(cell_a - cell), which is the displacement form of the
// ATOMS walks (the guard band's error bound covers it), and the atom's index
// in the molecule.
//
// Kernels: k_agrid_build (the lists of every frame, one search cell near the
// solute at a time per CTA, space reserved in a per-frame pool; a frame whose pool runs out loses its
// grid), k_agrid_real (real pass) and k_agrid_random (random insertion: the
// queries of the slots k_slot_filter listed and k_atoms_place placed), each
// followed by k_agrid_records.
// Frames without a grid take the walk path: k_agrid_real queues their
// molecule pairs for k_atoms_eval as k_atoms_filter does, and k_atoms_place
// queues their slots.
#pragma once
#include "cm_atoms32.cuh"

namespace cmk {

constexpr int kAgridMaxK = 6;          // fine cells per search-cell axis
constexpr int kAgridBuckets = 8;       // each list ordered by bucket of the atom's smallest distance to the fine cell
static_assert(kAgridStarts == kAgridBuckets + 1, "starts of a list");
constexpr int kAgridStage = 2560;      // stencil atoms staged in shared memory at a time (40 KB, dynamic)
constexpr int kAgridRound = 2;         // stencil atoms each thread loads per staging round
constexpr int kAgridBuildThreads = 256;
constexpr int kAgridBuildCtas = 4;     // resident CTAs per SM (40 KB of stage and 12 KB more each, 61 registers a thread)
constexpr int kAgridRecThreads = 32;   // k_agrid_records: a few records per SM,
constexpr int kAgridRecLanes = 4;      // each on a group of lanes

// Largest distance from p to a point of the fine cell centred at c: squared
// for orthogonal cells, the distance to the centre squared otherwise (the
// bound is then that distance + R).
__device__ __forceinline__ float fine_far2(const FineCells &fc, const float *c, const float4 &p) {
    const float dx = fabsf(p.x - c[0]), dy = fabsf(p.y - c[1]), dz = fabsf(p.z - c[2]);
    if (fc.ortho) {
        const float vx = dx + fc.h[0], vy = dy + fc.h[1], vz = dz + fc.h[2];
        return fmaf(vz, vz, fmaf(vy, vy, vx * vx));
    }
    return fmaf(dz, dz, fmaf(dy, dy, dx * dx));
}

// Smallest distance from p to the fine cell, squared (orthogonal cells), or
// the squared distance to the centre (the bound is then that distance - R).
__device__ __forceinline__ float fine_near2(const FineCells &fc, const float *c, const float4 &p) {
    const float dx = fabsf(p.x - c[0]), dy = fabsf(p.y - c[1]), dz = fabsf(p.z - c[2]);
    if (fc.ortho) {
        const float ux = fmaxf(dx - fc.h[0], 0.f), uy = fmaxf(dy - fc.h[1], 0.f), uz = fmaxf(dz - fc.h[2], 0.f);
        return fmaf(uz, uz, fmaf(uy, uy, ux * ux));
    }
    return fmaf(dz, dz, fmaf(dy, dy, dx * dx));
}

// A square root for bucket numbers: its error (2 ulp) lies within the lists' slack.
__device__ __forceinline__ float sqrt_approx(float x) {
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Lists of the fine cells of one search cell at a time, claimed by a resident
// grid from the list of cells near the solute (k_atoms_near).  The CTA stages
// the cell's stencil atoms in shared memory; each warp takes fine cells in
// turn and its lanes split the staged atoms (warp reductions, and ballots for
// the compacted writes).  The CTA counts its lists by bucket, reserves their
// room in the frame's entry pool with one atomic, writes each fine cell's
// bucket starts and end to gstart and its bucket edges to gedge, then the
// entries.  A frame whose pool runs out loses its grid (its queries take the
// walk).
// Bound by instruction issue: each fine cell tests every staged atom three
// times.  So (a) the grid holds only the near cells, one CTA per cell of the
// box spent most of a sparse frame on cells with nothing to do; (b) stencil
// cells farther than the own atoms' bound are dropped before their atoms are
// loaded; (c) bucket positions stay in lanes 0 .. 7 and ballots find a
// bucket's lanes, where match_any and a shared-memory update did.  us, before
// and after: 20,000-atom chain in water 656 and 513, in 14-site cosolvent
// 1,105 and 824, 24 systems of up to 10,000 atoms 3,234 and 1,741, 50 frames
// of 2,150 atoms 723 and 568.  Four CTAs of 256 threads with 40 KB of stage
// (rounds of two atoms a thread); three with 48 KB and rounds of four: 498,
// 835, 1,955 and 617; four with 32 KB: 553, 901, 1,805 and 580.
__device__ __forceinline__ void k_agrid_build_body(const uint3 blockIdx, const dim3 gridDim, const DevSys &S, const Bufs &B) {
    extern __shared__ float4 s_at[];  // kAgridStage entries
    __shared__ int s_pre[kAgridMaxStencil + 1];
    __shared__ int s_beg[kAgridMaxStencil];
    __shared__ short s_oi[kAgridMaxStencil];
    __shared__ float s_far[kAgridMaxK * kAgridMaxK * kAgridMaxK], s_near[kAgridMaxK * kAgridMaxK * kAgridMaxK];
    __shared__ int s_pos[kAgridMaxK * kAgridMaxK * kAgridMaxK][kAgridBuckets];
    __shared__ int s_wsum[kAgridBuildThreads / 32];
    __shared__ int s_base;
    __shared__ float s_tmax;
    __shared__ FineCells s_fc;
    __shared__ int s_item, s_cells;
    const int K = B.agk, K3 = K * K * K;
    const int t = threadIdx.x;
    const int lane = t & 31, warp = t >> 5, nwarps = blockDim.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    const int nitems = B.counters[11], per_frame = (int)(B.gfs / K3);
    for (;;) {
    __syncthreads();  // the previous cell's shared arrays are read no more
    if (t == 0) s_item = atomicAdd(B.counters + 12, 1);
    __syncthreads();
    if (s_item >= nitems) return;
    const int item = B.galist[s_item];
    const int f = item / per_frame, c = item - f * per_frame;
    const FrameGeom &G = B.G[f];
    const FrameScratch &F = B.FS[f];
    const int64_t gbase = ((int64_t)f * B.gfs + (int64_t)c * K3) * (kAgridBuckets + 1);  // bucket starts and end
    const int64_t ebase = (int64_t)f * B.gfs + (int64_t)c * K3;                            // fine-cell bucket edges
    const int La0 = F.La[0], La1 = F.La[1], La2 = F.La[2];
    const int nx = 2 * La0 + 1, ny = 2 * La1 + 1, nst = nx * ny * (2 * La2 + 1);
    const int cx = c % G.n[0], cy = (c / G.n[0]) % G.n[1], cz = c / (G.n[0] * G.n[1]);
    const int *cs = B.astart + (int64_t)f * B.as;  // solute molecule 0
    for (int i = t; i < nst; i += blockDim.x) {
        const int dx = i % nx - La0, dy = (i / nx) % ny - La1, dz = i / (nx * ny) - La2;
        const int cell = (wrap_cell(cz + dz, G.n[2]) * G.n[1] + wrap_cell(cy + dy, G.n[1])) * G.n[0] +
                         wrap_cell(cx + dx, G.n[0]);
        s_beg[i] = cs[cell];
        s_pre[i] = cs[cell + 1] - cs[cell];
        s_oi[i] = (short)off_index(dx, dy, dz);
    }
    const float4 *aq = B.asq32 + (int64_t)f * B.Ns;
    const float4 *off = B.off32 + (int64_t)f * kOffEntries;
    if (t == 0) {
        s_fc = F.fcells;  // the frame's fine-cell geometry (k_frame_consts)
        s_tmax = 0.f;
    }
    for (int g = t; g < K3; g += blockDim.x) {
        s_far[g] = INFINITY;
        s_near[g] = INFINITY;
    }
    __syncthreads();
    int N = 0, ncells = 0;  // atoms and cells of the stencil that are kept (below)
    // stencil atom kk: its position from this cell's origin
    auto atom_of = [&](int cell, int k) {
        const float4 q = aq[s_beg[cell] + k];
        const float4 o = off[s_oi[cell]];
        return make_float4(q.x + o.x, q.y + o.y, q.z + o.z, q.w);
    };
    auto atom_at = [&](int kk) {
        int lo = 0, hi = ncells - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (s_pre[mid] <= kk) lo = mid;
            else hi = mid - 1;
        }
        return atom_of(lo, kk - s_pre[lo]);
    };
    const FineCells fc = s_fc;
    auto centre = [&](int g, float *cen) {
        const float u0 = ((float)(g % K) + 0.5f), u1 = ((float)((g / K) % K) + 0.5f), u2 = ((float)(g / (K * K)) + 0.5f);
        for (int r = 0; r < 3; ++r) cen[r] = fmaf(fc.e[6 + r], u2, fmaf(fc.e[3 + r], u1, fc.e[r] * u0));
    };
    // a lower bound of the distance from p to this search cell: its box for
    // orthogonal cells, its bounding sphere otherwise
    float blo[3], bhi[3], cc[3];
    const float Rc = fc.R * (float)K;
    for (int r = 0; r < 3; ++r) {
        const float e = fc.e[4 * r] * (float)K;
        blo[r] = fminf(0.f, e);
        bhi[r] = fmaxf(0.f, e);
        cc[r] = 0.5f * (float)K * (fc.e[r] + fc.e[3 + r] + fc.e[6 + r]);
    }
    auto cell_near = [&](const float4 &p) {
        if (fc.ortho) {
            const float dx = fmaxf(fmaxf(blo[0] - p.x, p.x - bhi[0]), 0.f);
            const float dy = fmaxf(fmaxf(blo[1] - p.y, p.y - bhi[1]), 0.f);
            const float dz = fmaxf(fmaxf(blo[2] - p.z, p.z - bhi[2]), 0.f);
            return sqrtf(fmaf(dz, dz, fmaf(dy, dy, dx * dx)));
        }
        const float dx = p.x - cc[0], dy = p.y - cc[1], dz = p.z - cc[2];
        return fmaxf(sqrtf(fmaf(dz, dz, fmaf(dy, dy, dx * dx))) - Rc, 0.f);
    };
    // the next stencil atoms within `thr` of this cell, from atom `cursor` on,
    // compacted into s_at in stencil order (kAgridRound atoms per thread and
    // two barriers per round); returns how many
    auto stage_kept = [&](int &cursor, float thr) {
        int n = 0;
        const int round = kAgridRound * (int)blockDim.x;
        while (cursor < N && n + round <= kAgridStage) {
            float4 p[kAgridRound];
            unsigned m[kAgridRound];
            int mine_n = 0;
#pragma unroll
            for (int j = 0; j < kAgridRound; ++j) {
                const int kk = cursor + j * (int)blockDim.x + t;
                bool keep = false;
                p[j] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (kk < N) {
                    p[j] = atom_at(kk);
                    keep = cell_near(p[j]) <= thr;
                }
                m[j] = __ballot_sync(0xffffffffu, keep);
                mine_n += __popc(m[j]);
            }
            if (lane == 0) s_wsum[warp] = mine_n;
            __syncthreads();
            int before = 0, total = 0;
            for (int w = 0; w < nwarps; ++w) {
                const int cw = s_wsum[w];
                before += w < warp ? cw : 0;
                total += cw;
            }
            int at = n + before;
#pragma unroll
            for (int j = 0; j < kAgridRound; ++j) {
                if ((m[j] >> lane) & 1u) s_at[at + __popc(m[j] & below)] = p[j];
                at += __popc(m[j]);
            }
            n += total;
            cursor += round;
            __syncthreads();
        }
        return n;
    };
    auto warp_min = [&](float v) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
        return v;
    };
    const float cut = (float)S.cut;
    const float slack = 1e-3f * (1.0f + cut);
    const float margin = F.g.two_delta + slack;
    // the list threshold and bucket edges of fine cell g from its bounds
    auto thresh = [&](int g) { return fminf(fc.ortho ? sqrtf(s_far[g]) : sqrtf(s_far[g]) + fc.R, cut) + margin; };
    auto lowest = [&](int g) { return fc.ortho ? sqrtf(s_near[g]) : fmaxf(sqrtf(s_near[g]) - fc.R, 0.f); };
    int kept = -1;  // atoms of pass 1 still staged (-1 none yet, -2 several stages)
    {
        // the search cell's own atoms first: each fine cell's bound from them
        // limits the stencil atoms that can matter to those within the
        // largest bound of the cell (dense solutes: a few Angstrom)
        const int own = (La2 * ny + La1) * nx + La0, own_n = s_pre[own];
        for (int k0 = 0; k0 < own_n; k0 += kAgridStage) {
            const int nb = min(kAgridStage, own_n - k0);
            __syncthreads();
            for (int k = t; k < nb; k += blockDim.x) s_at[k] = atom_of(own, k0 + k);
            __syncthreads();
            for (int g = warp; g < K3; g += nwarps) {
                float cen[3];
                centre(g, cen);
                float far = INFINITY;
                for (int k = lane; k < nb; k += 32) far = fminf(far, fine_far2(fc, cen, s_at[k]));
                far = warp_min(far);
                if (lane == 0) s_far[g] = fminf(s_far[g], far);
            }
        }
        __syncthreads();
        for (int g = t; g < K3; g += blockDim.x) atomicMax((int *)&s_tmax, __float_as_int(thresh(g)));
        __syncthreads();
        const float thr1 = s_tmax + slack;
        // the stencil cells that hold atoms and (orthogonal cells) reach
        // within thr1 of this one, moved to the front; s_pre becomes the
        // exclusive scan of their counts
        if (t < 32) {
            int run = 0, cells = 0;
            for (int i0 = 0; i0 < nst; i0 += 32) {
                const int i = i0 + t;
                int v = i < nst ? s_pre[i] : 0;
                const int beg = i < nst ? s_beg[i] : 0;
                const short oi = i < nst ? s_oi[i] : (short)0;
                if (v > 0 && fc.ortho) {
                    const int dx = i % nx - La0, dy = (i / nx) % ny - La1, dz = i / (nx * ny) - La2;
                    const float gx = fmaxf((float)abs(dx) - 1.f, 0.f) * fabsf(fc.e[0]), gy = fmaxf((float)abs(dy) - 1.f, 0.f) * fabsf(fc.e[4]),
                                gz = fmaxf((float)abs(dz) - 1.f, 0.f) * fabsf(fc.e[8]);
                    if (sqrtf(fmaf(gz, gz, fmaf(gy, gy, gx * gx))) * (float)K > thr1 + slack) v = 0;
                }
                int incl = v;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, incl, o);
                    if (t >= o) incl += u;
                }
                const unsigned m = __ballot_sync(0xffffffffu, v > 0);
                __syncwarp();  // every lane has read its cell: the stores go to cells of this group or before it
                if (v > 0) {
                    const int at = cells + __popc(m & below);
                    s_pre[at] = run + incl - v;
                    s_beg[at] = beg;
                    s_oi[at] = oi;
                }
                __syncwarp();
                cells += __popc(m);
                run += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (t == 0) {
                s_pre[cells] = run;
                s_cells = cells;
            }
        }
        __syncthreads();
        ncells = s_cells;
        N = s_pre[ncells];
        // pass 1: an upper bound of the nearest atom's distance over each fine
        // cell, and the smallest distance of any atom to it
        int cursor = 0;
        while (cursor < N) {
            const int nb = stage_kept(cursor, thr1);
            kept = kept == -1 && cursor >= N ? nb : -2;  // one stage held every atom that passed
            for (int g = warp; g < K3; g += nwarps) {
                float cen[3];
                centre(g, cen);
                float far = INFINITY, near = INFINITY;
                for (int k = lane; k < nb; k += 32) {
                    const float4 p = s_at[k];
                    far = fminf(far, fine_far2(fc, cen, p));
                    near = fminf(near, fine_near2(fc, cen, p));
                }
                far = warp_min(far);
                near = warp_min(near);
                if (lane == 0) {
                    s_far[g] = fminf(s_far[g], far);
                    s_near[g] = fminf(s_near[g], near);
                }
            }
            __syncthreads();
        }
        for (int g = t; g < K3; g += blockDim.x) B.gedge[ebase + g] = make_float2(lowest(g), thresh(g));
        __syncthreads();
        if (t == 0) s_tmax = 0.f;
        __syncthreads();
    }
    // pass 2: the atoms whose smallest distance to the fine cell is within T,
    // by bucket of that distance: counted, then written
    auto LT = [&](int g, float &L, float &T) {
        L = lowest(g);
        T = thresh(g);
    };
    for (int g = t; g < K3; g += blockDim.x) {
        float L, T;
        LT(g, L, T);
        atomicMax((int *)&s_tmax, __float_as_int(T));
#pragma unroll
        for (int b = 0; b < kAgridBuckets; ++b) s_pos[g][b] = 0;
    }
    __syncthreads();
    const float thr2 = s_tmax + slack;
    float4 *ent = B.gent + (int64_t)f * B.gcap;
    // one stage of atoms through every fine cell: lane k of a group of 32
    // tests atom k; counting sums the buckets, filling writes each bucket's
    // atoms in stage order after its start.  Lane b < 8 keeps the position of
    // bucket b, and three ballots of the bucket's bits give every lane the
    // lanes of any bucket.
    auto pass2 = [&](int nb, bool fill) {
        for (int g = warp; g < K3; g += nwarps) {
            float cen[3];
            centre(g, cen);
            float L, T;
            LT(g, L, T);
            const float lim2 = fc.ortho ? T * T : (T + fc.R) * (T + fc.R);
            const float inv = T > L ? (float)kAgridBuckets / (T - L) : 0.f;
            int pos = s_pos[g][lane & (kAgridBuckets - 1)];
            for (int k0 = 0; k0 < nb; k0 += 32) {
                const int k = k0 + lane;
                const float4 p = s_at[min(k, nb - 1)];
                const float d2 = fine_near2(fc, cen, p);
                const bool in = k < nb && d2 <= lim2;
                const unsigned m = __ballot_sync(0xffffffffu, in);
                if (m == 0u) continue;
                const float d = sqrt_approx(d2);
                const int bk = min(kAgridBuckets - 1, max(0, (int)(((fc.ortho ? d : fmaxf(d - fc.R, 0.f)) - L) * inv)));
                const unsigned b0 = __ballot_sync(0xffffffffu, bk & 1), b1 = __ballot_sync(0xffffffffu, bk & 2),
                               b2 = __ballot_sync(0xffffffffu, bk & 4);
                auto of = [&](int q) { return m & (q & 1 ? b0 : ~b0) & (q & 2 ? b1 : ~b1) & (q & 4 ? b2 : ~b2); };
                if (fill) {
                    const int at = __shfl_sync(0xffffffffu, pos, bk) + __popc(of(bk) & below);
                    if (in) ent[at] = p;
                }
                pos += __popc(of(lane));
            }
            __syncwarp();
            if (lane < kAgridBuckets) s_pos[g][lane] = pos;
        }
    };
    // pass 1's single stage holds every atom that passes thr2 (thr2 <= thr1),
    // and the others fail the bucket test: counting and filling reuse it
    auto sweep = [&](bool fill) {
        int cursor = 0;
        if (kept >= 0) {
            pass2(kept, fill);
            cursor = N;
        }
        while (cursor < N) {
            const int nb = stage_kept(cursor, thr2);
            pass2(nb, fill);
            __syncthreads();
        }
        __syncthreads();
    };
    sweep(false);
    // the CTA's lists: offsets by (fine cell, bucket), one reservation in the
    // frame's pool, the starts and each fine cell's end
    int tot = 0;
    if (t < K3) {
#pragma unroll
        for (int b = 0; b < kAgridBuckets; ++b) {
            const int n = s_pos[t][b];
            s_pos[t][b] = tot;
            tot += n;
        }
    }
    int incl = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) s_wsum[warp] = incl;
    __syncthreads();
    int wbefore = 0, all = 0;
    for (int w = 0; w < nwarps; ++w) {
        wbefore += w < warp ? s_wsum[w] : 0;
        all += s_wsum[w];
    }
    if (t == 0) {
        const int base = atomicAdd(B.gpool + f, all);
        if ((int64_t)base + all > B.gcap) {
            B.FS[f].agrid = 0;  // this frame's queries take the walk
            atomicAdd(S.stats + ST_AGRID_OVF, 1ull);
            atomicMax(S.stats + ST_AGRID_NEED, (unsigned long long)((int64_t)base + all));
            s_base = -1;
        } else {
            s_base = base;
        }
    }
    __syncthreads();
    if (s_base < 0) continue;
    if (t < K3) {
        const int start = s_base + wbefore + incl - tot;
        int *st = B.gstart + gbase + (int64_t)t * (kAgridBuckets + 1);
#pragma unroll
        for (int b = 0; b < kAgridBuckets; ++b) {
            s_pos[t][b] += start;
            st[b] = s_pos[t][b];
        }
        st[kAgridBuckets] = start + tot;
    }
    __syncthreads();
    sweep(true);
    }
}

__global__ void __launch_bounds__(kAgridBuildThreads, kAgridBuildCtas) k_agrid_build(DevSys S, Bufs B) {
    k_agrid_build_body(blockIdx, gridDim, S, B);
}

// A site's fine cell (FP32 position q in search cell (cx, cy, cz)): its list's
// bucket starts and the smallest distance and width of its buckets.
struct AgridCell {
    const int *st;  // kAgridBuckets + 1 starts in the frame's entries
    float lo, w;
};

__device__ __forceinline__ AgridCell agrid_cell(const Bufs &B, const FrameGeom &G, const FrameScratch &F, int f, int packed,
                                                float4 q) {
    const int K = B.agk;
    const int cx = packed & 1023, cy = (packed >> 10) & 1023, cz = packed >> 20;
    int gi[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float u = fmaf(F.hin[3 * k + 2], q.z, fmaf(F.hin[3 * k + 1], q.y, F.hin[3 * k] * q.x));
        gi[k] = min(max((int)floorf(u * (float)K), 0), K - 1);
    }
    const int64_t fine = (int64_t)((cz * G.n[1] + cy) * G.n[0] + cx) * (K * K * K) + (gi[2] * K + gi[1]) * K + gi[0];
    const float2 edge = B.gedge[(int64_t)f * B.gfs + fine];
    AgridCell c;
    c.st = B.gstart + ((int64_t)f * B.gfs + fine) * (kAgridBuckets + 1);
    c.lo = edge.x;
    c.w = (edge.y - edge.x) * (1.0f / (float)kAgridBuckets);
    return c;
}

// One site's query: the top-2 update over its fine cell's list (p1 holds the
// solute atom index in the molecule), bucket by bucket of the entries'
// smallest distance to the fine cell.  A bucket whose smallest distance
// exceeds the running minimum (for the reference site, also its own minimum)
// by more than `band` holds no atom that can be the minimum, be within the
// guard band of it or lower the reference row, and neither do the buckets
// after it.
// GL lanes (gl = 0 .. GL - 1) split the list; each ends with its own entries' values.
template <int GL>
__device__ __forceinline__ void agrid_query(int gl, const Bufs &B, const FrameGeom &G, const FrameScratch &F, int f, int packed,
                                            float4 q, int b, bool isref, float band, Top2 &T, long long &evals) {
    const AgridCell c = agrid_cell(B, G, F, f, packed, q);
    const float4 *e = B.gent + (int64_t)f * B.gcap;
    int i = c.st[0], next = c.st[1];
    const int last = c.st[kAgridBuckets];
    if (i >= last) return;
    int k = 0;
#pragma unroll 1
    for (;;) {
        while (i >= next) {  // the bucket of entry i
            ++k;
            next = c.st[k + 1];
        }
        const float thr = fmaxf(sqrtf(T.m1), isref ? sqrtf(T.r1) : 0.f) + band;
        if (fmaf(c.w, (float)k, c.lo) > thr) break;
        // four entries in flight: past the end the last one again, as infinity
        float4 a[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) a[j] = e[min(i + GL * j + gl, last - 1)];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float ex = a[j].x - q.x, ey = a[j].y - q.y, ez = a[j].z - q.z;
            float d2 = fmaf(ez, ez, fmaf(ey, ey, ex * ex));
            if (GL > 1 || j > 0) d2 = i + GL * j + gl < last ? d2 : INFINITY;
            T.m2 = fminf(T.m2, fmaxf(T.m1, d2));
            const bool lt = d2 < T.m1;
            T.p1 = lt ? __float_as_int(a[j].w) : T.p1;
            T.b1 = lt ? b : T.b1;
            T.m1 = fminf(T.m1, d2);
            if (isref) T.r1 = fminf(T.r1, d2);
        }
        if (GL == 1) evals += min(4, last - i);
        else evals += gl == 0 ? min(4 * GL, last - i) : 0;
        i += 4 * GL;
        if (i >= last) break;
    }
}

// Exact scan of a slot's or molecule's sites over their lists: every list
// entry whose FP32 squared distance is within thr_arg (or, for the reference
// site, thr_r1) is evaluated exactly (exact_d2 on the input coordinates) and
// kept by the reference's tie rule -- the pairs of atoms_exact's stencil walk
// for the same thresholds.  The thresholds come from the query's minima plus
// 2 delta, so each such atom lies within (nearest distance + 3 delta) of its
// site, which the list's margin covers, and the buckets past sqrt(thr) + band
// hold none of them.  A group of GL lanes (gl the lane in it) splits the lists;
// every lane of the warp calls it (both thresholds negative: nothing to scan).
template <int GL>
__device__ __noinline__ void agrid_exact(int gl, const DevSys &S, const Bufs &B, const FrameGeom &G, const FrameScratch &F,
                                         int f, ExactMol &X, const int *vc, const float4 *vq, float band, float thr_arg,
                                         float thr_r1, Best64 &Bst, double &rr1, long long &evals) {
    best_init(Bst);
    rr1 = INFINITY;
    evals = 0;
    const int apv = fmaxf(thr_arg, thr_r1) >= 0.f ? S.apv : 0;
    const float4 *e = B.gent + (int64_t)f * B.gcap;
    for (int b = 0; b < apv; ++b) {
        const bool isref = b == S.iref;
        const float thr = isref ? fmaxf(thr_arg, thr_r1) : thr_arg;
        if (!(thr >= 0.f)) continue;
        const float4 q = vq[b];
        const AgridCell c = agrid_cell(B, G, F, f, vc[b], q);
        const float lim = sqrtf(thr) + band;
        double yb[3];
        bool have_y = false;
        const int i0 = c.st[0];
        int last = i0;  // the end of the buckets that can hold such an atom
        for (int k = 0; k < kAgridBuckets && fmaf(c.w, (float)k, c.lo) <= lim; ++k) last = c.st[k + 1];
        for (int i = i0; i < last; i += 4 * GL) {
            float4 a[4];
            unsigned need = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) a[j] = e[min(i + GL * j + gl, last - 1)];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float ex = a[j].x - q.x, ey = a[j].y - q.y, ez = a[j].z - q.z;
                const float d2f = fmaf(ez, ez, fmaf(ey, ey, ex * ex));
                if (i + GL * j + gl < last && (d2f <= thr_arg || (isref && d2f <= thr_r1))) need |= 1u << j;
            }
            for (; need; need &= need - 1) {
                const int j = __ffs(need) - 1;
                if (!have_y) {
                    exact_solvent_atom(B, G, X, b, yb);
                    have_y = true;
                }
                const int ai = __float_as_int(j == 0 ? a[0].w : j == 1 ? a[1].w : j == 2 ? a[2].w : a[3].w);
                double xa[3];
                exact_solute_atom(B, X, ai, xa);
                const double d2 = exact_d2(G, xa, yb);
                evals++;
                if (d2 <= S.cut2) {
                    if (isref) rr1 = fmin(rr1, d2);
                    best_update<false>(Bst, d2, ai, b);
                }
            }
        }
    }
    if (GL > 1) {
        // the group's smallest d = sqrt(d2), among equal d the larger (a, b); every lane ends with it
        double d = Bst.d2 <= S.cut2 ? best_d(Bst) : INFINITY;
#pragma unroll
        for (int o = GL / 2; o > 0; o >>= 1) {
            const double od = __shfl_xor_sync(0xffffffffu, d, o), od2 = __shfl_xor_sync(0xffffffffu, Bst.d2, o);
            const int oa = __shfl_xor_sync(0xffffffffu, Bst.a, o), ob = __shfl_xor_sync(0xffffffffu, Bst.b, o);
            if (od < d || (od == d && (oa > Bst.a || (oa == Bst.a && ob > Bst.b)))) {
                if (od < d) Bst.d2 = od2;
                d = od;
                Bst.a = oa;
                Bst.b = ob;
            }
            rr1 = fmin(rr1, __shfl_xor_sync(0xffffffffu, rr1, o));
            evals += __shfl_xor_sync(0xffffffffu, evals, o);
        }
        Bst.d = d <= 1e300 ? d : -1.0;
    }
}

// The record of a query's top-2 when every value is farther than the band
// from its decision boundary (the unambiguous branch of atoms_decide):
// 0 = no record within the cutoff, 1 = record r, 2 = inside the band (the
// record is then agrid_record's).
__device__ __forceinline__ int agrid_decide(const DevSys &S, const Guard &g, const Top2 &T, int64_t vb, DirRec &r) {
    r = dir_none(S);
    if (!(T.m1 <= g.cutp2)) return 0;
    const float d1 = sqrtf(T.m1);
    if (T.m1 >= g.cutm2 || (sqrtf(T.m2) - d1) <= g.two_delta) return 2;
    const int bin = bin_of(g, d1);
    if (bin < 0 || (S.usecutoff && d1 >= g.dbulk_lo && d1 <= g.dbulk_hi)) return 2;
    r.within = 1;
    r.i_local = T.p1;
    r.j = vb + T.b1;
    r.bin = bin;
    r.bulk = S.usecutoff ? (d1 > g.dbulk_hi) : 0;
    if (T.r1 <= g.cutp2) {
        const int rb = T.r1 < g.cutm2 ? bin_of(g, sqrtf(T.r1)) : -1;
        if (rb < 0) return 2;
        r.ref = 1;
        r.rbin = rb;
    }
    return 1;
}

// The record of a query inside the band (agrid_decide's 2), decided by
// atoms_decide's rules with the exact scans over the sites' lists (agrid_exact)
// instead of the stencil walk: v the solvent molecule (sample < 0) or the
// slot of sample `sample`, whose placement is drawn again in FP64.  Every lane
// of the warp calls it (active: the lane's group has a record), so that the
// groups go through the FP64 chain together; the GL lanes of a group share the
// scan and return the same record, the first one counts the statistics.
template <int GL>
__device__ __forceinline__ DirRec agrid_record(int gl, bool active, const DevSys &S, const Bufs &B, const FrameGeom &G,
                                               const FrameScratch &F, int f, int v, int sample, const int *vc,
                                               const float4 *vq, const Top2 &T, LocalStats &st) {
    const Guard &g = F.g;
    const float band = g.list_band;
    const int64_t vb = (int64_t)v * S.apv;
    ExactMol X;
    if (active) {
        if (sample < 0) {
            X = exact_mol(S, f, 0, v);
        } else {
            const Sample sm = B.samples[sample];
            const Placement P = draw_placement(S, G.frame_id, sm, v, B.bulk + (int64_t)f * B.ndist * B.mv,
                                               B.nbulk + (int64_t)f * B.ndist);
            uint64_t rs = P.st;
            double R[9];
            draw_rotation(rs, R);
            X = exact_mol_placed(S, G, f, sm.s, P.jmol, P.fc, R);
            exact_mol_ready(B, G, X);
        }
    }
    __syncwarp();
    DirRec r = dir_none(S);
    active = active && T.m1 <= g.cutp2;
    const float d1 = sqrtf(T.m1);
    // amb: the closest pair or the cutoff decision needs the exact scan; else
    // the search's minimum pair is the exact minimum pair
    const bool amb = active && (T.m1 >= g.cutm2 || (sqrtf(T.m2) - d1) <= g.two_delta);
    int bin = active && !amb ? bin_of(g, d1) : -1;
    const bool edge = active && !amb && (bin < 0 || (S.usecutoff && d1 >= g.dbulk_lo && d1 <= g.dbulk_hi));
    const bool ref = active && T.r1 <= g.cutp2;
    int rb = ref && !amb && T.r1 < g.cutm2 ? bin_of(g, sqrtf(T.r1)) : -1;
    const bool rscan = ref && rb < 0;
    Best64 Bst;
    double rr1;
    long long ev;
    agrid_exact<GL>(gl, S, B, G, F, f, X, vc, vq, band, amb ? r_sq_ru(d1 + g.two_delta) : -1.f,
                    rscan ? r_sq_ru(sqrtf(T.r1) + g.two_delta) : -1.f, Bst, rr1, ev);
    double d64 = -1.0;
    if (edge) d64 = sqrt(exact_pair_d2(B, G, X, T.p1, T.b1));
    if (!active) return r;
    if (gl == 0) {
        if (amb || rscan) {
            st.guard++;
            st.guard_pairs += ev;
        }
        if (edge) {
            st.guard++;
            st.guard_pairs++;
        }
    }
    r.within = 1;
    if (amb) {
        if (!(Bst.d2 <= S.cut2)) {
            r.within = 0;
            return r;
        }
        d64 = best_d(Bst);
        r.i_local = Bst.a;
        r.j = vb + Bst.b;
    } else {
        r.i_local = T.p1;
        r.j = vb + T.b1;
    }
    if (amb || edge) {
        if (gl == 0) st.maxerr = fmax(st.maxerr, fabs((double)d1 - d64));
        bin = setbin0(d64, S.binstep);
    }
    r.bin = bin;
    r.bulk = S.usecutoff ? (d64 >= 0.0 ? (d64 > S.dbulk) : (d1 > g.dbulk_hi)) : 0;
    if (rscan) rb = rr1 <= S.cut2 ? setbin0(sqrt(rr1), S.binstep) : -1;
    if (rb >= 0) {
        r.ref = 1;
        r.rbin = rb;
    }
    return r;
}

// Top-2 of a molecule's or slot's sites over their lists (vc, vq: its sites'
// cells and positions); false when no listed atom was met.  With GL > 1 every
// lane of the warp calls it (active: the lane's group has a query) and a group
// ends with the same values.
template <int GL>
__device__ __forceinline__ bool agrid_top2(int gl, bool active, const DevSys &S, const Bufs &B, const FrameGeom &G, const FrameScratch &F, int f,
                                           const int *vc, const float4 *vq, Top2 &T, long long &ev) {
    top2_init(T);
    ev = 0;
    const float band = F.g.list_band;
    const int apv = active ? S.apv : 0;
    for (int b = 0; b < apv; ++b) agrid_query<GL>(gl, B, G, F, f, vc[b], vq[b], b, b == S.iref, band, T, ev);
    if (GL > 1) {
        // the group's top-2; every lane ends with it
#pragma unroll
        for (int o = GL / 2; o > 0; o >>= 1) {
            const float m1 = __shfl_xor_sync(0xffffffffu, T.m1, o), m2 = __shfl_xor_sync(0xffffffffu, T.m2, o);
            const int p1 = __shfl_xor_sync(0xffffffffu, T.p1, o), b1 = __shfl_xor_sync(0xffffffffu, T.b1, o);
            T.m2 = fminf(fmaxf(T.m1, m1), fminf(T.m2, m2));
            if (m1 < T.m1 || (m1 == T.m1 && (p1 < T.p1 || (p1 == T.p1 && b1 < T.b1)))) {
                T.p1 = p1;
                T.b1 = b1;
            }
            T.m1 = fminf(T.m1, m1);
            T.r1 = fminf(T.r1, __shfl_xor_sync(0xffffffffu, T.r1, o));
        }
        return __shfl_sync(0xffffffffu, (int)(ev != 0), 0, GL) != 0;
    }
    return ev != 0;
}

// A query inside the band: listed for k_agrid_records (counters[9] entries in
// adefer, which holds every query of a launch).  About one query in a hundred
// is inside the band, and decided on the spot it left its warp on one lane of
// dependent FP64 operations in a third of the warp's rounds.
__device__ __forceinline__ void agrid_defer(const Bufs &B, int entry) {
    B.adefer[atomicAdd(B.counters + 9, 1)] = entry;
}

// Real pass of a single solute molecule, GL lanes per (frame, solvent
// molecule), persistent grid; frames without a grid queue their near pairs
// for k_atoms_eval (k_atoms_filter's rule).
template <int GL>
__device__ __forceinline__ void agrid_real(const DevSys &S, const Bufs &B) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned int *hbase = (unsigned int *)smem_raw;
    shist_zero(S, hbase);
    __syncthreads();
    const SHist h = shist_bind(S, hbase);
    LocalStats st;
    const int apv = S.apv;
    const int64_t n = (int64_t)B.nf * S.mv;
    auto put = [&](const DirRec &r, int f, int v) {
        st.molpairs++;
        if (r.within) {
            apply_hit(S, h, false, r.bin, r.i_local, r.j, r.ref, r.rbin);
            st.hits++;
            if (B.slot) {
                const int sl = B.slot[(int64_t)f * B.ms];
                if (sl >= 0) B.flags[((int64_t)f * B.ndist + sl) * S.mv + v] = flag_code(r);
            }
        }
    };
    const int lane = threadIdx.x & 31, gl = lane % GL;
    auto one_molecule = [&](int it, bool active) {
        const int f = it / S.mv, v = it - f * S.mv;
        const FrameScratch &F = B.FS[f];
        const FrameGeom &G = B.G[f];
        const int *vc = B.avcell + (int64_t)f * B.Nv + (int64_t)v * apv;
        if (!F.agrid && active) {
            active = false;
            if (gl == 0) {
                if (!F.ok) raise_err(S, ERR_STENCIL);
                else if (atoms_near(B, G, f, 0, vc, apv)) atoms_push(S, B, make_int4(v, 0, f, 0));
            }
        }
        const float4 *vq = B.avq32 + (int64_t)f * B.Nv + (int64_t)v * apv;
        Top2 T;
        long long ev;
        if (!agrid_top2<GL>(gl, active, S, B, G, F, f, vc, vq, T, ev)) return;
        DirRec r;
        if (gl != 0) return;
        if (agrid_decide(S, F.g, T, (int64_t)v * apv, r) == 2) {
            agrid_defer(B, it);
            return;
        }
        st.atompairs += (unsigned long long)ev;
        put(r, f, v);
    };
    // warps take their molecules from counters[6] (zeroed with the
    // chunk's counters), as k_agrid_random takes its slots; nf mv < 2^31 (the
    // fallback's queue holds every item of the chunk)
    for (;;) {
        long long at = 0;
        if (lane == 0) at = (long long)atomicAdd((unsigned long long *)(B.counters + 6), (unsigned long long)(32 / GL));
        at = __shfl_sync(0xffffffffu, at, 0) + lane / GL;
        if (at - lane / GL >= n) break;
        one_molecule((int)(at < n ? at : n - 1), at < n);
        __syncwarp();
    }
    stats_flush(S, st, false);
    __syncthreads();
    shist_flush(S, h, false);
}

// Lanes per query: one for small solvent molecules, whose slots are many;
// four for larger ones (more than four sites), whose lists are long and whose
// slots do not fill the SMs (181 14-site molecules, 20 frames, 10 samples:
// 235 us with one lane, 96 with four; 2,000 around a 20,000-atom chain, 16
// frames: 891 and 436).  Four resident CTAs per SM: the queries wait on their
// list entries.
template <int GL>
__global__ void __launch_bounds__(256, 4) k_agrid_real(DevSys S, Bufs B) {
    agrid_real<GL>(S, B);
}

// Random insertion of a single solute molecule, last pass: GL lanes per
// slot that k_atoms_place placed, in the order of the slots' fine cells;
// persistent grid.  The slot's sites are queried and the record is decided, or
// listed for k_agrid_records when it lies inside the band.  k_atoms_place has
// queued the near slots of the frames without a grid for k_atoms_eval.
//
// The loads of the lists bound it: a 16-byte load of 32 lanes from 32 lists
// takes about 11 cycles of the SM's L1 port, four times the arithmetic on it.
// Slots of a fine cell read the same lists, so in fine-cell order a warp's
// lanes share their lines and finish their lists together, and four entries
// per lane in flight then pay.  On a 43,000-atom system (50 frames, 10
// samples) the queries went from 2,850 to 1,980 us sorted and four wide, to
// 1,250 us (978 here, 274 in k_agrid_records) with the records inside the
// band apart and 4 M slots a launch instead of 32 samples.
template <int GL>
__device__ __forceinline__ void agrid_random(const DevSys &S, const Bufs &B, int sample0) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned int *hbase = (unsigned int *)smem_raw;
    shist_zero(S, hbase);
    __syncthreads();
    const SHist h = shist_bind(S, hbase);
    LocalStats st;
    const int apv = S.apv;
    const int lane = threadIdx.x & 31, gl = lane % GL;
    const int n = min(B.counters[8], B.aslot_cap);
    auto put = [&](const DirRec &r) {
        st.molpairs++;
        if (r.within) {
            apply_hit(S, h, true, r.bin, r.i_local, r.j, r.ref, r.rbin);
            st.hits++;
        }
    };
    auto one_slot = [&](int e, bool active) {
        const int y = e / S.mv, k = e - y * S.mv;
        const int f = B.samples[sample0 + y].pad;
        const FrameScratch &F = B.FS[f];
        const FrameGeom &G = B.G[f];
        const int64_t base = (int64_t)y * B.Nv + (int64_t)k * apv;
        Top2 T;
        long long ev;
        if (!agrid_top2<GL>(gl, active, S, B, G, F, f, B.pcell + base, B.pq32 + base, T, ev)) return;
        DirRec r;
        if (gl != 0) return;
        if (agrid_decide(S, F.g, T, (int64_t)k * apv, r) == 2) {
            agrid_defer(B, e);
            return;
        }
        st.atompairs += (unsigned long long)ev;
        put(r);
    };
    // warps take their slots from counters[6] (zeroed with the slot list): a
    // fixed share per thread left the CTAs' warps waiting for their slowest one
    for (;;) {
        int at = 0;
        if (lane == 0) at = atomicAdd(B.counters + 6, 32 / GL);
        at = __shfl_sync(0xffffffffu, at, 0);
        if (at >= n) break;
        at += lane / GL;
        one_slot(B.sslot[min(at, n - 1)], at < n);
        __syncwarp();
    }
    stats_flush(S, st, true);
    __syncthreads();
    shist_flush(S, h, true);
}

template <int GL>
__global__ void __launch_bounds__(256, 4) k_agrid_random(DevSys S, Bufs B, int sample0) {
    agrid_random<GL>(S, B, sample0);
}

// The listed queries inside the band, a group of lanes each: queried again and
// decided by agrid_record, the groups of a warp in step (left to run apart
// they took 176 us instead of 51 on 50,000 slots of 1,200 atoms).  RANDOM: entries y mv + slot of the piece from
// sample sample0 on; else entries frame mv + molecule.  Its time is the
// latency of one record's FP64 chain; the list holds a few per SM, so they run
// side by side.
template <bool RANDOM>
__device__ __forceinline__ void k_agrid_records_body(const uint3 blockIdx, const dim3 gridDim, const DevSys &S, const Bufs &B, int sample0) {
    const int n = B.counters[9];
    if ((int64_t)blockIdx.x * (blockDim.x / kAgridRecLanes) >= n) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned int *hbase = (unsigned int *)smem_raw;
    shist_zero(S, hbase);
    __syncthreads();
    const SHist h = shist_bind(S, hbase);
    LocalStats st;
    const int gl = threadIdx.x % kAgridRecLanes;
    const int per = blockDim.x / kAgridRecLanes;
    // every lane takes every round: the groups stay together
    for (int i0 = blockIdx.x * per; i0 < n; i0 += gridDim.x * per) {
        const int it = i0 + threadIdx.x / kAgridRecLanes;
        const bool active = it < n;
        const int e = B.adefer[min(it, n - 1)];
        const int row = e / S.mv, v = e - row * S.mv;
        const int f = RANDOM ? B.samples[sample0 + row].pad : row;
        const FrameScratch &F = B.FS[f];
        const FrameGeom &G = B.G[f];
        const int64_t base = (int64_t)row * B.Nv + (int64_t)v * S.apv;
        const int *vc = (RANDOM ? B.pcell : B.avcell) + base;
        const float4 *vq = (RANDOM ? B.pq32 : B.avq32) + base;
        Top2 T;
        long long ev;
        agrid_top2<kAgridRecLanes>(gl, active, S, B, G, F, f, vc, vq, T, ev);
        const DirRec r = agrid_record<kAgridRecLanes>(gl, active, S, B, G, F, f, v, RANDOM ? sample0 + row : -1, vc, vq, T, st);
        if (!active || gl != 0) continue;
        st.molpairs++;
        st.atompairs += (unsigned long long)ev;
        if (r.within) {
            apply_hit(S, h, RANDOM, r.bin, r.i_local, r.j, r.ref, r.rbin);
            st.hits++;
            if (!RANDOM && B.slot) {
                const int sl = B.slot[(int64_t)f * B.ms];
                if (sl >= 0) B.flags[((int64_t)f * B.ndist + sl) * S.mv + v] = flag_code(r);
            }
        }
    }
    stats_flush(S, st, RANDOM);
    __syncthreads();
    shist_flush(S, h, RANDOM);
}

template <bool RANDOM>
__global__ void __launch_bounds__(kAgridRecThreads) k_agrid_records(DevSys S, Bufs B, int sample0) {
    k_agrid_records_body<RANDOM>(blockIdx, gridDim, S, B, sample0);
}

}  // namespace cmk
