// cm_fixed.h -- integer positions for the FP32 search's preparation kernels.
//
// The FP32 search starts from cell indices and cell-relative positions rounded
// to FP32.  Computed in FP64 they cost about 45 operations an atom, and an FP64
// instruction occupies a quarter of an SM for 64 cycles on this GPU: the prep
// kernels ran with the FP64 pipe 84 % busy and nothing else above 10 %.  Here
// a coordinate is an integer in units of 2^-40 Angstrom (exact for FP32 inputs
// above 2^-17 A and FP64 inputs above 2^12 A, truncated by less than 2^-40 A
// otherwise; below 2^22 A), H^-1 an integer in units of 2^-64, and the fractional coordinate
// their product modulo 1 in units of 2^-64: its upper bits times the cell count
// are the cell, the rest the position in it.  A position is within
//   3 (2^-40 A + |x| 2^-64 |H|) + |H| 2^-62
// of the one an exact evaluation of the same H^-1 gives, and its FP32
// cell-relative form within (1 + 2^-20) u of its magnitude (u = 2^-24): far
// below the bounds the guard band uses for the FP64 chain (eps of
// k_frame_consts, at least 512 2^-53 (X + 16 |H|)) and for the rounding.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#include "cm_geom.h"

namespace cmgeom {

constexpr int kFixBits = 40;  // position unit 2^-40 Angstrom

struct FixedGeom {
    int64_t A[9];         // row-major H^-1 in units of 2^-64
    int64_t H[9];         // column-major H in units of 2^-40 A
    float hn[9], hl[9];   // column-major cell edge vectors, FP32 and what that leaves
    float hi[9];          // row-major H^-1
    int n[3];
    int ortho;            // H diagonal
    int set, bad;         // filled in; with an entry out of range
};

CM_HD int64_t fix_mulhi(int64_t a, int64_t b) {
#if defined(__CUDA_ARCH__)
    return __mul64hi(a, b);
#else
    return (int64_t)(((__int128)a * (__int128)b) >> 64);
#endif
}

CM_HD float fix_fma(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
    return __fmaf_rn(a, b, c);
#else
    return fmaf(a, b, c);
#endif
}

// Entry i (0-8) of the matrices; false (the FP64 chain is used) for a cell
// narrower than about 2 A or beyond 2^20 A.
CM_HD bool fixed_geometry_entry(const FrameGeom &G, FixedGeom &X, int i) {
    const double a = G.Hi[i], h = G.H[i];
    const bool ok = fabs(a) < 0.49 && fabs(h) < 1048576.0;
    X.A[i] = ok ? (int64_t)(a * 18446744073709551616.0) : 0;
    X.H[i] = ok ? (int64_t)rint(h * 1099511627776.0) : 0;
    X.hn[i] = (float)G.Hn[i];
    X.hl[i] = (float)(G.Hn[i] - (double)X.hn[i]);
    X.hi[i] = (float)a;
    return ok;
}

// The coordinate as an integer; false when it is not finite or beyond the limit.
CM_HD bool fixed_of(float x, int64_t &X) {
    uint32_t b;
    memcpy(&b, &x, 4);
    const int e = (int)((b >> 23) & 255u);
    const int64_t m = (int64_t)((b & 0x7fffffu) | (e ? 0x800000u : 0u));
    const int s = (e ? e : 1) - (150 - kFixBits);
    const int64_t v = s >= 0 ? m << (s < 39 ? s : 0) : m >> (-s < 63 ? -s : 63);
    X = (b >> 31) ? -v : v;
    return e < 149;
}
CM_HD bool fixed_of(double x, int64_t &X) {
    uint64_t b;
    memcpy(&b, &x, 8);
    const int e = (int)((b >> 52) & 2047u);
    const int64_t m = (int64_t)((b & 0xfffffffffffffull) | (e ? 0x10000000000000ull : 0ull));
    const int s = (e ? e : 1) - (1075 - kFixBits);
    const int64_t v = s >= 0 ? m << (s < 10 ? s : 0) : m >> (-s < 63 ? -s : 63);
    X = (b >> 63) ? -v : v;
    return e < 1045;
}

// An upper bound of |X| in Angstrom, FP32.
CM_HD float fixed_abs(int64_t X) {
    const uint64_t a = (uint64_t)(X < 0 ? -X : X);
    return ((float)(uint32_t)(a >> 32) + 1.0f) * (1.0f + 0x1.0p-22f) * 0x1.0p-8f;
}

// X 2^-40 A in FP32, one rounding.
CM_HD float fixed_f32(int64_t X) {
    const int64_t h = X >> 20;
    if (h >= (1 << 24) || h <= -(1 << 24)) return (float)X * 0x1.0p-40f;
    return fix_fma((float)(int32_t)h, 0x1.0p-20f, (float)(int32_t)(X & 0xfffff) * 0x1.0p-40f);
}

// Hn (gh + gl), gh the leading 24 bits of a position in a cell (grid units) and
// gl the rest, rounded to FP32.
CM_HD void fixed_lat(const FixedGeom &X, const float *gh, const float *gl, float *q) {
    for (int m = 0; m < 3; ++m) {
        if (X.ortho) {
            const float h = X.hn[4 * m];
            q[m] = fix_fma(h, gh[m], fix_fma(h, gl[m], X.hl[4 * m] * gh[m]));
            continue;
        }
        float s = 0.f, c = 0.f;  // the sum and its compensation
        for (int k = 0; k < 3; ++k) {
            const float h = X.hn[3 * k + m];
            const float p = h * gh[k];
            c += fix_fma(h, gh[k], -p) + fix_fma(h, gl[k], X.hl[3 * k + m] * gh[k]);
            const float t = s + p, z = t - s;
            c += (s - (t - z)) + (p - z);
            s = t;
        }
        q[m] = s + c;
    }
}

// The leading 24 bits and the rest of a fraction in units of 2^-64.
CM_HD void fixed_split(uint64_t r, float &gh, float &gl) {
    gh = (float)(uint32_t)(r >> 40) * 0x1.0p-24f;
    gl = (float)(uint32_t)((r >> 16) & 0xffffffu) * 0x1.0p-48f;
}

// Cell and FP32 position in it of an integer position.
CM_HD void bin_fixed(const FixedGeom &X, int64_t x0, int64_t x1, int64_t x2, int *c, float *q) {
    const int64_t x[3] = {x0, x1, x2};
    float gh[3], gl[3];
    for (int k = 0; k < 3; ++k) {
        uint64_t f = 0;
        for (int j = 0; j < 3; ++j) {
            if (X.ortho && j != k) continue;
            const int64_t a = X.A[3 * k + j];
            f += ((uint64_t)fix_mulhi(x[j], a) << (64 - kFixBits)) | (((uint64_t)x[j] * (uint64_t)a) >> kFixBits);
        }
        c[k] = (int)cmfeed::mulhi64(f, (uint64_t)X.n[k]);
        fixed_split(f * (uint64_t)X.n[k], gh[k], gl[k]);
    }
    fixed_lat(X, gh, gl, q);
}

// d -> d - H rint(H^-1 d) for a displacement; false when an image index is too
// near a half for FP32 to decide (or the displacement beyond 2,000 A).
CM_HD bool fixed_unwrap(const FixedGeom &X, int64_t *d) {
    float v[3];
    for (int k = 0; k < 3; ++k) {
        if (d[k] >= (int64_t(1) << 51) || d[k] <= -(int64_t(1) << 51)) return false;
        v[k] = fixed_f32(d[k]);
    }
    float n[3];
    for (int k = 0; k < 3; ++k) {
        const float f = fix_fma(X.hi[3 * k + 2], v[2], fix_fma(X.hi[3 * k + 1], v[1], X.hi[3 * k] * v[0]));
        n[k] = rintf(f);
        if (!(fabsf(f - n[k]) < 0.499f) || fabsf(n[k]) > 1000.f) return false;
    }
    if (n[0] == 0.f && n[1] == 0.f && n[2] == 0.f) return true;
    for (int m = 0; m < 3; ++m)
        d[m] -= (int64_t)(int)n[0] * X.H[m] + (int64_t)(int)n[1] * X.H[3 + m] + (int64_t)(int)n[2] * X.H[6 + m];
    return true;
}

// sum += d for |d| below 2^51; false once the sum leaves (-2^62, 2^62), which a
// few thousand atoms far from their molecule's reference atom can make it do
// (2^62 units are 4.2 10^6 A).
CM_HD bool fixed_add(int64_t &sum, int64_t d) {
    sum = (int64_t)((uint64_t)sum + (uint64_t)d);
    return sum < (int64_t(1) << 62) && sum > -(int64_t(1) << 62);
}

// sum / n for n >= 1, within one unit.
CM_HD int64_t fixed_mean(int64_t sum, int n) {
    if (n == 1) return sum;
    const uint64_t r = ~0ull / (uint64_t)n;
    const int64_t v = (int64_t)cmfeed::mulhi64((uint64_t)sum, r);
    return sum < 0 ? v - (int64_t)r : v;
}

// Bounds of the FP32 search's displacement components in units of u = 2^-24
// (k_frame_consts): of an atom pair of the search, and what a slot of the
// random insertion adds when it is placed in FP32 (r: the molecule radius) or
// in FP64 from the molecule's FP32 offsets (their rounding, rotated).
CM_HD double fp32_pair_units(double Q, double OFF, double rs, double rv, double cut) {
    return (5.0 * Q + 4.0 * OFF + 2.0 * rv + rs + cut + 1.0) * (1.0 + 0x1.0p-19);
}
CM_HD double fp32_slot_units(double Q, double r) { return 5.0 * Q + 44.0 * r; }
CM_HD double fp32_offset_units(double r) { return r * (1.0 + 0x1.0p-19); }

}  // namespace cmgeom
