// Biot-Savart sums close to FP64's on the FP32 pipe: every quantity of a pair is an unevaluated sum
// hi + lo of two FP32 values (about 48 bits), two segments per packed instruction.
//
// GB300's FP64 pipe runs at 1/64 of the FP32 rate: 21 FP64 operations a pair end at 29 Gpairs/s.
// The same pair takes 150 FP32 lane operations here.  The rounding of a pair is about 1e-14 of its
// term, unbiased, so that the error of a point's field is close to kDfError sqrt(sum |term|^2),
// while every sum over more than 32 segments is taken in FP64.  That is used only where it is no more
// than what FP64 sums left:
//   Fields: the bound is summed beside the field (|term| <= |kl| |r|^-2), and the field is good only
//   where it is below what one FP64 sum over tiles of 256 segments left at least, whose rounding grew
//   with the root of their number: kDfLimit sqrt(n / 256) of |B| (measured 3.0e-17 in the dipole's bore
//   and up to 1 m outside, 3.8e-17 to 5.3e-17 along sections of 60 to 600 segments a turn, 7e-17 and more
//   for 5000 segments).  Elsewhere -- coarse windings, points outside, where terms cancel -- the caller
//   sums in FP64 (f64.cuh).
//   Tracks: a sub-block that is close to the point, and so has a good part of that sum, is taken in
//   FP64, unless all of it is below the rounding of the particle's velocity (df_reach).
//
// A sub-block is 32 consecutive segments with an origin o (the midpoint of its middle segment):
//   B = A x (p - o) - M,  A = sum kl |r|^-3,  M = sum (kl x (p0 - o)) |r|^-3.
// The bias of a rounding matters where its size would not: a sum rounded at 2^-49 of its value
// 46 080 times the same way is an error of 2^-49.  So every rounded low-order sum takes in a product
// with random low bits: the low part of a square alone (an odd number squared is 1 modulo 8) or a
// term below half an ulp added alone would be rounded the same way every time.
//
// Where the bound does not hold, or FP32's range does not, a warp sums the sub-block in FP64
// (df_plain): a point within 4 segment spacings of one of its segments, far out (10 km), currents
// far from ordinary ones, non-finite values; in tracks, a point within df_reach of it.
#pragma once

#include <type_traits>

#include "f64.cuh"
#include "tile.cuh"

namespace cctgpu {

constexpr int kDfSub = kSub64;         // segments of a sub-block
constexpr int kDfMinSegments = 2048;   // fewer terms hardly ever average their rounding enough
constexpr double kDfError = 1.4e-14;   // 1.0e-14 to 1.4e-14 measured, bores to 5 m outside (of the bound)
constexpr double kDfLimit = 3.0e-17;   // of |B|, by the root of the 256-segment tiles
__host__ inline double df_weight(int64_t n_seg) { return kDfError / kDfLimit * (kDfError / kDfLimit) * 256.0 / (double)n_seg; }
constexpr float kDfFar2 = 1.0e8f;      // squared distance (m^2) from which a sub-block is summed in FP64
constexpr float kDfSpacings2 = 16.0f;  // squared distance in segment spacings below which it is, too

// One sub-block in shared memory: per segment kl (hi, lo), m = kl x (p0 - o) (hi, lo), o - p0 (hi, lo).
struct __align__(16) DfSub {
    float v[18][kDfSub];
    double o[3];
    float near2;   // squared distance of the nearest segment below which FP64 takes over (inf: always)
    int count;
    float strength;            // (sum |kl|^2)^(1/4)
    float pad;
};
// For fields, with |kl|.
struct DfFieldSub : DfSub {
    float k[kDfSub];
};
__device__ __forceinline__ float *df_sizes(DfSub &) { return nullptr; }
__device__ __forceinline__ float *df_sizes(DfFieldSub &D) { return D.k; }

// x = hi + lo, hi the nearest FP32 (ties away from zero), by integer operations: a conversion to or
// from FP64 runs at the FP64 pipe's rate.  Exact to 2^-49 |x| for 2^-74 < |x| < 2^127; smaller
// magnitudes lose lo, then hi (below 2^-126).
__device__ __forceinline__ void df_split(double x, float &hi, float &lo) {
    const unsigned xh = (unsigned)__double2hiint(x), sign = xh & 0x80000000u;
    const unsigned long long r = (unsigned long long)__double_as_longlong(x) + (1ull << 28);
    const unsigned e = (xh >> 20) & 0x7ffu;
    const unsigned rh = (unsigned)(r >> 32), rl = (unsigned)r;
    const unsigned f = __funnelshift_l(rl, rh, 3) - (384u << 23);   // exponent rebased, low 9 bits of it kept
    const int d = (int)(rl & 0x1fffffffu) - (1 << 28);
    hi = e > 896u ? __uint_as_float((f & 0x7fffffffu) | sign) : 0.0f;
    const float scale = e > 948u ? __uint_as_float(((e - 948u) << 23) | sign) : 0.0f;   // 2^(e - 1075), signed
    lo = __fmul_rn((float)d, scale);
}

// FP32 -> FP64 by integer operations (zero and subnormals to zero; finite values only).
__device__ __forceinline__ double df_widen(float x) {
    const unsigned b = __float_as_uint(x), m = b & 0x7fffffffu;
    const unsigned h = m < 0x00800000u ? 0u : (m >> 3) + 0x38000000u;
    return __hiloint2double((int)(h | (b & 0x80000000u)), m < 0x00800000u ? 0 : (int)(b << 29));
}

// The calling warp writes the sub-block of its lanes' segments (converged; the caller synchronises).
template <class Sub>
__device__ __forceinline__ void df_stage(Sub &D, const SegRaw &R, int cnt) {
    const int lane = threadIdx.x & 31;
    const bool mine = lane < cnt;
    double q[3], m[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) q[c] = R.p[c] - R.o[c];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int d = (c + 1) % 3, e = (c + 2) % 3;
        m[c] = R.k[d] * q[e] - R.k[e] * q[d];
    }
    float qf[3], k2 = 0.0f;
    unsigned kmax = 0u;   // largest |kl| component, high word of the FP64 value
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        float hi, lo;
        df_split(R.k[c], hi, lo);
        k2 = __fmaf_rn(hi, hi, k2);
        D.v[c][lane] = mine ? hi : 0.0f;
        D.v[3 + c][lane] = mine ? lo : 0.0f;
        df_split(m[c], hi, lo);
        D.v[6 + c][lane] = mine ? hi : 0.0f;
        D.v[9 + c][lane] = mine ? lo : 0.0f;
        df_split(q[c], hi, lo);
        qf[c] = hi;
        D.v[12 + c][lane] = mine ? -hi : -1.0e9f;   // padding: no current, far away
        D.v[15 + c][lane] = mine ? -lo : 0.0f;
        kmax = max(kmax, (unsigned)__double2hiint(R.k[c]) & 0x7fffffffu);
        // a coordinate out of FP32's range counts as out of range too
        if (((unsigned)__double2hiint(q[c]) & 0x7fffffffu) >= 0x43000000u) kmax = 0x7fffffffu;
    }
    if (float *sizes = df_sizes(D)) sizes[lane] = mine ? __fsqrt_rn(k2) : 0.0f;
    // spacing: a segment's distance to its nearer neighbour, so that a jump from one winding layer
    // to the next does not count
    float len2 = 0.0f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float d = __shfl_down_sync(0xffffffffu, qf[c], 1) - qf[c];
        len2 = __fmaf_rn(d, d, len2);
    }
    if (lane + 1 >= cnt) len2 = __int_as_float(0x7f800000);
    const float before = __shfl_up_sync(0xffffffffu, len2, 1);
    len2 = fminf(len2, lane > 0 ? before : __int_as_float(0x7f800000));
    if (!mine || cnt == 1) len2 = 0.0f;
    if (!mine) k2 = 0.0f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        len2 = fmaxf(len2, __shfl_xor_sync(0xffffffffu, len2, o));
        k2 += __shfl_xor_sync(0xffffffffu, k2, o);
        kmax = max(kmax, __shfl_xor_sync(0xffffffffu, kmax, o));
    }
    if (lane == 0) {
        // |kl| of 1e-12 to 1e12 (or none at all), so that no term leaves FP32's range
        const bool in_range = kmax == 0u || (kmax >= 0x3d719799u && kmax < 0x426d1a94u);
        D.near2 = in_range && cnt > 1 ? fmaxf(kDfSpacings2 * len2, 1.0e-10f) : __int_as_float(0x7f800000);
        D.count = cnt;
        D.strength = __fsqrt_rn(__fsqrt_rn(k2));
#pragma unroll
        for (int c = 0; c < 3; ++c) D.o[c] = R.o[c];
    }
}

// FP64 sum of the sub-block for the points of a warp (every lane).
static __device__ __noinline__ void df_plain(const double *__restrict__ kls, const double *__restrict__ p0s, int64_t a,
                                             int cnt, double px, double py, double pz, double *b) {
    double bx = 0.0, by = 0.0, bz = 0.0;
    for (int64_t s = a; s < a + cnt; ++s) {
        const double kx = __ldg(kls + 3 * s), ky = __ldg(kls + 3 * s + 1), kz = __ldg(kls + 3 * s + 2);
        const double rx = px - __ldg(p0s + 3 * s), ry = py - __ldg(p0s + 3 * s + 1), rz = pz - __ldg(p0s + 3 * s + 2);
        const double inv = rsqrt(rx * rx + ry * ry + rz * rz);
        const double inv3 = inv * inv * inv;
        bx += (ky * rz - kz * ry) * inv3;
        by += (kz * rx - kx * rz) * inv3;
        bz += (kx * ry - ky * rx) * inv3;
    }
    b[0] = bx;
    b[1] = by;
    b[2] = bz;
}

// The same for the few lanes in `need`, one after the other, with a lane a segment (at most 32): 37 FP64
// instructions each where the loop above takes 22 a segment whatever the lanes (5 protons through the section
// of 120 segments a turn, pieces of 16 segments of which now and then one proton is close: 6.1 -> 5.5 ms).
// A lane's a, cnt and p are its own; its sum goes to b.  Called by whole warps.
static __device__ __noinline__ void df_plain_few(unsigned need, const double *__restrict__ kls, const double *__restrict__ p0s,
                                                 int64_t a, int cnt, double px, double py, double pz, double *b) {
    const int lane = threadIdx.x & 31;
    for (; need; need &= need - 1) {
        const int from = __ffs(need) - 1;
        const int64_t s = __shfl_sync(0xffffffffu, a, from) + lane;
        const int n = __shfl_sync(0xffffffffu, cnt, from);
        const double x = __shfl_sync(0xffffffffu, px, from), y = __shfl_sync(0xffffffffu, py, from),
                     z = __shfl_sync(0xffffffffu, pz, from);
        double t[3] = {0.0, 0.0, 0.0};
        if (lane < n) {
            const double kx = __ldg(kls + 3 * s), ky = __ldg(kls + 3 * s + 1), kz = __ldg(kls + 3 * s + 2);
            const double rx = x - __ldg(p0s + 3 * s), ry = y - __ldg(p0s + 3 * s + 1), rz = z - __ldg(p0s + 3 * s + 2);
            const double inv = rsqrt(rx * rx + ry * ry + rz * rz);
            const double inv3 = inv * inv * inv;
            t[0] = (ky * rz - kz * ry) * inv3;
            t[1] = (kz * rx - kx * rz) * inv3;
            t[2] = (kx * ry - ky * rx) * inv3;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int c = 0; c < 3; ++c) t[c] += __shfl_xor_sync(0xffffffffu, t[c], o);
        if (lane == from)
#pragma unroll
            for (int c = 0; c < 3; ++c) b[c] = t[c];
    }
}

// a + b = s + e exactly (Knuth)
__device__ __forceinline__ f2 df_two_sum(f2 a, f2 b, f2 &e) {
    const f2 s = f2_add(a, b), t = f2_sub(s, a);
    e = f2_add(f2_sub(a, f2_sub(s, t)), f2_sub(b, t));
    return s;
}

// Tracks: a sub-block is summed in FP64 for points closer to its nearest segment than strength * reach.  Its
// part in the sum of |term|^2 is at most strength^4 d^-4 at that distance d; hi + lo pairs are for the
// sub-blocks that have at most kDfShare / n of a field's square, n sub-blocks in all.  With |B| for that
// field, against 80-bit sums in the bores: dipole 0.75e-16 of |B| (FP64 sums over tiles of 128 segments
// 0.85e-16, pairs everywhere 1.7e-16), sections of 60 / 120 / 360 / 600 segments a turn 0.5 / 0.4 / 0.4 /
// 0.4e-16 (1.2 / 1.1 / 0.8 / 0.7; 3.5 / 3.2 / 1.8 / 1.4), 9 % to 27 % of the sub-blocks in FP64: less than
// 1e-16.  The field is the largest that the particle has met, or if that is larger the one of which 1e-16
// turns the particle over a whole step by 2^-57 (df_idle_field: 16 T for a proton of 215 MeV in steps of 10
// mm, 160 T at 1 mm).  Such errors, at random over a step's stages, are a part in seven of the rounding of
// the particle's velocity and add 1 % to it: tracks are as good as with FP64 sums.
constexpr float kDfShare = 5.0e-4f;
__device__ __forceinline__ float df_reach(int64_t n, double b2) {
    return __fsqrt_rn(__fsqrt_rn(__fdiv_rn((float)n, kDfShare * (float)b2)));
}
// (kq: charge over mass; the field's square)
__device__ __forceinline__ double df_idle_field(double kq, double dt) {
    const double b = 0.0694 / (kq * dt);      // 2^-57 / 1e-16
    return b * b;
}

// Field of segments 2 j0 .. 2 j1 - 1 of sub-block D (segments a .. a + count - 1 of kls / p0s) at the lane's
// point p.  Fields: also the sum of their (|kl| |r|^-2)^2 as far as the pairs are hi + lo (q).  Called by
// whole warps.
template <class Sub>
__device__ __forceinline__ void df_sub_sum(const Sub &D, const double *__restrict__ kls, const double *__restrict__ p0s,
                                           int64_t a, const double (&p)[3], double (&b)[3], double &q, float reach, int j0,
                                           int j1) {
    constexpr bool TRACK = !std::is_same<Sub, DfFieldSub>::value;
    const float near2 = D.near2;
    bool plain = !(near2 < __int_as_float(0x7f800000));
    if (!plain) {
        double w[3];
        f2 wh[3], wl[3];
        float far2 = 0.0f;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            w[c] = p[c] - D.o[c];
            float hi, lo;
            df_split(w[c], hi, lo);
            wh[c] = f2_pack(hi, hi);
            wl[c] = f2_pack(lo, lo);
            // beyond FP32's exponents (or NaN): far
            far2 = __fmaf_rn(hi, hi, far2);
            if (((unsigned)__double2hiint(w[c]) & 0x7fffffffu) >= 0x41000000u) far2 = __int_as_float(0x7f800000);
        }
        if (TRACK) {
            // (o is a segment's midpoint: this close, so is that segment)
            const float least = D.strength * reach;
            plain = far2 < least * least || far2 >= kDfFar2;
        }
        if (!TRACK || !plain) {
            f2 S[6], E[6], R[6], Q = 0ull;
#pragma unroll
            for (int c = 0; c < 6; ++c) S[c] = E[c] = R[c] = 0ull;
            float near_lo = __int_as_float(0x7f800000), near_hi = near_lo;
            const f2 one = f2_pack(1.0f, 1.0f), half = f2_pack(0.5f, 0.5f), c15 = f2_pack(1.5f, 1.5f), c1875 = f2_pack(1.875f, 1.875f);
#pragma unroll 2
            for (int j = j0; j < j1; ++j) {
                auto at = [&](int c) { return reinterpret_cast<const f2 *>(D.v[c])[j]; };
                // r = h + l
                f2 h[3], l[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    f2 e;
                    h[c] = df_two_sum(wh[c], at(12 + c), e);
                    l[c] = f2_add(f2_add(wl[c], at(15 + c)), e);
                }
                // |r|^2 = s + e
                f2 s, e, e1, e2;
                {
                    const f2 px = f2_mul(h[0], h[0]), py = f2_mul(h[1], h[1]), pz = f2_mul(h[2], h[2]);
                    const f2 ex = f2_fma(l[0], h[0], f2_fma(h[0], h[0], f2_neg(px)));
                    const f2 ey = f2_fma(l[1], h[1], f2_fma(h[1], h[1], f2_neg(py)));
                    const f2 ez = f2_fma(l[2], h[2], f2_fma(h[2], h[2], f2_neg(pz)));
                    f2 t = f2_fma(l[2], l[2], f2_fma(l[1], l[1], f2_mul(l[0], l[0])));
                    t = f2_fma(l[2], h[2], f2_fma(l[1], h[1], f2_fma(l[0], h[0], t)));
                    s = df_two_sum(df_two_sum(px, py, e1), pz, e2);
                    e = f2_add(f2_add(f2_add(f2_add(ex, ey), ez), t), f2_add(e1, e2));
                }
                float s0, s1;
                f2_unpack(s, s0, s1);
                near_lo = fminf(near_lo, s0);
                near_hi = fminf(near_hi, s1);
                // |r|^-3 = c + d: y ~ |r|^-1 (MUFU and a Newton step, so that v is small and its own rounding
                // with it), v = 1 - |r|^2 y^2, |r|^-3 = y^3 (1 + 3/2 v + 15/8 v^2 + O(v^3))
                f2 cc, d;
                {
                    const f2 y0 = f2_pack(rsqrt_mufu(s0), rsqrt_mufu(s1)), ns = f2_neg(s);
                    const f2 y = f2_fma(f2_mul(y0, half), f2_fma(ns, f2_mul(y0, y0), one), y0);
                    const f2 y2 = f2_mul(y, y), ye = f2_fma(y, y, f2_neg(y2));
                    if constexpr (!TRACK) {
                        const f2 u = f2_mul(reinterpret_cast<const f2 *>(D.k)[j], y2);
                        Q = f2_fma(u, u, Q);
                    }
                    f2 v = f2_fma(ns, y2, one);
                    v = f2_fma(ns, ye, v);
                    v = f2_fma(f2_neg(e), y2, v);
                    const f2 corr = f2_fma(c1875, f2_mul(v, v), f2_mul(c15, v));
                    const f2 c0 = f2_mul(y2, y);
                    d = f2_fma(ye, y, f2_fma(y2, y, f2_neg(c0)));            // y^3 = c0 + d
                    d = f2_fma(c0, corr, f2_fma(d, corr, d));
                    cc = f2_add(c0, d);
                    d = f2_sub(d, f2_sub(cc, c0));
                }
                // A += kl |r|^-3, M += m |r|^-3
#pragma unroll
                for (int c = 0; c < 6; ++c) {
                    const int at0 = c < 3 ? c : c + 3;
                    const f2 xh = at(at0), xl = at(at0 + 3);
                    const f2 t = f2_mul(xh, cc);
                    const f2 te = f2_fma(xl, cc, f2_fma(xh, d, f2_fma(xh, cc, f2_neg(t))));
                    f2 er;
                    S[c] = df_two_sum(S[c], t, er);
                    E[c] = f2_add(E[c], te);
                    R[c] = f2_add(R[c], er);
                }
            }
            // halves together, to FP64, A x w - M
            double T[6];
            float check = 0.0f;
#pragma unroll
            for (int c = 0; c < 6; ++c) {
                float s0, s1, e0, e1;
                f2_unpack(S[c], s0, s1);
                f2_unpack(E[c], e0, e1);
                float r0, r1;
                f2_unpack(R[c], r0, r1);
                const float s = __fadd_rn(s0, s1), t = __fsub_rn(s, s0), e = __fadd_rn(e0, e1);
                const float r = __fadd_rn(__fadd_rn(__fsub_rn(s0, __fsub_rn(s, t)), __fsub_rn(s1, t)), __fadd_rn(r0, r1));
                check = __fmaf_rn(r + e, 0.0f, check);   // NaN unless every sum is finite
                T[c] = df_widen(s) + (df_widen(r) + df_widen(e));
            }
            b[0] = (T[1] * w[2] - T[2] * w[1]) - T[3];
            b[1] = (T[2] * w[0] - T[0] * w[2]) - T[4];
            b[2] = (T[0] * w[1] - T[1] * w[0]) - T[5];
            float q0, q1;
            f2_unpack(Q, q0, q1);
            q = df_widen(__fadd_rn(q0, q1));
            const float least = TRACK ? fmaxf(near2, D.strength * reach * (D.strength * reach)) : near2;
            plain = !(fminf(near_lo, near_hi) > least && far2 < kDfFar2 && check == 0.0f);
        }
    }
    const unsigned need = __ballot_sync(0xffffffffu, plain);
    if (need) {
        double t[3];
        const int64_t from = a + 2 * j0;
        const int cnt = min(D.count, 2 * j1) - 2 * j0;
        if (TRACK && 37 * __popc(need) < 22 * 2 * (j1 - j0)) df_plain_few(need, kls, p0s, from, cnt, p[0], p[1], p[2], t);
        else df_plain(kls, p0s, from, cnt, p[0], p[1], p[2], t);
        if (plain) {      // (a field point's field does not depend on its neighbours)
#pragma unroll
            for (int c = 0; c < 3; ++c) b[c] = t[c];
            q = 0.0;
        }
    }
}

__device__ __forceinline__ void df_sub_field(const DfFieldSub &D, const double *__restrict__ kls, const double *__restrict__ p0s,
                                             int64_t a, const double (&p)[3], double (&b)[3], double &q) {
    df_sub_sum(D, kls, p0s, a, p, b, q, 0.0f, 0, kDfSub / 2);
}

__device__ __forceinline__ void df_track_field(const DfSub &D, const double *__restrict__ kls, const double *__restrict__ p0s,
                                               int64_t a, const double (&p)[3], float reach, double (&b)[3], int j0 = 0,
                                               int j1 = kDfSub / 2) {
    double q;
    df_sub_sum(D, kls, p0s, a, p, b, q, reach, j0, j1);
}

}  // namespace cctgpu
