// FP64 Biot-Savart sums over sub-blocks of 32 consecutive segments, staged in shared memory by a warp.
//
// With the midpoint of its middle segment as the origin o of a sub-block,
//   B = A x (p - o) - M,  A = sum kl |r|^-3,  M = sum (kl x (p0 - o)) |r|^-3  (moment form).
// Bound by the FP64 pipe (GB300: 1/64 of the FP32 rate), so operations and idle lanes are what count:
// 21 operations a pair here, 26 with kl x r formed a pair.  The cancellation in A x w - M costs
// |w| / |r| roundings, w = p - o: an origin a sub-block rather than a tile of 128 or 256 segments, and
// sums of 32 terms, leave 4e-17 to 7e-17 of |B| in the bores of the dipole and of sections of 60 to
// 600 segments a turn (tiles of 128: 0.6e-16 to 1.1e-16, of 256: 3.6e-16 to 2.3e-15; 80-bit reference).
#pragma once

#include <stdint.h>

namespace cctgpu {

constexpr int kSub64 = 32;             // segments of a sub-block

// A segment's FP64 values as a lane loads them ahead of their sub-block.
struct SegRaw {
    double k[3], p[3], o[3];
};

// One sub-block in shared memory: per segment kl, m = kl x (p0 - o), p0 - o.
struct __align__(16) F64Sub {
    double v[9][kSub64];
    double o[3];
    double pad;
};

// The calling warp loads the segments a .. a + cnt - 1 (cnt >= 1) and their origin.
__device__ __forceinline__ void sub_load(SegRaw &R, const double *__restrict__ kls, const double *__restrict__ p0s,
                                         int64_t a, int cnt) {
    const int lane = threadIdx.x & 31;
    const int64_t s = a + min(lane, cnt - 1), m = a + cnt / 2;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        R.k[c] = __ldg(kls + 3 * s + c);
        R.p[c] = __ldg(p0s + 3 * s + c);
        R.o[c] = __ldg(p0s + 3 * m + c);
    }
}

// The calling warp writes the sub-block of its lanes' segments (converged; the caller synchronises).
__device__ __forceinline__ void f64_stage(F64Sub &D, const SegRaw &R, int cnt) {
    const int lane = threadIdx.x & 31;
    const bool mine = lane < cnt;
    double q[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) q[c] = R.p[c] - R.o[c];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int d = (c + 1) % 3, e = (c + 2) % 3;
        D.v[c][lane] = mine ? R.k[c] : 0.0;
        D.v[3 + c][lane] = mine ? R.k[d] * q[e] - R.k[e] * q[d] : 0.0;
        D.v[6 + c][lane] = mine ? q[c] : 1.0e18;     // padding: no current, far away
    }
    if (lane == 0)
#pragma unroll
        for (int c = 0; c < 3; ++c) D.o[c] = R.o[c];
}

// Field of the sub-block's cnt segments at p in an order that does not depend on how it is cut up: four
// sums of 8 segments, added in pairs, by W = 1, 2 or 4 neighbouring lanes (the same point; lane h of them
// takes sums h * 4 / W on).  Called by whole warps; every lane gets the field.
__device__ __forceinline__ void f64_sub_field_by(const F64Sub &D, int cnt, const double (&p)[3], int W, int h, double (&b)[3]) {
    constexpr int E = kSub64 / 4;
    double w[3], T[6];
#pragma unroll
    for (int c = 0; c < 3; ++c) w[c] = p[c] - D.o[c];
    auto eight = [&](int j0, double (&S)[6]) {
#pragma unroll
        for (int c = 0; c < 6; ++c) S[c] = 0.0;
        if (j0 >= cnt) return;      // (padding only)
#pragma unroll 4
        for (int j = j0; j < j0 + E; ++j) {
            const double rx = w[0] - D.v[6][j], ry = w[1] - D.v[7][j], rz = w[2] - D.v[8][j];
            const double inv = rsqrt(rx * rx + ry * ry + rz * rz);
            const double inv3 = inv * inv * inv;
#pragma unroll
            for (int c = 0; c < 6; ++c) S[c] += D.v[c][j] * inv3;
        }
    };
    auto sixteen = [&](int j0, double (&S)[6]) {
        double X[6];
        eight(j0, S);
        eight(j0 + E, X);
#pragma unroll
        for (int c = 0; c < 6; ++c) S[c] += X[c];
    };
    if (W == 1) {
        double X[6];
        sixteen(0, T);
        sixteen(2 * E, X);
#pragma unroll
        for (int c = 0; c < 6; ++c) T[c] += X[c];
    } else {
        if (W == 2) {
            sixteen(2 * E * h, T);
        } else {
            eight(E * h, T);
#pragma unroll
            for (int c = 0; c < 6; ++c) T[c] += __shfl_xor_sync(0xffffffffu, T[c], 1);
        }
#pragma unroll
        for (int c = 0; c < 6; ++c) T[c] += __shfl_xor_sync(0xffffffffu, T[c], W / 2);
    }
    b[0] = (T[1] * w[2] - T[2] * w[1]) - T[3];
    b[1] = (T[2] * w[0] - T[0] * w[2]) - T[4];
    b[2] = (T[0] * w[1] - T[1] * w[0]) - T[5];
}

// Sums of sub-block fields: 16 at a time, so that no long sum runs in one accumulator (the rounding
// of 1440 additions to it would exceed that of the sub-blocks).
struct SubSum {
    double b[3], g[3];
    int n;
    __device__ __forceinline__ SubSum() : b{0.0, 0.0, 0.0}, g{0.0, 0.0, 0.0}, n(0) {}
    __device__ __forceinline__ void add(const double (&x)[3]) {
#pragma unroll
        for (int c = 0; c < 3; ++c) g[c] += x[c];
        if (++n == 16) flush();
    }
    __device__ __forceinline__ void flush() {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            b[c] += g[c];
            g[c] = 0.0;
        }
        n = 0;
    }
};

}  // namespace cctgpu
