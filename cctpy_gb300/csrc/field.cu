// Biot-Savart field of CCT winding segments (+ analytic QS magnets) at field points.
//
//   B(p) = sum_i kl_i x r_i / |r_i|^3,  r_i = p - p0_i,  kl_i = 1e-7 I (w[i+1]-w[i]),
//   p0_i = (w[i+1]+w[i])/2            -- cctpy final_code/packages/cct.py:157-164, :249-285
//
// Two forms:
//  * field_df_kernel    FP64 (the drop-in for CCT.magnetic_field_at), one thread per field point,
//    field_f64_kernel   in moment form about each 32-segment sub-block's middle: first with the pair
//                       terms as hi + lo pairs of FP32 values, everything longer in FP64, and a bound
//                       of their rounding (df.cuh); points whose bound is above FP64's rounding are
//                       then summed in FP64 (f64.cuh).
//  * field_f32c_kernel  FP32 arithmetic on per-tile local offsets: each tile of 128 segments
//                       carries a double-float origin, point-minus-origin is taken in
//                       double-float, the pair terms run as packed FP32x2 (two segments
//                       per instruction; rsqrt on the MUFU pipe) in the moment form
//                       (sums of kl |r|^-3 and (kl x p0) |r|^-3 per 32-segment
//                       sub-block, crossed with the point once per sub-block), summed into
//                       a Kahan-compensated (S, C) pair resolved in FP64 at the end
//                       (tile.cuh).  Tiles are streamed into
//                       shared memory by the TMA bulk-copy engine through an mbarrier
//                       ring.
// Too few points to fill the GPU: the segments are cut into splits as well (grid y).  FP64: each
// CTA writes fields of sub-blocks, chunks or its split to a workspace and field_combine_kernel adds
// them, and the analytic magnets.  FP32c: each CTA writes every tile's FP32
// field, and field_tiles_kernel takes the same compensated sum over the tiles in the same order
// as an unsplit CTA, so that a field does not depend on how the call was cut.
#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <vector>

#include "cctgpu_internal.cuh"
#include "df.cuh"
#include "qs.cuh"
#include "tile.cuh"

namespace cctgpu {

// FP32c field kernel shape (chosen at the kernel below)
constexpr int kF32Block = 128;
constexpr int kF32Ppt = 3;
constexpr int kF32Warps = kF32Block / 32;
constexpr int kF32Points = kF32Block * kF32Ppt;   // points of a CTA

// Largest FP32c workspace (12 bytes a point and tile); a larger call runs unsplit.
constexpr int64_t kMaxTileBytes = 2LL << 30;

// ===================================================================== FP64
// A point's field is the same, bit for bit, however many points its call has and however the call is
// cut up: a sub-block's field does not depend on that (df.cuh, f64.cuh), four of them are a chunk and
// four chunks a group, summed in their order, and the groups are summed in hi + lo pairs of FP64 values,
// whose rounding (2^-106) leaves the order no trace.
constexpr int kF64Block = 128;
constexpr int kF64Warps = kF64Block / 32;
constexpr int kF64Blocks = 4;          // CTAs a SM (128 registers)
constexpr int kChunkSubs = 4;          // sub-blocks of a chunk
constexpr int kGroupSubs = 16;         // sub-blocks of a group
static_assert(kChunkSubs == 4 && kGroupSubs == 16, "four chunks of four sub-blocks: field_combine_kernel");
constexpr int kEntry = 4;              // doubles of a sub-block's or chunk's field: x, y, z, bound
constexpr int64_t kMaxSplitBytes = 64LL << 20;   // of the splits of points left to FP64
constexpr int kSplit = 7;              // doubles of a split's field: x, y, z, their low parts, bound

// x of a point's field while it has to be summed in FP64 (a NaN that no arithmetic makes)
constexpr unsigned long long kRedo = 0x7ff8c3a5e1d20b47ull;

// How a call's sums reach field_combine_kernel: entries of `level` sub-blocks (1 or kChunkSubs), or
// sums of gridDim.y splits (level 0; one split: straight to B).
struct FieldCut {
    int64_t subs;
    int level, splits;
    double weight;      // df_weight: a field is good if its bound, so weighted, is below |B|^2
};

// hi + lo += x
__device__ __forceinline__ void wide_add(double &s, double &e, double x) {
    const double t = s + x, z = t - s;
    e += (s - (t - z)) + (x - z);
    s = t;
}

// A point's field as its sums give it, if it is good, with the analytic magnets, to B; DF and not good:
// kRedo.
template <bool DF>
__device__ __forceinline__ void field_finish(const double (&s)[3], const double (&e)[3], double q, double weight,
                                             const double *__restrict__ qs, int n_qs, const double (&p)[3],
                                             double *__restrict__ B) {
    double b[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) b[c] = isfinite(e[c]) ? s[c] + e[c] : s[c];      // (e of an infinite s is NaN)
    if (DF) {
        if (!(q * weight <= b[0] * b[0] + b[1] * b[1] + b[2] * b[2])) {
            *reinterpret_cast<unsigned long long *>(B) = kRedo;
            return;
        }
    }
    for (int i = 0; i < n_qs; ++i) qs_field_add(qs + kQsRecord * i, p[0], p[1], p[2], b[0], b[1], b[2]);
#pragma unroll
    for (int c = 0; c < 3; ++c) B[c] = b[c];
}

// Every point in hi + lo FP32 pairs (df.cuh), with the bound of their rounding: split blockIdx.y of
// gridDim.y.  NARROW: the CTA's four warps share 32 points and take an entry of C.level sub-blocks
// each, staging it themselves; else the CTA has 128 points and every warp passes every sub-block, a
// chunk staged at a time, a sub-block by each warp (a sub-block's staging then serves four times the
// points).  The next sub-block's segments are loaded before the staged ones are summed.
//
// Bound by the FP32 pipe (df.cuh): 77 824 points x 46 080 segments 19.7 ms, 182
// Gpairs/s.  4 CTAs a SM at 128
// registers; 3 at 168 were 2 % slower, 5 at 96 (spills) 13 %.  Error against 80-bit sums, 2-norm over
// points kept: dipole bore 1.7e-16 (FP64 in one sum over tiles of 256 segments: 4.0e-16), along sections
// of 60 / 120 / 360 / 600 segments a turn 2.8 / 3.0 / 4.3 / 5.1e-16 (6.8e-16 / 1.0 / 1.3 / 1.8e-15).
template <bool NARROW>
__global__ void __launch_bounds__(kF64Block, kF64Blocks) field_df_kernel(
    const double *__restrict__ kls, const double *__restrict__ p0s, int64_t n_seg, const double *__restrict__ qs,
    int n_qs, const double *__restrict__ pts, int64_t n, double *__restrict__ B, double *__restrict__ part, FieldCut C) {
    constexpr int LP = NARROW ? 32 : kF64Block;         // points of the CTA
    __shared__ DfFieldSub sub[NARROW ? 1 : 2][kF64Warps];
    __shared__ double wide[NARROW ? 1 : kSplit][kF64Block];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t idx = (int64_t)blockIdx.x * LP + (NARROW ? lane : tid), from = min(idx, n - 1);
    const double p[3] = {pts[3 * from], pts[3 * from + 1], pts[3 * from + 2]};
    auto count = [&](int64_t s) { return (int)min((int64_t)kDfSub, n_seg - s * kDfSub); };
    auto add = [&](const DfFieldSub &D, int64_t s, double (&t)[kEntry]) {
        double b[3], q;
        df_sub_field(D, kls, p0s, s * kDfSub, p, b, q);
#pragma unroll
        for (int c = 0; c < 3; ++c) t[c] += b[c];
        t[3] += q;
    };
    auto put = [&](int64_t entry, const double (&t)[kEntry]) {
        if (idx >= n) return;
        double *out = part + kEntry * (entry * n + idx);
#pragma unroll
        for (int c = 0; c < kEntry; ++c) out[c] = t[c];
    };
    SegRaw raw;
    if constexpr (NARROW) {
        const int64_t entries = (C.subs + C.level - 1) / C.level, stride = (int64_t)gridDim.y * kF64Warps;
        int64_t entry = (int64_t)blockIdx.y * kF64Warps + warp;
        if (entry < entries) sub_load(raw, kls, p0s, entry * C.level * kDfSub, count(entry * C.level));
        for (; entry < entries; entry += stride) {
            double t[kEntry] = {0.0, 0.0, 0.0, 0.0};
            const int64_t end = min((entry + 1) * C.level, C.subs);
            for (int64_t s = entry * C.level; s < end; ++s) {
                __syncwarp();
                df_stage(sub[0][warp], raw, count(s));
                __syncwarp();
                const int64_t next = s + 1 < end ? s + 1 : (entry + stride) * C.level;
                if (next < C.subs) sub_load(raw, kls, p0s, next * kDfSub, count(next));
                add(sub[0][warp], s, t);
            }
            put(entry, t);
        }
    } else {
        static_assert(kChunkSubs == kF64Warps, "a warp stages a sub-block of the chunk");
        constexpr int kOf = kGroupSubs / kChunkSubs;        // chunks of a group
        const int64_t chunks = (C.subs + kChunkSubs - 1) / kChunkSubs, groups = (C.subs + kGroupSubs - 1) / kGroupSubs;
        const int64_t first = C.level ? chunks * blockIdx.y / gridDim.y : groups * blockIdx.y / gridDim.y * kOf;
        const int64_t end = C.level ? chunks * (blockIdx.y + 1) / gridDim.y
                                    : min(groups * (blockIdx.y + 1) / gridDim.y * kOf, chunks);
#pragma unroll
        for (int c = 0; c < kSplit; ++c) wide[c][tid] = 0.0;
        double g[kEntry] = {0.0, 0.0, 0.0, 0.0};
        int64_t s0 = first * kChunkSubs;
        if (first < end && s0 + warp < C.subs) sub_load(raw, kls, p0s, (s0 + warp) * kDfSub, count(s0 + warp));
        for (int64_t k = first; k < end; ++k, s0 += kChunkSubs) {
            const int64_t own = s0 + warp, next = own + kChunkSubs;
            DfFieldSub *buf = sub[k & 1];
            if (own < C.subs) df_stage(buf[warp], raw, count(own));
            if (k + 1 < end && next < C.subs) sub_load(raw, kls, p0s, next * kDfSub, count(next));
            __syncthreads();   // (the other buffer's readers passed the previous round's barrier)
            double t[kEntry] = {0.0, 0.0, 0.0, 0.0};
            for (int w = 0; w < kChunkSubs && s0 + w < C.subs; ++w) add(buf[w], s0 + w, t);
            if (C.level) {
                put(k, t);
                continue;
            }
#pragma unroll
            for (int c = 0; c < kEntry; ++c) g[c] += t[c];
            if (k % kOf == kOf - 1 || k + 1 == end) {
#pragma unroll
                for (int c = 0; c < 3; ++c) wide_add(wide[c][tid], wide[3 + c][tid], g[c]);
                wide[6][tid] += g[3];
#pragma unroll
                for (int c = 0; c < kEntry; ++c) g[c] = 0.0;
            }
        }
        if (C.level || idx >= n) return;
        if (gridDim.y == 1) {
            const double s[3] = {wide[0][tid], wide[1][tid], wide[2][tid]}, e[3] = {wide[3][tid], wide[4][tid], wide[5][tid]};
            field_finish<true>(s, e, wide[6][tid], C.weight, qs, n_qs, p, B + 3 * idx);
        } else {
            double *out = part + kSplit * ((int64_t)blockIdx.y * n + idx);
#pragma unroll
            for (int c = 0; c < kSplit; ++c) out[c] = wide[c][tid];
        }
    }
}

// FP64 (f64.cuh), of every point (all) or of those that B marks, in CTAs of 32 points: split blockIdx.y of
// gridDim.y.  The points left are moved together, W lanes a point.  A warp takes an entry of C.level
// sub-blocks at a time, or groups, whose sums the four warps then put together (level 0).  apart:
// the warps have 32 points each instead, for calls whose points alone fill the GPU.
//
// Bound by the FP64 pipe, 21 operations a pair and some 55 a sub-block: 155 648 points x 2000 segments run at
// 27.7 Gpairs/s, x 300 at 26.8 (a thread a point and tiles of 256 segments: 29.9 where the points made whole
// waves, 3.8 for 10 000 points, here 24), 77 824 points 1 m from the dipole, the pass over them in hi + lo
// pairs included, at 24.  Error against 80-bit sums: 5e-17 to 1e-16 in bores, 1.5e-15 at 50 m and more from
// the dipole (one sum over tiles of 256 segments: 4e-16 to 2e-15, 5e-15).
__global__ void __launch_bounds__(kF64Block, kF64Blocks) field_f64_kernel(
    const double *__restrict__ kls, const double *__restrict__ p0s, int64_t n_seg, const double *__restrict__ qs,
    int n_qs, const double *__restrict__ pts, int64_t n, double *__restrict__ B, double *__restrict__ part, FieldCut C,
    int all, int apart) {
    __shared__ F64Sub sub[kF64Warps];
    __shared__ double sums[kF64Warps][6][32];
    __shared__ int list[kF64Warps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t base = (apart ? (int64_t)blockIdx.x * kF64Warps + warp : (int64_t)blockIdx.x) * 32;
    const bool left = base + lane < n && (all || reinterpret_cast<const unsigned long long *>(B)[3 * (base + lane)] == kRedo);
    const unsigned votes = __ballot_sync(0xffffffffu, left);
    const int points = __popc(votes);
    if (points == 0) return;      // (the whole CTA, or a warp apart)
    if (left) list[warp][__popc(votes & ((1u << lane) - 1u))] = lane;
    __syncwarp();
    const int W = points <= 8 ? 4 : points <= 16 ? 2 : 1, slot = lane / W, h = lane % W;
    const bool mine = slot < points && h == 0;
    const int64_t idx = base + list[warp][slot < points ? slot : 0];
    const double p[3] = {pts[3 * idx], pts[3 * idx + 1], pts[3 * idx + 2]};
    auto count = [&](int64_t s) { return (int)min((int64_t)kSub64, n_seg - s * kSub64); };
    const int level = C.level ? C.level : kGroupSubs;
    const int64_t entries = (C.subs + level - 1) / level, stride = (int64_t)gridDim.y * (apart ? 1 : kF64Warps);
    int64_t entry = apart ? (int64_t)blockIdx.y : (int64_t)blockIdx.y * kF64Warps + warp;
    double s[3] = {0.0, 0.0, 0.0}, e[3] = {0.0, 0.0, 0.0};
    SegRaw raw;
    if (entry < entries) sub_load(raw, kls, p0s, entry * level * kSub64, count(entry * level));
    for (; entry < entries; entry += stride) {
        double g[3] = {0.0, 0.0, 0.0}, t[3] = {0.0, 0.0, 0.0};
        const int64_t end = min((entry + 1) * level, C.subs);
        for (int64_t k = entry * level; k < end; ++k) {
            __syncwarp();
            f64_stage(sub[warp], raw, count(k));
            __syncwarp();
            const int64_t next = k + 1 < end ? k + 1 : (entry + stride) * level;
            if (next < C.subs) sub_load(raw, kls, p0s, next * kSub64, count(next));
            double b[3];
            f64_sub_field_by(sub[warp], count(k), p, W, h, b);
            const bool chunk = k % kChunkSubs == kChunkSubs - 1 || k + 1 == end;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                t[c] += b[c];
                if (chunk) {
                    g[c] += t[c];
                    t[c] = 0.0;
                }
            }
        }
        if (C.level) {
            if (mine) {
                double *out = part + kEntry * (entry * n + idx);
#pragma unroll
                for (int c = 0; c < 3; ++c) out[c] = g[c];
                out[3] = 0.0;
            }
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) wide_add(s[c], e[c], g[c]);
        }
    }
    if (C.level) return;
    if (!apart) {
        if (mine)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                sums[warp][c][slot] = s[c];
                sums[warp][3 + c][slot] = e[c];
            }
        __syncthreads();
        if (warp != 0) return;
        if (mine)
            for (int w = 1; w < kF64Warps; ++w)
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    wide_add(s[c], e[c], sums[w][c][slot]);
                    e[c] += sums[w][3 + c][slot];
                }
    }
    if (!mine) return;
    if (gridDim.y == 1) {
        field_finish<false>(s, e, 0.0, C.weight, qs, n_qs, p, B + 3 * idx);
    } else {
        double *out = part + kSplit * ((int64_t)blockIdx.y * n + idx);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            out[c] = s[c];
            out[3 + c] = e[c];
        }
        out[6] = 0.0;
    }
}

// A handful of points: a thread a segment instead of a thread a point (a point alone used one
// thread of one CTA for all segments: 120 ms for 46 080).  CTA x takes the segments x * kFewBlock
// + thread, + gridDim.x * kFewBlock, ...; pair terms kl x r |r|^-3 in FP64; the CTA's sum per
// point goes to split blockIdx.x.
constexpr int kFewPoints = 4;
constexpr int kFewBlock = 128;

template <int NP>
__global__ void __launch_bounds__(kFewBlock) field_f64_few_kernel(const double *__restrict__ kls,
                                                                  const double *__restrict__ p0s, int64_t n_seg,
                                                                  const double *__restrict__ pts, int64_t n,
                                                                  double *__restrict__ part) {
    __shared__ double red[kFewBlock / 32][NP][3];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double p[NP][3], b[NP][3];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        const int64_t j = min((int64_t)i, n - 1);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            p[i][c] = pts[3 * j + c];
            b[i][c] = 0.0;
        }
    }
    for (int64_t s = (int64_t)blockIdx.x * kFewBlock + threadIdx.x; s < n_seg; s += (int64_t)gridDim.x * kFewBlock) {
        const double kx = kls[3 * s], ky = kls[3 * s + 1], kz = kls[3 * s + 2];
        const double qx = p0s[3 * s], qy = p0s[3 * s + 1], qz = p0s[3 * s + 2];
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            const double rx = p[i][0] - qx, ry = p[i][1] - qy, rz = p[i][2] - qz;
            const double inv = rsqrt(rx * rx + ry * ry + rz * rz);
            const double inv3 = inv * inv * inv;
            b[i][0] += (ky * rz - kz * ry) * inv3;
            b[i][1] += (kz * rx - kx * rz) * inv3;
            b[i][2] += (kx * ry - ky * rx) * inv3;
        }
    }
#pragma unroll
    for (int i = 0; i < NP; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double v = b[i][c];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0) red[warp][i][c] = v;
        }
    __syncthreads();
    if (threadIdx.x < 3 * NP) {
        const int i = threadIdx.x / 3, c = threadIdx.x % 3;
        double v = red[0][i][c];
        for (int w = 1; w < kFewBlock / 32; ++w) v += red[w][i][c];
        if (i < n) part[3 * ((int64_t)blockIdx.x * n + i) + c] = v;
    }
}

// Its splits' fields (part[split][point][3]) together, plus the analytic magnets: a warp a point, a fixed
// order of additions.
__global__ void __launch_bounds__(128) field_few_combine_kernel(const double *__restrict__ part, int splits,
                                                            const double *__restrict__ qs, int n_qs,
                                                            const double *__restrict__ pts, int64_t n,
                                                            double *__restrict__ B) {
    const int64_t t = (int64_t)blockIdx.x * 128 + threadIdx.x;
    const int64_t idx = t / 32;
    const int lane = (int)(t % 32);
    if (idx >= n) return;   // (whole warps)
    double b[3] = {0.0, 0.0, 0.0};
    for (int s = lane; s < splits; s += 32)
#pragma unroll
        for (int c = 0; c < 3; ++c) b[c] += part[3 * ((int64_t)s * n + idx) + c];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) b[c] += __shfl_down_sync(0xffffffffu, b[c], o);
    if (lane != 0) return;
    const double px = pts[3 * idx], py = pts[3 * idx + 1], pz = pts[3 * idx + 2];
    for (int q = 0; q < n_qs; ++q) qs_field_add(qs + kQsRecord * q, px, py, pz, b[0], b[1], b[2]);
#pragma unroll
    for (int c = 0; c < 3; ++c) B[3 * idx + c] = b[c];
}

// Field of every point (FP64: of every point, or those that B marks) from its entries or splits: LANES
// threads a point (128: a CTA).
template <bool DF, int LANES>
__global__ void __launch_bounds__(128) field_combine_kernel(const double *__restrict__ part, FieldCut C,
                                                            const double *__restrict__ qs, int n_qs,
                                                            const double *__restrict__ pts, int64_t n,
                                                            double *__restrict__ B, int all) {
    const int64_t t = (int64_t)blockIdx.x * 128 + threadIdx.x;
    const int64_t idx = t / LANES;
    const int lane = (int)(t % LANES);
    if (idx >= n) return;   // (whole warps leave)
    if (!DF && !all && reinterpret_cast<const unsigned long long *>(B)[3 * idx] != kRedo) return;
    double s[3] = {0.0, 0.0, 0.0}, e[3] = {0.0, 0.0, 0.0}, q = 0.0;
    if (C.level) {
        const int64_t groups = (C.subs + kGroupSubs - 1) / kGroupSubs, entries = (C.subs + C.level - 1) / C.level;
        // four entries at a time, so that 16 loads are in flight: a chunk's sub-blocks, or a group's chunks
        const int of = kGroupSubs / C.level, turns = of / 4;
        for (int64_t k = lane; k < groups; k += LANES) {
            double g[kEntry] = {0.0, 0.0, 0.0, 0.0};
            for (int i = 0; i < turns; ++i) {
                double v[4][kEntry], u[kEntry] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int64_t entry = k * of + 4 * i + j;
                    const double *at = part + kEntry * (min(entry, entries - 1) * n + idx);
#pragma unroll
                    for (int c = 0; c < kEntry; ++c) v[j][c] = entry < entries ? at[c] : 0.0;
                }
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int c = 0; c < kEntry; ++c) u[c] += v[j][c];
#pragma unroll
                for (int c = 0; c < kEntry; ++c) g[c] += u[c];
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) wide_add(s[c], e[c], g[c]);
            q += g[3];
        }
    } else {
        for (int k = lane; k < C.splits; k += LANES) {
            const double *v = part + kSplit * ((int64_t)k * n + idx);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                wide_add(s[c], e[c], v[c]);
                e[c] += v[3 + c];
            }
            q += v[6];
        }
    }
    if (LANES >= 32)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const double s1 = __shfl_down_sync(0xffffffffu, s[c], o), e1 = __shfl_down_sync(0xffffffffu, e[c], o);
                wide_add(s[c], e[c], s1);
                e[c] += e1;
            }
            q += __shfl_down_sync(0xffffffffu, q, o);
        }
    if (LANES == 128) {      // the warps' sums
        __shared__ double sums[3][kSplit];
        if (threadIdx.x % 32 == 0 && lane > 0) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                sums[lane / 32 - 1][c] = s[c];
                sums[lane / 32 - 1][3 + c] = e[c];
            }
            sums[lane / 32 - 1][6] = q;
        }
        __syncthreads();
        if (lane == 0)
            for (int w = 0; w < 3; ++w) {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    wide_add(s[c], e[c], sums[w][c]);
                    e[c] += sums[w][3 + c];
                }
                q += sums[w][6];
            }
    }
    if (lane != 0) return;
    const double p[3] = {pts[3 * idx], pts[3 * idx + 1], pts[3 * idx + 2]};
    field_finish<DF>(s, e, q, C.weight, qs, n_qs, p, B + 3 * idx);
}

// ---------------------------------------------------------------- launch shape
// CTAs the GPU holds at once, by precision: the splits fill them about once.
static int field_slots(int precision) {
    static const int per_sm[2] = {kF64Blocks, 3};     // resident CTAs a SM (field_f64_kernel, field_f32c_kernel)
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        (void)cudaGetLastError();
        sms = 152;
    }
    return sms * per_sm[precision];
}

static int64_t tiles_for(int64_t n_seg) { return (n_seg + kTile - 1) / kTile; }

// Splits where the points alone leave the GPU idle: one point of 46 080 segments took 119.8 ms
// unsplit and takes 0.06 ms (the whole Python call), 351 points of 119 520 segments 310 ms and 1.6 ms
// (FP64); 517 points of 597 600 segments 17.0 ms and 0.35 ms (FP32c, split up to one wave: 175 104
// points).
FieldPlan plan_field(int precision, int64_t n_seg, int64_t n, int64_t work_bytes) {
    FieldPlan P{kFieldFull, 1, 0, 0, 1};
    if (n <= 0 || n_seg <= 0) return P;
    const int slots = field_slots(precision);
    if (precision == 0) {
        const int64_t wide = (n + kF64Block - 1) / kF64Block, narrow = (n + 31) / 32;
        const int64_t subs = (n_seg + kDfSub - 1) / kDfSub, chunks = (subs + kChunkSubs - 1) / kChunkSubs,
                      groups = (subs + kGroupSubs - 1) / kGroupSubs;
        // up to kFewPoints a thread a segment (at least 2 a thread)
        if (n <= kFewPoints) {
            const int64_t want = std::min<int64_t>(slots, (n_seg + 2 * kFewBlock - 1) / (2 * kFewBlock));
            const int64_t splits = std::min(want, work_bytes / (24 * n));
            if (splits > 0) return FieldPlan{kFieldFew, (int)splits, 24 * n * splits, 0, 1};
        }
        // narrow CTAs where their fuller lanes outweigh staging every sub-block for 32 points instead of
        // 128 (a twelfth of its sum), or wide ones would be fewer than a wave (100 points x 300 segments 102
        // -> 37 us).  Single sub-blocks to a warp as long as chunks would not make one and a
        // half waves of warps (200 points of 46 080 segments 113 -> 99 us: one wave and a bit had most SMs
        // wait for a few; 351 points 140 -> 145)
        if (13 * narrow < 48 * wide || wide * chunks < slots) {
            for (int level : {1, kChunkSubs}) {
                const int64_t entries = level == 1 ? subs : chunks;
                if (level == 1 && 2 * narrow * chunks >= 3 * (int64_t)slots * kF64Warps) continue;
                if (entries > work_bytes / (8 * kEntry * n)) continue;
                const int splits = (int)std::min((entries + kF64Warps - 1) / kF64Warps, (8 * slots + narrow - 1) / narrow);
                return FieldPlan{kFieldNarrow, splits, 8 * kEntry * n * entries, level, splits};
            }
        }
        // else at least four waves of CTAs, so that their ends even out (the warp schedulers favour some
        // CTAs of an SM over others: 77 824 points of 46 080 segments run 9 % slower in one wave), with the
        // same number of whole groups each (4096 points 1.31 -> 1.11 ms against one or two); where there are
        // too few groups for that, entries of chunks.  The FP64 sums of points left over: as many splits as
        // its warps have groups for, of up to kMaxSplitBytes (CTAs without such points leave at once).
        if (wide * groups < 4 * slots && chunks <= work_bytes / (8 * kEntry * n)) {
            const int64_t splits = std::min((8 * slots + wide - 1) / wide, chunks);
            return FieldPlan{kFieldFull, (int)splits, 8 * kEntry * n * chunks, kChunkSubs, (int)((chunks + kF64Warps - 1) / kF64Warps)};
        }
        const int64_t per = std::max<int64_t>(wide * groups / (4 * slots), 1), waves = (groups + per - 1) / per;
        const int64_t most = std::min((groups + kF64Warps - 1) / kF64Warps, std::min(work_bytes, kMaxSplitBytes) / (8 * kSplit * n));
        const int left = (int)std::max<int64_t>(most, 1);
        const int64_t left_bytes = left > 1 ? 8 * kSplit * n * left : 0;
        const int64_t splits = std::max<int64_t>(std::min(waves, work_bytes / (8 * kSplit * n)), 1);
        return FieldPlan{kFieldFull, (int)splits, std::max(splits > 1 ? 8 * kSplit * n * splits : 0, left_bytes), 0, left};
    }
    // FP32c: the workspace holds every tile's field of every point
    const int64_t tiles = tiles_for(n_seg), need = 12 * n * tiles;
    const int64_t wide = (n + kF32Points - 1) / kF32Points, narrow = (n + 31) / 32;
    if (wide > slots || need > work_bytes || need > kMaxTileBytes) return P;
    // warps of 32 points at 1 point a thread run at about 3/4 of the rate of 3 points a thread
    const bool few = 4 * 32 * narrow < 3 * kF32Points * wide;
    const int64_t units = few ? (tiles + kF32Warps - 1) / kF32Warps : tiles;
    const int64_t splits = std::min(std::max<int64_t>(slots / (few ? narrow : wide), 1), units);
    if (!few && splits < 2) return P;
    return FieldPlan{few ? kFieldFew : kFieldFull, (int)splits, need, 0, 1};
}

template <bool DF>
static int launch_combine(const FieldCut &C, const double *qs, int n_qs, const double *pts, int64_t n, double *B,
                          const double *part, int all, cudaStream_t st) {
    if (!C.level && C.splits == 1) return CCT_OK;
    // few points: as many threads as there are groups, since each costs a trip to L2
    const int64_t terms = C.level ? (C.subs + kGroupSubs - 1) / kGroupSubs : C.splits;
    if (terms > 32 && n <= 1024)
        field_combine_kernel<DF, 128><<<(unsigned)n, 128, 0, st>>>(part, C, qs, n_qs, pts, n, B, all);
    else if (terms > 8)
        field_combine_kernel<DF, 32><<<(unsigned)((32 * n + 127) / 128), 128, 0, st>>>(part, C, qs, n_qs, pts, n, B, all);
    else
        field_combine_kernel<DF, 1><<<(unsigned)((n + 127) / 128), 128, 0, st>>>(part, C, qs, n_qs, pts, n, B, all);
    CCT_TRY_CUDA(cudaGetLastError());
    return CCT_OK;
}

int launch_field_f64(const double *kls, const double *p0s, int64_t n_seg, const double *qs, int n_qs,
                     const double *pts, int64_t n, double *B, void *work, int64_t work_bytes, cudaStream_t st) {
    if (n == 0) return CCT_OK;
    const FieldPlan P = plan_field(0, n_seg, n, work ? work_bytes : 0);
    const int64_t wide = (n + kF64Block - 1) / kF64Block, narrow = (n + 31) / 32;
    if (narrow > 0x7fffffff) return set_error(CCT_ERR_ARG, "too many field points (%lld)", (long long)n);
    double *part = static_cast<double *>(work);
    if (P.shape == kFieldFew) {
        if (n <= 1) field_f64_few_kernel<1><<<P.splits, kFewBlock, 0, st>>>(kls, p0s, n_seg, pts, n, part);
        else if (n <= 2) field_f64_few_kernel<2><<<P.splits, kFewBlock, 0, st>>>(kls, p0s, n_seg, pts, n, part);
        else field_f64_few_kernel<kFewPoints><<<P.splits, kFewBlock, 0, st>>>(kls, p0s, n_seg, pts, n, part);
        CCT_TRY_CUDA(cudaGetLastError());
        field_few_combine_kernel<<<(unsigned)((32 * n + 127) / 128), 128, 0, st>>>(part, P.splits, qs, n_qs, pts, n, B);
        CCT_TRY_CUDA(cudaGetLastError());
        return CCT_OK;
    }
    // FP64 alone: few segments, and fields written over their points, which a second pass would miss
    const bool all = n_seg < kDfMinSegments || (B < pts + 3 * n && pts < B + 3 * n);
    const FieldCut C{(n_seg + kDfSub - 1) / kDfSub, P.level, P.splits, df_weight(std::max<int64_t>(n_seg, 1))};
    if (!all) {
        if (P.shape == kFieldNarrow)
            field_df_kernel<true><<<dim3((unsigned)narrow, P.splits), kF64Block, 0, st>>>(kls, p0s, n_seg, qs, n_qs, pts, n,
                                                                                         B, part, C);
        else
            field_df_kernel<false><<<dim3((unsigned)wide, P.splits), kF64Block, 0, st>>>(kls, p0s, n_seg, qs, n_qs, pts, n,
                                                                                        B, part, C);
        CCT_TRY_CUDA(cudaGetLastError());
        const int rc = launch_combine<true>(C, qs, n_qs, pts, n, B, part, 0, st);
        if (rc != CCT_OK) return rc;
    }
    const bool apart = !P.level && narrow >= 4 * field_slots(0);
    const FieldCut L{C.subs, P.level, all && apart ? 1 : P.left, 0.0};
    const unsigned ctas = (unsigned)(apart ? (narrow + kF64Warps - 1) / kF64Warps : narrow);
    field_f64_kernel<<<dim3(ctas, L.splits), kF64Block, 0, st>>>(kls, p0s, n_seg, qs, n_qs, pts, n, B, part, L, all, apart);
    CCT_TRY_CUDA(cudaGetLastError());
    return launch_combine<false>(L, qs, n_qs, pts, n, B, part, all, st);
}

// ===================================================================== FP32c pack
// Packs FP64 segments into FP32c tiles (layout in tile.cuh).  The tile origin is the
// centroid of the tile's midpoints rounded to a double-float (hi, lo) pair; offsets are
// taken from that represented origin, so point - origin needs no FP64 in the kernels.  Each
// 32-segment sub-block gets its own FP32 origin (centroid of its offsets), about which the
// moments kl x (p0 - origin - sub-block origin) are formed in FP64 and rounded once.
__global__ void __launch_bounds__(kTile) pack_f32c_kernel(const double *__restrict__ kls,
                                                          const double *__restrict__ p0s,
                                                          unsigned char *__restrict__ packed) {
    const int64_t n_designs = reinterpret_cast<const int64_t *>(packed)[1];
    const int64_t *tile_off = reinterpret_cast<const int64_t *>(packed + kPackedHeaderBytes);
    const int64_t *seg_off = tile_off + (n_designs + 1);
    unsigned char *tiles = packed + kPackedHeaderBytes + packed_index_bytes((int)n_designs);
    const int64_t t = blockIdx.x;
    // design holding tile t: last d with tile_off[d] <= t
    int64_t lo = 0, hi = n_designs - 1;
    while (lo < hi) {
        const int64_t mid = (lo + hi + 1) / 2;
        if (tile_off[mid] <= t) lo = mid; else hi = mid - 1;
    }
    const int64_t d = lo;
    const int64_t s0 = seg_off[d] + (t - tile_off[d]) * kTile;
    const int cnt = (int)min((int64_t)kTile, seg_off[d + 1] - s0);
    const int i = threadIdx.x;

    __shared__ double red[3][kTile];
    double k[3] = {0.0, 0.0, 0.0}, p[3] = {0.0, 0.0, 0.0};
    if (i < cnt) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            k[c] = kls[3 * (s0 + i) + c];
            p[c] = p0s[3 * (s0 + i) + c];
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) red[c][i] = p[c];
    __syncthreads();
    for (int w = kTile / 2; w > 0; w >>= 1) {   // fixed-order tree: deterministic origin
        if (i < w) {
#pragma unroll
            for (int c = 0; c < 3; ++c) red[c][i] += red[c][i + w];
        }
        __syncthreads();
    }
    float ohi[3], olo[3];
    double o[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        split_df(cnt > 0 ? red[c][0] / cnt : 0.0, ohi[c], olo[c]);
        o[c] = (double)ohi[c] + (double)olo[c];
    }
    // sub-block origins: FP32 centroid of the sub-block's offsets from the tile origin
    double off[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) off[c] = p[c] - o[c];
    __syncthreads();                              // everyone has read red[c][0]
#pragma unroll
    for (int c = 0; c < 3; ++c) red[c][i] = i < cnt ? off[c] : 0.0;
    __syncthreads();
    for (int w = kSub / 2; w > 0; w >>= 1) {      // fixed-order tree within each sub-block
        if (i % kSub < w) {
#pragma unroll
            for (int c = 0; c < 3; ++c) red[c][i] += red[c][i + w];
        }
        __syncthreads();
    }
    const int sbk = i / kSub;
    const int cnt_sb = min(max(cnt - sbk * kSub, 0), kSub);
    float so[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) so[c] = cnt_sb > 0 ? (float)(red[c][sbk * kSub] / cnt_sb) : 0.0f;

    unsigned char *tile = tiles + t * (int64_t)kTileBytes;
    TileHeader *hdr = reinterpret_cast<TileHeader *>(tile);
    float *f = reinterpret_cast<float *>(tile + kTileHeaderBytes);
    if (i == 0) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            hdr->o_hi[c] = ohi[c];
            hdr->o_lo[c] = olo[c];
        }
        hdr->count = cnt;
        hdr->pad = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) hdr->pad2[c] = 0.0f;
    }
    if (i % kSub == 0) {
#pragma unroll
        for (int c = 0; c < 3; ++c) hdr->sub_o[sbk][c] = so[c];
    }
    if (i < cnt) {
        // kl x (p0 - origin - sub-block origin), in FP64, rounded once
        const double e[3] = {off[0] - (double)so[0], off[1] - (double)so[1], off[2] - (double)so[2]};
        const double m[3] = {k[1] * e[2] - k[2] * e[1], k[2] * e[0] - k[0] * e[2], k[0] * e[1] - k[1] * e[0]};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            f[c * kTile + i] = (float)k[c];
            f[(3 + c) * kTile + i] = (float)m[c];
            f[(6 + c) * kTile + i] = (float)off[c];
        }
    } else {   // padding: zero current element far away (contributes exactly 0)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            f[c * kTile + i] = 0.0f;
            f[(3 + c) * kTile + i] = 0.0f;
            f[(6 + c) * kTile + i] = kPadOffset;
        }
    }
}

int launch_pack_f32c(const double *kls, const double *p0s, const int64_t *h_seg_off, int n_designs,
                     void *packed, int64_t packed_bytes, cudaStream_t st) {
    std::vector<int64_t> hdr(kPackedHeaderBytes / 8 + 2 * (n_designs + 1), 0);
    int64_t *tile_off = hdr.data() + kPackedHeaderBytes / 8;
    int64_t *seg_off = tile_off + (n_designs + 1);
    tile_off[0] = 0;
    for (int d = 0; d < n_designs; ++d) {
        const int64_t ns = h_seg_off[d + 1] - h_seg_off[d];
        tile_off[d + 1] = tile_off[d] + (ns + kTile - 1) / kTile;
    }
    for (int d = 0; d <= n_designs; ++d) seg_off[d] = h_seg_off[d];
    hdr[0] = kPackedMagic;
    hdr[1] = n_designs;
    hdr[2] = tile_off[n_designs];
    const int64_t need = kPackedHeaderBytes + packed_index_bytes(n_designs) + tile_off[n_designs] * kTileBytes;
    if (packed_bytes < need)
        return set_error(CCT_ERR_ARG, "packed buffer holds %lld bytes, needs %lld", (long long)packed_bytes,
                         (long long)need);
    CCT_TRY_CUDA(cudaMemcpyAsync(packed, hdr.data(), hdr.size() * 8, cudaMemcpyHostToDevice, st));
    if (tile_off[n_designs] > 0) {
        pack_f32c_kernel<<<(unsigned)tile_off[n_designs], kTile, 0, st>>>(kls, p0s,
                                                                         static_cast<unsigned char *>(packed));
        CCT_TRY_CUDA(cudaGetLastError());
    }
    // the header copy reads a host vector that goes out of scope here
    CCT_TRY_CUDA(cudaStreamSynchronize(st));
    return CCT_OK;
}

// ===================================================================== FP32c field
// Launch shape from a sweep of (threads, points per thread, CTAs per SM, unroll, ring depth)
// on the 2^20-point field map: 3 points per thread, 3 CTAs of 4 warps per SM (146 registers),
// the sub-block's 8-iteration segment loop fully unrolled.  CTAs of 3 or 6 warps were 20 %
// slower (their warps leave one SM sub-partition idle).
constexpr int kF32Blocks = 3;
constexpr int kF32Unroll = 8;
constexpr int kStages = 3;
constexpr bool kF32Rcp = false;   // |r|^-3 as rsqrt x rcp (tile.cuh inv_r3)
constexpr uint32_t kWaitPolls = 1u << 22;

__device__ int g_field_status;   // last non-OK status seen by a field kernel (sticky)

// PPT points a thread.  SPLIT = false: the sums over all tiles of the design, and the analytic
// magnets, into B.  SPLIT = true: tiles [first, first + nt) of split blockIdx.y of gridDim.y, each
// tile's field into tile_f[tile][c][point] (nothing if the design has more than `room` tiles).  SHARED (few points, PPT 1): the warps share the CTA's
// 32 points and take every kF32Warps-th tile (a ring slot then belongs to one warp), else a CTA's
// warps have 32 * PPT points each and all pass every tile.
template <int PPT, bool SPLIT, bool SHARED>
__global__ void __launch_bounds__(kF32Block, kF32Blocks) field_f32c_kernel(const unsigned char *__restrict__ packed,
                                                                  int design, const double *__restrict__ qs,
                                                                  int n_qs, const double *__restrict__ pts,
                                                                  int64_t n, double *__restrict__ B,
                                                                  float *__restrict__ tile_f, int64_t room) {
    constexpr int NS = SHARED ? kF32Warps : kStages;       // ring slots
    constexpr int WPT = SHARED ? 1 : kF32Warps;            // warps that use a tile
    constexpr int LP = SHARED ? 32 : kF32Block;            // points side by side in a CTA
    static_assert(!SHARED || (SPLIT && PPT == 1), "shared points: one a lane, tile fields written");
    __shared__ __align__(128) unsigned char buf[NS][kTileBytes];
    __shared__ __align__(8) uint64_t full[NS];
    __shared__ int64_t last_issued[NS];        // tile index last copied into each slot (-1: none)
    __shared__ int released[NS];               // warps done with the slot's current tile
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int pt = SHARED ? lane : tid;        // this thread's (first) point in the CTA
    const int64_t magic = reinterpret_cast<const int64_t *>(packed)[0];
    const int64_t n_designs = reinterpret_cast<const int64_t *>(packed)[1];
    const int64_t base = (int64_t)blockIdx.x * LP * PPT;
    if (magic != kPackedMagic || design >= n_designs) {   // not a packed set, or no such design
        if (tid == 0 && blockIdx.x == 0) atomicExch(&g_field_status, (int)CCT_ERR_ARG);
        if (SPLIT) return;                     // field_tiles_kernel writes the NaN
        for (int i = 0; i < PPT; ++i) {
            const int64_t idx = base + pt + (int64_t)i * LP;
            if (idx < n) B[3 * idx] = B[3 * idx + 1] = B[3 * idx + 2] = __longlong_as_double(0x7ff8000000000000LL);
        }
        return;
    }
    const int64_t *tile_off = reinterpret_cast<const int64_t *>(packed + kPackedHeaderBytes);
    const int64_t all = tile_off[design + 1] - tile_off[design];
    if (SPLIT && all > room) {                 // (field_tiles_kernel writes the NaN)
        if (tid == 0 && blockIdx.x == 0) atomicExch(&g_field_status, (int)CCT_ERR_ARG);
        return;
    }
    const int64_t first = SPLIT ? all * blockIdx.y / gridDim.y : 0;
    const int64_t nt = SPLIT ? all * (blockIdx.y + 1) / gridDim.y - first : all;
    const unsigned char *tiles = packed + kPackedHeaderBytes + packed_index_bytes((int)n_designs) +
                                 (tile_off[design] + first) * (int64_t)kTileBytes;

    if (tid == 0) {
        for (int s = 0; s < NS; ++s) {
            cctdev::mbar_init(&full[s], 1);
            released[s] = 0;
            last_issued[s] = -1;
        }
        cctdev::mbar_fence_init();
    }
    __syncthreads();
    if (tid == 0) {
        for (int s = 0; s < NS && s < nt; ++s) {
            last_issued[s] = s;
            cctdev::mbar_arrive_expect_tx(&full[s], kTileBytes);
            cctdev::bulk_g2s(buf[s], tiles + (int64_t)s * kTileBytes, kTileBytes, &full[s]);
        }
    }

    // each thread's points as double-float pairs in shared memory (only that thread reads them):
    // spt[c][i][tid], c = hi x, y, z, lo x, y, z
    __shared__ float spt[6][PPT][kF32Block];
#pragma unroll
    for (int i = 0; i < PPT; ++i) {
        int64_t idx = base + pt + (int64_t)i * LP;
        if (idx >= n) idx = n - 1;
#pragma unroll
        for (int c = 0; c < 3; ++c) split_df(pts[3 * idx + c], spt[c][i][tid], spt[3 + c][i][tid]);
    }
    F32cAcc<PPT> acc;
    acc.zero();

    // Warps run through the ring independently: a warp waits only for its next tile to land;
    // the last warp done with a slot refills it with the tile NS further on.
    bool failed = false;
    for (int64_t t = SHARED ? warp : 0; t < nt; t += SHARED ? kF32Warps : 1) {
        const int s = (int)(t % NS);
        const bool ok = cctdev::mbar_wait_bounded(&full[s], (uint32_t)((t / NS) & 1), kWaitPolls);
        if (!__all_sync(0xffffffffu, ok)) {
            failed = true;
            break;
        }
        f2 q[PPT][3];
        tile_offsets_smem<PPT>(buf[s], &spt[0][0][tid], PPT * kF32Block, kF32Block, q);
        if (SPLIT) {
            tile_field<PPT, kF32Unroll, kF32Rcp>(buf[s], q, 0, kTile / 4, [&](int i, int c, float v) {
                const int64_t idx = base + pt + (int64_t)i * LP;
                if (idx < n) tile_f[(3 * (first + t) + c) * n + idx] = v;
            });
        } else {
            tile_pairs<PPT, kF32Unroll, kF32Rcp>(buf[s], q, acc, 0, kTile / 4);
        }
        if (cctdev::ring_release_last(&released[s], WPT) && t + NS < nt) {
            last_issued[s] = t + NS;
            cctdev::fence_proxy_async();
            cctdev::mbar_arrive_expect_tx(&full[s], kTileBytes);
            cctdev::bulk_g2s(buf[s], tiles + (t + NS) * (int64_t)kTileBytes, kTileBytes, &full[s]);
        }
    }
    failed = __syncthreads_or(failed);
    if (failed && tid == 0) {
        // a warp gave up: let the last copy into every slot land before the CTA's shared
        // memory is released (earlier copies into a slot were consumed before its refill)
        for (int s = 0; s < NS; ++s)
            if (last_issued[s] >= 0)
                (void)cctdev::mbar_wait_bounded(&full[s], (uint32_t)((last_issued[s] / NS) & 1), kWaitPolls);
        atomicExch(&g_field_status, (int)CCT_ERR_TIMEOUT);
    }

    if (SPLIT) {   // a split that gave up is a NaN field of its first tile
        if (failed)
            for (int i = 0; i < PPT; ++i) {
                const int64_t idx = base + pt + (int64_t)i * LP;
                for (int c = 0; c < 3; ++c)
                    if (idx < n) tile_f[(3 * first + c) * n + idx] = __int_as_float(0x7fc00000);
            }
        return;
    }
#pragma unroll
    for (int i = 0; i < PPT; ++i) {
        const int64_t idx = base + pt + (int64_t)i * LP;
        if (idx >= n) continue;
        if (failed) {
            B[3 * idx] = B[3 * idx + 1] = B[3 * idx + 2] = __longlong_as_double(0x7ff8000000000000LL);
            continue;
        }
        double bx = acc.total(i, 0), by = acc.total(i, 1), bz = acc.total(i, 2);
        for (int q = 0; q < n_qs; ++q)
            qs_field_add(qs + kQsRecord * q, pts[3 * idx], pts[3 * idx + 1], pts[3 * idx + 2], bx, by, bz);
        B[3 * idx] = bx;
        B[3 * idx + 1] = by;
        B[3 * idx + 2] = bz;
    }
}

// Field of every point from the tiles' fields tile_f[tile][c][point], summed as an unsplit field_f32c_kernel does, plus the analytic magnets.  A thread a
// point and component: the chain of one compensated sum (about 20 cycles a tile) bounds it, the
// loads of kTilesAhead tiles being in flight ahead of it.
constexpr int kTilesAhead = 16;
constexpr int kTilesBlock = 96;   // 32 points x 3 components

__global__ void __launch_bounds__(kTilesBlock) field_tiles_kernel(const unsigned char *__restrict__ packed, int design,
                                                                  int64_t room, const float *__restrict__ tile_f,
                                                                  const double *__restrict__ qs, int n_qs,
                                                                  const double *__restrict__ pts, int64_t n,
                                                                  double *__restrict__ B) {
    __shared__ double b[3][32];
    const int lane = threadIdx.x & 31, c = threadIdx.x >> 5;
    const int64_t idx = (int64_t)blockIdx.x * 32 + lane;
    const int64_t *h = reinterpret_cast<const int64_t *>(packed);
    const bool ok = h[0] == kPackedMagic && design < h[1];
    const int64_t *tile_off = reinterpret_cast<const int64_t *>(packed + kPackedHeaderBytes);
    const int64_t nt = ok ? tile_off[design + 1] - tile_off[design] : 0;
    const bool fits = ok && nt <= room;
    float S = 0.0f, C = 0.0f;
    if (fits && idx < n) {
        const float *f = tile_f + c * n + idx;
        int64_t t = 0;
        for (; t + kTilesAhead <= nt; t += kTilesAhead) {
            float v[kTilesAhead];
#pragma unroll
            for (int k = 0; k < kTilesAhead; ++k) v[k] = f[3 * n * (t + k)];
#pragma unroll
            for (int k = 0; k < kTilesAhead; ++k) kahan_add(S, C, v[k]);
        }
        for (; t < nt; ++t) kahan_add(S, C, f[3 * n * t]);
    }
    b[c][lane] = fits ? (double)S - (double)C : __longlong_as_double(0x7ff8000000000000LL);
    __syncthreads();
    if (c != 0 || idx >= n) return;
    double bx = b[0][lane], by = b[1][lane], bz = b[2][lane];
    if (fits)
        for (int q = 0; q < n_qs; ++q)
            qs_field_add(qs + kQsRecord * q, pts[3 * idx], pts[3 * idx + 1], pts[3 * idx + 2], bx, by, bz);
    B[3 * idx] = bx;
    B[3 * idx + 1] = by;
    B[3 * idx + 2] = bz;
}

__device__ int g_field_status_taken;   // g_field_status as field_status_take_kernel last found it

__global__ void field_status_take_kernel() { g_field_status_taken = atomicExch(&g_field_status, 0); }

int take_field_status(cudaStream_t st, int *status) {
    field_status_take_kernel<<<1, 1, 0, st>>>();
    CCT_TRY_CUDA(cudaGetLastError());
    CCT_TRY_CUDA(cudaMemcpyFromSymbolAsync(status, g_field_status_taken, sizeof(int), 0, cudaMemcpyDeviceToHost, st));
    CCT_TRY_CUDA(cudaStreamSynchronize(st));
    return CCT_OK;
}

int launch_field_f32c(const void *packed, int design, int64_t n_seg, const double *qs, int n_qs, const double *pts,
                      int64_t n, double *B, void *work, int64_t work_bytes, cudaStream_t st) {
    if (n == 0) return CCT_OK;
    const FieldPlan P = plan_field(1, n_seg, n, work ? work_bytes : 0);
    const int64_t per = P.shape == kFieldFew ? 32 : kF32Points;
    const int64_t grid = (n + per - 1) / per;
    if (grid > 0x7fffffff) return set_error(CCT_ERR_ARG, "too many field points (%lld)", (long long)n);
    const unsigned char *pk = static_cast<const unsigned char *>(packed);
    float *tile_f = static_cast<float *>(work);
    const dim3 g((unsigned)grid, P.splits);
    if (P.shape == kFieldFew)
        field_f32c_kernel<1, true, true><<<g, kF32Block, 0, st>>>(pk, design, qs, n_qs, pts, n, B, tile_f,
                                                                        tiles_for(n_seg));
    else if (P.splits > 1)
        field_f32c_kernel<kF32Ppt, true, false><<<g, kF32Block, 0, st>>>(pk, design, qs, n_qs, pts, n, B, tile_f,
                                                                               tiles_for(n_seg));
    else
        field_f32c_kernel<kF32Ppt, false, false><<<g, kF32Block, 0, st>>>(pk, design, qs, n_qs, pts, n, B, nullptr,
                                                                                0);
    CCT_TRY_CUDA(cudaGetLastError());
    if (P.work_bytes > 0) {
        field_tiles_kernel<<<(unsigned)((n + 31) / 32), kTilesBlock, 0, st>>>(pk, design, tiles_for(n_seg), tile_f, qs,
                                                                             n_qs, pts, n, B);
        CCT_TRY_CUDA(cudaGetLastError());
    }
    return CCT_OK;
}

}  // namespace cctgpu
