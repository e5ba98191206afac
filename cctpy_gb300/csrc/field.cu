// Biot-Savart field of CCT winding segments (+ analytic QS magnets) at field points.
//
//   B(p) = sum_i kl_i x r_i / |r_i|^3,  r_i = p - p0_i,  kl_i = 1e-7 I (w[i+1]-w[i]),
//   p0_i = (w[i+1]+w[i])/2            -- cctpy final_code/packages/cct.py:157-164, :249-285
//
// Two forms:
//  * field_f64_kernel   FP64 (the drop-in for CCT.magnetic_field_at), one thread per field point,
//                       the pair terms as hi + lo pairs of FP32 values in moment form about
//                       each 32-segment sub-block's middle (df.cuh), everything longer in FP64.
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
// CTA writes the field of its split to a workspace and field_combine_kernel adds the splits of a
// point in a fixed order, and the analytic magnets.  FP32c: each CTA writes every tile's FP32
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
constexpr int kF64Block = 128;
constexpr int kF64Warps = kF64Block / 32;
constexpr int kF64Blocks = 4;          // CTAs a SM (128 registers)

// Split blockIdx.y of gridDim.y of the sub-blocks of 32 segments.  SHARED: the CTA's four warps
// share 32 points and take every fourth sub-block, each staging its own; else the CTA has 128
// points and every warp passes every sub-block, four staged at a time, one by each warp (a
// sub-block's staging then serves four times the points).  The next sub-block's segments are
// loaded before the staged ones are summed.  With one split the result (analytic magnets
// included) goes to B, else the split's field to part.
//
// Bound by the FP32 pipe: 148 lane operations a pair (df.cuh); 196 Gpairs/s is 72 % of it (77 824
// points x 46 080 segments 18.3 ms; the FP64 pipe's sum ran at 28.9).  4 CTAs a SM at 128 registers;
// 3 at 168 give 193, 5 at 96 (spills) 171.  Error against 80-bit and wider sums, 2-norm over
// points in the 46 080-segment dipole's bore: 2.7e-16 (plain FP64: 4.1e-16); along the gantry
// section of 360 segments a turn 2.6e-16 (2.2e-15), 120 a turn 4.2e-16 (1.4e-15).
template <bool SHARED>
__global__ void __launch_bounds__(kF64Block, kF64Blocks) field_f64_kernel(
    const double *__restrict__ kls, const double *__restrict__ p0s, int64_t n_seg, const double *__restrict__ qs,
    int n_qs, const double *__restrict__ pts, int64_t n, double *__restrict__ B, double *__restrict__ part) {
    constexpr int LP = SHARED ? 32 : kF64Block;         // points of the CTA
    __shared__ DfSub sub[SHARED ? 1 : 2][kF64Warps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t idx = (int64_t)blockIdx.x * LP + (SHARED ? lane : tid);
    const int64_t at = min(idx, n - 1);
    const double p[3] = {pts[3 * at], pts[3 * at + 1], pts[3 * at + 2]};
    const bool plain = n_seg < kDfMinSegments;
    const int64_t subs = (n_seg + kDfSub - 1) / kDfSub;
    const int64_t first = subs * blockIdx.y / gridDim.y, end = subs * (blockIdx.y + 1) / gridDim.y;
    auto count = [&](int64_t s) { return (int)min((int64_t)kDfSub, n_seg - s * kDfSub); };
    SubSum sum;
    SegRaw raw;
    if (first + warp < end) sub_load(raw, kls, p0s, (first + warp) * kDfSub, count(first + warp));
    for (int64_t s0 = first, k = 0; s0 < end; s0 += kF64Warps, ++k) {
        const int64_t mine = s0 + warp, next = mine + kF64Warps;
        DfSub *buf = sub[SHARED ? 0 : k & 1];
        if (mine < end) df_stage(buf[warp], raw, count(mine), plain);
        if (next < end) sub_load(raw, kls, p0s, next * kDfSub, count(next));
        double b[3];
        if (SHARED) {
            __syncwarp();
            if (mine < end) {
                df_sub_field(buf[warp], kls, p0s, mine * kDfSub, p, b);
                sum.add(b);
            }
            __syncwarp();
        } else {
            __syncthreads();   // (the other buffer's readers passed the previous round's barrier)
            for (int w = 0; w < kF64Warps && s0 + w < end; ++w) {
                df_sub_field(buf[w], kls, p0s, (s0 + w) * kDfSub, p, b);
                sum.add(b);
            }
        }
    }
    sum.flush();
    double b[3] = {sum.b[0], sum.b[1], sum.b[2]};
    if (SHARED) {
        __shared__ double red[kF64Warps][32][3];
#pragma unroll
        for (int c = 0; c < 3; ++c) red[warp][lane][c] = b[c];
        __syncthreads();
        if (warp != 0) return;
#pragma unroll
        for (int c = 0; c < 3; ++c)
            b[c] = (red[0][lane][c] + red[1][lane][c]) + (red[2][lane][c] + red[3][lane][c]);
    }
    if (idx >= n) return;
    double *out = gridDim.y > 1 ? part + 3 * (int64_t)blockIdx.y * n : B;
    if (gridDim.y == 1)
        for (int q = 0; q < n_qs; ++q) qs_field_add(qs + kQsRecord * q, p[0], p[1], p[2], b[0], b[1], b[2]);
#pragma unroll
    for (int c = 0; c < 3; ++c) out[3 * idx + c] = b[c];
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

// Field of every point from its splits' fields (part[split][point][3]) plus the analytic
// magnets: LANES threads a point (32 where there are many splits), a fixed order of additions.
template <int LANES>
__global__ void __launch_bounds__(128) field_combine_kernel(const double *__restrict__ part, int splits,
                                                            const double *__restrict__ qs, int n_qs,
                                                            const double *__restrict__ pts, int64_t n,
                                                            double *__restrict__ B) {
    const int64_t t = (int64_t)blockIdx.x * 128 + threadIdx.x;
    const int64_t idx = t / LANES;
    const int lane = (int)(t % LANES);
    if (idx >= n) return;   // LANES 32: whole warps leave
    double b[3] = {0.0, 0.0, 0.0};
    for (int s = lane; s < splits; s += LANES)
#pragma unroll
        for (int c = 0; c < 3; ++c) b[c] += part[3 * ((int64_t)s * n + idx) + c];
    if (LANES == 32)
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

static int launch_combine(const double *part, int splits, const double *qs, int n_qs, const double *pts, int64_t n,
                          double *B, cudaStream_t st) {
    if (splits > 8) {
        field_combine_kernel<32><<<(unsigned)((32 * n + 127) / 128), 128, 0, st>>>(part, splits, qs, n_qs, pts, n, B);
    } else {
        field_combine_kernel<1><<<(unsigned)((n + 127) / 128), 128, 0, st>>>(part, splits, qs, n_qs, pts, n, B);
    }
    CCT_TRY_CUDA(cudaGetLastError());
    return CCT_OK;
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
// unsplit and takes 0.11 ms (the whole Python call), 351 points of 119 520 segments 310 ms and 0.36 ms
// (FP64); 517 points of 597 600 segments 17.0 ms and 0.35 ms (FP32c, split up to one wave: 175 104
// points).
FieldPlan plan_field(int precision, int64_t n_seg, int64_t n, int64_t work_bytes) {
    FieldPlan P{kFieldFull, 1, 0};
    if (n <= 0 || n_seg <= 0) return P;
    const int slots = field_slots(precision);
    if (precision == 0) {
        // up to kFewPoints a thread a segment (at least 2 a thread); narrow CTAs where their fuller
        // lanes outweigh staging every sub-block for 32 points instead of 128 (a twelfth of its sum)
        const int64_t wide = (n + kF64Block - 1) / kF64Block, narrow = (n + 31) / 32;
        const FieldShape shape = n <= kFewPoints ? kFieldFew : 13 * narrow < 48 * wide ? kFieldNarrow : kFieldFull;
        const int64_t blocks = shape == kFieldFew ? 1 : shape == kFieldNarrow ? narrow : wide;
        const int64_t subs = (n_seg + kDfSub - 1) / kDfSub;
        // one wave of CTAs down to 4 sub-blocks a CTA; from 16 on four waves, so that their ends even
        // out (the warp schedulers favour some CTAs of an SM over others: 77 824 points of 46 080
        // segments run at 179 Gpairs/s in one wave and 196 in four)
        const int64_t one_wave = std::min((slots + blocks - 1) / blocks, (subs + 3) / 4);
        const int64_t four_waves = std::min((4 * slots + blocks - 1) / blocks, (subs + 15) / 16);
        const int64_t want = shape == kFieldFew ? std::min<int64_t>(slots, (n_seg + 2 * kFewBlock - 1) / (2 * kFewBlock))
                                                : std::max(one_wave, four_waves);
        const int64_t splits = std::min(want, work_bytes / (24 * n));
        if (shape == kFieldFew && splits < 1) return FieldPlan{kFieldNarrow, 1, 0};
        return FieldPlan{shape, (int)std::max<int64_t>(splits, 1),
                         shape == kFieldFew || splits > 1 ? 24 * n * splits : 0};
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
    return FieldPlan{few ? kFieldFew : kFieldFull, (int)splits, need};
}

int launch_field_f64(const double *kls, const double *p0s, int64_t n_seg, const double *qs, int n_qs,
                     const double *pts, int64_t n, double *B, void *work, int64_t work_bytes, cudaStream_t st) {
    if (n == 0) return CCT_OK;
    const FieldPlan P = plan_field(0, n_seg, n, work ? work_bytes : 0);
    const int64_t per = P.shape == kFieldNarrow ? 32 : kF64Block;
    const int64_t grid = (n + per - 1) / per;
    if (grid > 0x7fffffff) return set_error(CCT_ERR_ARG, "too many field points (%lld)", (long long)n);
    double *part = static_cast<double *>(work);
    if (P.shape == kFieldFew) {
        if (n <= 1) field_f64_few_kernel<1><<<P.splits, kFewBlock, 0, st>>>(kls, p0s, n_seg, pts, n, part);
        else if (n <= 2) field_f64_few_kernel<2><<<P.splits, kFewBlock, 0, st>>>(kls, p0s, n_seg, pts, n, part);
        else field_f64_few_kernel<kFewPoints><<<P.splits, kFewBlock, 0, st>>>(kls, p0s, n_seg, pts, n, part);
        CCT_TRY_CUDA(cudaGetLastError());
        return launch_combine(part, P.splits, qs, n_qs, pts, n, B, st);
    }
    const dim3 g((unsigned)grid, P.splits);
    if (P.shape == kFieldNarrow)
        field_f64_kernel<true><<<g, kF64Block, 0, st>>>(kls, p0s, n_seg, qs, n_qs, pts, n, B, part);
    else
        field_f64_kernel<false><<<g, kF64Block, 0, st>>>(kls, p0s, n_seg, qs, n_qs, pts, n, B, part);
    CCT_TRY_CUDA(cudaGetLastError());
    return P.splits > 1 ? launch_combine(part, P.splits, qs, n_qs, pts, n, B, st) : CCT_OK;
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
    if (SPLIT && all > room) return;
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
