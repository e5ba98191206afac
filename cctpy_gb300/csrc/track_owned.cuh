// The owned schedule: every CTA owns a share of the segments of one particle block for the whole
// launch, so that a stage has one hop between SMs and no work is handed out.  For launches whose
// particle blocks get several CTAs each (choose_owned).
//
// A CTA keeps its share in shared memory if it fits (else FP32c tiles stream through TMA rings, FP64
// sub-blocks are staged again) and its own copy of the block's RK4 state.  A stage is:
//   1. the warps sum the share's field at the block's positions;
//   2. the CTA's sum goes, as fixed-point integers, by atomic additions to the block's accumulators
//      in L2: (value << bits) + 1 a component, so that the low bits count the CTAs that have
//      arrived.  Integer sums do not depend on their order;
//   3. every CTA of the block reads the accumulators until every CTA has arrived -- the data is its
//      own flag: no fence, no counter, no second trip -- and advances its copy of the particles
//      (the same integers and the same FP64 arithmetic in all of them).
// FP32c: the share is a range of the planner's units (segment chunks).  Four warps (a quad) work as
// the CTA of the other schedules does, unit after unit, so that a unit's compensated sums are the
// same, bit for bit.  FP64: the share is every so manieth of the 32-segment sub-blocks (df.cuh; those close to
// the particles, which take longer, are then spread over the CTAs), dealt to the warps' groups of a lane a
// particle, whole or in pieces.
// The accumulators are never cleared: a stage's value is the difference from the reading of the
// last stage of the same parity.  They come in up to kOwnedCopies copies (the block's c-th CTA adds
// into copy c % copies), so that fewer additions queue on an address.  A stage's words cannot be
// touched by the stage after next before every CTA has read them: that stage's additions follow
// the next stage's complete arrival, and a CTA adds to the next stage only after reading this one.
//
// Fixed point, FP32c: 2^-54 T, of which an accumulator takes the whole multiples of 2^-52 T (2^-51 from 64
// CTAs a block on, 2^-49 from 128) and one more word the bits below of all three components, so that no
// bit of a warp's sum is lost on the way.  A sum rounded at 2^-44 T moves a proton by 1e-14, and the FP32
// field there by a rounding or two: of 200 drawn populations 10 came out further than 1e-9 (up to 1e-7)
// from FP64 sums of the same units in their objectives, at 2^-46 two, at 2^-48 none.  Batches of at most
// 64 protons are at 2^-44: their sums always were.  FP64: 2^-44 T and the remainder in a second word of
// 2^-86 T, so that its sums lose nothing of an FP64 field.  CTA fields beyond an equal share of the
// counted range (0.126 T at 127 CTAs a block, 0.21 T at 152 and 76, else more) go to a word without a
// count, those beyond that one's (16 T or more) and with sums of 2^59 units (32 T: a proton within half a
// millimetre of a filament, as lost ones of a population come) to four in units of 2^-54 to 2^108 T; the
// flag word says whether there are any.
//
// Bound by the latency of a stage (an L2 round of atomics and one of reads, three CTA barriers, the
// FP64 bookkeeping) and, for larger batches and FP64, by the FP32 or FP64 pipe.  A stage, single dipole
// of 46 080 segments, against the schedules this takes over from: FP32c 32 protons 9.1 -> 5.0 us, 100
// 22.3 -> 12.4, 512 38.8 -> 25.1, 2560 98 -> 69; FP64 1 proton 24 -> 7.4, 5 24 -> 8.7, 32 27 -> 16.2,
// 256 109 -> 77.
// Tried: CTAs of 4 warps, three a SM, for more blocks (speed test of 100 x 16: 48 us against 35 on
// dataflow); 2 to 20 additions an address (within 2 %); a flag word a component (6 % more at 256
// protons a block).
#pragma once

#include "track_common.cuh"

namespace cctgpu {

constexpr int kOwnedLowShift = 42;             // FP64: the remainder's extra bits
// x, y, z, flags, remainders (FP64 x, y, z; FP32c of all three, or none)
constexpr int kOwnedWords32 = 4, kOwnedWords32Rem = 5, kOwnedWords64 = 7;
constexpr int kOwnedFlagCount = 12, kOwnedFlagBig = 12, kOwnedFlagHuge = 24, kOwnedFlagBad = 36;
constexpr int kOwnedHugeUnits = 4;             // of sums beyond the counted range: 2^-54, 1, 2^54 and 2^108 T
constexpr int kOwnedWarps = 12;                         // warps of a CTA, one CTA a SM
constexpr int kOwnedThreads = 32 * kOwnedWarps;
constexpr int kOwnedSmemBytes = 215 << 10;     // its dynamic shared memory

// FP32 sums as fixed point of `shift` fraction bits, halves rounded away from zero, by integer operations
// (FP64 and 64-bit conversions run at GB300's low FP64 rate).  Sums of 2^59 units and more, infinities
// and NaN (as NaN) are kept as FP64 values, their bits moved (magnitude halved, sign last) to where neither one
// nor the number it makes with another sum is in the range of fixed point.
__device__ __forceinline__ bool fixed_in_range(long long v) {
    return (unsigned)((unsigned long long)v >> 32) + 0x08000000u < 0x10000000u;
}
__device__ __forceinline__ long long fixed_wide(double x) {      // |x| >= 32
    const unsigned long long b = isfinite(x) ? (unsigned long long)__double_as_longlong(x) : 0x7ff8000000000000ull;
    return (long long)(((b & 0x7fffffffffffffffull) >> 1 & ~1ull) | b >> 63);
}

__device__ __forceinline__ long long fixed_of(float x, int shift) {      // |x| < 2^(59 - shift)
    const unsigned b = __float_as_uint(x);
    const int e = (int)((b >> 23) & 0xffu);
    if (e == 0) return 0;                                   // zero, or below 2^-126
    const long long m = (long long)((b & 0x7fffffu) | 0x800000u);
    const int sh = e - (127 + 23) + shift;
    long long v = 0;
    if (sh >= 0) v = m << sh;
    else if (sh >= -24) v = (m + (1ll << (-sh - 1))) >> (-sh);
    return (b >> 31) ? -v : v;
}

__device__ __forceinline__ double fixed_value(long long v, int shift) {
    if (fixed_in_range(v)) return ldexp((double)v, -shift);
    return __longlong_as_double((long long)(((unsigned long long)v & ~1ull) << 1 | (unsigned long long)v << 63));
}

// a + b where one or the result is out of range.
static __device__ __noinline__ long long fixed_add_wide(long long a, long long b, int shift) {
    const double x = fixed_value(a, shift) + fixed_value(b, shift);
    return fabs(x) < ldexp(1.0, 58 - shift) ? __double2ll_rn(ldexp(x, shift)) : fixed_wide(x);
}

__device__ __forceinline__ long long fixed_add(long long a, long long b, int shift) {
    const long long r = (long long)((unsigned long long)a + (unsigned long long)b);
    return fixed_in_range(r) ? r : fixed_add_wide(a, b, shift);
}

// A compensated pair, S - C.
static __device__ __noinline__ long long fixed_pair_wide(float S, float C) { return fixed_wide((double)S - (double)C); }

__device__ __forceinline__ long long fixed_pair(float S, float C, int shift) {
    if ((int)((__float_as_uint(S) >> 23) & 0xffu) >= 127 + 59 - shift || !(fabsf(C) <= 1.0f)) return fixed_pair_wide(S, C);
    return fixed_of(S, shift) - fixed_of(C, shift);
}

// Fraction bits of a launch's fixed point: of the sums within a CTA, and `drop` fewer of the accumulators,
// with their count bits.  A CTA's counted range is `limit`.  FP32c: the bits dropped of a CTA's three sums
// go to one more word, drop + bits for each above the count.
struct OwnedScale {
    int shift, drop, bits;
    long long limit;
    __device__ __forceinline__ int remainder_at(int c) const { return bits + c * (drop + bits); }
};
constexpr int kOwnedShift64 = 44;              // FP64's first word

template <bool F64, int G, bool REM>
struct OwnedShape {
    static constexpr bool HALF = G == kHalfGroup;      // FP32c: lanes l and l + 16 hold a particle
    static constexpr int NS = F64 ? 32 / G : 1;        // FP64: sub-blocks a warp sums side by side
    static constexpr int PPT = !F64 && G >= 64 ? 2 : 1;
    static constexpr int NB = HALF ? 1 : G / (32 * PPT);   // FP32c: particle sub-blocks, one a warp
    static constexpr int S = 4 / NB;                       // FP32c: slices of a tile (HALF: see below)
    static constexpr int Q = F64 ? 1 : kOwnedWarps / 4;             // FP32c: quads
    static constexpr int W = F64 ? kOwnedWords64 : REM ? kOwnedWords32Rem : kOwnedWords32;
    static constexpr int R = REM ? 7 : W;                  // readings kept (the remainders' by each component's thread)
    static constexpr int T = kOwnedThreads;
    static constexpr int NI = (3 * G + T - 1) / T;         // components a thread updates
    static_assert(F64 ? G == 8 || G == 16 || G == 32 : G >= 16, "FP64 blocks of 8, 16 and 32");
};

template <bool F64, int G, bool REM>
struct OwnedSmem {
    using Sh = OwnedShape<F64, G, REM>;
    double y0[6][G], ys[6][G], ks[6][G];
    double h[3][G];                        // dt / 2, dt, dt / 6
    double kq[G], nsteps[G];
    double B[3][G];
    long long prev[2][Sh::R][G];           // last reading of each parity's words
    long long big_prev[2][3][G];
    unsigned flags[G];
    float reach[G];                        // FP64: the least df_reach so far
    int qs_hit[G];                         // a QS may act at the stage position
    float pts[6][G];                       // FP32c: stage positions as double-float
    union {
        long long fixed[kOwnedWarps][32 * Sh::PPT][3];
        double f64[kOwnedWarps][32][3];
    } red;
    // FP32c, a quad's tiles: all loaded at the start, or through a ring of kRing
    uint64_t loaded[Sh::Q], full[Sh::Q][kRing];
    int64_t last_issued[Sh::Q][kRing];     // streamed tile last copied into each slot (-1: none)
    int released[Sh::Q][kRing];            // warps done with the slot's current tile
    int give_up;
    int max_steps;
};

// The accumulators of a launch.
struct OwnedAcc {
    unsigned long long *words;    // [copies][2][words][particles]
    unsigned long long *big;      // [2][3][particles]
    unsigned long long *huge;     // [4][3 kOwnedHugeUnits][particles], cleared in the stage after the one that used them
    int64_t total;
    int copies, n_words;
    __device__ unsigned long long *at(int copy, int par, int w, int64_t pi) const {
        return words + (((int64_t)copy * 2 + par) * n_words + w) * total + pi;
    }
    __device__ unsigned long long *big_at(int par, int c, int64_t pi) const { return big + ((int64_t)par * 3 + c) * total + pi; }
    __device__ unsigned long long *huge_at(int set, int c, int64_t pi) const { return huge + ((int64_t)set * 3 * kOwnedHugeUnits + c) * total + pi; }
};

// FP32c: a quad's share, units [first, end) of its design's chunks; its tiles [0, nt) from `tiles` on,
// in `mem` for the whole launch or, from `held` = false on, through a ring there that the warps run
// through independently as in unit_sum_f32c, continuing over the stages: streamed tile k of the
// launch is tile k % nt.
struct OwnedQuad {
    int64_t first, end, ct, nt, total;     // total: tiles to stream over the whole launch
    const unsigned char *tiles;
    unsigned char *mem;
    bool held;
};

template <class SM>
static __device__ __forceinline__ void owned_issue(SM &sm, const OwnedQuad &R, int quad, int64_t k) {
    const int s = (int)(k % kRing);
    sm.last_issued[quad][s] = k;
    cctdev::fence_proxy_async();
    cctdev::mbar_arrive_expect_tx(&sm.full[quad][s], kTileBytes);
    cctdev::bulk_g2s(R.mem + s * (int64_t)kTileBytes, R.tiles + (k % R.nt) * (int64_t)kTileBytes, kTileBytes,
                     &sm.full[quad][s]);
}

// Thread 0, before the CTA gives up its shared memory early: the copies in flight land.
template <class SM>
static __device__ void owned_drain(SM &sm) {
    for (int q = 0; q < SM::Sh::Q; ++q)
        for (int s = 0; s < kRing; ++s)
            if (sm.last_issued[q][s] >= 0)
                (void)cctdev::mbar_wait_bounded(&sm.full[q][s], (uint32_t)((sm.last_issued[q][s] / kRing) & 1), kTmaPolls);
}

// FP32c: field of the quad's share at the block's particles, per warp in fixed point into
// sm.red.fixed; `before`: tiles streamed in the stages before.  A unit's slices and compensated
// sums are unit_sum_f32c's.  False (a tile wait gave up) only after every barrier of the quad.
template <int G, bool REM>
static __device__ bool owned_sum_f32c(OwnedSmem<false, G, REM> &sm, const OwnedQuad &R, int64_t before, int shift) {
    using Sh = OwnedShape<false, G, REM>;
    constexpr int PPT = Sh::PPT;
    constexpr bool HALF = Sh::HALF;
    constexpr int TS = HALF ? 2 : 1;           // tiles side by side in the quad, 4 / TS warps on each
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, quad = warp >> 2, wq = warp & 3;
    const int g0 = HALF ? (2 * (wq % 2) + (lane >> 4)) * (kSub / 4) : wq / Sh::NB * (kTile / 4 / Sh::S);
    const int g1 = g0 + (HALF ? kSub / 4 : kTile / 4 / Sh::S);
    const int pl0 = HALF ? lane & 15 : wq % Sh::NB * 32 * PPT + lane;
    float ph[PPT][3], pl[PPT][3];
#pragma unroll
    for (int i = 0; i < PPT; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            ph[i][c] = sm.pts[c][pl0 + 32 * i];
            pl[i][c] = sm.pts[3 + c][pl0 + 32 * i];
            if (R.first >= R.end && (!HALF || lane < 16)) sm.red.fixed[warp][lane + 32 * i][c] = 0;
        }
    bool ok = true;
    const int nt = (int)R.nt, ct = (int)R.ct;
    for (int t0 = 0; t0 < nt; t0 += ct) {      // a unit
        F32cAcc<PPT> acc;
        acc.zero();
        const int t1 = min(t0 + ct, nt);
        for (int t = t0 + (HALF ? wq / 2 : 0); t < t1; t += TS) {
            const unsigned k = (unsigned)before + (unsigned)t, s = k % kRing;
            const unsigned char *tile = R.mem + t * kTileBytes;
            if (!R.held) {
                const bool landed = ok && !*(volatile int *)&sm.give_up &&
                                    cctdev::mbar_wait_bounded(&sm.full[quad][s], (k / kRing) & 1u, kTmaPolls);
                if (!__all_sync(0xffffffffu, landed)) {
                    ok = false;
                    sm.give_up = 1;
                    break;
                }
                tile = R.mem + s * kTileBytes;
            }
            tile_f32c<PPT, kTrackUnroll, kTrackRcp>(tile, ph, pl, acc, g0, g1);
            if (!R.held && cctdev::ring_release_last(&sm.released[quad][s], 4 / TS)) {
                const int64_t next = before + t + kRing;
                if (next < R.total) owned_issue(sm, R, quad, next);
            }
        }
        // (HALF: a slot's tiles belong to one pair of warps only within a unit, and a phase parity
        // tells its tile from the last one only to a warp that has seen that one land)
        if (HALF && !R.held) {      // (constant barrier numbers: a register would reserve all sixteen)
            if (quad == 0) asm volatile("bar.sync 1, 128;" ::: "memory");
            else if (quad == 1) asm volatile("bar.sync 2, 128;" ::: "memory");
            else asm volatile("bar.sync 3, 128;" ::: "memory");
        }
#pragma unroll
        for (int i = 0; i < PPT; ++i)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                long long v = fixed_pair(acc.S[i][c], acc.C[i][c], shift);
                if (HALF) v = fixed_add(v, __shfl_down_sync(0xffffffffu, v, 16), shift);
                if (HALF && lane >= 16) continue;
                long long &sum = sm.red.fixed[warp][lane + 32 * i][c];      // (this lane's own)
                if (t0 > 0) v = fixed_add(v, sum, shift);
                sum = v;
            }
    }
    return ok;
}

// FP64, a share in shared memory: the lanes of a warp are `parts` = 32 / mine groups of a lane a
// particle, and each takes pieces (2^-log of a sub-block) of the n sub-blocks.  Pieces trade the
// length of a warp's chain (16 >> log pairs of segments) for its FP64 work a piece (worth 4.5 of
// them); the pipe time of a stage is that of the warps on an SM quarter, and a warp alone takes about
// twice its pipe time.  Without sub-blocks close to the particles, 5 protons: single dipole 10.3 -> 8.4 us
// (9 or 10 sub-blocks a CTA, in pieces of 4 pairs), gantry section 13.6 -> 10.9 us (24 or 25, in pieces of
// 8).  Of the four splits, the one taken was the fastest or within 4 % of it over 1 to 32 protons and 46 080
// to 358 560 segments.
__device__ __forceinline__ int owned_pieces_log(int64_t n, int parts) {
    int best = 0, best_cost = 0x7fffffff;
    for (int log = 0; log < 4; ++log) {
        const int warps = (int)(((n << log) + parts - 1) / parts), length = 16 >> log;
        const int cost = max((warps + 3) / 4 * (2 * length + 9), (warps + kOwnedWarps - 1) / kOwnedWarps * (4 * length + 12));
        if (cost < best_cost) {
            best_cost = cost;
            best = log;
        }
    }
    return best;
}

// FP64: field of the share's n sub-blocks (every stride-th from sub0 on of the design's ns segments)
// at the block's `mine` particles, per warp.  The first `held` sub-blocks are staged in shared memory
// for the whole launch; if that is not all, the others are staged every time in the warp's own slots
// and a warp takes 32 / G whole sub-blocks side by side, G lanes each.
template <int G>
static __device__ void owned_sum_f64(OwnedSmem<true, G, false> &sm, DfSub *hold, int64_t n, int64_t held, int64_t sub0,
                                     int64_t stride, int64_t ns, const double *kls, const double *p0s, int mine,
                                     int log) {
    constexpr int NS = OwnedShape<true, G, false>::NS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int width = n <= held ? mine : G, parts = n <= held ? 32 / mine : NS;
    const int slot = lane % width, part = lane / width;
    const int of = min(slot, mine - 1);      // (the block's last particle, in lanes that have none)
    const double p[3] = {sm.ys[0][of], sm.ys[1][of], sm.ys[2][of]};
    const float reach = sm.reach[of];
    auto at = [&](int64_t i) { return (sub0 + i * stride) * kDfSub; };      // first segment
    auto count = [&](int64_t i) { return (int)min((int64_t)kDfSub, ns - at(i)); };
    SubSum sum;
    if (n <= held) {
        const int items = (int)n << log, length = (kDfSub / 2) >> log;
        for (int i0 = warp * parts; i0 < items; i0 += kOwnedWarps * parts) {
            const bool work = part < parts && i0 + part < items;
            const int i = work ? i0 + part : i0, h = i >> log, j0 = (i - (h << log)) * length;
            double b[3];
            if (log == 0) df_track_field(hold[h], kls, p0s, at(h), p, reach, b);      // (a constant loop: 2 %)
            else df_track_field(hold[h], kls, p0s, at(h), p, reach, b, j0, j0 + length);
            if (!work) b[0] = b[1] = b[2] = 0.0;
            sum.add(b);
        }
    } else {
        DfSub *own = hold + held + warp * NS;
        SegRaw raw;
        bool loaded = false;        // raw holds the segments of the warp's next first sub-block
        for (int64_t i0 = warp * NS; i0 < n; i0 += kOwnedWarps * NS) {
            const DfSub *D = hold + i0;
            if (i0 >= held) {       // (held < n is a multiple of NS)
                __syncwarp();
                if (!loaded) sub_load(raw, kls, p0s, at(i0), count(i0));
                for (int k = 0; k < NS && i0 + k < n; ++k) {
                    df_stage(own[k], raw, count(i0 + k));
                    if (k + 1 < NS && i0 + k + 1 < n) sub_load(raw, kls, p0s, at(i0 + k + 1), count(i0 + k + 1));
                }
                __syncwarp();
                D = own;
            }
            const int64_t next = i0 + kOwnedWarps * NS;
            loaded = next >= held && next < n;
            if (loaded) sub_load(raw, kls, p0s, at(next), count(next));
            const int h = i0 + part < n ? part : 0;
            double b[3];
            df_track_field(D[h], kls, p0s, at(i0 + h), p, reach, b);
            if (h != part) b[0] = b[1] = b[2] = 0.0;
            sum.add(b);
        }
    }
    sum.flush();
    // the groups' sums together, the upper half of them onto the lower at a time
    for (int r = parts; r > 1;) {
        const int half = (r + 1) / 2;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double v = __shfl_down_sync(0xffffffffu, sum.b[c], half * width);
            if (part + half < r) sum.b[c] += v;
        }
        r = half;
    }
    if (lane < width)
#pragma unroll
        for (int c = 0; c < 3; ++c) sm.red.f64[warp][lane][c] = sum.b[c];
}

// A CTA's sum beyond the counted range: v units (an uncounted word holds `most` of every CTA), or
// (marked) s, in units of 2^-54 to 2^108 T; the flags it raises.
static __device__ __noinline__ unsigned long long owned_add_beyond(const OwnedAcc &A, int phase, int c, int64_t pi, long long v,
                                                                   double s, bool marked, long long most, int shift) {
    if (!marked && v <= most && v >= -most) {
        atomicAdd(A.big_at(phase & 1, c, pi), (unsigned long long)v);
        return 1ull << kOwnedFlagBig;
    }
    double x = marked ? s : ldexp((double)v, -shift);
    if (!(fabs(x) < ldexp(1.0, 54 * kOwnedHugeUnits - 54))) return 1ull << kOwnedFlagBad;
#pragma unroll 1
    for (int k = kOwnedHugeUnits - 1; k >= 0; --k) {       // (exact: 54 bits of x in each unit)
        const double r = rint(ldexp(x, 54 - 54 * k));
        if (r != 0.0) atomicAdd(A.huge_at(phase & 3, 3 * k + c, pi), (unsigned long long)__double2ll_rn(r));
        x -= ldexp(r, 54 * k - 54);
    }
    return 1ull << kOwnedFlagHuge;
}

// The CTA's sum of a component at slot, added to the accumulators of particle pi; the flags it raises.
template <bool F64, int G, bool REM>
static __device__ __forceinline__ unsigned long long owned_add_one(const OwnedAcc &A, const OwnedSmem<F64, G, REM> &sm, int copy,
                                                                  int phase, int c, int slot, int64_t pi, const OwnedScale &F,
                                                                  unsigned long long &remainder) {
    using Sh = OwnedShape<F64, G, REM>;
    unsigned long long note = 0ull;
    long long v = 0, low = 0;
    bool marked = false;
    double s = 0.0;
    if constexpr (F64) {
#pragma unroll
        for (int w = 0; w < kOwnedWarps; ++w) s += sm.red.f64[w][slot][c];
        marked = !(fabs(s) < (double)(1 << (54 - kOwnedShift64)));
        const double x = marked ? 0.0 : s * (double)(1ll << kOwnedShift64), r = rint(x);
        v = __double2ll_rn(r);
        low = __double2ll_rn((x - r) * (double)(1ll << kOwnedLowShift));
    } else {
        constexpr int PW = 32 * Sh::PPT;               // particles of a warp
#pragma unroll
        for (int w = 0; w < kOwnedWarps / Sh::NB; ++w) {
            const long long t = sm.red.fixed[slot / PW + w * Sh::NB][slot % PW][c];
            marked = marked || !fixed_in_range(t);
            v += t;
        }
    }
    if (REM) {
        remainder += (unsigned long long)(marked ? 0 : v & ((1ll << F.drop) - 1)) << F.remainder_at(c);
        v >>= F.drop;
    } else if (!F64 && F.drop > 0) {
        // (batches of few_particles drop nothing, but their kernels are 8 % slower where the compiler knows it)
        v = (v + (1ll << (F.drop - 1))) >> F.drop;
    }
    if (marked || v >= F.limit || v <= -F.limit) {
        if constexpr (!F64) {
            if (marked) {
                v = 0;
                for (int w = 0; w < kOwnedWarps / Sh::NB; ++w)
                    s += fixed_value(sm.red.fixed[slot / (32 * Sh::PPT) + w * Sh::NB][slot % (32 * Sh::PPT)][c], F.shift);
            }
        }
        note = owned_add_beyond(A, phase, c, pi, v, s, marked, F.limit << F.bits, F.shift - F.drop);
        v = 0;
    }
    if (note) __threadfence();        // before the flag that announces it
    const int par = phase & 1;
    atomicAdd(A.at(copy, par, c, pi), ((unsigned long long)v << F.bits) + 1ull);
    if (F64) atomicAdd(A.at(copy, par, 4 + c, pi), ((unsigned long long)low << F.bits) + 1ull);
    return note;
}

// All components of the block's `mine` particles from `first` on.  FP32c: a thread a particle.  FP64: warp 0, a
// lane a component as far as they fit, as a warp's FP64 instruction takes 64 cycles whatever its lanes
// (the twelve warps' sums and the conversions: 2.0 -> 0.7 us for blocks of 8).
template <bool F64, int G, bool REM>
static __device__ __forceinline__ void owned_add(const OwnedAcc &A, const OwnedSmem<F64, G, REM> &sm, int copy, int phase, int mine,
                                                 int64_t first, const OwnedScale &F) {
    const int tid = threadIdx.x, par = phase & 1;
    if constexpr (F64) {
        if (tid >= 32) return;
        unsigned long long note = 0ull, unused = 0ull;
        for (int i = tid; i < 3 * G; i += 32)
            if (i % G < mine) note += owned_add_one<F64, G, REM>(A, sm, copy, phase, i / G, i % G, first + i % G, F, unused);
        __syncwarp();
#pragma unroll
        for (int o = 16; o >= G; o >>= 1) note += __shfl_down_sync(0xffffffffu, note, o);
        if (note) __threadfence();      // (a lane's big values, announced by another's flag)
        if (tid < mine) atomicAdd(A.at(copy, par, 3, first + tid), note + 1ull);
    } else if (tid < mine) {
        unsigned long long note = 1ull, remainder = 1ull;
#pragma unroll
        for (int c = 0; c < 3; ++c) note += owned_add_one<F64, G, REM>(A, sm, copy, phase, c, tid, first + tid, F, remainder);
        if (REM) atomicAdd(A.at(copy, par, 4, first + tid), remainder);
        atomicAdd(A.at(copy, par, 3, first + tid), note);
    }
}

// Polls word w of particle pi (TWO: and word w2), all copies, until `want` additions of this stage
// have arrived (the low `bits` bits of the difference from the last reading count them); false:
// gave up.
template <bool TWO>
static __device__ __forceinline__ bool owned_poll(const TrackParams &P, const OwnedAcc &A, int par, int w, int w2, int64_t pi, int bits,
                                 unsigned want, long long *prev0, long long *prev1, unsigned long long (&diff)[2]) {
    const volatile int *err = reinterpret_cast<const volatile int *>(P.ctrl + CW_ERR);
    const unsigned long long mask = (1ull << bits) - 1ull;
    const unsigned long long p0 = (unsigned long long)*prev0, p1 = TWO ? (unsigned long long)*prev1 : 0ull;
    const unsigned long long *a0 = A.at(0, par, w, pi);
    const int64_t copy = 2 * A.n_words * A.total, up = (w2 - w) * A.total;
    unsigned long long t0 = 0;
    for (unsigned polls = 1;; ++polls) {
        unsigned long long s0 = 0, s1 = 0;
#pragma unroll
        for (int r = 0; r < kOwnedCopies; ++r)
            if (r < A.copies) {
                s0 += *(const volatile unsigned long long *)(a0 + r * copy);
                if (TWO) s1 += *(const volatile unsigned long long *)(a0 + r * copy + up);
            }
        diff[0] = s0 - p0;
        diff[1] = s1 - p1;
        if ((diff[0] & mask) == want && (!TWO || (diff[1] & mask) == want)) {
            *prev0 = (long long)s0;
            if (TWO) *prev1 = (long long)s1;
            return true;
        }
        if ((polls & 63u) == 0) {
            if (t0 == 0) t0 = global_ns();
            if (*err == CCT_ERR_TIMEOUT) return false;
            if (global_ns() - t0 > P.wait_ns) {
                set_timeout(P);
                return false;
            }
        }
        if (polls > 256) __nanosleep(64);
    }
}

// The same as a call: three copies of the loop cost the kernels with remainders 6 % (100 protons).
template <bool TWO>
static __device__ __noinline__ bool owned_poll_call(const TrackParams &P, const OwnedAcc &A, int par, int w, int w2, int64_t pi,
                                                    int bits, unsigned want, long long *prev0, long long *prev1,
                                                    unsigned long long (&diff)[2]) {
    return owned_poll<TWO>(P, A, par, w, w2, pi, bits, want, prev0, prev1, diff);
}

// What a stage's flag word says: whether any CTA has raised each flag (12 bits hold three a CTA of up to
// 255; the top flag has the word's last 28).
enum { kBig = 1u, kHuge = 2u, kBad = 4u };
__device__ __forceinline__ unsigned owned_flags(unsigned long long diff) {
    constexpr unsigned long long field = (1ull << 12) - 1ull;
    return ((diff >> kOwnedFlagBig & field) ? kBig : 0u) | ((diff >> kOwnedFlagHuge & field) ? kHuge : 0u) |
           (diff >> kOwnedFlagBad ? kBad : 0u);
}

// Signed value above the count bits.
__device__ __forceinline__ long long owned_value(unsigned long long diff, int bits) { return (long long)diff >> bits; }

// Whether a QS record may act at a point: conservative (the exact test follows in qs_field_add).
__device__ __forceinline__ bool qs_may_act(const double *q, double px, double py, double pz) {
    if (q[12] < 0.0 && isinf(q[12])) return true;
    const double z = q[9] * (px - q[0]) + q[10] * (py - q[1]) + q[11] * (pz - q[2]), e = 1e-6 + 1e-9 * fabs(z);
    return !(z < -e || z > fabs(q[12]) + e);
}

// The share of this CTA over the launch's steps.  REC: a checkpoint segment of the adjoint, from and to
// the particles' state and with their stages recorded (apart, as its code costs the others 1 %).  REM: FP32c with
// the remainders' word (all but batches of few_particles, which their code would cost 3 %).
template <bool F64, int G, bool REC, bool REM>
static __device__ void owned_track(const TrackParams &P, OwnedSmem<F64, G, REM> &sm, unsigned char *hold) {
    using Sh = OwnedShape<F64, G, REM>;
    constexpr int T = Sh::T;
    const int tid = threadIdx.x, warp = tid >> 5;
    if ((int64_t)blockIdx.x >= P.owned_off[P.n_designs]) return;
    int ud = 0, hi = P.n_designs - 1;          // design: last d with owned_off[d] <= CTA
    while (ud < hi) {
        const int mid = (ud + hi + 1) / 2;
        if (P.owned_off[mid] <= (int64_t)blockIdx.x) ud = mid; else hi = mid - 1;
    }
    const int cd = (int)P.owned_n[ud];                                // CTAs of the block
    const int ub = (int)(((int64_t)blockIdx.x - P.owned_off[ud]) / cd), ui = (int)(((int64_t)blockIdx.x - P.owned_off[ud]) % cd);
    const int64_t first = (int64_t)ud * P.n_p + (int64_t)ub * G;      // the block's first particle
    const int mine = (int)min((int64_t)G, P.n_p - (int64_t)ub * G);   // its particles
    const int64_t q0 = P.qs_off[ud], q1 = P.qs_off[ud + 1];
    OwnedAcc A{P.owned_acc, nullptr, nullptr, (int64_t)P.n_designs * P.n_p, P.owned_copies, Sh::W};
    A.big = A.words + (int64_t)A.copies * 2 * A.n_words * A.total;
    A.huge = A.big + 2 * 3 * A.total;
    const int copy = ui % A.copies;
    OwnedScale F{kOwnedShift64, 0, kOwnedCountBits, 0};
    if (!F64) {
        F.bits = 32 - __clz(cd);
        if (!few_particles(P.n_designs, P.n_p, P.G)) {
            F.shift = 54;
            F.drop = F.bits > 7 ? 5 : F.bits > 6 ? 3 : 2;
        }
    }
    F.limit = (1ll << (62 - F.bits)) / cd;
    const double unit = __longlong_as_double((long long)(1023 - (F.shift - F.drop)) << 52);
    const double fine = __longlong_as_double((long long)(1023 - F.shift) << 52);
    int huge_phase = -1;       // the stage before, if it raised flags

    if (tid == 0) {
        sm.give_up = 0;
        sm.max_steps = 0;
        for (int q = 0; q < Sh::Q; ++q) {
            cctdev::mbar_init(&sm.loaded[q], 1);
            for (int s = 0; s < kRing; ++s) {
                cctdev::mbar_init(&sm.full[q][s], 1);
                sm.last_issued[q][s] = -1;
                sm.released[q][s] = 0;
            }
        }
        cctdev::mbar_fence_init();
    }
    __syncthreads();
    // the block's state from the particle records, the step count as the CPU reference computes it; or
    // from the state of the launch before
    if (REC) {
        if (tid < G) {
            const double *S = P.state + (first + min(tid, mine - 1)) * kStateD;
#pragma unroll
            for (int c = 0; c < 6; ++c) sm.y0[c][tid] = sm.ys[c][tid] = S[ST_Y0 + c];
            sm.kq[tid] = S[ST_KQ];
            sm.reach[tid] = (float)S[ST_REACH];
            sm.nsteps[tid] = S[ST_NSTEPS];
            sm.h[0][tid] = S[ST_DT] / 2;
            sm.h[1][tid] = S[ST_DT];
            sm.h[2][tid] = S[ST_DT] / 6;
            if (tid < mine) atomicMax(&sm.max_steps, (int)S[ST_NSTEPS]);
        }
    } else if (tid < G) {
        const double *r = P.particles + (first + min(tid, mine - 1)) * 10;
#pragma unroll
        for (int c = 0; c < 6; ++c) sm.y0[c][tid] = sm.ys[c][tid] = r[c];
#pragma unroll
        for (int c = 0; c < 3; ++c) split_df(r[c], sm.pts[c][tid], sm.pts[3 + c][tid]);
        const double speed = r[8], dt0 = P.footstep / speed, t_end = P.distance / speed, steps = ceil(t_end / dt0);
        const bool ok = isfinite(steps) && steps >= 1.0 && steps < 5.0e8;   // (4 stages a step in an int)
        const double dt = ok ? t_end / steps : 0.0;
        sm.kq[tid] = r[7] / r[6];
        if (F64) sm.reach[tid] = df_reach(sub_blocks(P, ud), df_idle_field(r[7] / r[6], dt));
        sm.nsteps[tid] = ok ? steps : 0.0;
        sm.h[0][tid] = dt / 2;
        sm.h[1][tid] = dt;
        sm.h[2][tid] = dt / 6;
        if (tid < mine) {
            if (ok) atomicMax(&sm.max_steps, (int)steps);
            else if (ui == 0) atomicExch(P.ctrl + CW_NONFINITE, 1u);
        }
    }
    for (int i = tid; i < 2 * Sh::R * G; i += T) (&sm.prev[0][0][0])[i] = 0;
    for (int i = tid; i < 2 * 3 * G; i += T) (&sm.big_prev[0][0][0])[i] = 0;
    __syncthreads();
    const int step_end = REC ? min(sm.max_steps, P.step_end) : sm.max_steps;

    // the share
    constexpr int kHeldAt = (sizeof(OwnedSmem<F64, G, REM>) + 127) / 128 * 128;
    constexpr int kRoom = kOwnedSmemBytes - kHeldAt;
    constexpr int kRoomTiles = kRoom / Sh::Q / kTileBytes;             // of a quad
    constexpr int kRoomSubs = kRoom / (int)sizeof(DfSub);
    static_assert(kRoomTiles > kRing && kRoomSubs > Sh::NS * kOwnedWarps, "room for streaming");
    const int64_t seg0 = P.seg_off[ud], ns = P.seg_off[ud + 1] - seg0, nt = (ns + kTile - 1) / kTile;
    const double *kls = P.kls + 3 * seg0, *p0s = P.p0s + 3 * seg0;
    const int64_t subs = (ns + kDfSub - 1) / kDfSub, n_sub = (subs - ui + cd - 1) / cd;
    int64_t held = 0;
    int pieces = 0;
    OwnedQuad R{};
    bool ok = true;
    if constexpr (F64) {
        pieces = owned_pieces_log(n_sub, 32 / mine);
        held = n_sub <= kRoomSubs ? n_sub : (kRoomSubs - kOwnedWarps * Sh::NS) / Sh::NS * Sh::NS;
        for (int64_t i = warp; i < held; i += kOwnedWarps) {
            SegRaw raw;
            const int64_t a = (ui + i * cd) * kDfSub;
            const int cnt = (int)min((int64_t)kDfSub, ns - a);
            sub_load(raw, kls, p0s, a, cnt);
            df_stage(reinterpret_cast<DfSub *>(hold)[i], raw, cnt);
        }
    } else {
        const int quad = warp >> 2, nq = cd * Sh::Q, qi = ui * Sh::Q + quad;
        const int64_t units = P.chunks[ud];
        R.ct = P.chunk_tiles[ud];
        R.first = units * qi / nq;
        R.end = units * (qi + 1) / nq;
        const int64_t t0 = min(R.first * R.ct, nt);
        R.nt = R.end > R.first ? min(R.end * R.ct, nt) - t0 : 0;
        if (R.nt == 0) R.end = R.first;
        R.tiles = P.tiles + (P.tile_off[ud] + t0) * (int64_t)kTileBytes;
        R.mem = hold + quad * (kRoomTiles * kTileBytes);
        R.held = R.nt <= kRoomTiles;
        R.total = R.held ? 0 : R.nt * 4 * (int64_t)step_end;
        if ((tid & 127) == 0) {
            if (R.held && R.nt > 0) {
                cctdev::mbar_arrive_expect_tx(&sm.loaded[quad], (uint32_t)(R.nt * kTileBytes));
                for (int64_t t = 0; t < R.nt; ++t)
                    cctdev::bulk_g2s(R.mem + t * (int64_t)kTileBytes, R.tiles + t * (int64_t)kTileBytes, kTileBytes,
                                     &sm.loaded[quad]);
            }
            for (int64_t k = 0; k < kRing && k < R.total; ++k) owned_issue(sm, R, quad, k);
        }
        if (R.held && R.nt > 0) ok = cctdev::mbar_wait_bounded(&sm.loaded[quad], 0, kTmaPolls);
    }
    if (__syncthreads_or(!ok)) {
        if (!F64 && (tid & 127) == 0 && R.held && R.nt > 0) (void)cctdev::mbar_wait_bounded(&sm.loaded[warp >> 2], 0, kTmaPolls);
        if (tid == 0) {
            set_timeout(P);
            owned_drain(sm);
        }
        __syncthreads();
        return;
    }

    for (int step = REC ? P.step_begin : 0, phase = 0; step < step_end; ++step) {
        for (int stage = 0; stage < 4; ++stage, ++phase) {
            const int par = phase & 1;
            // 1. the share's field
            bool summed = true;
            if constexpr (F64)
                owned_sum_f64<G>(sm, reinterpret_cast<DfSub *>(hold), n_sub, held, ui, cd, ns, kls, p0s, mine, pieces);
            else
                summed = owned_sum_f32c<G, REM>(sm, R, phase * R.nt, F.shift);
            if (__syncthreads_or(!summed)) {
                if (tid == 0) {
                    set_timeout(P);
                    owned_drain(sm);
                }
                __syncthreads();
                return;
            }
            // 2. to the accumulators
            owned_add<F64, G, REM>(A, sm, copy, phase, mine, first, F);
            // what the update needs besides the field
            double x[Sh::NI][3], v[Sh::NI][3], y[Sh::NI][2], k[Sh::NI][2];
#pragma unroll
            for (int n = 0; n < Sh::NI; ++n) {
                const int i = tid + n * T, uc = i / G, us = i % G;
                if (uc >= 3) continue;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    x[n][c] = sm.ys[c][us];
                    v[n][c] = sm.ys[3 + c][us];
                }
                y[n][0] = sm.y0[uc][us];
                y[n][1] = sm.y0[3 + uc][us];
                k[n][0] = sm.ks[uc][us];
                k[n][1] = sm.ks[3 + uc][us];
            }
            const int qs_slot = T - 1 - tid;      // the last threads look for QS meanwhile
            if (qs_slot < G) {
                int hit = 0;
                for (int64_t q = q0; q < q1 && !hit; ++q)
                    hit = qs_may_act(P.qs + kQsRecord * q, sm.ys[0][qs_slot], sm.ys[1][qs_slot], sm.ys[2][qs_slot]);
                sm.qs_hit[qs_slot] = hit;
            }
            // 3. every CTA's, when they have arrived
            for (int i = tid; i < 4 * G; i += T) {
                const int uc = i / G, us = i % G;
                if (us >= mine) continue;
                unsigned long long d[2];
                const int64_t pi = first + us;
                const unsigned skew = (unsigned)P.flow_skew;      // (test hooks: an arrival that never comes)
                bool got;
                if (uc == 3) {
                    got = REM ? owned_poll_call<false>(P, A, par, 3, 3, pi, kOwnedFlagCount, (unsigned)cd + skew,
                                                       &sm.prev[par][3][us], nullptr, d)
                              : owned_poll<false>(P, A, par, 3, 3, pi, kOwnedFlagCount, (unsigned)cd + skew,
                                                  &sm.prev[par][3][us], nullptr, d);
                    sm.flags[us] = owned_flags(d[0]);
                } else {
                    double b;
                    if constexpr (REM) {
                        got = owned_poll_call<true>(P, A, par, uc, 4, pi, F.bits, (unsigned)cd + skew, &sm.prev[par][uc][us],
                                                    &sm.prev[par][4 + uc][us], d);
                        const long long low = (long long)(d[1] >> F.remainder_at(uc)) & ((1ll << (F.drop + F.bits)) - 1);
                        b = __ll2double_rn((owned_value(d[0], F.bits) << F.drop) + low) * fine;
                    } else {
                        got = owned_poll<F64>(P, A, par, uc, F64 ? 4 + uc : uc, pi, F.bits, (unsigned)cd + skew, &sm.prev[par][uc][us],
                                              &sm.prev[par][F64 ? 4 + uc : 0][us], d);
                        b = __ll2double_rn(owned_value(d[0], F.bits)) * unit;
                        if (F64) b += __ll2double_rn(owned_value(d[1], F.bits)) * (unit / (double)(1ll << kOwnedLowShift));
                    }
                    sm.B[uc][us] = b;
                }
                if (!got) sm.give_up = 1;
            }
            __syncthreads();
            if (sm.give_up) {
                if (tid == 0) owned_drain(sm);
                __syncthreads();
                return;
            }
            // every CTA has read the last stage's huge sums, and none adds to their set before this one's
            // stage after next
            if (huge_phase >= 0 && ui == 0) {
                for (int i = tid; i < 3 * kOwnedHugeUnits * mine; i += T)
                    *(volatile unsigned long long *)A.huge_at(huge_phase & 3, i / mine, first + i % mine) = 0ull;
                __threadfence();
            }
            huge_phase = -1;
            bool flagged = false;
#pragma unroll
            for (int n = 0; n < Sh::NI; ++n) {
                const int i = tid + n * T, uc = i / G, us = i % G;
                if (uc >= 3 || us >= mine || !((double)step < sm.nsteps[us])) continue;
                const unsigned fl = sm.flags[us];
                double B[3] = {sm.B[0][us], sm.B[1][us], sm.B[2][us]};
                if (fl) {       // fields beyond the usual range, or not finite
                    flagged = true;
                    __threadfence();
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const long long now = *(const volatile long long *)A.big_at(par, c, first + us);
                        B[c] += __ll2double_rn(now - sm.big_prev[par][c][us]) * unit;
                        if (fl & kHuge)
#pragma unroll 1
                            for (int k = 0; k < kOwnedHugeUnits; ++k)
                                B[c] += ldexp((double)*(const volatile long long *)A.huge_at(phase & 3, 3 * k + c, first + us), 54 * k - 54);
                        if (fl & kBad) B[c] = __longlong_as_double(0x7ff8000000000000LL);
                    }
                }
                if (sm.qs_hit[us])
                    for (int64_t q = q0; q < q1; ++q)
                        qs_field_add(P.qs + kQsRecord * q, x[n][0], x[n][1], x[n][2], B[0], B[1], B[2]);
                if (REC && P.record && ui == 0) {
                    double *rec = P.record + (((int64_t)(step - P.step_begin) * 4 + stage) * A.total + first + us) * kRec;
                    rec[uc] = uc == 0 ? x[n][0] : uc == 1 ? x[n][1] : x[n][2];
                    rec[3 + uc] = uc == 0 ? v[n][0] : uc == 1 ? v[n][1] : v[n][2];
                    rec[6 + uc] = uc == 0 ? B[0] : uc == 1 ? B[1] : B[2];
                }
                if (F64 && uc == 0) sm.reach[us] = fminf(sm.reach[us], df_reach(subs, B[0] * B[0] + B[1] * B[1] + B[2] * B[2]));
                // k = [v, kq (v x B)], component uc of both halves
                const double *vn = v[n];
                const double hk = sm.h[stage == 2 ? 1 : stage == 3 ? 2 : 0][us];
                const double vc = uc == 0 ? vn[0] : uc == 1 ? vn[1] : vn[2];
                const double a1 = uc == 0 ? vn[1] : uc == 1 ? vn[2] : vn[0], a2 = uc == 0 ? vn[2] : uc == 1 ? vn[0] : vn[1];
                const double b1 = uc == 0 ? B[1] : uc == 1 ? B[2] : B[0], b2 = uc == 0 ? B[2] : uc == 1 ? B[0] : B[1];
                const double kk[2] = {vc, __dmul_rn(__dadd_rn(__dmul_rn(a1, b2), -__dmul_rn(a2, b1)), sm.kq[us])};
                bool finite = true;
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const double kn = stage == 0 ? kk[j] : __dadd_rn(k[n][j], stage == 3 ? kk[j] : __dmul_rn(2.0, kk[j]));
                    const double yn = __dadd_rn(y[n][j], __dmul_rn(hk, stage == 3 ? kn : kk[j]));
                    finite = finite && isfinite(yn);
                    sm.ks[3 * j + uc][us] = kn;
                    sm.ys[3 * j + uc][us] = yn;
                    if (stage == 3) sm.y0[3 * j + uc][us] = yn;
                    if (!F64 && j == 0) split_df(yn, sm.pts[uc][us], sm.pts[3 + uc][us]);
                }
                if (stage == 3 && !finite && ui == 0) atomicExch(P.ctrl + CW_NONFINITE, 1u);
            }
            if (__syncthreads_or(flagged)) {       // (every component's thread has read big_prev)
                huge_phase = phase;
#pragma unroll
                for (int n = 0; n < Sh::NI; ++n) {
                    const int i = tid + n * T, uc = i / G, us = i % G;
                    if (uc < 3 && us < mine && sm.flags[us])
                        sm.big_prev[par][uc][us] = *(const volatile long long *)A.big_at(par, uc, first + us);
                }
                __syncthreads();
            }
        }
    }
    if (REC && ui == 0 && tid < mine) {
        double *S = P.state + (first + tid) * kStateD;
#pragma unroll
        for (int c = 0; c < 6; ++c) S[ST_Y0 + c] = S[ST_YS + c] = sm.y0[c][tid];
        S[ST_REACH] = sm.reach[tid];
    }
    if ((!REC || P.write_back) && ui == 0 && tid < mine && sm.nsteps[tid] > 0.0) {
        double *r = P.particles + (first + tid) * 10;
#pragma unroll
        for (int c = 0; c < 6; ++c) r[c] = sm.y0[c][tid];
        r[9] = r[9] + P.distance;
    }
}

template <bool F64, int G, bool REC = false, bool REM = false>
__global__ void __launch_bounds__(kOwnedThreads, 1) track_owned_kernel(TrackParams P) {
    extern __shared__ __align__(128) unsigned char owned_mem[];
    using SM = OwnedSmem<F64, G, REM>;
    // the device-side plan rejected the inputs, or chose another schedule
    if (*(volatile unsigned *)(P.ctrl + CW_ERR) != 0) return;
    if (P.planned_on_device && *(volatile unsigned *)(P.ctrl + CW_OWNED) == 0u) return;
    owned_track<F64, G, REC, REM>(P, *reinterpret_cast<SM *>(owned_mem), owned_mem + (sizeof(SM) + 127) / 128 * 128);
}

// The kernel of a launch, by particle block (track_owned_f32c.cu, track_owned_f64.cu).
using TrackKernel = void (*)(TrackParams);
TrackKernel owned_kernel_f32c(int G, bool few);
TrackKernel owned_kernel_f64(int G);
TrackKernel owned_kernel_f64_rec(int G);      // (track_owned_f64_rec.cu)

}  // namespace cctgpu
