// Small batches (at most kTinyMax particles in fewer than kFlowMinBlocks particle blocks): latency,
// not throughput, sets the time of an RK4 stage, so the schedule has one hop between SMs a stage.
//
// One CTA of 12 warps a SM owns one unit (design, particle block, segment chunk) for the whole
// launch.  It keeps the chunk in shared memory (as much as fits) and its own copy of the block's
// RK4 state.  A stage is:
//   1. the warps sum the chunk's field at the block's positions (FP32c tile slices, or FP64
//      sub-blocks, df.cuh);
//   2. the CTA's sum goes, as fixed-point integers, by atomic additions to the block's accumulators
//      in L2: (value << 10) + 1 a component, so that the low 10 bits count the units that have
//      arrived.  Integer sums do not depend on their order;
//   3. every CTA of the block reads the accumulators until every unit has arrived -- the data is its
//      own flag: no fence, no counter, no second trip -- and advances its copy of the particles
//      (the same integers and the same FP64 arithmetic in all of them).
// The accumulators are never cleared: a stage's value is the difference from the reading of the
// last stage of the same parity.  They come in up to kTinyCopies copies (the unit of chunk c adds
// into copy c % copies), so that fewer additions queue on an address.  A stage's words cannot be
// touched by the stage after next before every CTA has read them: that stage's additions follow
// the next stage's complete arrival, and a CTA adds to the next stage only after reading this one.
//
// Fixed point: 2^-44 T; FP64 keeps the remainder in a second word of 2^-86 T, so that its sums lose
// nothing of an FP64 unit field.  Unit fields of 2^52 / chunks units and more (2.1 T for 120 chunks)
// go to a word of their own without a count (up to 2^18 T, beyond that the particle becomes NaN);
// the flag word, which counts 3 arrivals a unit, says whether there are any.
//
// Bound by the latency of a stage (one L2 round of atomics, one of reads, three CTA barriers, FP64
// bookkeeping).  Measured, a stage of the 46 080-segment dipole: 32 protons FP32c 9.1 -> 6.8 us, 16
// and fewer 8.3 -> 5.9 (before: three CTAs a SM, each with the state of every particle, a fence,
// unit counters and a second read); FP64 32 protons 28 -> 16.4 us, 16 and fewer 25 -> 12.2 (before:
// grid barriers); 5 protons, 119 520 segments, FP64: 51 -> 20 us.
#pragma once

#include "track_common.cuh"

namespace cctgpu {

constexpr int kTinyThreads = 384;
constexpr int kTinyWarps = kTinyThreads / 32;
constexpr int kTinyGroup = 64;                 // largest particle block
constexpr int kTinySmemBytes = 215 << 10;      // dynamic shared memory: one CTA a SM
constexpr int kTinyCountBits = 10;
constexpr int kTinyLowShift = 42;              // FP64: the remainder's extra bits
constexpr int kTinyWords32 = 4, kTinyWords64 = 7;   // x, y, z, flags (, remainders x, y, z)
constexpr int kTinyFlagCount = 12, kTinyFlagBig = 12, kTinyFlagBad = 24;

struct TinySmem {
    double y0[6][kTinyGroup], ys[6][kTinyGroup], ks[6][kTinyGroup];
    double h[3][kTinyGroup];                   // dt / 2, dt, dt / 6
    double kq[kTinyGroup], nsteps[kTinyGroup];
    double B[3][kTinyGroup];
    long long prev[2][7][kTinyGroup];          // last reading of each parity's words
    long long big_prev[2][3][kTinyGroup];
    unsigned flags[kTinyGroup];
    int qs_hit[kTinyGroup];                    // a QS may act at the stage position
    float pts[6][kTinyGroup];                  // FP32c: stage positions as double-float
    union {
        long long fixed[kTinyWarps][kTinyGroup][3];
        double f64[kTinyWarps][kTinyGroup][3];
    } red;
    uint64_t loaded, full[2];
    int give_up;
    int max_steps;
};
constexpr int kTinyHeld = (sizeof(TinySmem) + 127) / 128 * 128;    // the chunk follows
constexpr int kTinyStream = 3;                                     // FP32c tiles a streamed group (HALF: 6)
constexpr int kTinyRoomTiles = (kTinySmemBytes - kTinyHeld) / kTileBytes;
constexpr int kTinyRoomSubs = (kTinySmemBytes - kTinyHeld) / (int)sizeof(DfSub);
static_assert(kTinyRoomTiles > 4 * kTinyStream && kTinyRoomSubs > 2 * kTinyWarps, "room for streaming");

// The accumulators of a launch.
struct TinyAcc {
    unsigned long long *words;    // [copies][2][words][particles]
    unsigned long long *big;      // [2][3][particles]
    int64_t total;
    int copies, n_words;
    __device__ unsigned long long *at(int copy, int par, int w, int64_t pi) const {
        return words + (((int64_t)copy * 2 + par) * n_words + w) * total + pi;
    }
    __device__ unsigned long long *big_at(int par, int c, int64_t pi) const { return big + ((int64_t)par * 3 + c) * total + pi; }
};

// FP32c: fields of the unit's tiles [0, nt) at the block's particles, per warp in fixed point.
// A warp takes the same slice of every kTinyWarps / 4-th tile (HALF: 2 sub-blocks, one a half-warp,
// of every kTinyWarps / 2-th); a tile slice is summed as in unit_sum_f32c.
template <int PPT, bool HALF>
static __device__ bool tiny_sum_f32c(TinySmem &sm, unsigned char *hold, int64_t nt,
                                     int64_t held, const unsigned char *tiles, uint32_t &groups_done) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int IPT = HALF ? 2 : 4;                       // items of a tile
    constexpr int SP = kTinyWarps / IPT;                    // tiles side by side
    constexpr int GT = kTinyWarps / IPT;                    // tiles of a streamed group: an item a warp
    const int r = warp % IPT;
    const int g0 = HALF ? (2 * r + (lane >> 4)) * (kSub / 4) : r * (kSub / 4), g1 = g0 + kSub / 4;
    const int pl0 = HALF ? lane & 15 : lane;
    float ph[PPT][3], pl[PPT][3];
#pragma unroll
    for (int i = 0; i < PPT; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            ph[i][c] = sm.pts[c][pl0 + 32 * i];
            pl[i][c] = sm.pts[3 + c][pl0 + 32 * i];
        }
    F32cAcc<PPT> acc;
    acc.zero();
    const int64_t streamed = nt - held, n_groups = (streamed + GT - 1) / GT;
    unsigned char *buf = hold + held * (int64_t)kTileBytes;
    auto issue = [&](int64_t g) {   // thread 0: the tiles of group g into buffer g & 1
        const int64_t t0 = g * GT, n = min((int64_t)GT, streamed - t0);
        const int b = (int)((groups_done + g) & 1);
        cctdev::fence_proxy_async();
        cctdev::mbar_arrive_expect_tx(&sm.full[b], (uint32_t)(n * kTileBytes));
        for (int64_t t = 0; t < n; ++t)
            cctdev::bulk_g2s(buf + (b * GT + t) * (int64_t)kTileBytes, tiles + (held + t0 + t) * (int64_t)kTileBytes,
                             kTileBytes, &sm.full[b]);
    };
    if (tid == 0)
        for (int64_t g = 0; g < 2 && g < n_groups; ++g) issue(g);
    for (int64_t t = warp / IPT; t < held; t += SP)
        tile_f32c<PPT, kTrackUnroll, kTrackRcp>(hold + t * (int64_t)kTileBytes, ph, pl, acc, g0, g1);
    bool ok = true;
    for (int64_t g = 0; g < n_groups; ++g) {
        const uint32_t k = groups_done + (uint32_t)g;
        ok = ok && cctdev::mbar_wait_bounded(&sm.full[k & 1], (k >> 1) & 1u, kTmaPolls);
        const int64_t t = g * GT + warp / IPT;
        if (ok && t < streamed)
            tile_f32c<PPT, kTrackUnroll, kTrackRcp>(buf + ((k & 1) * GT + warp / IPT) * (int64_t)kTileBytes, ph, pl,
                                                    acc, g0, g1);
        if (__syncthreads_or(!ok)) {
            ok = false;
            // the copies in flight land before the CTA gives up its shared memory
            if (tid == 0) {
                (void)cctdev::mbar_wait_bounded(&sm.full[k & 1], (k >> 1) & 1u, kTmaPolls);
                if (g + 1 < n_groups)
                    (void)cctdev::mbar_wait_bounded(&sm.full[(k + 1) & 1], ((k + 1) >> 1) & 1u, kTmaPolls);
            }
            break;
        }
        if (tid == 0 && g + 2 < n_groups) issue(g + 2);
    }
    groups_done += (uint32_t)n_groups;
#pragma unroll
    for (int i = 0; i < PPT; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            long long v = fixed44_pair(acc.S[i][c], acc.C[i][c]);
            if (HALF) {
                const long long o = __shfl_down_sync(0xffffffffu, v, 16);
                v = (v == kTinyBad || o == kTinyBad) ? kTinyBad : (long long)((unsigned long long)v + (unsigned long long)o);
            }
            if (!HALF || lane < 16) sm.red.fixed[warp][pl0 + 32 * i][c] = v;
        }
    return ok;
}

// FP64: fields of the unit's sub-blocks [0, n) (segments from a on, ns of them in the design) at the
// block's particles, per warp.  The first `held` sub-blocks are
// staged in shared memory for the whole launch, the others every time, in the warp's own slots.
template <bool HALF>
static __device__ void tiny_sum_f64(TinySmem &sm, DfSub *hold, int64_t n, int64_t held, int64_t sub0, int64_t ns,
                                    const double *kls, const double *p0s, bool plain) {
    constexpr int NS = HALF ? 2 : 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int slot = HALF ? lane & 15 : lane, half = HALF ? lane >> 4 : 0;
    const double p[3] = {sm.ys[0][slot], sm.ys[1][slot], sm.ys[2][slot]};
    DfSub *own = hold + held + warp * NS;
    auto count = [&](int64_t i) { return (int)min((int64_t)kDfSub, ns - (sub0 + i) * kDfSub); };
    DfSum sum;
    for (int64_t i0 = warp * NS; i0 < n; i0 += kTinyWarps * NS) {
        const DfSub *D = hold + i0;
        if (i0 >= held) {       // (held < n is a multiple of NS)
            __syncwarp();
            for (int k = 0; k < NS && i0 + k < n; ++k) {
                DfRaw raw;
                df_load(raw, kls, p0s, (sub0 + i0 + k) * kDfSub, count(i0 + k));
                df_stage(own[k], raw, count(i0 + k), plain);
            }
            __syncwarp();
            D = own;
        }
        const int h = i0 + half < n ? half : 0;
        double b[3];
        df_sub_field(D[h], kls, p0s, (sub0 + i0 + h) * kDfSub, p, b);
        if (h != half) b[0] = b[1] = b[2] = 0.0;
        sum.add(b);
    }
    sum.flush();
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double v = sum.b[c];
        if (HALF) v += __shfl_down_sync(0xffffffffu, v, 16);
        if (!HALF || lane < 16) sm.red.f64[warp][slot][c] = v;
    }
}

// The CTA's sum of component c at slot, added to the accumulators of particle pi.
template <bool F64>
static __device__ void tiny_add(const TinyAcc &A, const TinySmem &sm, int copy, int par, int slot, int c, int64_t pi,
                                long long limit) {
    long long v = 0, low = 0;
    bool bad = false;
    if (F64) {
        double s = 0.0;
        for (int w = 0; w < kTinyWarps; ++w) s += sm.red.f64[w][slot][c];
        bad = !(fabs(s) < (double)(1 << kTinyRange));
        const double x = bad ? 0.0 : s * kTinyScale, r = rint(x);
        v = __double2ll_rn(r);
        low = __double2ll_rn((x - r) * (double)(1ll << kTinyLowShift));
    } else {
        for (int w = 0; w < kTinyWarps; ++w) {
            const long long t = sm.red.fixed[w][slot][c];
            bad = bad || t == kTinyBad;
            v = (long long)((unsigned long long)v + (unsigned long long)t);
        }
        if (bad) v = 0;
    }
    const bool big = v >= limit || v <= -limit;
    if (big) {
        atomicAdd(A.big_at(par, c, pi), (unsigned long long)v);
        __threadfence();      // before the flag that announces it
    }
    atomicAdd(A.at(copy, par, c, pi), ((unsigned long long)(big ? 0 : v) << kTinyCountBits) + 1ull);
    if (F64) atomicAdd(A.at(copy, par, 4 + c, pi), ((unsigned long long)low << kTinyCountBits) + 1ull);
    atomicAdd(A.at(copy, par, 3, pi), 1ull + (big ? 1ull << kTinyFlagBig : 0ull) + (bad ? 1ull << kTinyFlagBad : 0ull));
}

// Polls word w of particle pi (TWO: and word w + 4), all copies, until `want` additions of this stage
// have arrived (the low `bits` bits of the difference from the last reading count them); false:
// gave up.
template <bool TWO>
static __device__ bool tiny_poll(const TrackParams &P, const TinyAcc &A, int par, int w, int64_t pi, int bits,
                                 unsigned want, long long *prev0, long long *prev1, unsigned long long (&diff)[2]) {
    const volatile int *err = reinterpret_cast<const volatile int *>(P.ctrl + CW_ERR);
    const unsigned long long mask = (1ull << bits) - 1ull;
    const unsigned long long p0 = (unsigned long long)*prev0, p1 = TWO ? (unsigned long long)*prev1 : 0ull;
    const unsigned long long *a0 = A.at(0, par, w, pi);
    const int64_t copy = 2 * A.n_words * A.total, up = 4 * A.total;
    unsigned long long t0 = 0;
    for (unsigned polls = 1;; ++polls) {
        unsigned long long s0 = 0, s1 = 0;
#pragma unroll
        for (int r = 0; r < kTinyCopies; ++r)
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

// Signed value above the count bits.
__device__ __forceinline__ long long tiny_value(unsigned long long diff) { return (long long)diff >> kTinyCountBits; }

// Whether a QS record may act at a point: conservative (the exact test follows in qs_field_add).
__device__ __forceinline__ bool qs_may_act(const double *q, double px, double py, double pz) {
    if (q[12] < 0.0 && isinf(q[12])) return true;
    const double z = q[9] * (px - q[0]) + q[10] * (py - q[1]) + q[11] * (pz - q[2]), e = 1e-6 + 1e-9 * fabs(z);
    return !(z < -e || z > fabs(q[12]) + e);
}

template <bool F64, int PPT, bool HALF>
static __device__ void tiny_track(const TrackParams &P, TinySmem &sm, unsigned char *hold) {
    const int tid = threadIdx.x, warp = tid >> 5;
    constexpr int G = HALF ? 16 : PPT == 2 ? 64 : 32;
    static_assert(G <= kTinyGroup, "blocks of at most kTinyGroup");
    const int64_t n_units = P.unit_off[P.n_designs];
    if ((int64_t)blockIdx.x >= n_units) return;
    const UnitRef U = locate_unit(P, blockIdx.x);
    const int64_t first = (int64_t)U.d * P.n_p + U.b * G;             // the block's first particle
    const int mine = (int)min((int64_t)G, P.n_p - U.b * G);           // its particles
    const unsigned cd = (unsigned)P.chunks[U.d];
    const int64_t q0 = P.qs_off[U.d], q1 = P.qs_off[U.d + 1];
    TinyAcc A{reinterpret_cast<unsigned long long *>(P.tiny_acc), nullptr, (int64_t)P.n_designs * P.n_p, P.tiny_copies,
              F64 ? kTinyWords64 : kTinyWords32};
    A.big = A.words + (int64_t)A.copies * 2 * A.n_words * A.total;
    const int copy = (int)(U.c % A.copies);
    const long long limit = (1ll << 52) / cd;

    // the block's state from the particle records, the step count as the CPU reference computes it
    if (tid == 0) {
        sm.give_up = 0;
        sm.max_steps = 0;
        cctdev::mbar_init(&sm.loaded, 1);
        cctdev::mbar_init(&sm.full[0], 1);
        cctdev::mbar_init(&sm.full[1], 1);
        cctdev::mbar_fence_init();
    }
    __syncthreads();
    if (tid < G) {
        const double *r = P.particles + (first + min(tid, mine - 1)) * 10;
#pragma unroll
        for (int c = 0; c < 6; ++c) sm.y0[c][tid] = sm.ys[c][tid] = r[c];
#pragma unroll
        for (int c = 0; c < 3; ++c) split_df(r[c], sm.pts[c][tid], sm.pts[3 + c][tid]);
        const double speed = r[8], dt0 = P.footstep / speed, t_end = P.distance / speed, steps = ceil(t_end / dt0);
        const bool ok = isfinite(steps) && steps >= 1.0 && steps < 5.0e8;   // (4 stages a step in an int)
        const double dt = ok ? t_end / steps : 0.0;
        sm.kq[tid] = r[7] / r[6];
        sm.nsteps[tid] = ok ? steps : 0.0;
        sm.h[0][tid] = dt / 2;
        sm.h[1][tid] = dt;
        sm.h[2][tid] = dt / 6;
        if (tid < mine) {
            if (ok) atomicMax(&sm.max_steps, (int)steps);
            else if (U.c == 0) atomicExch(P.ctrl + CW_NONFINITE, 1u);
        }
    }
    for (int i = tid; i < 2 * 7 * kTinyGroup; i += kTinyThreads) (&sm.prev[0][0][0])[i] = 0;
    for (int i = tid; i < 2 * 3 * kTinyGroup; i += kTinyThreads) (&sm.big_prev[0][0][0])[i] = 0;

    // the chunk, as much as fits
    const int64_t seg0 = P.seg_off[U.d], ns = P.seg_off[U.d + 1] - seg0;
    const int64_t nt = max(U.t_end - U.t_beg, (int64_t)0);
    const unsigned char *tiles = F64 ? nullptr : P.tiles + (P.tile_off[U.d] + U.t_beg) * (int64_t)kTileBytes;
    const double *kls = P.kls + 3 * seg0, *p0s = P.p0s + 3 * seg0;
    constexpr int kSubs = kTile / kDfSub;
    const int64_t sub0 = U.t_beg * kSubs;
    const int64_t n_sub = max(min(U.t_end * kSubs, (ns + kDfSub - 1) / kDfSub) - sub0, (int64_t)0);
    const bool plain = ns < kDfMinSegments;
    int64_t held;
    bool ok = true;
    if (F64) {
        constexpr int NS = HALF ? 2 : 1;
        held = n_sub <= kTinyRoomSubs ? n_sub : (kTinyRoomSubs - kTinyWarps * NS) / NS * NS;
        for (int64_t i = warp; i < held; i += kTinyWarps) {
            DfRaw raw;
            const int cnt = (int)min((int64_t)kDfSub, ns - (sub0 + i) * kDfSub);
            df_load(raw, kls, p0s, (sub0 + i) * kDfSub, cnt);
            df_stage(reinterpret_cast<DfSub *>(hold)[i], raw, cnt, plain);
        }
    } else {
        held = nt <= kTinyRoomTiles ? nt : kTinyRoomTiles - 2 * (HALF ? 2 * kTinyStream : kTinyStream);
        if (held > 0) {
            if (tid == 0) {
                cctdev::mbar_arrive_expect_tx(&sm.loaded, (uint32_t)(held * kTileBytes));
                for (int64_t t = 0; t < held; ++t)
                    cctdev::bulk_g2s(hold + t * (int64_t)kTileBytes, tiles + t * (int64_t)kTileBytes, kTileBytes, &sm.loaded);
            }
            ok = cctdev::mbar_wait_bounded(&sm.loaded, 0, kTmaPolls);
        }
    }
    if (__syncthreads_or(!ok)) {
        if (tid == 0) {
            set_timeout(P);
            (void)cctdev::mbar_wait_bounded(&sm.loaded, 0, kTmaPolls);
        }
        __syncthreads();
        return;
    }

    const int step_end = sm.max_steps;
    uint32_t groups_done = 0;
    const int uc = tid / G, us = tid % G;               // a thread's component and slot, in 2 and 3
    for (int step = 0, phase = 0; step < step_end; ++step) {
        for (int stage = 0; stage < 4; ++stage, ++phase) {
            const int par = phase & 1;
            // 1. the chunk's field
            if (F64) {
                tiny_sum_f64<HALF>(sm, reinterpret_cast<DfSub *>(hold), n_sub, held, sub0, ns, kls, p0s, plain);
            } else if (!tiny_sum_f32c<PPT, HALF>(sm, hold, nt, held, tiles, groups_done)) {
                if (tid == 0) set_timeout(P);
                __syncthreads();
                return;
            }
            __syncthreads();
            // 2. to the accumulators
            if (uc < 3 && us < mine) tiny_add<F64>(A, sm, copy, par, us, uc, first + us, limit);
            // what the update needs besides the field
            double x[3], v[3], y[2], k[2], hk = 0.0, kq = 0.0;
            bool active = false;
            if (uc < 3) {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    x[c] = sm.ys[c][us];
                    v[c] = sm.ys[3 + c][us];
                }
                y[0] = sm.y0[uc][us];
                y[1] = sm.y0[3 + uc][us];
                k[0] = sm.ks[uc][us];
                k[1] = sm.ks[3 + uc][us];
                hk = sm.h[stage == 2 ? 1 : stage == 3 ? 2 : 0][us];
                kq = sm.kq[us];
                active = us < mine && (double)step < sm.nsteps[us];
            }
            const int qs_slot = tid - (kTinyThreads - G);    // the last threads look for QS meanwhile
            if (qs_slot >= 0) {
                int hit = 0;
                for (int64_t q = q0; q < q1 && !hit; ++q)
                    hit = qs_may_act(P.qs + kQsRecord * q, sm.ys[0][qs_slot], sm.ys[1][qs_slot], sm.ys[2][qs_slot]);
                sm.qs_hit[qs_slot] = hit;
            }
            // 3. every unit's, when they have arrived
            if (uc < 4 && us < mine) {
                unsigned long long d[2];
                const int64_t pi = first + us;
                const unsigned skew = (unsigned)P.flow_skew;      // (test hooks: an arrival that never comes)
                bool got;
                if (uc == 3) {
                    got = tiny_poll<false>(P, A, par, 3, pi, kTinyFlagCount, 3 * cd + skew, &sm.prev[par][3][us], nullptr, d);
                    sm.flags[us] = (unsigned)(d[0] >> kTinyFlagBig);
                } else {
                    got = tiny_poll<F64>(P, A, par, uc, pi, kTinyCountBits, cd + skew, &sm.prev[par][uc][us],
                                         &sm.prev[par][4 + (F64 ? uc : 0)][us], d);
                    double b = __ll2double_rn(tiny_value(d[0])) * (1.0 / kTinyScale);
                    if (F64) b += __ll2double_rn(tiny_value(d[1])) * (1.0 / kTinyScale / (double)(1ll << kTinyLowShift));
                    sm.B[uc][us] = b;
                }
                if (!got) sm.give_up = 1;
            }
            __syncthreads();
            if (sm.give_up) return;
            const unsigned fl = active ? sm.flags[us] : 0u;
            if (active) {
                double B[3] = {sm.B[0][us], sm.B[1][us], sm.B[2][us]};
                if (fl) {       // unit fields beyond the usual range, or not finite
                    __threadfence();
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const long long now = *(const volatile long long *)A.big_at(par, c, first + us);
                        B[c] += __ll2double_rn(now - sm.big_prev[par][c][us]) * (1.0 / kTinyScale);
                        if (fl >> (kTinyFlagBad - kTinyFlagBig)) B[c] = __longlong_as_double(0x7ff8000000000000LL);
                    }
                }
                if (sm.qs_hit[us])
                    for (int64_t q = q0; q < q1; ++q)
                        qs_field_add(P.qs + kQsRecord * q, x[0], x[1], x[2], B[0], B[1], B[2]);
                // k = [v, kq (v x B)], component uc of both halves
                const double vc = uc == 0 ? v[0] : uc == 1 ? v[1] : v[2];
                const double a1 = uc == 0 ? v[1] : uc == 1 ? v[2] : v[0], a2 = uc == 0 ? v[2] : uc == 1 ? v[0] : v[1];
                const double b1 = uc == 0 ? B[1] : uc == 1 ? B[2] : B[0], b2 = uc == 0 ? B[2] : uc == 1 ? B[0] : B[1];
                const double kk[2] = {vc, __dmul_rn(__dadd_rn(__dmul_rn(a1, b2), -__dmul_rn(a2, b1)), kq)};
                bool finite = true;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    k[i] = stage == 0 ? kk[i] : __dadd_rn(k[i], stage == 3 ? kk[i] : __dmul_rn(2.0, kk[i]));
                    const double n = __dadd_rn(y[i], __dmul_rn(hk, stage == 3 ? k[i] : kk[i]));
                    finite = finite && isfinite(n);
                    sm.ks[3 * i + uc][us] = k[i];
                    sm.ys[3 * i + uc][us] = n;
                    if (stage == 3) sm.y0[3 * i + uc][us] = n;
                    if (i == 0) split_df(n, sm.pts[uc][us], sm.pts[3 + uc][us]);
                }
                if (stage == 3 && !finite && U.c == 0) atomicExch(P.ctrl + CW_NONFINITE, 1u);
            }
            if (__syncthreads_or(fl != 0u)) {      // (every component's thread has read big_prev)
                if (fl) sm.big_prev[par][uc][us] = *(const volatile long long *)A.big_at(par, uc, first + us);
                __syncthreads();
            }
        }
    }
    if (U.c == 0 && P.write_back && tid < mine && sm.nsteps[tid] > 0.0) {
        double *r = P.particles + (first + tid) * 10;
#pragma unroll
        for (int c = 0; c < 6; ++c) r[c] = sm.y0[c][tid];
        r[9] = r[9] + P.distance;
    }
}

template <bool F64>
__global__ void __launch_bounds__(kTinyThreads, 1) track_tiny_kernel(TrackParams P) {
    extern __shared__ __align__(128) unsigned char tiny_mem[];
    TinySmem &sm = *reinterpret_cast<TinySmem *>(tiny_mem);
    unsigned char *hold = tiny_mem + kTinyHeld;
    if (*(volatile unsigned *)(P.ctrl + CW_ERR) != 0) return;   // the device-side plan rejected the inputs
    if (P.G == kHalfGroup) tiny_track<F64, 1, true>(P, sm, hold);
    else if (F64 || P.ppt == 1) tiny_track<F64, 1, false>(P, sm, hold);
    else tiny_track<F64, 2, false>(P, sm, hold);
}

}  // namespace cctgpu
