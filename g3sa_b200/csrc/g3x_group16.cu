// g3x_group16.cu -- group-per-job sm_100a kernel for batched ksw_extend2 in int16x2
// (bwa/src/ksw.cu:303-401), for batches too small to fill the lane-per-job kernel.
//
// The lane-per-job kernel (g3x_lane16.cu) needs tens of thousands of jobs: a lane walks its row
// block by block, 2,000-3,400 cycles a row for 200 columns, so a batch lasts as long as its
// longest job (0.5-0.6 ms at 250 bases) however few jobs it has.  Here a group of G lanes runs a
// job and a row is one step: lane r of the group holds B eight-column blocks of the row buffer
// (ksw.cu:310), columns 8 B r on, in registers for the whole job, as the same four int16x2 words of
// H and four of E per block, with the blocks' query codes beside them.  B G = 4, 8, 16 or 32 by query
// length (up to 31, 63, 127, 255 bases: the group holds column qlen too), so a warp runs 8 B to B
// jobs.  Nothing of a row touches memory.
//
// One row: every lane runs the block recurrence of g3x_lane16.cuh; the F that enters each lane
// is a max-plus prefix over the group (g3x_group.cuh); H of the column left of a lane's first block
// comes from the lane before it by one shuffle; the row maximum with its last column is one max over
// (H << 16 | column) keys; and the trim of end (ksw.cu:390-391) takes the last lane of a ballot over
// the lanes' non-zero column masks.  Band edges follow g3x_lane16.cuh: columns left of beg hold
// zeros (the words the band clamp cuts off are zeroed), columns right of end keep their words, column
// end gets {H(i, end-1), 0}, which the shifted H words of its block hold already.
//
// What bounds it: latency for small batches -- a warp alone takes 600 cycles over a row's 220
// dependent-heavy instructions --, the ALU pipe beyond a few thousand jobs (84% busy at 20k jobs).
// 62 jobs 598 us -> 113, 20k 800 -> 323 against the lane classes.
#include <cuda_runtime.h>
#include "g3x_core.h"
#include "g3x_group.cuh"
#include "g3x_internal.h"
#include "g3x_lane16.cuh"
#include "g3x_stage.cuh"

namespace g3x {

namespace {

using namespace l16;

constexpr int kBlockWarps = 2;
constexpr int kOneBlockJobs = 32768;

// Masks by h = clamp(end - first column of the block, -1, 8), entry h + 1: the pair words of
// the columns left of end and right of end, and the bits of the columns up to end.
struct EdgeTable {
    uint4 left[10], right[10];
    uint32_t upto[10];
};

// No row yet: below every row's key but those of rows without a positive cell (columns stay below
// 256).
constexpr int32_t kNoRow = 0xFFFF;
constexpr int32_t kNoGscore = -2;   // no to-end score in a row: below gscore's start

// v >> n for any n as an unsigned shift amount: 0 from 32 on.
__device__ __forceinline__ uint32_t shr_clamp(uint32_t v, uint32_t n) {
    uint32_t r;
    asm("shr.b32 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(n));
    return r;
}

// One group's job (uniform over its lanes, but for gscore and max_ie, which count only in the
// lane that holds column qlen).
struct GroupJob {
    int32_t job;                   // -1: none
    int32_t qlen, tlen, w;
    int32_t i;                     // the next row
    int32_t hv;                    // h0 - o_del - e_del (i + 1)
    uint32_t t_off;
    bool trev;
    int32_t best, best_i, best_d;  // the maximum, its row, its diagonal (row - column)
    int32_t max_off, gscore, max_ie, cells;
    uint32_t qsel;                 // prmt selector of column qlen's H from words 0-1 or 2-3
};

// Runs the jobs order[0 .. n) (order null: 0 .. n) of one class with groups of G lanes, taken from
// *queue.  misfit non-null: jobs that do not fit (query, int16) go to misfit[0 .. *misfits)
// instead of being refused.
//
// The row loop is rotated so that the parts of a row that only decide (its maximum, z-drop, the
// next band) overlap the next row's blocks, whose inputs they are not: an iteration starts with
// row i's blocks and F prefix, then finishes row i - 1's bookkeeping from the reductions issued at
// its end, and then completes row i within the band that this gives.
template <int G, int B, bool kSym>
__device__ __forceinline__ void run_groups(const LaunchDesc& d, const ScoreParams& sp, const PairConst& pc,
                                           const EdgeTable& tab, const uint2* pools, const int32_t* order, int n,
                                           int32_t* queue, int32_t* misfit, int32_t* misfits, int lane,
                                           unsigned long long& busy, unsigned long long& idle,
                                           unsigned long long& waves) {
    constexpr int kGroups = 32 / G;
    const int r = lane & (G - 1), gb = lane & ~(G - 1);
    const unsigned gmask = (G == 32 ? kAll : ((1u << G) - 1u)) << gb;
    unsigned leaders = 0;
#pragma unroll
    for (int k = 0; k < kGroups; ++k) leaders |= 1u << (k * G);
    const int col0 = 8 * B * r;
    const int32_t zdrop = sp.zdrop > 0 ? sp.zdrop : 0x7FFFFFFF;

    GroupJob J = {};
    J.job = -1;
    uint32_t H[B][4], E[B][4];
    uint32_t qw[B], tw = 0;       // query codes of the blocks; target codes of rows 8 (r + G c) ..
#pragma unroll
    for (int b = 0; b < B; ++b) {
        qw[b] = 0u;
#pragma unroll
        for (int p = 0; p < 4; ++p) H[b][p] = E[b][p] = 0u;
    }
    uint2 pl = pools[0];          // score pools of row i
    // row i - 1: (maximum << 16 | its last column), its to-end score, and its last lane with
    // non-zero columns with their mask
    int32_t key = kNoRow, gval = kNoGscore;
    int ll = 0;
    uint32_t nzl = 1u;
    int32_t beg = 0;              // kept for the cell counts only (see g3x_lane16.cuh)
    bool exhausted = false, all_idle = true;
    int32_t iters = 0;
    unsigned long long rows = 0;
    for (;;) {
        // ---- row i: the blocks with F from zero, and the F entering each ----
        RowState rs;
        rs.plo = pl.x; rs.phi = pl.y;
        BlockA a[B];
        uint32_t ne[B][4];
        int32_t x = 0;                                   // F leaving the lane's blocks
#pragma unroll
        for (int b = 0; b < B; ++b) {
            phase_a<kSym>(H[b], E[b], qw[b], rs, pc, a[b], ne[b]);
            const int32_t xb = (int32_t)__viaddmax_s16x2(a[b].L2[3] << 16, pc.n4, a[b].L2[3]);
            x = b ? __viaddmax_s32(x, decay_hi(sp.e_ins, 1), xb) : xb;
        }
        rs.fr = (uint32_t)f_entering<G>(x, r, B * sp.e_ins);
        rs.hlast = 0u;
        // score pools of row i + 1: lane r holds the target codes of rows i0 + 8r .. + 7, i0 the
        // last multiple of 8 G rows
        const int32_t i1 = J.i + 1;
        if ((i1 & (8 * G - 1)) == 0) {
            if (J.job >= 0) tw = codes8(d.codes, d.nmask, J.t_off, J.tlen, J.trev, i1 + 8 * r);
        }
        // (the funnel shift takes its amount modulo 32)
        const uint32_t t8 = __shfl_sync(kAll, tw, gb | ((i1 >> 3) & (G - 1)));
        pl = pools[__funnelshift_r(t8, 0u, i1 << 2) & 7u];

        // ---- row i - 1's bookkeeping (ksw.cu:371-386) ----
        J.max_ie = gval >= J.gscore ? J.i - 1 : J.max_ie;
        J.gscore = max(J.gscore, gval);
        const int32_t m = key >> 16, dg = J.i - 1 - (key & 0xFFFF);
        const bool up = m > J.best;
        // z-drop: best - m, less the gap between the diagonals (never for a new maximum)
        const int32_t t = dg - J.best_d;
        const bool zstop = J.best - m - max(t * sp.e_del, -t * sp.e_ins) > zdrop;
        J.max_off = max(J.max_off, up ? abs(dg) : 0);
        J.best = max(J.best, m);
        J.best_i = up ? J.i - 1 : J.best_i;
        J.best_d = up ? dg : J.best_d;
        // no positive cell, z-drop or the last row; or no job in any group
        const bool stop = J.job >= 0 ? (uint32_t)key < (uint32_t)kNoRow || zstop || J.i >= J.tlen : all_idle;
        if (__any_sync(kAll, stop)) {
            const int owner = gb + J.qlen / (8 * B);          // holds column qlen
            const int32_t gs = __shfl_sync(kAll, J.gscore, owner & 31), gi = __shfl_sync(kAll, J.max_ie, owner & 31);
            if (stop && J.job >= 0) {
                if (r == 0) {
                    d.out[J.job] = g3x_ext_t{J.best, J.best_i - J.best_d + 1, J.best_i + 1, gi + 1, gs, J.max_off};
                    d.status[J.job] = G3X_OK;
                    if (d.cells) d.cells[J.job] = J.cells;
                    if (d.rows) d.rows[J.job] = J.i;
                    rows += J.i;
                }
                J.job = -1;
            }
            // refill together once half of the groups are idle: a refill waits for two dependent
            // global loads, and jobs of a class and length come one after another
            const unsigned idle = __ballot_sync(kAll, J.job < 0);
            if (exhausted ? idle == kAll : 2 * __popc(idle) >= 32) {
                if (exhausted) break;
                const unsigned want = idle & leaders;
                int first = 0;
                if (lane == 0) first = atomicAdd(queue, __popc(want));
                first = __shfl_sync(kAll, first, 0);
                exhausted = first + __popc(want) >= n;
                ++waves;
                const int slot = first + __popc(want & ((1u << gb) - 1u));
                bool fresh = false;
                if (J.job < 0 && slot < n) {
                    const int job = order ? order[slot] : slot;
                    const g3x_job_t jb = d.jobs[job];
                    JobConst c;
                    c.qlen = jb.qlen; c.tlen = jb.tlen; c.h0 = jb.h0;
                    c.o_del = sp.o_del; c.e_del = sp.e_del; c.o_ins = sp.o_ins; c.e_ins = sp.e_ins;
                    c.oe_del = sp.oe_del; c.oe_ins = sp.oe_ins; c.zdrop = sp.zdrop;
                    c.w = clamp_w(jb.w, c.qlen, sp.max_sc, sp.end_bonus, sp.o_del, sp.e_del, sp.o_ins, sp.e_ins);
                    const bool fits = c.qlen < 8 * B * G && job_fits_int16(c, sp.max_sc);
                    const bool too_long = c.qlen > d.qmax || c.tlen > d.tmax || !fits;
                    const bool outside = !job_in_planes(jb, d.n_bases);
                    if (!fits && misfit) {
                        if (r == 0) misfit[atomicAdd(misfits, 1)] = job;
                    } else if (too_long || outside || c.tlen == 0 || c.w < 0) {
                        // refused before any base is read, or no cells
                        if (r == 0) finish_unrun(d, job, c, too_long ? G3X_ERR_TOO_LONG : outside ? G3X_ERR_INVALID : G3X_OK);
                    } else {
                        fresh = true;
                        J.job = job;
                        J.qlen = c.qlen; J.tlen = c.tlen; J.w = c.w;
                        J.i = 0;
                        J.hv = c.h0 - c.oe_del;
                        J.t_off = jb.t_off;
                        J.trev = (jb.flags & G3X_JOB_TREV) != 0;
                        J.best = c.h0; J.best_i = J.gscore = J.max_ie = -1;
                        J.best_d = J.max_off = J.cells = 0;
                        // column t of a block: half t >> 2 of word t & 3
                        const uint32_t b2 = ((c.qlen & 1) ? 0x54u : 0x10u) + ((c.qlen & 4) ? 0x22u : 0u);
                        J.qsel = b2 | (8u | b2 >> 4) * 0x1100u;      // zero-extended by H's sign
                        // the blocks' query codes, the first rows' target codes and row -1
                        // (ksw.cu:317-319)
                        tw = codes8(d.codes, d.nmask, J.t_off, c.tlen, J.trev, 8 * r);
#pragma unroll
                        for (int b = 0; b < B; ++b) {
                            qw[b] = codes8(d.codes, d.nmask, jb.q_off, c.qlen, (jb.flags & G3X_JOB_QREV) != 0, col0 + 8 * b);
#pragma unroll
                            for (int p = 0; p < 4; ++p) {
                                const int j = col0 + 8 * b + p;
                                const uint32_t lo = j <= c.qlen + 1 ? (uint32_t)init_h(j, c) : 0u;
                                const uint32_t hi = j + 4 <= c.qlen + 1 ? (uint32_t)init_h(j + 4, c) : 0u;
                                H[b][p] = (lo & 0xFFFFu) | (hi << 16);
                                E[b][p] = 0u;
                            }
                        }
                        // the band of row 0: all of [0, qlen)
                        ll = gb + 64; nzl = 1u;
                        beg = 0;
                    }
                }
                // start the iteration anew: nothing is left of row i - 1, and a new job's blocks
                // are still to come
                const uint32_t t0 = __shfl_sync(kAll, tw, gb);
                pl = fresh ? pools[t0 & 7u] : make_uint2(rs.plo, rs.phi);
                all_idle = __all_sync(kAll, J.job < 0);
                key = J.best << 16 | kNoRow;
                gval = kNoGscore;
                continue;
            }
        }
        ++iters;

        // ---- the band of row i (ksw.cu:388-391, then 335-345) ----
        const int32_t cut = J.i - J.w;
        const int32_t end = min(min(8 * B * (ll - gb) + msb32(nzl) + 2, J.i + J.w + 1), J.qlen);
        const int32_t h1 = cut <= 0 ? max(J.hv, 0) : 0;
        J.hv -= sp.e_del;
        // ---- the rest of the row: F and H, the row maximum, the new words ----
        uint32_t nh[B][4], h2[B][4];
#pragma unroll
        for (int b = 0; b < B; ++b) phase_b(a[b], rs, pc, nh[b], h2[b]);
        const uint32_t hl = __shfl_up_sync(kAll, rs.hlast, 1, G);
        key = 0;
        uint32_t nz = 0u;
#pragma unroll
        for (int b = 0; b < B; ++b) {
            const int h = max(min(end - col0 - 8 * b, 8), -1) + 1;
            const uint4 lv = tab.left[h], rv = tab.right[h];
            const uint32_t left[4] = {lv.x, lv.y, lv.z, lv.w}, right[4] = {rv.x, rv.y, rv.z, rv.w};
            int32_t kk[8];
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                const uint32_t v = h2[b][p] & left[p];
                kk[p] = (int32_t)(v * sp.k16 + (uint32_t)(8 * b + p));
                kk[p + 4] = (int32_t)prmt((uint32_t)(8 * b + p + 4), v, 0x7610u);
            }
            key = max3_i32(max3_i32(key, kk[0], kk[1]), max3_i32(kk[2], kk[3], kk[4]), max3_i32(kk[5], kk[6], kk[7]));
            if (b == 0) nh[0][0] = prmt(r ? hl : (uint32_t)h1 << 16, h2[0][3], 0x5432u);
            // columns beyond end keep their words, column end has E = 0 (ksw.cu:371)
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                H[b][p] = (nh[b][p] & ~right[p]) | (H[b][p] & right[p]);
                E[b][p] = (ne[b][p] & left[p]) | (E[b][p] & right[p]);
            }
            nz |= nonzero_mask(H[b], E[b], tab.upto[h]) << (8 * b);
        }
        key = max_of_group<G>(key + col0);
        const unsigned bal = __ballot_sync(kAll, nz != 0u) & gmask;
        ll = msb32(bal);
        nzl = __shfl_sync(kAll, nz, ll & 31);
        if (d.cells) {
            J.cells += max(end - max(beg, cut), 0);
            const int fl = ffs32(bal) - 1;
            beg = 8 * B * (fl - gb) + ffs32(__shfl_sync(kAll, nz, fl & 31)) - 1;
        }
        // to-end score: H(i, qlen - 1) is the H word of column qlen (used in its lane only)
        {
            const bool w2 = (J.qlen & 2) != 0;
            uint32_t lo = w2 ? H[0][2] : H[0][0], hi = w2 ? H[0][3] : H[0][1];
#pragma unroll
            for (int b = 1; b < B; ++b) {
                const bool mine = ((J.qlen >> 3) & (B - 1)) == b;
                lo = mine ? (w2 ? H[b][2] : H[b][0]) : lo;
                hi = mine ? (w2 ? H[b][3] : H[b][1]) : hi;
            }
            const int32_t v = (int32_t)prmt(lo, hi, J.qsel);
            gval = end == J.qlen ? v : kNoGscore;
        }
        // the column that the band clamp cuts off in row i + 1 (ksw.cu:338) becomes zero
        const int cc = cut - col0;
        if (__any_sync(kAll, shr_clamp(nz, (uint32_t)cc) & 1u)) {
#pragma unroll
            for (int b = 0; b < B; ++b)
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const uint32_t keep = cc == 8 * b + p ? 0xFFFF0000u : cc == 8 * b + p + 4 ? 0x0000FFFFu : 0xFFFFFFFFu;
                    H[b][p] &= keep;
                    E[b][p] &= keep;
                }
        }
        ++J.i;
    }
    busy += rows;
    idle += (lane == 0 ? (unsigned long long)iters * kGroups : 0ull) - rows;
}

// B = 0: jobs 0 .. n in the given order (or d.order's), one warp each; misfit non-null (see
// run_groups).  Else classes 0-3 of a sorted batch (order_off: [offset, count] pairs), widest first,
// B blocks a lane.
template <int B, bool kSym>
__global__ void __launch_bounds__(32 * kBlockWarps, B == 2 ? 8 : 1) group16_kernel(LaunchDesc d, ScoreParams sp, int32_t* misfit,
                                                                  int32_t* misfits) {
    pdl_trigger();
    __shared__ EdgeTable tab;
    __shared__ uint2 pools[8];
    for (int t = threadIdx.x; t < 10; t += 32 * kBlockWarps) {
        const int h = t - 1;
        uint32_t lw[4], rw[4];
        for (int p = 0; p < 4; ++p) {
            lw[p] = ~ge_word(h < 0 ? 0 : h, p);
            rw[p] = ge_word(h + 1, p);
        }
        tab.left[t] = make_uint4(lw[0], lw[1], lw[2], lw[3]);
        tab.right[t] = make_uint4(rw[0], rw[1], rw[2], rw[3]);
        tab.upto[t] = h < 0 ? 0u : (h < 8 ? (2u << h) - 1u : 0xFFu) & 0xFFu;
    }
    if (threadIdx.x < 8) {
        uint32_t lo[5], hi[5];
        score_pools(sp, lo, hi);
        const int a = threadIdx.x < 4 ? threadIdx.x : 4;
#pragma unroll
        for (int t = 0; t < 5; ++t)
            if (a == t) pools[threadIdx.x] = make_uint2(lo[t], hi[t]);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const PairConst pc = pair_const(sp);
    unsigned long long busy = 0, idle = 0, waves = 0;
    if constexpr (B == 0) {
        const int n = d.count ? *d.count : d.n;
        run_groups<32, 1, kSym>(d, sp, pc, tab, pools, d.order, n, d.queue, misfit, misfits, lane, busy, idle, waves);
    } else {
        const int32_t* oc = d.order_off;
        run_groups<32 / B, B, kSym>(d, sp, pc, tab, pools, d.order + oc[6], oc[7], d.queue + 3, nullptr, nullptr, lane, busy, idle, waves);
        run_groups<16 / B, B, kSym>(d, sp, pc, tab, pools, d.order + oc[4], oc[5], d.queue + 2, nullptr, nullptr, lane, busy, idle, waves);
        run_groups<8 / B, B, kSym>(d, sp, pc, tab, pools, d.order + oc[2], oc[3], d.queue + 1, nullptr, nullptr, lane, busy, idle, waves);
        run_groups<4 / B, B, kSym>(d, sp, pc, tab, pools, d.order + oc[0], oc[1], d.queue, nullptr, nullptr, lane, busy, idle, waves);
    }
    if (d.stats) add_warp_stats(d.stats, busy, idle, waves, lane);
    pdl_chain_end();
}

}  // namespace

// The classes of a sorted group16 batch: queries up to 8 G - 1 bases in groups of G lanes, then
// everything the groups cannot take.
void group16_tiles(TileTable& t) {
    const int w[] = {31, 63, 127, 255, 0x7FFFFFFF};
    t.n = 5;
    t.by_rows = 1;
    for (int k = 0; k < 5; ++k) {
        t.width[k] = w[k]; t.lanes[k] = k < 4 ? 1 : 32; t.tile[k] = k < 4 ? 2 : 9;
        t.warp_batch[k] = 0; t.refill[k] = 1;
    }
}

int launch_group16(const LaunchDesc& d, const ScoreParams& sp, int32_t* misfit, int32_t* misfits,
                   cudaStream_t stream) {
    const bool sym = sp.oe_del == sp.oe_ins;
    // Blocks per lane in a sorted batch: two halve what a row costs beyond its blocks (half the lanes a
    // job) and take longer over a row.  One against two: 19.8k jobs 376 and 411 us, 39.6k 690 and 634;
    // right extensions 20k 479 and 449, 40k 897 and 809; seed calls of 40k 1473 and 1360, 60k 2118 and
    // 1884, chains of 39k seeds 1324 and 1375.
    auto kern = !d.order_off ? (sym ? group16_kernel<0, true> : group16_kernel<0, false>)
                : d.n <= kOneBlockJobs ? (sym ? group16_kernel<1, true> : group16_kernel<1, false>)
                                       : (sym ? group16_kernel<2, true> : group16_kernel<2, false>);
    const int per_sm = resident_blocks(kern, 32 * kBlockWarps, 0);
    const int need = (d.n + kBlockWarps - 1) / kBlockWarps;
    const int full = sm_count() * (per_sm > 0 ? per_sm : 1);
    const int blocks = need < full ? need : full;
    if (blocks < 1) return G3X_OK;
    kern<<<blocks, 32 * kBlockWarps, 0, stream>>>(d, sp, misfit, misfits);
    return cudaPeekAtLastError() == cudaSuccess ? G3X_OK : G3X_ERR_CUDA;
}

}  // namespace g3x
