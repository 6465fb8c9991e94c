// g3x_band.cu -- group-per-job sm_100a kernel for batched ksw_extend2 on wide bands
// (bwa/src/ksw.cu:303-401), int32.
//
// A group of G = 8, 16 or 32 lanes runs one job through the reference's row loop, one target row
// per step, the warp's groups together, with the row buffer eh[] (ksw.cu:310) held in registers
// over a window of G R columns that slides with the band: at row i, window index d holds column
// i - w + d, and lane r of the group owns indices r R .. r R + R - 1.  The band of row i lies in columns [i - w, i + w + 1) (ksw.cu:338-340), so
// 2w + 1 columns hold it.  H(i, j) is what the cell (i+1, j+1) reads as its diagonal
// (eh[j+1].h), and that cell has the same index: H stays where it is.  E(i+1, j) (eh[j].e) and the
// query codes move one index down per row, one shuffle each.  No shared memory holds the row.
//
// Per row: M = H(i-1,j-1) + S and E need only the previous row, and F is the max-plus recurrence
// F(j+1) = max(F(j) - e_ins, max(M(j) - oe_ins, 0)), F(beg) = 0, an exact prefix maximum with linear
// decay.  Pass 1 forms, per column, L = F leaving it from 0 at its segment's start, the row's E
// entry, and Z = max(M, E, L of the column before); a scan over the lanes gives the F entering
// each lane; pass 2 is H = max(F entering - k e_ins, Z), one instruction a column, and the row's
// maximum and last column with H > 0.
//
// What the reference's band edges need of the buffer, besides the band's own cells:
//  * Left of beg every entry is zero: row 0's columns < 0 are, the trim (ksw.cu:388-389) passes only
//    zero entries, a zero entry left of beg stays zero (its M is at most 0, its E and F are 0), and
//    the columns the clamp cuts off leave the window.  So beg itself is not needed, except
//    for the cell count, and h1 = H(i, -1) matters only while it is positive: then column 0 holds
//    it, so the band starts at 0 until the clamp moves it (row w).
//  * An entry is non-zero only where H(i, j-1) > 0 or E(i+1, j) > 0, and E(i+1, j) > 0 implies
//    H(i, j) > 0.  So the last non-zero entry of ksw.cu:390 is the column after the last H > 0.
//  * Right of end the entries are zero or still row -1: row 0's band starts full (w + 1 columns), and
//    a later row's end passes only entries that the trim found zero.  Row -1 is non-zero beyond
//    column w + 1 only for seed scores above o_ins + w e_ins, and only while the window holds those
//    columns; those rows (tail_rows) restore the columns never reached from row -1's closed form
//    (ksw.cu:317-319), all others store zeros.
//
// Query and target codes come straight from the bit planes: each lane of a group loads eight of the
// codes that enter the window (or the rows) next, every 8 G rows.
//
// What bounds it: the integer ALU pipe, about 11 instructions per column and row beside 3
// multiply-adds, and about 100 per row of a warp, whatever its groups.  The form that kept eh[] at its
// own index, one warp per job and every edge in per-column selects took 34 a column: 20,000
// segments of 500-5,000 bases at w = 100 21.5 ms, now 8.2 (895 GCUPS); 1,500 at w = 500 6.4 ms.
#include <cuda_runtime.h>
#include "g3x_core.h"
#include "g3x_group.cuh"
#include "g3x_internal.h"
#include "g3x_stage.cuh"

namespace g3x {

namespace {

// prmt.b32 in its default mode, where a selector nibble with bit 3 set replicates the sign of
// the byte it selects (__byte_perm ignores that bit).
__device__ __forceinline__ uint32_t permute(uint32_t lo, uint32_t hi, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(lo), "r"(hi), "r"(sel));
    return r;
}
// Score of byte b of four score bytes, sign-extended.
template <int b>
__device__ __forceinline__ int32_t score_byte(uint32_t sc4) {
    return (int32_t)permute(sc4, 0u, (uint32_t)b | (8u | b) << 4 | (8u | b) << 8 | (8u | b) << 12);
}

// The job's band (2w' + 2 entries, w' the clamped width) fits the window, and its scores stay
// below 2^21 (the row maximum travels as score << 10 | window index in one 32-bit reduction):
// every H is at most h0 + qlen * max_score.
__device__ __forceinline__ bool band_fits(const JobConst& c, int32_t max_sc, int W) {
    return 2 * c.w + 2 <= W && (int64_t)c.qlen * max_sc + (c.h0 > 0 ? c.h0 : 0) < (1 << 21);
}

// F entering each lane of a group: exclusive prefix over the lanes of the F leaving each lane's R
// columns, dec = R e_ins.  A lane that a shuffle leaves alone meets its own value, decayed.
template <int G>
__device__ __forceinline__ int32_t f_into_lane(int32_t x, int r, int32_t dec) {
    const int32_t y = __shfl_up_sync(kAll, x, 1, G);
    int32_t f = r ? y : 0;
    if constexpr (G < 32) {
#pragma unroll
        for (int o = 1; o < G; o <<= 1) f = addmax_i32(__shfl_up_sync(kAll, f, o, G), -o * dec, f);
    } else {
#pragma unroll
        for (int o = 1; o < 16; o <<= 2) {
            const int32_t a = __shfl_up_sync(kAll, f, o), b = __shfl_up_sync(kAll, f, 2 * o);
            const int32_t c = __shfl_up_sync(kAll, f, 3 * o);
            f = addmax_i32(a, -o * dec, f);
            f = addmax_i32(b, -2 * o * dec, f);
            f = addmax_i32(c, -3 * o * dec, f);
        }
        f = addmax_i32(__shfl_up_sync(kAll, f, 16), -16 * dec, f);
    }
    return f;
}

// A group's job: its constants and where its sequences lie.
struct BandJob {
    int32_t job;                 // -1: none
    JobConst c;
    uint32_t q_off, t_off;
    bool qrev, trev;
};

// One job per group of G lanes over windows of G * R columns (2 w + 1 <= G R), the warp's groups row
// by row together.  kSym: oe_del == oe_ins (BWA's defaults), so E reuses F's max(M - oe, 0).
template <int G, int R, bool kSym>
__device__ __forceinline__ void run_band(const LaunchDesc& d, const ScoreParams& sp, const BandJob& J, const uint2* pools,
                                         int lane, unsigned long long& rows_run) {
    constexpr int W = G * R, kSegs = (R + 7) / 8;
    const int r = lane & (G - 1), gb = lane & ~(G - 1);
    const JobConst& c = J.c;
    // F and H stay below 2^21, so a larger extension decays them all the same
    const int32_t e_ins = sp.e_ins < (1 << 21) ? sp.e_ins : 1 << 21;
    const int32_t e_del = sp.e_del, oe_ins = sp.oe_ins, oe_del = sp.oe_del;
    const int32_t zdrop = sp.zdrop > 0 ? sp.zdrop : 0x7FFFFFFF;
    const uint32_t two = sp.k16 >> 15, k32 = sp.k16 >> 11;   // run-time 2 and 32: multiply-adds, beside the ALU pipe
    bool run = J.job >= 0;
    int32_t D[R], E[R];                  // eh[j].h and eh[j].e of the window's columns
    uint32_t q[kSegs];                   // their query codes, a nibble each
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const int32_t j = r * R + k - c.w;
        D[k] = run && j >= 0 && j <= c.qlen + 1 ? init_h(j, c) : 0;
        E[k] = 0;
    }
#pragma unroll
    for (int g = 0; g < kSegs; ++g)
        q[g] = run ? codes8(d.codes, d.nmask, J.q_off, c.qlen, J.qrev, r * R + 8 * g - c.w) : 0u;
    // lane r: the codes that enter the window at its right end in rows 8 (e0 + r) .., and the
    // target's of those rows
    uint32_t ext = 0u, tw = 0u, ext8 = 0u, t8 = 0u;
    int32_t end = c.qlen, hv = c.h0 - c.oe_del;
    // rows whose window may hold columns beyond w + 1 that no band has reached, with row -1's
    // scores in them (v1 - (j - 1) e_ins at column j)
    const int32_t v1 = c.h0 > c.oe_ins ? c.h0 - c.oe_ins : 0;
    const int32_t zero_from = v1 > 0 ? (v1 - 1) / sp.e_ins + 2 : 1;
    const int32_t tail = run && c.qlen > c.w + 1 && zero_from > c.w + 1 ? zero_from + c.w + 1 : 0;
    const int32_t tail_rows = (int32_t)__reduce_max_sync(kAll, (uint32_t)tail);
    int32_t max_end = 0, beg = 0;              // beg: kept for the cell count only
    int32_t best = c.h0, best_i = -1, best_d = 0, max_off = 0, gscore = -1, max_ie = -1;
    int64_t cells = 0;

    for (int32_t i = 0; __any_sync(kAll, run); ++i) {
        if ((i & 7) == 0) {
            const int e = i >> 3;
            if ((e & (G - 1)) == 0 && run) {
                ext = codes8(d.codes, d.nmask, J.q_off, c.qlen, J.qrev, W - c.w + 8 * (e + r));
                tw = codes8(d.codes, d.nmask, J.t_off, c.tlen, J.trev, 8 * (e + r));
            }
            ext8 = __shfl_sync(kAll, ext, gb | (e & (G - 1)));
            t8 = __shfl_sync(kAll, tw, gb | (e & (G - 1)));
        }
        const int sh = (i & 7) << 2;
        const uint2 pl = pools[(t8 >> sh) & 7u];
        const int32_t base = i - c.w;                    // column of window index 0
        end = min(min(end, i + c.w + 1), c.qlen);        // ksw.cu:338-340
        const int32_t j0 = base + r * R;                 // this lane's first column
        const int32_t hi = end - j0;                     // its cells: k < hi (left of beg all are zero)

        // ---- pass 1 ----
        int32_t Z[R], out[kSegs], e_first = 0;
#pragma unroll
        for (int g = 0; g < kSegs; ++g) {
            const uint32_t sc[2] = {permute(pl.x, pl.y, q[g]), permute(pl.x, pl.y, q[g] >> 16)};
            int32_t L = 0;                               // F entering the column, from 0 at the segment
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const int k = 8 * g + t;
                if (k < R) {
                    const int32_t s = (t & 3) == 0 ? score_byte<0>(sc[t >> 2]) : (t & 3) == 1 ? score_byte<1>(sc[t >> 2])
                                    : (t & 3) == 2 ? score_byte<2>(sc[t >> 2]) : score_byte<3>(sc[t >> 2]);
                    const int32_t M = addmin_i32(D[k], s, (int32_t)((uint32_t)D[k] * sp.k8));
                    const int32_t T = addmax_i32(M, -oe_ins, 0);
                    Z[k] = max3_i32(M, E[k], L);
                    L = addmax_i32(L, -e_ins, T);
                    const int32_t En = addmax_i32(E[k], -e_del, kSym ? T : addmax_i32(M, -oe_del, 0));
                    if (k == 0) e_first = En; else E[k - 1] = En;
                }
            }
            out[g] = L;
        }
        if (i < tail_rows) {                             // columns from end on may hold row -1's scores
#pragma unroll
            for (int k = 1; k < R; ++k) E[k - 1] = k < hi ? E[k - 1] : 0;
            e_first = hi > 0 ? e_first : 0;
        }
        // ---- F along the row, and the window's move: E and the codes one index down ----
        int32_t f = out[0];
#pragma unroll
        for (int g = 1; g < kSegs; ++g) f = addmax_i32(f, -(R - 8 * g < 8 ? R - 8 * g : 8) * e_ins, out[g]);
        f = f_into_lane<G>(f, r, R * e_ins);
        const int32_t e_in = __shfl_down_sync(kAll, e_first, 1, G);
        E[R - 1] = r < G - 1 ? e_in : 0;
        {
            uint32_t in = __shfl_down_sync(kAll, q[0], 1, G);
            in = r < G - 1 ? in : ext8 >> sh;
#pragma unroll
            for (int g = 0; g < kSegs; ++g) {
                if (g + 1 < kSegs) q[g] = __funnelshift_r(q[g], q[g + 1], 4);
                else if (R % 8 == 0) q[g] = __funnelshift_r(q[g], in, 4);
                else q[g] = (q[g] & ((1u << (4 * (R & 7))) - 1u)) >> 4 | (in & 0xFu) << (4 * ((R - 1) & 7));
            }
        }
        // ---- pass 2: H; row max as H * 32 + k (ties: larger k); the columns with H > 0 ----
        int32_t lkey = 0;
        uint32_t pos = 0u;
#pragma unroll
        for (int g = 0; g < kSegs; ++g) {
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const int k = 8 * g + t;
                if (k < R) {
                    // 1 for the columns left of end, 0 for the others: a multiply-add pipe operand
                    const int32_t in = __viaddmin_s32_relu(hi, -k, 1);
                    D[k] = addmax_i32(f, -t * e_ins, Z[k]) * in;
                    lkey = addmax_i32((int32_t)((uint32_t)D[k] * k32), k, lkey);
                    pos = pos * two + (uint32_t)min(D[k], 1);        // column k in bit R - 1 - k
                }
            }
            f = addmax_i32(f, -8 * e_ins, out[g]);       // F entering the next segment
        }
        const int32_t key = max_of_group<G>((lkey >> 5) << 10 | (r * R + (lkey & 31)));
        const int32_t last = max_of_group<G>(pos ? r * R + R + 1 - __ffs((int)pos) : 0);

        // ---- row end (ksw.cu:371-386) ----
        const int32_t m = key >> 10, dg = i - (base + (key & 1023));
        // H(i, -1), column 0's entry, while the band starts there (ksw.cu:342-345)
        const int32_t h1 = i <= c.w ? max(hv, 0) : 0;
        hv -= e_del;
        if (d.cells) {
            // the first non-zero entry: column 0 by h1, else the first column whose E entry is, else
            // the column after the first H > 0
            cells += run ? max(end - max(beg, base), 0) : 0;
            int32_t fk = 0x7FFFFFF;
#pragma unroll
            for (int k = R - 1; k >= 0; --k) {
                const int32_t e = k ? E[k - 1] : e_first;
                fk = D[k] > 0 ? j0 + k + (e > 0 ? 0 : 1) : fk;
            }
            const int32_t first = -max_of_group<G>(-fk);     // (every lane of the warp takes part)
            beg = h1 > 0 ? 0 : first;
        }
        if (__any_sync(kAll, run && end == c.qlen)) {
            // the to-end score H(i, qlen - 1), 0 left of beg; no later cell reads it as its diagonal
            const int32_t at = c.qlen - 1 - j0;
            int32_t v = 0;
#pragma unroll
            for (int k = 0; k < R; ++k) {
                v = at == k ? D[k] : v;
                D[k] = at == k ? 0 : D[k];
            }
            v = max_of_group<G>(v);
            if (c.qlen == 0) v = h1;
            if (end == c.qlen) {
                max_ie = v >= gscore ? i : max_ie;
                gscore = max(gscore, v);
            }
        }
        const bool up = m > max(best, 0);                // (a negative seed score ends at its first row)
        const int32_t t = dg - best_d;                   // z-drop (never for a new maximum)
        const bool zstop = best - m - (t > 0 ? t * e_del : -t * sp.e_ins) > zdrop;
        max_off = max(max_off, up ? abs(dg) : 0);
        best = up ? m : best;
        best_i = up ? i : best_i;
        best_d = up ? dg : best_d;
        if (run && (m == 0 || zstop || i + 1 >= c.tlen)) {
            if (r == 0) {
                d.out[J.job] = g3x_ext_t{best, best_i - best_d + 1, best_i + 1, max_ie + 1, gscore, max_off};
                d.status[J.job] = G3X_OK;
                if (d.cells) d.cells[J.job] = (int32_t)cells;
                if (d.rows) d.rows[J.job] = i + 1;
                rows_run += i + 1;
            }
            run = false;
        }
        // ---- the next row's buffer and band ----
        if (__any_sync(kAll, h1 > 0 && i < c.w)) {       // column -1 of this row is the diagonal of column 0
            const int32_t at = h1 > 0 ? -1 - j0 : -1;
#pragma unroll
            for (int k = 0; k < R; ++k) D[k] = at == k ? h1 : D[k];
        }
        if (i < tail_rows) {                             // columns never reached: row -1
            max_end = max(max_end, end);
            const int32_t v = v1 - j0 * e_ins;           // of column j0 + 1
#pragma unroll
            for (int k = 0; k < R; ++k)
                if (k >= hi && j0 + k + 1 > max_end) D[k] = addmax_i32(v, -k * e_ins, 0);
        }
        end = base + last + 2;                           // ksw.cu:390-391: two past the last non-zero entry
    }
}

// d.tile columns W, groups of G lanes (launch_band).
template <int W, int G, bool kSym>
__global__ void __launch_bounds__(64) band_kernel(LaunchDesc d, ScoreParams sp) {
    pdl_trigger();
    static_assert(W <= 1024, "window index must fit 10 bits");
    constexpr int kGroups = 32 / G;
    __shared__ uint2 pools[8];
    if (threadIdx.x < 8) {
        uint32_t lo[5], hi[5];
        score_pools(sp, lo, hi);
        const int a = threadIdx.x < 4 ? threadIdx.x : 4;
#pragma unroll
        for (int t = 0; t < 5; ++t)
            if (a == t) pools[threadIdx.x] = make_uint2(lo[t], hi[t]);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, r = lane & (G - 1), gb = lane & ~(G - 1);
    unsigned leaders = 0;
#pragma unroll
    for (int k = 0; k < kGroups; ++k) leaders |= 1u << (k * G);
    const int n = d.count ? *d.count : d.n;
    const int* order = d.order ? d.order + (d.order_off ? *d.order_off : 0) : nullptr;
    unsigned long long rows_run = 0, jobs_run = 0;
    int static_slot = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kGroups;
    const int static_stride = gridDim.x * (blockDim.x >> 5) * kGroups;

    for (bool more = true; more;) {
        // ---- a job for every group ----
        BandJob J;
        J.job = -1;
        J.c = JobConst{};
        J.q_off = J.t_off = 0;
        J.qrev = J.trev = false;
        for (;;) {
            const unsigned want = __ballot_sync(kAll, J.job < 0) & leaders;
            if (!want || !more) break;
            int first = 0;
            if (d.persistent) {
                if (lane == 0) first = atomicAdd(d.queue, __popc(want));
                first = __shfl_sync(kAll, first, 0);
            } else {                                     // __popc(want) == kGroups: nothing is taken twice
                first = static_slot;
                static_slot += static_stride;
            }
            more = first + (d.persistent ? __popc(want) : static_stride) < n;
            const int slot = first + __popc(want & ((1u << gb) - 1u));
            if (J.job < 0 && slot < n) {
                const int job = order ? order[slot] : slot;
                const g3x_job_t jb = d.jobs[job];
                JobConst c;
                c.qlen = jb.qlen; c.tlen = jb.tlen; c.h0 = jb.h0;
                c.o_del = sp.o_del; c.e_del = sp.e_del; c.o_ins = sp.o_ins; c.e_ins = sp.e_ins;
                c.oe_del = sp.oe_del; c.oe_ins = sp.oe_ins; c.zdrop = sp.zdrop;
                c.w = clamp_w(jb.w, c.qlen, sp.max_sc, sp.end_bonus, sp.o_del, sp.e_del, sp.o_ins, sp.e_ins);
                // the checks of stage_job (M = min(H + S, 256 H) needs h0 >= 0 or h0 <= -max_score),
                // and a band that fits the window
                const bool bad = (jb.h0 < 0 && jb.h0 > -sp.max_sc) || !job_in_planes(jb, d.n_bases);
                const bool too_long = c.qlen > d.qmax || c.tlen > d.tmax || c.qlen > 65534 || !band_fits(c, sp.max_sc, W);
                if (d.split && band_window(c.w, c.qlen, c.h0, sp.max_sc) != W) {
                    // another kernel's
                } else if (bad || too_long || c.tlen == 0 || c.w < 0) {
                    if (r == 0) finish_unrun(d, job, c, bad ? G3X_ERR_INVALID : too_long ? G3X_ERR_TOO_LONG : G3X_OK);
                } else {
                    J.job = job;
                    J.c = c;
                    J.q_off = jb.q_off; J.t_off = jb.t_off;
                    J.qrev = (jb.flags & G3X_JOB_QREV) != 0;
                    J.trev = (jb.flags & G3X_JOB_TREV) != 0;
                }
            }
            if (!d.persistent) break;
        }
        const unsigned have = __ballot_sync(kAll, J.job >= 0) & leaders;
        if (!have) continue;
        jobs_run += __popc(have);
        // the narrowest registers that hold the warp's bands: a row costs about 11 instructions a column.
        // 224 is there for w = 100, BWA's default: 20k segments 8.2 ms, in 256 columns 8.9.  (192 beside it
        // measured 7.3 against 8.1 for 20k at w = 90 and 4.0 against 4.4 for 3,000, where 256 takes 3.9.)
        const int cols = 2 * __reduce_max_sync(kAll, J.c.w) + 1;
#define G3X_BAND(R) run_band<G, (R), kSym>(d, sp, J, pools, lane, rows_run)
        if constexpr (W == 256) {
            if (cols <= 64) G3X_BAND(64 / G);
            else if (cols <= 128) G3X_BAND(128 / G);
            else if (cols <= 224) G3X_BAND(224 / G);
            else G3X_BAND(256 / G);
        } else {
            if (cols <= W / 4 * 3) G3X_BAND(W / 4 * 3 / G);
            else G3X_BAND(W / G);
        }
#undef G3X_BAND
    }
    if (d.stats) {
        if (r == 0 && rows_run) atomicAdd(d.stats + 0, rows_run);
        if (lane == 0 && jobs_run) atomicAdd(d.stats + 2, jobs_run);
    }
    pdl_chain_end();
}

}  // namespace

template <int W, int G, bool kSym>
static int launch_band_t(const LaunchDesc& d, const ScoreParams& sp, cudaStream_t stream) {
    auto kern = band_kernel<W, G, kSym>;
    constexpr int kWarps = 2, kJobs = 32 / G * kWarps;     // per block
    const int per_sm = resident_blocks(kern, 32 * kWarps, 0);
    int blocks = d.blocks > 0 ? d.blocks : sm_count() * (per_sm > 0 ? per_sm : 1);
    const int need = (d.n + kJobs - 1) / kJobs;
    blocks = need < blocks ? need : blocks;
    if (blocks == 0) return G3X_OK;
    return launch_class_kernel(kern, blocks, 32 * kWarps, 0, stream, d, sp) == cudaSuccess ? G3X_OK : G3X_ERR_CUDA;
}

template <int W, int G>
static int launch_band_w(const LaunchDesc& d, const ScoreParams& sp, cudaStream_t stream) {
    return sp.oe_del == sp.oe_ins ? launch_band_t<W, G, true>(d, sp, stream) : launch_band_t<W, G, false>(d, sp, stream);
}

// d.tile is the window W (256, 512 or 1024 columns): jobs whose band 2w' + 2 exceeds it get
// G3X_ERR_TOO_LONG.
//
// Lanes per job: a row's work beyond its columns (the scan, the reductions, the bookkeeping: about
// 100 instructions) is done once per warp, so narrow groups share it, but a batch needs enough
// jobs to fill the schedulers with them, and a warp's jobs end together.  Long segments of 500-5,000
// bases, 32, 16 and 8 lanes: w = 100, 20k jobs 11.8, 10.5 and 9.1 ms, 10k 6.3, 5.9 and 6.7, 5k 4.7, 5.5
// and 6.8; w = 240, 6k 7.0 and 7.0, w = 170, 3k 4.8 and 6.5 (16 lanes hold 512 columns, 8 hold 256).
// d.n counts the whole batch: a table's classes run side by side.
constexpr int kBandNarrow = 16000, kBandHalf = 8000;
int launch_band(const LaunchDesc& d, const ScoreParams& sp, cudaStream_t stream) {
    const bool narrow = d.n >= kBandNarrow, half = d.n >= kBandHalf;
    switch (d.tile) {
        case 256: return narrow ? launch_band_w<256, 8>(d, sp, stream) : half ? launch_band_w<256, 16>(d, sp, stream)
                                                                     : launch_band_w<256, 32>(d, sp, stream);
        case 512: return half ? launch_band_w<512, 16>(d, sp, stream) : launch_band_w<512, 32>(d, sp, stream);
        case 1024: return launch_band_w<1024, 32>(d, sp, stream);
        default: return G3X_ERR_INVALID;
    }
}

}  // namespace g3x
