// g3x_sw.cu -- batched striped local Smith-Waterman with 16-bit cells, as ksw_align2 computes
// it (bwa/src/ksw.cu:271-292 over the profile of ksw_qinit, :18-64, and the pass of ksw_i16,
// :155-262; the reference stops ksw_align2 at its first statement, :276, and this is the
// function as written after it).
//
// Four lanes per job (a quad), eight jobs per warp.  ksw_i16 works on vectors of eight 16-bit
// cells; here a vector is the quad's four int16x2 words (lane p holds cells 2p and 2p+1), so
// each vector step of the reference is one DPX/SIMD instruction per lane:
//   adds, then max with E and F      -> __viaddmax_s16x2(H, S, max(E, F))
//   max of non-negative cells        -> __vimax_s16x2_relu
//   "subtract, 0 if not positive"    -> __viaddmax_s16x2_relu with the negated penalty
//   "any cell of F beats H - oe"      -> max(F, H - oe) != H - oe
//   the one-cell shift                -> one quad shuffle and a byte permute
// (only DPX forms: the SIMD-video intrinsics are instruction sequences on this architecture).
// The query profile is not stored: segment j's word of lane p is the score of the row's target
// base against query positions j + 2p*slen and j + (2p+1)*slen, one sign-extending byte
// permute (prmt) of the score row by a selector built once per job.  The job's H and E rows
// live in registers: segment j sits in slot MAXSEG - slen + j, so the last segment, which the
// next row shifts in, is always the last slot.
//
// Exactness: the reference's int16 arithmetic wraps; every cell here stays in [0, 32639]
// (H <= max(mat) * qlen <= 127 * 256, plus one score) for queries up to 256 bases, so the
// wrapping and non-wrapping forms agree, and "subtract, 0 if not positive" of a non-negative
// cell never wraps.  Longer queries get G3X_ERR_TOO_LONG.
//
// Jobs are sorted by segment count and rows (a device counting sort), so a warp's eight jobs have
// the same segments and about the same rows; each of three launches (registers for 8, 16, 32
// segments) takes its classes of four segment counts from device counters.  The second pass for the start positions (KSW_XSTART) has
// its own sort and launches.
#include <cuda_runtime.h>
#include <stdint.h>
#include <algorithm>
#include <type_traits>
#include "g3x_core.h"
#include "g3x_internal.h"
#include "g3x_stage.cuh"

namespace g3x {
namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr int kQuads = 8;                 // jobs per warp
constexpr int kWarps = 4;                 // warps per block
constexpr int kRowBins = 128;             // rows, eight bins per doubling
constexpr int kSegBins = 32;              // segments 1..32
constexpr int kClasses = kSegBins / 4;    // 29-32 segments first
constexpr int kBins = kSegBins * kRowBins + 1;   // + the bin of rejected jobs (qlen 0 or > 256)
constexpr int kNoScore = 0x10000;         // minsc / endsc when the flag is absent (ksw.cu:176-177)

struct SwDesc {
    const g3x_job_t* jobs;
    const uint32_t* codes;
    const uint32_t* nmask;
    const int32_t* order;      // job indices, sorted
    const int32_t* range;      // [offset, count] in `order` of each class of four segment counts
    int32_t* queue;            // the classes' slot counters (zeroed)
    g3x_swr_t* out;
    int32_t* status;
    uint32_t* sub;             // XSUBO: row maxima per job (imax << 16 | row), sub_stride each
    int32_t sub_stride;
    int32_t xtra, maxmat;
    uint32_t tab[10];          // per target base: score bytes (lo: codes 0-3, hi: N, then 0)
    uint32_t nedel, noedel, neins, noeins;   // -e_del, -(o_del+e_del), ... as int16x2
    // the carried F (sw_rows): its decay of segment 0 and the step to the next segment's, e_ins to
    // add, and 1 (a run-time value keeps the step a multiply-add, beside the saturated ALU pipe);
    // one == 0: the WIDE form, with nstep the saturating step.  carry_e: the decay per segment.
    uint32_t dec0, step, peins, one, nstep;
    int32_t carry_e;
    int64_t n_bases;           // bases the planes hold: jobs reaching past them are refused
};

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// The vector moved up one cell (cell 0 gets 0), ksw.cu:86-97.
__device__ __forceinline__ uint32_t shift_up(uint32_t w, int p) {
    const uint32_t up = __shfl_up_sync(kFull, w, 1, 4);
    return __byte_perm(p ? up : 0u, w, 0x5432);
}

// Selector nibbles for one word: cell codes c0, c1 (5 = past the query, score 0); the high byte
// of each half replicates the sign of its low byte.
__device__ __forceinline__ uint32_t sel_of(uint32_t c0, uint32_t c1) {
    return c0 | (c0 | 8u) << 4 | c1 << 8 | (c1 | 8u) << 12;
}

__device__ __forceinline__ int quad_max(int v) {
    v = max(v, __shfl_xor_sync(kFull, v, 1));
    return max(v, __shfl_xor_sync(kFull, v, 2));
}
__device__ __forceinline__ int quad_min(int v) {
    v = min(v, __shfl_xor_sync(kFull, v, 1));
    return min(v, __shfl_xor_sync(kFull, v, 2));
}

// The quad's query codes, one byte per position: 0-3, 4 for N, 5 from len up to the 8 slen cells of its
// vectors.  A lane takes every fourth 16-base chunk, so the quad waits for one or two memory
// latencies (base by base they were a quarter of a 90-base job's time).
__device__ __forceinline__ void stage_query(const SwDesc& d, uint32_t off, int len, bool rev, int cells, int p,
                                            uint8_t* qc) {
    for (int b = 16 * p; b < cells; b += 64) {
        uint64_t v = 0;
        if (b < len) {
            uint32_t x, nb;
            load16(d.codes, d.nmask, off, len, b >> 4, rev, x, nb);
            v = nibbles16(x, nb);
        }
        uint32_t w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t h = (uint32_t)(v >> (16 * u)) & 0xFFFFu, t = (h & 0xFFu) | (h & 0xFF00u) << 8;
            const uint32_t c = (t | t << 4) & 0x0F0F0F0Fu, n = c >> 2 & 0x01010101u;
            const int valid = len - (b + 4 * u);
            const uint32_t past = valid >= 4 ? 0u : valid <= 0 ? kFull : kFull << (8 * valid);
            w[u] = (c & ~(n | n << 1) & ~past) | (0x05050505u & past);
        }
        *reinterpret_cast<uint4*>(qc + b) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// Target rows of a pass: row i is base i of the job's target, or, in the second pass, base
// te - i for i <= te (the prefix 0..te reversed, ksw.cu:287).  Lane p of the quad holds rows 64 c + 16 p
// .. + 15 as nibbles (4-7 for N).
struct Rows {
    uint32_t off, roff;
    int len, rlen, flip;       // flip: rows 0..flip-1 come from the reversed prefix
    bool rev, rrev;
    uint32_t w0, w1;
    __device__ __forceinline__ void refill(const uint32_t* codes, const uint32_t* nmask, int i, int p) {
        const int b = i + 16 * p;
        uint64_t v = 0;
        uint32_t x, nb;
        if (b < flip) {
            load16(codes, nmask, roff, rlen, b >> 4, rrev, x, nb);
            v = nibbles16(x, nb);
        }
        if (b + 16 > flip && b < len) {
            load16(codes, nmask, off, len, b >> 4, rev, x, nb);
            const uint64_t keep = b < flip ? ((uint64_t)1 << (4 * (flip - b))) - 1u : 0u;
            v = (v & keep) | (nibbles16(x, nb) & ~keep);
        }
        w0 = (uint32_t)v;
        w1 = (uint32_t)(v >> 32);
    }
    __device__ __forceinline__ uint32_t code(int i, int lane) const {
        const uint32_t w = __shfl_sync(kFull, (i & 8) ? w1 : w0, (lane & ~3) | (i >> 4 & 3));
        return w >> ((i & 7) << 2) & 7u;
    }
};

// Selectors of the segments' scores: one per register up to 16 segments, two beyond (registers
// bound the resident warps there).
__host__ __device__ constexpr int sel_words(int maxseg) { return maxseg > 16 ? maxseg / 2 : maxseg; }
template <int MAXSEG, int S>
__device__ __forceinline__ uint32_t sel_at(const uint32_t (&sel)[sel_words(MAXSEG)]) {
    if constexpr (MAXSEG <= 16) return sel[S];
    else return (S & 1) ? sel[S >> 1] >> 16 : sel[S >> 1];
}

// The int16x2 word of -v in both halves, at most 2^15 - 1.
__device__ __forceinline__ uint32_t neg_pair(int64_t v) {
    const uint32_t n = (uint32_t)-(int32_t)(v < 0x7FFF ? v : 0x7FFF) & 0xFFFFu;
    return n | n << 16;
}

struct PassOut {
    int score, te, qe;
};

// Constants of a pass: the score steps of SwDesc as int16x2 and what a job's segment count makes of
// the insertion extension.
struct PassConst {
    uint32_t last;             // decay of the carried F up to the last segment
    uint32_t d1, d2, d4;       // decay of F over 1, 2 and 4 cells of the vector (slen segments each)
};

// The segments of a row, slots S .. MAXSEG - 1 (S0: the row's first).
template <int MAXSEG, int S0, bool SYM, bool WIDE, int S = S0>
__device__ __forceinline__ void seg_steps(const SwDesc& d, const uint2 pool, const uint32_t (&sel)[sel_words(MAXSEG)],
                                          int base, uint32_t (&H)[MAXSEG], uint32_t (&E)[MAXSEG], uint32_t& hd,
                                          uint32_t& f, uint32_t& mx, uint32_t& dec, uint32_t& fc) {
    if constexpr (S < MAXSEG) {
        const bool mine = S >= S0 + 3 || S >= base;      // (known for all but three slots)
        const uint32_t sc = prmt(pool.x, pool.y, sel_at<MAXSEG, S>(sel));
        uint32_t h = __viaddmax_s16x2(hd, sc, __vimax_s16x2_relu(E[S], f));
        uint32_t raised, fc2 = fc, dec2 = dec;
        if constexpr (WIDE) {
            raised = __vimax_s16x2_relu(H[S], fc);
            fc2 = __viaddmax_s16x2_relu(fc, d.nstep, 0u);
        } else {
            raised = __viaddmax_s16x2(fc, dec, H[S]);
            dec2 = dec * d.one + d.step;
        }
        if constexpr (S < S0 + 3) {
            h = mine ? h : 0u;
            raised = mine ? raised : hd;
            fc2 = mine ? fc2 : fc;
            dec2 = mine ? dec2 : dec;
        }
        hd = raised; fc = fc2; dec = dec2;
        // two segments at a time
        if constexpr (S & 1) mx = __vimax3_s16x2(mx, H[S - 1], h);
        H[S] = h;
        const uint32_t td = __viaddmax_s16x2_relu(h, d.noedel, 0u);
        E[S] = __viaddmax_s16x2(E[S], d.nedel, td);
        f = __viaddmax_s16x2(f, d.neins, SYM ? td : __viaddmax_s16x2_relu(h, d.noeins, 0u));
        seg_steps<MAXSEG, S0, SYM, WIDE, S + 1>(d, pool, sel, base, H, E, hd, f, mx, dec, fc);
    }
}

// The row loop of one pass over registers H, E (slot MAXSEG - slen + j = segment j), over the last V
// slots: every live quad of the warp has V - 3 .. V segments, so only the first three slots ask
// whether they are the quad's (a slot before its first segment holds zeros: score 0, no H, E or F),
// and the others are straight code.  (One jump per row to a first slot common to the warp, and a guard
// in every slot where there was none, took 390 instructions a row of 12 segments.)  A quad that is
// not running computes on slots it never reads back.  SYM: equal insertion and deletion costs, so
// E and F share H - (o + e).  WIDE: see below.
//
// The lazy-F loop (ksw.cu:209-220) in closed form.  It moves F up one cell, folds it into H segment
// by segment as it decays, E untouched, round after round, until no cell's F - e beats its
// H - (o + e).  With o > 0 it can only stop where every F it still holds is dominated by the F
// that the row's own pass had computed from there on (F > H - o - e fails for a cell that F itself
// has just raised), so stopping early changes nothing and the loop's result is
//   H(j) = max(H(j), C - j e),   C(cell) = max over the cells before it of their F at the end of
//                                the pass, less slen e per cell in between.
// C is a prefix over the vector's eight cells, three shuffles a row, and the row maximum and the
// best row's position never come from a raised cell (it stays below the H it descends from).  So
// H is stored as the pass leaves it, and the next row raises each segment as it reads it (one
// addition and maximum) -- no loop, no ballot.  The decay -(j + 1) e of segment j (C is kept as
// C + e) is one 32-bit addition a segment on both halves, exact while it fits 16 bits.  WIDE: gap
// extensions above 1000 decay C by a saturating step instead; so does o = 0, where the loop stops
// after the first segment of the first round and raises nothing else.
template <int MAXSEG, int V, bool SYM, bool WIDE>
__device__ __forceinline__ void sw_rows(const SwDesc& d, bool live, int tlen, Rows& rows, int minsc, int endsc,
                                        uint32_t* sub, int& n_b, uint32_t (&H)[MAXSEG], uint32_t (&E)[MAXSEG],
                                        const uint32_t (&sel)[sel_words(MAXSEG)], const PassConst& pc, int base,
                                        uint32_t* hm, const uint2* tab, int lane, int& gmax, int& te) {
    constexpr int S0 = MAXSEG - V;
    const int p = lane & 3;
    int last_row = -2, last_v = 0;
    bool run = live;
    uint32_t fc = 0u;             // the carried F of the row before (WIDE: C, else C + e_ins)
    for (int i = 0;; ++i) {
        run = run && i < tlen;
        if (!__any_sync(kFull, run)) break;
        if ((i & 63) == 0 && run) rows.refill(d.codes, d.nmask, i, p);
        uint2 pool = tab[rows.code(i, lane)];
        if (!run) pool = make_uint2(0u, 0u);
        uint32_t hd = shift_up(__viaddmax_s16x2(fc, pc.last, H[MAXSEG - 1]), p);
        uint32_t f = 0u, mx = 0u, dec = d.dec0;
        // the row (ksw.cu:193-208): M = H(i-1, j-1) + S, H = max(M, E, F), E' and F' from H
        seg_steps<MAXSEG, S0, SYM, WIDE>(d, pool, sel, base, H, E, hd, f, mx, dec, fc);
        // the F carried into each cell (a lane a shuffle leaves alone meets its own, decayed)
        f = shift_up(f, p);
        f = __viaddmax_s16x2(shift_up(f, p), pc.d1, f);
        f = __viaddmax_s16x2(__shfl_up_sync(kFull, f, 1, 4), pc.d2, f);
        f = __viaddmax_s16x2(__shfl_up_sync(kFull, f, 2, 4), pc.d4, f);
        fc = WIDE ? f : __viaddmax_s16x2(f, d.peins, 0u);
        uint32_t m2 = __vimax_s16x2_relu(mx, __shfl_xor_sync(kFull, mx, 1));
        m2 = __vimax_s16x2_relu(m2, __shfl_xor_sync(kFull, m2, 2));
        const int im = max((int)(int16_t)(m2 & 0xFFFFu), (int)(int16_t)(m2 >> 16));
        if (run) {
            if (sub && im >= minsc && p == 0) {     // ksw.cu:223-232
                if (n_b == 0 || last_row + 1 != i) {
                    sub[n_b++] = (uint32_t)im << 16 | (uint32_t)i;
                    last_row = i; last_v = im;
                } else if (last_v < im) {
                    sub[n_b - 1] = (uint32_t)im << 16 | (uint32_t)i;
                    last_row = i; last_v = im;
                }
            }
            if (im > gmax) {                        // ksw.cu:233-238
                gmax = im; te = i;
#pragma unroll
                for (int S = S0; S < MAXSEG; ++S) hm[S * 32 + lane] = H[S];
                if (gmax >= endsc) run = false;
            }
        }
    }
}

// One pass of ksw_i16 (ksw.cu:155-262) for the quad's job (live), query codes qc (stage_query).  With `sub`, row maxima >= minsc go to the job's list (ksw.cu:223-232; lane p = 0
// keeps it) and *nb receives its length.
template <int MAXSEG, int V>
__device__ __forceinline__ PassOut sw_pass(const SwDesc& d, bool live, int qlen, int tlen, const uint8_t* qc, Rows rows,
                                           int minsc, int endsc, uint32_t* sub, int* nb, uint32_t* hm,
                                           const uint2* tab, int lane) {
    const int p = lane & 3;
    const int slen = live ? (qlen + 7) >> 3 : 0;
    const int base = MAXSEG - slen;
    uint32_t H[MAXSEG], E[MAXSEG], sel[sel_words(MAXSEG)];
#pragma unroll
    for (int s = 0; s < MAXSEG; s += 2) {
        uint32_t v = 0;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int j = s + u - base;
            uint32_t c0 = 5u, c1 = 5u;
            if (live && j >= 0) {
                const int p0 = j + 2 * p * slen, p1 = p0 + slen;
                c0 = qc[p0];
                c1 = qc[p1];
            }
            v |= sel_of(c0, c1) << (16 * u);
        }
        if constexpr (MAXSEG <= 16) {
            sel[s] = v & 0xFFFFu;
            sel[s + 1] = v >> 16;
        } else {
            sel[s >> 1] = v;
        }
        H[s] = H[s + 1] = 0u;
        E[s] = E[s + 1] = 0u;
    }
    int gmax = 0, te = -1, n_b = 0;
    const int64_t seg = (int64_t)slen * d.carry_e;
    const bool wide = d.one == 0u;
    const PassConst pc{neg_pair(wide ? seg - d.carry_e : seg), neg_pair(seg), neg_pair(2 * seg), neg_pair(4 * seg)};
#define G3X_SW_ROWS(SYM, WIDE)                                                                                    \
    sw_rows<MAXSEG, V, SYM, WIDE>(d, live, tlen, rows, minsc, endsc, sub, n_b, H, E, sel, pc, base, hm, tab, lane, gmax, te)
    // SYM: equal insertion and deletion costs, so E and F share H - (o + e)
    if (wide) G3X_SW_ROWS(false, true);
    else if (d.noedel == d.noeins) G3X_SW_ROWS(true, false);
    else G3X_SW_ROWS(false, false);
#undef G3X_SW_ROWS
    __syncwarp();
    // end on the query: the smallest position holding the best row's largest cell, cells read
    // as uint16 (ksw.cu:244-248); with no best row the cells are all 0 and it is position 0
    const bool has = live && te >= 0;      // quad-uniform; every lane takes part in the shuffles
    int best = 0;
#pragma unroll
    for (int s = 0; s < MAXSEG; ++s)
        if (has && s >= base) {
            const uint32_t v = hm[s * 32 + lane];
            best = max(best, (int)max(v & 0xFFFFu, v >> 16));
        }
    best = quad_max(best);
    int pos = 0x7FFFFFFF;
#pragma unroll
    for (int s = 0; s < MAXSEG; ++s)
        if (has && s >= base) {
            const uint32_t v = hm[s * 32 + lane];
            const int j = s - base;
            if ((int)(v & 0xFFFFu) == best) pos = min(pos, j + 2 * p * slen);
            if ((int)(v >> 16) == best) pos = min(pos, j + (2 * p + 1) * slen);
        }
    pos = quad_min(pos);
    const int qe = has ? pos : 0;
    if (nb) *nb = n_b;
    return PassOut{gmax, te, qe};
}

// SECOND false: the first pass of every job.  SECOND: the start positions (ksw.cu:286-291) of the jobs
// that want them, sorted anew by the segments and rows of their second pass: the query prefix
// 0..qe and the target with its prefix 0..te reversed, stopping at the first score.  (Run by the warp
// that ran the first pass, the second passes of eight jobs of one segment count have eight
// segment counts, and each of a segment's steps ran once for every few of them: 15.8 of 32 lanes active,
// and both passes of 200k windows took 4.91 ms; 2.15 with this launch and the finer bins of rows.)
template <int MAXSEG, bool SECOND>
__global__ void __launch_bounds__(128, MAXSEG == 32 ? 4 : MAXSEG == 16 ? 6 : 8) sw_kernel(SwDesc d) {
    constexpr int QMAX = 8 * MAXSEG;
    __shared__ __align__(16) uint8_t qcodes[kWarps][kQuads][QMAX];
    __shared__ uint32_t snap[kWarps][MAXSEG * 32];
    __shared__ uint2 tab[8];
    pdl_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, quad = lane >> 2, p = lane & 3;
    if (threadIdx.x < 8) {
        const int a = threadIdx.x < 4 ? threadIdx.x : 4;
        tab[threadIdx.x] = make_uint2(d.tab[2 * a], d.tab[2 * a + 1]);
    }
    __syncthreads();
    uint8_t* qc = qcodes[warp][quad];
    uint32_t* hm = snap[warp];
    const bool subo = (d.xtra & G3X_KSW_XSUBO) != 0;
    const int minsc = subo ? d.xtra & 0xFFFF : kNoScore;
    const int endsc = (d.xtra & G3X_KSW_XSTOP) ? d.xtra & 0xFFFF : kNoScore;
    // the jobs of V - 3 .. V segments, class k of the sort
    auto run_class = [&](auto v, int k) {
    constexpr int V = decltype(v)::value;
    const int off = d.range[2 * k], cnt = d.range[2 * k + 1];
    for (;;) {
        int first = 0;
        if (lane == 0) first = atomicAdd(d.queue + k, kQuads);
        first = __shfl_sync(kFull, first, 0);
        if (first >= cnt) break;
        const int slot = first + quad;
        const int job = slot < cnt ? d.order[off + slot] : -1;
        int qlen = 0, tlen = 0;
        bool live = false;
        g3x_job_t jb;
        if (job >= 0) {
            jb = d.jobs[job];
            qlen = jb.qlen; tlen = jb.tlen;
            int st = G3X_OK;
            if (qlen < 1) st = G3X_ERR_INVALID;     // the reference reads before its buffers
            else if (!job_in_planes(jb, d.n_bases)) st = G3X_ERR_INVALID;   // past the planes: unread
            else if (qlen > 8 * kSegBins || (subo && tlen > d.sub_stride)) st = G3X_ERR_TOO_LONG;
            if (st != G3X_OK) {                     // (first pass only: the second takes none of them)
                if (p == 0) {
                    d.out[job] = g3x_swr_t{0, -1, -1, -1, -1, -1, -1};
                    d.status[job] = st;
                }
            } else {
                live = true;
            }
        }
        const bool trev = live && (jb.flags & G3X_JOB_TREV) != 0, qrev = live && (jb.flags & G3X_JOB_QREV) != 0;
        Rows rows;
        rows.off = live ? jb.t_off : 0u; rows.len = tlen; rows.rev = trev;
        rows.roff = 0u; rows.rlen = 0; rows.rrev = false; rows.flip = 0;
        rows.w0 = rows.w1 = 0u;
        if constexpr (!SECOND) {
            if (live) stage_query(d, jb.q_off, qlen, qrev, (qlen + 7) & ~7, p, qc);
            __syncwarp();
            uint32_t* sub = subo && live ? d.sub + (int64_t)job * d.sub_stride : nullptr;
            int n_b = 0;
            const PassOut r = sw_pass<MAXSEG, V>(d, live, qlen, tlen, qc, rows,
                                              minsc, endsc, sub, &n_b, hm, tab, lane);
            g3x_swr_t o{r.score, r.te, r.qe, -1, -1, -1, -1};
            // second best: list entries more than ceil(score / max(mat)) rows from te (ksw.cu:249-256)
            if (live && p == 0 && n_b > 0) {
                const int c = (r.score + d.maxmat - 1) / d.maxmat, low = r.te - c, high = r.te + c;
                for (int k = 0; k < n_b; ++k) {
                    const uint32_t v = sub[k];
                    const int e = (int)(v & 0xFFFFu), sc = (int)(v >> 16);
                    if ((e < low || e > high) && sc > o.score2) { o.score2 = sc; o.te2 = e; }
                }
            }
            if (live && p == 0) {
                d.out[job] = o;
                d.status[job] = G3X_OK;
            }
        } else {
            int score = 0, te = -1, qe = 0;
            if (live) { score = d.out[job].score; te = d.out[job].te; qe = d.out[job].qe; }
            const int lq = live ? qe + 1 : 0, lt = te + 1;
            // the query's prefix 0..qe backwards
            if (live) stage_query(d, qrev ? jb.q_off + (uint32_t)(qlen - lq) : jb.q_off, lq, !qrev, (lq + 7) & ~7, p, qc);
            __syncwarp();
            rows.flip = lt;
            rows.rlen = lt;
            if (!trev) { rows.roff = rows.off; rows.rrev = true; }
            else { rows.roff = rows.off + (uint32_t)(tlen - lt); rows.rrev = false; }
            const PassOut rr = sw_pass<MAXSEG, V>(d, live, lq, tlen, qc, rows,
                                               kNoScore, score, nullptr, nullptr, hm, tab, lane);
            if (live && p == 0 && rr.score == score) {      // kept when it finds the same score
                d.out[job].tb = te - rr.te;
                d.out[job].qb = qe - rr.qe;
            }
        }
        __syncwarp();
    }
    };
#define G3X_SW_CLASS(V) run_class(std::integral_constant<int, (V)>(), (kSegBins - (V)) / 4)
    if constexpr (MAXSEG == 32) {
        G3X_SW_CLASS(32);
        G3X_SW_CLASS(28);
        G3X_SW_CLASS(24);
        G3X_SW_CLASS(20);
    } else {
        G3X_SW_CLASS(MAXSEG);
        G3X_SW_CLASS(MAXSEG - 4);
    }
#undef G3X_SW_CLASS
    pdl_chain_end();
}

// Sort bins: segment count descending, then rows descending; the last bin holds the jobs the first
// pass rejects, or (res set: the second pass) those without one -- refused ones and, under
// KSW_XSUBO, scores below the threshold.
__global__ void sw_bin_kernel(const g3x_job_t* __restrict__ jobs, int n, const g3x_swr_t* __restrict__ res,
                              const int32_t* __restrict__ status, int min_score, int32_t* __restrict__ bin,
                              int32_t* __restrict__ hist) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const g3x_job_t jb = jobs[k];
    int qlen = jb.qlen, rows = jb.tlen;
    if (res) {
        const g3x_swr_t r = res[k];
        qlen = status[k] == G3X_OK && r.score >= min_score ? r.qe + 1 : 0;
        if (r.te >= 0) rows = r.te + 1;
    }
    int b = kBins - 1;
    if (qlen >= 1 && qlen <= 8 * kSegBins) {
        const int slen = (qlen + 7) >> 3;
        const int rb = (int)(log2f(1.0f + (float)rows) * 8.0f);
        b = (kSegBins - slen) * kRowBins + (kRowBins - 1 - min(rb, kRowBins - 1));
    }
    bin[k] = b;
    const unsigned peers = __match_any_sync(__activemask(), b);
    if ((threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(hist + b, __popc(peers));
}

// Exclusive scan of the bins (one block) and the classes' ranges, the last (1-4 segments) in the
// first pass together with the rejected bin (with_last).
__global__ void __launch_bounds__(1024) sw_scan_kernel(const int32_t* __restrict__ hist, int32_t* __restrict__ cursor,
                                                       int32_t* __restrict__ range, int with_last) {
    constexpr int kPer = (kBins + 1023) / 1024;
    __shared__ int32_t part[1024];
    const int t = threadIdx.x;
    int32_t v[kPer], sum = 0;
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        v[u] = t * kPer + u < kBins ? hist[t * kPer + u] : 0;
        sum += v[u];
    }
    part[t] = sum;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const int x = t >= o ? part[t - o] : 0;
        __syncthreads();
        part[t] += x;
        __syncthreads();
    }
    int32_t at = part[t] - sum;
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        if (t * kPer + u < kBins) cursor[t * kPer + u] = at;
        at += v[u];
    }
    __syncthreads();
    if (t < kClasses) {
        const int lo = cursor[4 * t * kRowBins];
        const int hi = cursor[4 * (t + 1) * kRowBins] + (t == kClasses - 1 && with_last ? hist[kBins - 1] : 0);
        range[2 * t] = lo;
        range[2 * t + 1] = hi - lo;
    }
}

__global__ void sw_scatter_kernel(const int32_t* __restrict__ bin, int n, int32_t* __restrict__ cursor,
                                  int32_t* __restrict__ order) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int b = bin[k];
    const unsigned peers = __match_any_sync(__activemask(), b);
    const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
    int at = 0;
    if (lane == leader) at = atomicAdd(cursor + b, __popc(peers));
    at = __shfl_sync(peers, at, leader) + __popc(peers & ((1u << lane) - 1u));
    order[at] = k;
}

uint32_t pack16(int v) { return (uint32_t)(uint16_t)(int16_t)v * 0x10001u; }

template <int MAXSEG, bool SECOND>
int launch_classes(const SwDesc& d, bool first, cudaStream_t st) {
    auto kern = sw_kernel<MAXSEG, SECOND>;
    const int per_sm = resident_blocks(kern, 32 * kWarps, 0);
    // the classes of a pass run side by side: programmatic dependents of one another
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(sm_count() * std::max(per_sm, 1)));
    cfg.blockDim = dim3(32 * kWarps);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = first ? 0 : 1;
    return cudaLaunchKernelEx(&cfg, kern, d) == cudaSuccess ? G3X_OK : G3X_ERR_CUDA;
}

// One pass over the jobs: sorted, then a launch per class.
template <bool SECOND>
int run_pass(const SwDesc& d0, int32_t n, int32_t* buf, cudaStream_t st) {
    int32_t* bin = buf;
    int32_t* order = bin + n;
    int32_t* hist = order + n;
    int32_t* cursor = hist + kBins;
    int32_t* range = cursor + kBins;
    int32_t* queue = range + 2 * kClasses;
    SwDesc d = d0;
    d.order = order; d.range = range; d.queue = queue;
    if (cudaMemsetAsync(hist, 0, sizeof(int32_t) * kBins, st) != cudaSuccess ||
        cudaMemsetAsync(queue, 0, sizeof(int32_t) * kClasses, st) != cudaSuccess)
        return G3X_ERR_CUDA;
    const int min_score = (d.xtra & G3X_KSW_XSUBO) ? d.xtra & 0xFFFF : -1;
    const int tb = 256, nb = (n + tb - 1) / tb;
    sw_bin_kernel<<<nb, tb, 0, st>>>(d.jobs, n, SECOND ? d.out : nullptr, d.status, min_score, bin, hist);
    sw_scan_kernel<<<1, 1024, 0, st>>>(hist, cursor, range, SECOND ? 0 : 1);
    sw_scatter_kernel<<<nb, tb, 0, st>>>(bin, n, cursor, order);
    if (cudaPeekAtLastError() != cudaSuccess) return G3X_ERR_CUDA;
    int rc;
    if ((rc = launch_classes<32, SECOND>(d, true, st))) return rc;
    if ((rc = launch_classes<16, SECOND>(d, false, st))) return rc;
    return launch_classes<8, SECOND>(d, false, st);
}

}  // namespace
}  // namespace g3x

extern "C" int g3x_ksw_align2_batch(g3x_ctx* ctx, const g3x_score_t* score, const g3x_job_t* d_jobs, int32_t n,
                                    const uint32_t* d_codes, const uint32_t* d_nmask, int64_t n_bases, int32_t xtra,
                                    int32_t max_tlen,
                                    g3x_swr_t* d_out, int32_t* d_status, void* stream) {
    using namespace g3x;
    if (!ctx || !score || n < 0 || max_tlen < 0) return G3X_ERR_INVALID;
    // the reference fills an 8-bit profile for KSW_XBYTE and then reads it as 16-bit cells
    if (xtra & G3X_KSW_XBYTE) return G3X_ERR_INVALID;
    if (n == 0) return G3X_OK;
    if (!d_jobs || !d_codes || !d_nmask || !d_out || !d_status) return G3X_ERR_INVALID;
    if (n_bases < 1 || n_bases > 0x100000000ll) return G3X_ERR_INVALID;
    ScoreParams sp;
    int rc = score_params(score, &sp);
    if (rc) return rc;
    if (sp.oe_del > 32767 || sp.oe_ins > 32767) return G3X_ERR_SCORE;
    const bool subo = (xtra & G3X_KSW_XSUBO) != 0;
    if (subo && sp.max_sc < 1) return G3X_ERR_SCORE;   // ceil(score / max(mat)) of ksw.cu:250
    const int dev = ctx_device(ctx);
    if (cudaSetDevice(dev) != cudaSuccess) return G3X_ERR_CUDA;
    SwScratch& s = ctx_sw(ctx);
    const int64_t need = (int64_t)2 * n + 2 * kBins + 3 * kClasses;
    const int64_t sub_need = subo ? (int64_t)n * std::max(max_tlen, 1) : 0;
    if (s.cap < need || s.sub_cap < sub_need) {
        const int64_t cap = std::max(need, s.cap), sub_cap = std::max(sub_need, s.sub_cap);
        cudaFree(s.buf); cudaFree(s.sub);
        s.buf = nullptr; s.sub = nullptr; s.cap = 0; s.sub_cap = 0;
        if (cudaMalloc(&s.buf, (size_t)cap * sizeof(int32_t)) != cudaSuccess ||
            (sub_cap && cudaMalloc(&s.sub, (size_t)sub_cap * sizeof(uint32_t)) != cudaSuccess)) {
            cudaFree(s.buf); s.buf = nullptr; cudaGetLastError();
            return G3X_ERR_NOMEM;
        }
        s.cap = cap; s.sub_cap = sub_cap;
    }
    const cudaStream_t st = (cudaStream_t)stream;
    SwDesc d;
    memset(&d, 0, sizeof(d));
    d.jobs = d_jobs; d.codes = d_codes; d.nmask = d_nmask;
    d.out = d_out; d.status = d_status;
    d.sub = subo ? s.sub : nullptr;
    d.sub_stride = subo ? std::max(max_tlen, 1) : 0;
    d.xtra = xtra; d.maxmat = sp.max_sc; d.n_bases = n_bases;
    for (int a = 0; a < 5; ++a) {
        uint32_t lo = 0;
        for (int c = 0; c < 4; ++c) lo |= (uint32_t)(uint8_t)sp.mat[a * 5 + c] << (8 * c);
        d.tab[2 * a] = lo;
        d.tab[2 * a + 1] = (uint32_t)(uint8_t)sp.mat[a * 5 + 4];   // byte 5 (past the query) = 0
    }
    d.nedel = pack16(-sp.e_del); d.noedel = pack16(-sp.oe_del);
    d.neins = pack16(-sp.e_ins); d.noeins = pack16(-sp.oe_ins);
    d.one = sp.o_ins > 0 && sp.e_ins <= 1000 ? 1u : 0u;
    d.carry_e = sp.o_ins > 0 ? sp.e_ins : 0x7FFF;
    // two's complement of both halves at once: -k in each is 2^16 - k (2^16 + 1)
    d.step = 0u - (uint32_t)sp.e_ins * 0x10001u;
    d.dec0 = 0x10000u + d.step;
    d.peins = pack16(sp.e_ins);
    d.nstep = pack16(-d.carry_e);
    if ((rc = run_pass<false>(d, n, s.buf, st))) return rc;
    return (xtra & G3X_KSW_XSTART) ? run_pass<true>(d, n, s.buf, st) : G3X_OK;
}
