// g3x_global16.cu -- banded global alignment with backtrack (ksw_global2, bwa/src/ksw.cu:706-809),
// a group of lanes per job, int16x2.
//
// The lane-per-job kernel (g3x_global.cu) walks a row cell by cell, so a call lasts as long as its
// widest job's rows x columns however few jobs it has.  Here a group of G = 2, 4, 8, 16 or 32 lanes
// holds the whole band of a job, eight columns a lane, and a row is one step; a warp runs 16 to 1
// jobs, row i of all of them together.
//
// The row buffer lives in registers over a window that slides with the band: at row i, index d
// holds column i - w + d, d = 0 .. 2w.  H(i, j) is the diagonal of (i+1, j+1), which has the same
// index, so H stays where it is; E(i+1, j) moves one index down (one shuffle a row), and so do
// the query codes (one shuffle every eight rows).  Blocks and F as in g3x_lane16.cuh, the F entering
// a block by a prefix over the group (g3x_group.cuh).
//
// Values are biased by 2^14 with 0 for the reference's -2^30 outside the band: a batch comes here
// only when every value inside the band stays within 8000 (g3x_ksw_global2_batch), so each one is
// positive, sums are clipped at 0 as in the extension kernels, and every comparison goes the way of
// the reference's.  Cells left of column 0 (the first w rows) are masked: M and E are 0, and H
// keeps H(i, -1) of the row that will need it as its diagonal.  Cells right of the query need no
// mask: F flows right, E stays in its column.  E entering at index 2w is 0.
//
// A cell's direction is four bits: H is not M, H is not E, E and F continue (ksw.cu:753-776: M
// before E before F), each the difference of a maximum and one of its operands, formed by
// multiply-adds (the bias keeps both halves non-negative, so one 32-bit subtraction serves both)
// and clipped to 0 or 1.  A
// lane's eight cells make one word, a warp's row one 128-byte line of scratch.  The backtrack
// (ksw.cu:783-806) stays on one index while it moves diagonally, so the group reads 32 rows of that
// index at a time and takes the run of matches up to the first gap from a ballot; gaps go cell by
// cell.
#include <cuda_runtime.h>
#include "g3x_core.h"
#include "g3x_global.cuh"
#include "g3x_group.cuh"
#include "g3x_internal.h"
#include "g3x_lane16.cuh"
#include "g3x_stage.cuh"

namespace g3x {

namespace {

using namespace l16;

constexpr int32_t kBias = 0x4000;

// One 16-bit half of the block words, offset t of the block.
__device__ __forceinline__ int32_t half_of(const uint32_t (&w)[4], int t) {
    const uint32_t lo = (t & 1) ? w[1] : w[0], hi = (t & 1) ? w[3] : w[2];
    const uint32_t v = (t & 2) ? hi : lo;
    return (int32_t)((t & 4) ? v >> 16 : v & 0xFFFFu);
}

// Runs the jobs order[0 .. n) (order null: 0 .. n), taken from *queue; z: the warp's direction
// scratch, 32 words a row.
template <int G, bool kSym>
__device__ __forceinline__ void run_pairs(const GlobalDesc& d, const ScoreParams& sp, const PairConst& pc,
                                          const uint4* from, const uint2* pools, const int32_t* order, int n,
                                          int32_t* queue, uint32_t* z, int lane) {
    constexpr int kGroups = 32 / G, K = 32 / G;     // K: rows a lane looks up at a time in the backtrack
    const int r = lane & (G - 1), gb = lane & ~(G - 1);
    const unsigned gmask = (G == 32 ? kAll : ((1u << G) - 1u)) << gb;
    const uint32_t minus = 0u - sp.k16 / 65536u;      // run-time -1: subtract on the multiply-add pipe
    for (;;) {
        int first = 0;
        if (lane == 0) first = atomicAdd(queue, kGroups);
        first = __shfl_sync(kAll, first, 0);
        if (first >= n) break;
        const int slot = first + lane / G;
        int job = -1, qlen = 0, tlen = 0, w = 0;
        uint32_t q_off = 0, t_off = 0, flags = 0;
        if (slot < n) {
            job = order ? order[slot] : slot;
            const g3x_job_t jb = d.jobs[job];
            const bool outside = !job_in_planes(jb, d.n_bases);   // refused before any base is read
            qlen = jb.qlen; tlen = jb.tlen; w = jb.w; flags = jb.flags; q_off = jb.q_off; t_off = jb.t_off;
            const int wide = min(w, max(qlen, tlen));             // a wider band holds no more cells
            if (qlen > d.qmax || tlen > d.tmax || w < 0 || w > d.wmax || outside || 2 * wide + 1 > 8 * G) {
                if (r == 0) {
                    d.score[job] = 0; d.n_cigar[job] = 0;
                    d.status[job] = outside ? G3X_ERR_INVALID : G3X_ERR_TOO_LONG;
                    if (d.nm) { d.nm[job] = 0; d.md[(int64_t)job * d.md_stride] = 0; }
                }
                job = -1;
                qlen = tlen = 0;
            }
            w = wide;
        }
        const bool qrev = (flags & G3X_JOB_QREV) != 0, trev = (flags & G3X_JOB_TREV) != 0;
        // the last cell lies in the band of the last row; otherwise the score is a border value or
        // outside the band, and there is no matrix to fill
        const bool inside = qlen > 0 && tlen > 0 && tlen + w >= qlen && tlen - w <= qlen;
        const int rows = inside ? tlen : 0;
        const int max_rows = (int)__reduce_max_sync(kAll, (unsigned)rows);
        const int max_w = (int)__reduce_max_sync(kAll, (unsigned)(inside ? w : 0));
        int next_end = (int)__reduce_min_sync(kAll, rows > 0 ? (unsigned)rows : 0x7FFFFFFFu);
        int32_t score = kBias + kNegInf;

        uint32_t H[4], E[4] = {0u, 0u, 0u, 0u}, em[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            uint32_t v2 = 0u;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int k = 8 * r + p + 4 * u, j = k - w;       // row 0: index k is column j
                // j <= 0: H(-1 - j, -1), the diagonal of column 0 at row -j; else H(-1, j - 1)
                const int32_t v = j < 0 ? -(sp.o_del - sp.e_del * j) : j == 0 ? 0 : -(sp.oe_ins + sp.e_ins * (j - 1));
                if (k <= 2 * w) v2 |= ((uint32_t)(v + kBias) & 0xFFFFu) << (16 * u);
            }
            H[p] = v2;
        }
        {
            const uint4 g = from[max(min(2 * w - 8 * r, 8), 0)];
            em[0] = ~g.x; em[1] = ~g.y; em[2] = ~g.z; em[3] = ~g.w;
        }
        // query codes of the block's columns and of the next eight; ext: lane r holds the eight
        // codes that enter the window at its right end in rows 8 (e0 + r) ..
        uint32_t qlo = rows ? codes8(d.codes, d.nmask, q_off, qlen, qrev, 8 * r - w) : 0u, qhi = 0u, ext = 0u, tw = 0u, t8 = 0u;
        uint32_t* zr = z + lane;
        for (int i = 0; i < max_rows; ++i, zr += 32) {
            if ((i & 7) == 0) {
                const int e = i >> 3;
                if ((e & (G - 1)) == 0) {
                    ext = tw = 0u;
                    if (i < rows) {
                        ext = codes8(d.codes, d.nmask, q_off, qlen, qrev, i - w + 8 * (G + r));
                        const int ch = (e + r) >> 1;
                        if (ch << 4 < tlen) {
                            uint32_t x, nb;
                            load16(d.codes, d.nmask, t_off, tlen, ch, trev, x, nb);
                            tw = (uint32_t)(nibbles16(x, nb) >> (((e + r) & 1) << 5));
                        }
                    }
                }
                if (i) qlo = qhi;
                const int src = gb | (e & (G - 1));
                const uint32_t in = __shfl_sync(kAll, ext, src), dn = __shfl_down_sync(kAll, qlo, 1, G);
                qhi = r == G - 1 ? in : dn;
                t8 = __shfl_sync(kAll, tw, src);
            }
            const int sh = (i & 7) << 2;
            const uint32_t qw = __funnelshift_r(qlo, qhi, sh);
            const uint2 pl = pools[(t8 >> sh) & 7u];

            // M, the F prefix from 0 over each half of the block, E of the next row
            const uint32_t sc_lo = prmt(pl.x, pl.y, qw), sc_hi = prmt(pl.x, pl.y, qw >> 16);
            const uint32_t S2[4] = {pair_score<0>(sc_lo, sc_hi), pair_score<1>(sc_lo, sc_hi),
                                    pair_score<2>(sc_lo, sc_hi), pair_score<3>(sc_lo, sc_hi)};
            uint32_t M[4];
#pragma unroll
            for (int p = 0; p < 4; ++p) M[p] = __viaddmax_s16x2(H[p], S2[p], 0u);
            uint32_t keep[4] = {kAll, kAll, kAll, kAll};
            if (i < max_w) {                                      // columns left of 0
                const uint4 g = from[max(min(w - i - 8 * r, 8), 0)];
                keep[0] = g.x; keep[1] = g.y; keep[2] = g.z; keep[3] = g.w;
#pragma unroll
                for (int p = 0; p < 4; ++p) M[p] &= keep[p];
            }
            uint32_t T[4], L[4], Td[4], En[4];
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                T[p] = __viaddmax_s16x2(M[p], pc.noe_ins, 0u);
                L[p] = p == 0 ? T[p] : __viaddmax_s16x2(L[p - 1], pc.ne_ins, T[p]);
                Td[p] = kSym ? T[p] : __viaddmax_s16x2(M[p], pc.noe_del, 0u);
                En[p] = __viaddmax_s16x2(E[p], pc.ne_del, Td[p]);
            }
            const uint32_t fr = (uint32_t)f_entering<G>((int32_t)__viaddmax_s16x2(L[3] << 16, pc.n4, L[3]), r, sp.e_ins);
            const uint32_t x = __viaddmax_s16x2(prmt(fr, fr, 0x3232u), pc.n4, L[3]);   // low half: F(4)
            uint32_t F[5];
            F[0] = prmt(fr, x, 0x5432u);
#pragma unroll
            for (int p = 1; p < 4; ++p) F[p] = __viaddmax_s16x2(F[0], pc.nt[p], L[p - 1]);
            F[4] = prmt(F[0], __viaddmax_s16x2(F[0], pc.n4, L[3]), 0x7632u);           // (F(4), F(8))

            // H and the directions: bits 0-3 of each half for the pair's two cells
            uint32_t dir = 0u;
#pragma unroll
            for (int p = 3; p >= 0; --p) {
                const uint32_t h = __vimax3_s16x2(M[p], E[p], F[p]);
                const uint32_t one = 0x00010001u;
                const uint32_t b0 = __vimin3_u16x2(M[p] * minus + h, one, one), b1 = __vimin3_u16x2(E[p] * minus + h, one, one);
                const uint32_t b2 = __vimin3_u16x2(Td[p] * minus + En[p], one, one);
                const uint32_t b3 = __vimin3_u16x2(T[p] * minus + F[p + 1], one, one);
                dir = dir * 16u + (b0 + 2u * b1 + 4u * b2 + 8u * b3);
                H[p] = i < max_w ? (h & keep[p]) | (H[p] & ~keep[p]) : h;
            }
            if (i < rows) *zr = dir;
            // E one index down
            const uint32_t e0 = __shfl_down_sync(kAll, En[0], 1, G);
            E[0] = En[1] & em[0];
            E[1] = En[2] & em[1];
            E[2] = En[3] & em[2];
            E[3] = prmt(En[0], e0, 0x5432u) & em[3];
            if (i + 1 == next_end) {                              // some job's last row: its score
                const int k = qlen - tlen + w;                    // index of column qlen - 1
                const int32_t v = __shfl_sync(kAll, half_of(H, k & 7), gb | ((k >> 3) & (G - 1)));
                if (rows == next_end) score = v;
                next_end = (int)__reduce_min_sync(kAll, rows > next_end ? (unsigned)rows : 0x7FFFFFFFu);
            }
        }
        __syncwarp();

        // ---- score and backtrack (ksw.cu:781-806) ----
        score -= kBias;
        bool finite = inside;
        if (job >= 0 && !inside) {          // borders: H(tlen - 1, -1), H(-1, qlen - 1) or no path
            if (qlen == 0 && tlen <= w + 1) { finite = true; score = tlen ? -(sp.o_del + sp.e_del * tlen) : 0; }
            else if (tlen == 0 && qlen <= w) { finite = true; score = -(sp.oe_ins + sp.e_ins * (qlen - 1)); }
            else score = kNegInf;
        }
        int i = tlen - 1, k = qlen - 1, which = 0, n_ops = 0, op = -1, len = 0;
        bool full = false, bad = false;
        uint32_t* cg = d.cigar + (int64_t)(job >= 0 ? job : 0) * d.stride;
        auto push = [&](int o, int l) {     // the run being built is entry n_ops - 1
            if (o == op) {
                len += l;
            } else if (n_ops < d.stride) {
                if (n_ops && r == 0) cg[n_ops - 1] = (uint32_t)len << 4 | (uint32_t)op;
                ++n_ops;
                op = o; len = l;
            } else {
                full = true;
            }
        };
        while (__any_sync(kAll, inside && i >= 0 && k >= 0 && !full && !bad)) {
            const bool go = inside && i >= 0 && k >= 0 && !full && !bad;
            const int dk = k - i + w;                             // index, the same along a diagonal
            if (go && (dk < 0 || dk > 2 * w)) bad = true;         // never on a path with a finite score
            const int cells = min(min(i, k) + 1, which ? 1 : 32); // a gap goes on cell by cell
            // lane r: rows i - K r .. i - K r - (K - 1); its first cell that is no match, and the
            // operation there: from H (M, else E, else F), or the gap going on or not
            uint32_t dirs[K];
#pragma unroll
            for (int t = 0; t < K; ++t) {
                dirs[t] = 0u;
                if (go && !bad && K * r + t < cells) dirs[t] = z[(int64_t)(i - K * r - t) * 32 + gb + (dk >> 3)];
            }
            int stop_at = K, o = 0;
#pragma unroll
            for (int t = K - 1; t >= 0; --t) {
                const uint32_t nib = dirs[t] >> ((dk & 7) << 2);
                const int ot = which == 0 ? ((nib & 1u) ? 1 + (int)(nib >> 1 & 1u) : 0) : (nib >> (which + 1)) & 1u ? which : 0;
                o = ot ? ot : o;
                stop_at = ot ? t : stop_at;
            }
            const unsigned gap = __ballot_sync(kAll, stop_at < K) & gmask;
            const int at = gap ? __ffs(gap) - 1 : 0;
            const int og = __shfl_sync(kAll, o, at);
            const int before = __shfl_sync(kAll, stop_at, at) + K * (at - gb);
            if (go && !bad) {
                const int run = gap ? before : cells;
                if (run) { push(0, run); i -= run; k -= run; which = 0; }
                if (gap && !full) {
                    if (og == 1) { push(2, 1); --i; } else { push(1, 1); --k; }
                    which = og;
                }
            }
        }
        if (job >= 0) {
            if (finite && !bad && !full) {
                if (i >= 0) push(2, i + 1);
                if (k >= 0) push(1, k + 1);
            }
            if (r == 0) {
                if (n_ops) cg[n_ops - 1] = (uint32_t)len << 4 | (uint32_t)op;
                for (int a = 0; a < n_ops >> 1; ++a) {
                    const uint32_t t = cg[a]; cg[a] = cg[n_ops - 1 - a]; cg[n_ops - 1 - a] = t;
                }
                d.score[job] = score;
                d.n_cigar[job] = full || bad ? 0 : n_ops;
                int32_t st = full ? G3X_ERR_TOO_LONG : bad ? G3X_ERR_INTERNAL : G3X_OK;
                if (d.nm && st == G3X_OK) {
                    int cq = -1, ct = -1;
                    uint64_t vq = 0, vt = 0;
                    auto qchunk = [&](int c) -> uint64_t {
                        if (c != cq) {
                            uint32_t x, nb;
                            load16(d.codes, d.nmask, q_off, qlen, cq = c, qrev, x, nb);
                            vq = plain_nibbles(nibbles16(x, nb));
                        }
                        return vq;
                    };
                    auto tchunk = [&](int c) -> uint64_t {
                        if (c != ct) {
                            uint32_t x, nb;
                            load16(d.codes, d.nmask, t_off, tlen, ct = c, trev, x, nb);
                            vt = plain_nibbles(nibbles16(x, nb));
                        }
                        return vt;
                    };
                    if (!write_nm_md(d, job, flags, cg, n_ops, qchunk, tchunk)) st = G3X_ERR_TOO_LONG;
                } else if (d.nm) {
                    d.nm[job] = 0;
                    d.md[(int64_t)job * d.md_stride] = 0;
                }
                d.status[job] = st;
            }
        }
        __syncwarp();
    }
}

// d.range null: the jobs as they are numbered, a warp each.  Else [offset, count] of the classes
// of d.order, class k in groups of 2 << k lanes, the widest first.
template <bool kSym>
__global__ void __launch_bounds__(32 * kGlobal16Warps, 11) global16_kernel(GlobalDesc d, ScoreParams sp) {
    __shared__ uint4 from[9];          // pair words of the columns at or right of an offset
    __shared__ uint2 pools[8];
    if (threadIdx.x < 9) {
        const int o = threadIdx.x;
        from[o] = make_uint4(ge_word(o, 0), ge_word(o, 1), ge_word(o, 2), ge_word(o, 3));
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
    uint32_t* z = reinterpret_cast<uint32_t*>(d.z + (blockIdx.x * kGlobal16Warps + (threadIdx.x >> 5)) * d.zwarp);
    if (!d.range) {
        run_pairs<32, kSym>(d, sp, pc, from, pools, nullptr, d.n, d.queue, z, lane);
    } else {
        const int32_t* oc = d.range;
        run_pairs<32, kSym>(d, sp, pc, from, pools, d.order + oc[8], oc[9], d.queue + 4, z, lane);
        run_pairs<16, kSym>(d, sp, pc, from, pools, d.order + oc[6], oc[7], d.queue + 3, z, lane);
        run_pairs<8, kSym>(d, sp, pc, from, pools, d.order + oc[4], oc[5], d.queue + 2, z, lane);
        run_pairs<4, kSym>(d, sp, pc, from, pools, d.order + oc[2], oc[3], d.queue + 1, z, lane);
        run_pairs<2, kSym>(d, sp, pc, from, pools, d.order + oc[0], oc[1], d.queue, z, lane);
    }
}

}  // namespace

int global16_blocks() {
    const int per_sm = resident_blocks(global16_kernel<true>, 32 * kGlobal16Warps, 0);
    return sm_count() * (per_sm > 0 ? per_sm : 1);
}

int launch_global16(const GlobalDesc& d, const ScoreParams& sp, int blocks, cudaStream_t st) {
    auto kern = sp.oe_del == sp.oe_ins ? global16_kernel<true> : global16_kernel<false>;
    kern<<<blocks, 32 * kGlobal16Warps, 0, st>>>(d, sp);
    return cudaPeekAtLastError() == cudaSuccess ? G3X_OK : G3X_ERR_CUDA;
}

}  // namespace g3x
