// g3x_global.cu -- banded global alignment with backtrack (ksw_global2, bwa/src/ksw.cu:706-809)
// for batches of alignments on the GPU.
//
// Two kernels.  Jobs whose band fits a group of lanes and whose scores fit int16 run in
// g3x_global16.cu; this file holds the call and the kernel for the others.
//
// One job per lane.  The jobs are first ordered by decreasing row count and row width (the
// scheduler's counting sort); a warp takes 32 consecutive ones and runs their target rows
// together (row i of every job in the same step); in a row each lane walks its own band
// [max(i-w, 0), min(i+w+1, qlen)) column by column (the reference's scalar recurrence, in int32
// with -2^30 outside the band, ksw.cu:548; see Ring for the int16 form of short batches).  The
// band has a fixed width and never trims, so the
// row buffer of H(i-1, j-1) and E(i, j) (ksw.cu:299-301) is a ring of R >= 2w+3 columns per lane
// in shared memory: a row reads columns [beg, end) and writes column end, and a column enters
// the ring either from the first row's fill (columns 0..w) or from the row end that precedes its
// first read.  Each cell's direction byte (ksw.cu:753-776: h from M, E or F in bits 0-1, E and F
// continuing in bits 2 and 4-5) goes to global scratch, laid out [row][band column][lane] per
// warp so that the 32 lanes of a step write one 32-byte sector.  The backtrack then walks each
// lane's bytes from the last cell (ksw.cu:783-806) and writes the CIGAR, merging runs as
// push_cigar does (ksw.cu:694-704); on request NM and the MD string follow, as the traceback
// stage computes them (bwa/src/aux.cu:2831-2860).
#include <cuda_runtime.h>
#include <algorithm>
#include "g3x_core.h"
#include "g3x_global.cuh"
#include "g3x_internal.h"
#include "g3x_stage.cuh"

namespace g3x {

namespace {

__device__ __forceinline__ int32_t sbyte0(uint32_t x) { return (int32_t)(int8_t)(x & 0xFFu); }

// The ring's H and E: int32 pairs with the reference's -2^30 outside the band, or, for batches
// whose every value fits (compact_fits), int16 pairs in one word with -2^14 outside the band.
// Every value outside the band is that constant plus a sum of scores and penalties, the same sum
// in both forms, and every value inside stays above -2^13 while every value outside stays below
// it: each comparison goes the same way in both, and a score from outside the band maps back to
// the reference's -2^30 plus the same sum.
template <bool C16> struct Ring;
template <> struct Ring<false> {
    static constexpr int32_t kNeg = kNegInf;
    static constexpr int kSlotBytes = 8;
    int2* p;
    __device__ __forceinline__ int2 ld(int k) const { return p[k]; }
    __device__ __forceinline__ void st(int k, int32_t h, int32_t e) const { p[k] = make_int2(h, e); }
};
template <> struct Ring<true> {
    static constexpr int32_t kNeg = -0x4000;
    static constexpr int kSlotBytes = 4;
    uint32_t* p;
    __device__ __forceinline__ int2 ld(int k) const {
        const uint32_t v = p[k];
        return make_int2((int32_t)(int16_t)(v & 0xFFFFu), (int32_t)v >> 16);
    }
    __device__ __forceinline__ void st(int k, int32_t h, int32_t e) const {
        p[k] = (uint32_t)(uint16_t)h | ((uint32_t)e << 16);
    }
};

template <bool C16>
__global__ void __launch_bounds__(64) global_kernel(GlobalDesc d, ScoreParams sp) {
    extern __shared__ __align__(16) char smem[];
    using RingT = Ring<C16>;
    constexpr int32_t kNeg = RingT::kNeg;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int nq = (d.qmax + 7) / 8 + 1;                       // query words (8 codes each)
    uint32_t* qn = reinterpret_cast<uint32_t*>(
        smem + (size_t)warp * ((size_t)nq * 128 + (size_t)d.ring * 32 * RingT::kSlotBytes));
    RingT he;                                                   // ring slot s of lane L: index s*32 + L
    he.p = reinterpret_cast<decltype(he.p)>(qn + nq * 32);
    const int wslot = blockIdx.x * (blockDim.x >> 5) + warp;
    uint8_t* z = d.z + (int64_t)wslot * d.zwarp;
    uint32_t lo[5], hi[5];
    score_pools(sp, lo, hi);
    const int32_t oe_del = sp.o_del + sp.e_del, oe_ins = sp.o_ins + sp.e_ins;
    const int R = d.ring;
    const int n_jobs = d.range[1];
    const int32_t* order = d.order + d.range[0];

    for (;;) {
        int first = 0;
        if (lane == 0) first = atomicAdd(d.queue, 32);
        first = __shfl_sync(0xFFFFFFFFu, first, 0);
        if (first >= n_jobs) break;
        const int job = first + lane < n_jobs ? order[first + lane] : -1;
        int32_t qlen = 0, tlen = 0, w = 0;
        uint32_t t_off = 0, flags = 0;
        bool trev = false, live = false;
        if (job >= 0) {
            const g3x_job_t jb = d.jobs[job];
            qlen = jb.qlen; tlen = jb.tlen; w = jb.w; flags = jb.flags;
            t_off = jb.t_off; trev = (jb.flags & G3X_JOB_TREV) != 0;
            const bool outside = !job_in_planes(jb, d.n_bases);   // refused before any base is read
            if (qlen > d.qmax || tlen > d.tmax || w < 0 || w > d.wmax || outside) {
                d.score[job] = 0; d.n_cigar[job] = 0; d.status[job] = outside ? G3X_ERR_INVALID : G3X_ERR_TOO_LONG;
                if (d.nm) { d.nm[job] = 0; d.md[(int64_t)job * d.md_stride] = 0; }
            } else {
                live = true;
                stage_own_query(d.codes, d.nmask, jb.q_off, qlen, (jb.flags & G3X_JOB_QREV) != 0,
                                (qlen + 15) >> 4, qn, lane);
                // the first row (ksw.cu:721-724): columns 0..min(w, qlen)
                const int top = qlen < w ? qlen : w;
                for (int j = 0; j <= top; ++j)
                    he.st((j % R) * 32 + lane, j == 0 ? 0 : -(oe_ins + sp.e_ins * (j - 1)), kNeg);
            }
        }
        __syncwarp();
        const int rows = __reduce_max_sync(0xFFFFFFFFu, (unsigned)(live ? tlen : 0));
        uint32_t tx = 0, tn = 0;
        for (int i = 0; i < rows; ++i) {
            const bool run = live && i < tlen;
            int beg = 0, end = 0;
            uint32_t plo = 0, phi = 0;
            int32_t h1 = kNeg, f = kNeg;
            if (run) {
                beg = i > w ? i - w : 0;
                end = i + w + 1 < qlen ? i + w + 1 : qlen;
                h1 = beg == 0 ? -(sp.o_del + sp.e_del * (i + 1)) : kNeg;
                if ((i & 15) == 0) load16(d.codes, d.nmask, t_off, tlen, i >> 4, trev, tx, tn);
                uint32_t code = (tx >> ((i & 15) << 1)) & 3u;
                if ((tn >> (i & 15)) & 1u) code = 4;
                plo = lo[code]; phi = hi[code];
            }
            const int width = run && end > beg ? end - beg : 0;   // rows past qlen + w have no cells
            const int wmax = __reduce_max_sync(0xFFFFFFFFu, (unsigned)width);
            uint8_t* zrow = z + (int64_t)i * d.ncol * 32 + lane;
            int s = run ? beg % R : 0;
            uint32_t qw = 0;
            for (int t = 0; t < wmax; ++t) {
                if (t < width) {
                    const int j = beg + t;
                    if (t == 0 || (j & 7) == 0) qw = qn[(j >> 3) * 32 + lane];
                    const int32_t sc = sbyte0(__byte_perm(plo, phi, (qw >> ((j & 7) << 2)) & 0xFu));
                    int2 c = he.ld(s * 32 + lane);
                    const int32_t m = c.x + sc;
                    int32_t e = c.y;
                    c.x = h1;
                    uint32_t dir = m >= e ? 0u : 1u;
                    int32_t h = m >= e ? m : e;
                    if (h < f) { dir = 2u; h = f; }
                    h1 = h;
                    int32_t tt = m - oe_del;
                    e -= sp.e_del;
                    if (e > tt) dir |= 1u << 2; else e = tt;
                    c.y = e;
                    he.st(s * 32 + lane, c.x, c.y);
                    tt = m - oe_ins;
                    f -= sp.e_ins;
                    if (f > tt) dir |= 2u << 4; else f = tt;
                    zrow[(int64_t)t * 32] = (uint8_t)dir;
                    s = s + 1 == R ? 0 : s + 1;
                }
            }
            if (run) he.st((end % R) * 32 + lane, h1, kNeg);   // ksw.cu:779
            __syncwarp();
        }
        // score and backtrack (ksw.cu:781-806)
        if (live) {
            // H of column qlen: written by the last row's end when its band reaches qlen, else
            // still the first row's value
            const int32_t init = qlen == 0 ? 0 : (qlen <= w ? -(oe_ins + sp.e_ins * (qlen - 1)) : kNeg);
            const int32_t score = tlen > 0 && tlen + w >= qlen ? he.ld((qlen % R) * 32 + lane).x : init;
            const bool finite = score > kNeg / 2;
            d.score[job] = finite ? score : kNegInf + (score - kNeg);
            uint32_t* cg = d.cigar + (int64_t)job * d.stride;
            int n = 0;
            bool full = false;
            auto push = [&](int op, int len) {
                if (n > 0 && (int)(cg[n - 1] & 0xFu) == op) cg[n - 1] += (uint32_t)len << 4;
                else if (n < d.stride) cg[n++] = (uint32_t)len << 4 | (uint32_t)op;
                else full = true;
            };
            bool bad = false;
            if (finite) {
                int i = tlen - 1, k = (i + w + 1 < qlen ? i + w + 1 : qlen) - 1, which = 0;
                while (i >= 0 && k >= 0 && !full) {
                    const int bi = i > w ? i - w : 0;
                    if (k - bi < 0 || k - bi >= d.ncol) { bad = true; break; }   // never on a path with a finite score
                    which = (z[((int64_t)i * d.ncol + (k - bi)) * 32 + lane] >> (which << 1)) & 3;
                    if (which == 0) { push(0, 1); --i; --k; }
                    else if (which == 1) { push(2, 1); --i; }
                    else { push(1, 1); --k; }
                }
                if (!bad && i >= 0) push(2, i + 1);
                if (!bad && k >= 0) push(1, k + 1);
                for (int a = 0; a < n >> 1; ++a) {
                    const uint32_t t = cg[a]; cg[a] = cg[n - 1 - a]; cg[n - 1 - a] = t;
                }
            }
            d.n_cigar[job] = full || bad ? 0 : n;
            int32_t stj = full ? G3X_ERR_TOO_LONG : bad ? G3X_ERR_INTERNAL : G3X_OK;
            if (d.nm && stj == G3X_OK) {
                // the query from its codes in shared memory, the target from the planes
                int cy = -1;
                uint64_t vy = 0;
                auto qchunk = [&](int c) -> uint64_t {
                    return plain_nibbles((uint64_t)qn[2 * c * 32 + lane] | (uint64_t)qn[(2 * c + 1) * 32 + lane] << 32);
                };
                auto tchunk = [&](int c) -> uint64_t {
                    if (c != cy) {
                        uint32_t x, nb;
                        load16(d.codes, d.nmask, t_off, tlen, cy = c, trev, x, nb);
                        vy = plain_nibbles(nibbles16(x, nb));
                    }
                    return vy;
                };
                if (!write_nm_md(d, job, flags, cg, n, qchunk, tchunk)) stj = G3X_ERR_TOO_LONG;
            } else if (d.nm) {
                d.nm[job] = 0;
                d.md[(int64_t)job * d.md_stride] = 0;
            }
            d.status[job] = stj;
        }
        __syncwarp();
    }
}

// Up to here the group kernel takes the jobs as they come, a warp each; beyond, sorted by band
// width, up to sixteen a warp.  CIGAR only, direct and sorted: 128 pairs 87 and 113 us, 1,024 105 and 132,
// 2,048 152 and 171, 4,096 211 and 233, 8,192 324 and 234.  The line lies well below the crossing: from
// there on the sorted form's time hardly moves with the count, the direct one's grows with it.
constexpr int kDirectPairs = 1024;

// Large batches of very short pairs stay in the lane kernel, which has 32 of them a warp where the groups
// have sixteen at most and one lane of each walks the CIGAR and MD.  Lane kernel and groups, us: up to 8
// bases 100k pairs with MD 86 and 86, 130k 91 and 97, 190k 103 and 123, without 91 and 103; 12 bases 160k
// with MD 130 and 133, 190k 133 and 153, without 114 and 119; 16 bases 190k with MD 163 and 177, without 141
// and 134; 20 bases 160k 193 and 192, 190k 203 and 216; 23 bases 190k 240 and 239.
static bool short_pairs(int qmax, bool md, int64_t n) {
    return qmax <= (md ? 20 : 12) && n > (qmax <= 8 ? 114688 : 163840);
}

}  // namespace

}  // namespace g3x

extern "C" int g3x_ksw_global2_batch(g3x_ctx* ctx, const g3x_score_t* score, const g3x_job_t* d_jobs, int32_t n,
                                     const uint32_t* d_codes, const uint32_t* d_nmask, int64_t n_bases, int32_t max_qlen,
                                     int32_t max_tlen, int32_t max_w, int32_t* d_score, uint32_t* d_cigar,
                                     int32_t cigar_stride, int32_t* d_n_cigar, int32_t* d_nm, char* d_md,
                                     int32_t md_stride, int32_t* d_status, void* stream) {
    using namespace g3x;
    if (!ctx || !score || n < 0 || max_qlen < 0 || max_tlen < 0 || max_w < 0 || cigar_stride <= 0)
        return G3X_ERR_INVALID;
    if ((d_nm != nullptr) != (d_md != nullptr) || (d_nm && md_stride < 2)) return G3X_ERR_INVALID;
    if (n == 0) return G3X_OK;
    if (n_bases < 1 || n_bases > 0x100000000ll) return G3X_ERR_INVALID;
    if (!d_jobs || !d_codes || !d_nmask || !d_score || !d_cigar || !d_n_cigar || !d_status) return G3X_ERR_INVALID;
    ScoreParams sp;
    int rc = score_params(score, &sp);
    if (rc) return rc;
    const int dev = ctx_device(ctx);
    if (cudaSetDevice(dev) != cudaSuccess) return G3X_ERR_CUDA;
    GlobalDesc d;
    d.jobs = d_jobs; d.codes = d_codes; d.nmask = d_nmask; d.score = d_score; d.cigar = d_cigar;
    d.n_cigar = d_n_cigar; d.status = d_status; d.n = n;
    d.nm = d_nm; d.md = d_md; d.md_stride = md_stride; d.n_bases = n_bases;
    d.qmax = std::max(max_qlen, 1); d.tmax = std::max(max_tlen, 1); d.wmax = max_w;
    d.ncol = std::max(1, std::min(d.qmax, 2 * max_w + 1));
    d.ring = ((2 * max_w + 3) + 3) & ~3;
    d.stride = cigar_stride;
    // int16 ring when every value of the batch fits: |inside-band values| <= bound <= 8000
    int max_abs = 0;
    for (int k = 0; k < 25; ++k) max_abs = std::max(max_abs, std::abs((int)sp.mat[k]));
    const int64_t bound = 2 * (int64_t)std::max(sp.o_del, sp.o_ins) +
                          (int64_t)std::max(sp.e_del, sp.e_ins) * (d.qmax + d.tmax + 2) +
                          (int64_t)max_abs * (std::min(d.qmax, d.tmax) + 1);
    const bool c16 = bound <= 8000;
    auto kern = c16 ? global_kernel<true> : global_kernel<false>;
    const int nq = (d.qmax + 7) / 8 + 1;
    const size_t warp_smem = (size_t)nq * 128 + (size_t)d.ring * 32 * (c16 ? 4 : 8);
    size_t max_smem = 0;
    if (allow_max_smem(kern, &max_smem) != cudaSuccess) return G3X_ERR_CUDA;
    if (warp_smem > max_smem) return G3X_ERR_TOO_LONG;
    // The group kernel takes the jobs that fit it; the lane kernel is launched when there may be
    // others: values beyond int16, or bands beyond the widest group (a band is cut to the longer
    // sequence).  may: which of them calls of these bounds launch at some number of pairs.
    const bool brief = short_pairs(d.qmax, d_nm != nullptr, n), may_brief = short_pairs(d.qmax, d_nm != nullptr, 0x7FFFFFFF);
    const bool groups = c16 && !brief;
    const bool lanes = !groups || std::min(max_w, std::max(d.qmax, d.tmax)) > kGlobalGroupMaxW;
    const bool may_groups = c16, may_lanes = lanes || may_brief;
    const int64_t cap = (int64_t)8 << 30;
    int wpb = 0, blocks = 0, gblocks = 0;
    int64_t need = 0;
    const int64_t zlane = (int64_t)d.tmax * d.ncol * 32, zgroup = global16_warp_bytes(d.tmax);
    // scratch: the resident warps' directions, at most 8 GiB; the two kernels run one after the
    // other and share it.  It is sized by the bounds alone, for the whole device and whatever n is: a call
    // captured after a smaller one of the same bounds must find its scratch.
    if (may_lanes) {
        wpb = 2 * warp_smem <= max_smem ? 2 : 1;
        const int per_sm = resident_blocks(kern, 32 * wpb, wpb * warp_smem);
        blocks = sm_count() * std::max(per_sm, 1);
        while (blocks > 1 && (int64_t)blocks * wpb * zlane > cap) blocks = blocks / 2;
        need = (int64_t)blocks * wpb * zlane;
    }
    const bool direct = groups && !lanes && n <= kDirectPairs;
    if (may_groups) {
        gblocks = global16_blocks();
        while (gblocks > 1 && (int64_t)gblocks * kGlobal16Warps * zgroup > cap) gblocks = gblocks / 2;
        need = std::max(need, (int64_t)gblocks * kGlobal16Warps * zgroup);
        gblocks = std::min(gblocks, (n + kGlobal16Warps - 1) / kGlobal16Warps);
    }
    GlobalScratch& gs = ctx_global(ctx);
    if (gs.bytes < need || !gs.queue) {
        cudaFree(gs.z); cudaFree(gs.queue);
        gs.z = nullptr; gs.queue = nullptr; gs.bytes = 0;
        if (cudaMalloc(&gs.z, (size_t)need) != cudaSuccess ||
            cudaMalloc(&gs.queue, (kGlobalGroupClasses + 1) * sizeof(int32_t)) != cudaSuccess) {
            cudaFree(gs.z); gs.z = nullptr; cudaGetLastError();
            return G3X_ERR_NOMEM;
        }
        gs.bytes = need;
    }
    d.z = gs.z;
    const cudaStream_t st = (cudaStream_t)stream;
    d.range = nullptr;
    d.order = nullptr;
    if (!direct && (rc = pair_order(ctx, d_jobs, n, groups ? kGlobalGroupClasses : 0, lanes, st, &d.order, &d.range)))
        return rc;
    if (cudaMemsetAsync(gs.queue, 0, (kGlobalGroupClasses + 1) * sizeof(int32_t), st) != cudaSuccess) return G3X_ERR_CUDA;
    if (groups) {
        GlobalDesc g = d;
        g.zwarp = zgroup;
        g.queue = gs.queue;
        if ((rc = launch_global16(g, sp, gblocks, st))) return rc;
    }
    if (lanes) {
        d.zwarp = zlane;
        d.queue = gs.queue + kGlobalGroupClasses;
        d.range += 2 * (groups ? kGlobalGroupClasses : 0);
        kern<<<blocks, 32 * wpb, wpb * warp_smem, st>>>(d, sp);
    }
    return cudaPeekAtLastError() == cudaSuccess ? G3X_OK : G3X_ERR_CUDA;
}
