// g3x_global.cuh -- what the two global-alignment kernels share (g3x_global.cu: a job per lane;
// g3x_global16.cu: a job per group of lanes).
#pragma once
#include <cuda_runtime.h>
#include "g3x_core.h"
#include "g3x_internal.h"
#include "g3x_stage.cuh"

namespace g3x {

constexpr int32_t kNegInf = -0x40000000;   // outside the band (ksw.cu:548)

struct GlobalDesc {
    const g3x_job_t* jobs;
    const uint32_t* codes;
    const uint32_t* nmask;
    int32_t* score;
    uint32_t* cigar;
    int32_t* n_cigar;
    int32_t* status;
    uint8_t* z;            // direction bytes: per warp slot zwarp bytes
    int64_t zwarp;
    int32_t* queue;
    const int32_t* order;  // queue slot -> job, jobs alike in row count and width together
    const int32_t* range;  // [offset, count] of this launch's jobs in order, per class
    int32_t* nm;           // optional: NM per job
    char* md;              // optional: MD string per job, md_stride bytes each
    int32_t n, qmax, tmax, wmax, ncol, ring, stride, md_stride;
    int64_t n_bases;       // bases the planes hold: jobs reaching past them are refused
};

// Appends the decimal digits of v (>= 0) to buf[l ...] while they fit below cap.
__device__ __forceinline__ bool put_uint(char* buf, int& l, int cap, int v) {
    char tmp[12];
    int k = 0;
    do { tmp[k++] = (char)('0' + v % 10); v /= 10; } while (v);
    if (l + k >= cap) return false;
    while (k) buf[l++] = tmp[--k];
    return true;
}

// Sixteen codes as nibbles with every N as 4, whatever its 2-bit code.
__device__ __forceinline__ uint64_t plain_nibbles(uint64_t v) {
    const uint64_t n = v >> 2 & 0x1111111111111111ull;
    return v & ~(n | n << 1);
}

// NM and the MD string along a CIGAR (aux.cu:2831-2860), by one lane: qchunk(c) and tchunk(c) are the
// codes of bases 16 c .. 16 c + 15 of the query and the target (plain_nibbles).  A run of matches
// is compared up to sixteen bases at a time (base by base this was 28% of a batch of 200k pairs).
// Returns false when MD does not fit; md is then empty.
template <typename Q, typename T>
__device__ __forceinline__ bool write_nm_md(const GlobalDesc& d, int job, uint32_t flags, const uint32_t* cg, int n,
                                            Q qchunk, T tchunk) {
    const char* alpha = (flags & 4u) ? "TGCAN" : "ACGTN";
    char* md = d.md + (int64_t)job * d.md_stride;
    int x = 0, y = 0, u = 0, n_mm = 0, n_gap = 0, l = 0;
    bool ok = true;
    for (int k = 0; k < n && ok; ++k) {
        const int op = (int)(cg[k] & 0xFu), len = (int)(cg[k] >> 4);
        if (op == 0) {
            for (int i = 0; i < len && ok;) {
                const int xo = (x + i) & 15, yo = (y + i) & 15;
                const int m = min(16 - max(xo, yo), len - i);
                const uint64_t b = tchunk((y + i) >> 4) >> (4 * yo);
                uint64_t diff = (qchunk((x + i) >> 4) >> (4 * xo)) ^ b;
                if (m < 16) diff &= ((uint64_t)1 << (4 * m)) - 1u;
                int done = 0;
                while (diff && ok) {
                    const int at = (__ffsll((long long)diff) - 1) >> 2;
                    ok = put_uint(md, l, d.md_stride - 1, u + at - done);
                    if (ok && l + 1 < d.md_stride) md[l++] = alpha[(b >> (4 * at)) & 7u]; else ok = false;
                    ++n_mm; u = 0; done = at + 1;
                    diff &= ~((uint64_t)0xF << (4 * at));
                }
                u += m - done;
                i += m;
            }
            x += len; y += len;
        } else if (op == 2) {
            if (k > 0 && k < n - 1) {
                ok = put_uint(md, l, d.md_stride - 1, u);
                if (ok && l + 1 < d.md_stride) md[l++] = '^'; else ok = false;
                for (int i = 0; i < len && ok; ++i) {
                    if (l + 1 < d.md_stride) md[l++] = alpha[(tchunk((y + i) >> 4) >> (4 * ((y + i) & 15))) & 7u];
                    else ok = false;
                }
                u = 0; n_gap += len;
            }
            y += len;
        } else if (op == 1) {
            x += len; n_gap += len;
        }
    }
    ok = ok && put_uint(md, l, d.md_stride - 1, u);
    md[ok ? l : 0] = 0;
    d.nm[job] = ok ? n_mm + n_gap : 0;
    return ok;
}

// The group kernel (g3x_global16.cu): classes of a sorted batch by the band's columns, and the
// largest half band it holds.
constexpr int kGlobalGroupClasses = 5;     // groups of 2, 4, 8, 16, 32 lanes: 16 .. 256 columns
constexpr int kGlobalGroupMaxW = 127;      // 2 w + 1 columns in 256
int launch_global16(const GlobalDesc& d, const ScoreParams& sp, int blocks, cudaStream_t st);
int global16_blocks();                     // blocks that fill the device
constexpr int kGlobal16Warps = 2;          // warps per block
// Direction nibbles of one warp: 32 lanes x 8 columns a row.
inline int64_t global16_warp_bytes(int tmax) { return (int64_t)tmax * 128; }

}  // namespace g3x
