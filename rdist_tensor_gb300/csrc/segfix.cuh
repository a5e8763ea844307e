// Carry fix-up of the chunked segmented reductions over row-sorted hits
// (sort_lookup.hpp:347-371 computes the same row sums serially): rows that
// cross a chunk border are summed from the chunks' carries in chunk order.
#pragma once
#include "engine.cuh"

namespace exafac {

constexpr uint32_t kNoRow = 0xffffffffu;  // rows are < 2^32 - 1
constexpr int kLongSpan = 256;             // chunks from which an FP64 row takes a whole block
constexpr int kLongBatch = 8;               // chunks a warp looks at before the block sums the long rows among them

// Crossing rows, one warp per chunk c0 whose last row continues: the row's
// carries carry_last[c0] + sum over c in (c0, c1] of carry_first[c], c1 the
// last chunk that starts inside the row: the chunk of the row's last hit,
// seg_start[carry_seg[c0] + 1] - 1, when the run starts are given (one load
// however long the row); otherwise the chunks that do form a prefix of c0+1,
// c0+2, ..., whose end is searched.  Spans of up to 32 chunks
// (almost every row): lane = column, chunks summed in order.  Longer spans
// (the hot rows): lane l sums chunks c0+1+l, c0+1+l+32, ... over all 32 padded
// columns, then a butterfly reduce-scatter leaves column l's total in lane l.
// FP64 spans of more than kLongSpan chunks take the whole block.  The order of
// a row's sum depends on its span alone, so results are reproducible run to run.
// carry_seg != null: Mc is compact and the row's output index is carry_seg[c0].
template <typename TA, int kChunk, int CB = 1>  // CB column blocks of 32 (carry stride 32 CB)
__global__ void __launch_bounds__(256) segfix_kernel(int R, int ldm, const int64_t* __restrict__ counters, int64_t cap,
                                                     const uint32_t* __restrict__ carry_row,
                                                     const uint32_t* __restrict__ carry_seg,
                                                     const int64_t* __restrict__ seg_start,
                                                     const uint32_t* __restrict__ keys,
                                                     const TA* __restrict__ carry_first,
                                                     const TA* __restrict__ carry_last, TA* __restrict__ Mc) {
    pdl_wait();
    pdl_trigger();
    const int64_t H = min(counters[1], cap);
    const int64_t nchunks = (H + kChunk - 1) / kChunk;
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const unsigned full = 0xffffffffu;
    constexpr bool kBlockSpans = sizeof(TA) == 8;
    __shared__ int nlong;
    __shared__ int64_t longs[kBlockSpans ? 8 * kLongBatch : 1][2];
    auto one = [&](int64_t c0) {
        const uint32_t row = carry_row[c0];
        if (row == kNoRow) return;
        const int64_t out = carry_seg ? (int64_t)carry_seg[c0] : (int64_t)row;
        int64_t c1 = c0;
        if (seg_start) {
            c1 = (min(seg_start[out + 1], H) - 1) / kChunk;
        } else {
            // the last chunk that starts inside the row: the keys ascend, so a
            // 32-way search (a row of 1e6 nonzeros spans 8000 chunks)
            int64_t lo = c0, hi = nchunks;  // keys[lo kChunk ..] on (or c0), hi off (or the end)
            while (hi - lo > 1) {
                const int64_t step = (hi - lo + 31) / 32;
                const int64_t m = lo + (lane + 1) * step;
                const bool on = m < hi && keys[m * kChunk] == row;
                const int cnt = __popc(__ballot_sync(full, on));
                hi = min(hi, lo + (cnt + 1) * step);
                lo += cnt * step;
            }
            c1 = lo;
        }
        // Columns R .. ldm - 1 of a padded FP32 row are written as zeros: the
        // solve reads whole rows, and the row's memory holds whatever the
        // workspace held before (a NaN there would survive the product with
        // Phi's zero padding).
        if (c1 - c0 <= 32) {  // short span: column per lane, chunks in order
            for (int cb = 0; cb < CB; cb++) {
                const int col = 32 * cb + lane;
                if (col >= R) {
                    if (col < ldm) Mc[out * ldm + col] = TA(0);
                    continue;
                }
                TA v = carry_last[c0 * (32 * CB) + col];
#pragma unroll 4
                for (int64_t m = c0 + 1; m <= c1; m++) v += carry_first[m * (32 * CB) + col];
                Mc[out * ldm + col] = v;
            }
            return;
        }
        if (kBlockSpans && c1 - c0 > kLongSpan) {  // a hot row: left to the whole block, below
            if (lane == 0) {
                const int at = atomicAdd(&nlong, 1);
                longs[at][0] = c0;
                longs[at][1] = c1;
            }
            return;
        }
        for (int cb = 0; cb < CB; cb++) {
            TA acc[32];
#pragma unroll
            for (int k = 0; k < 32; k++) acc[k] = 0;
            for (int64_t m = c0 + 1 + lane; m <= c1; m += 32) {
                const TA* src = carry_first + m * (32 * CB) + 32 * cb;
#pragma unroll
                for (int k = 0; k < 32; k++) acc[k] += src[k];
            }
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) {
                const bool upper = (lane & off) != 0;
#pragma unroll
                for (int k = 0; k < off; k++) {
                    const TA send = upper ? acc[k] : acc[k + off];
                    const TA keep = upper ? acc[k + off] : acc[k];
                    acc[k] = keep + __shfl_xor_sync(full, send, off);
                }
            }
            const int col = 32 * cb + lane;
            if (col < R) Mc[out * ldm + col] = carry_last[c0 * (32 * CB) + col] + acc[0];
            else if (col < ldm) Mc[out * ldm + col] = TA(0);
        }
    };
    if (!kBlockSpans) {
        for (int64_t c0 = warp; c0 < nchunks; c0 += nwarps) one(c0);
        return;
    }
    // A block's warps look at kLongBatch chunks each, then the block sums the
    // long rows among them: warp w takes the chunks c0 + 1 + w, + 8, ... with
    // lane = column, the warps' sums are added in warp order (one warp took 0.9
    // ms over the hottest row of 1e7 Zipf nonzeros, the block 0.05)
    __shared__ TA wsum[8][32];
    const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int64_t b0 = (int64_t)blockIdx.x * nw; b0 < nchunks; b0 += kLongBatch * nwarps) {
        if (threadIdx.x == 0) nlong = 0;
        __syncthreads();
        for (int k = 0; k < kLongBatch; k++) {
            const int64_t c0 = b0 + w + k * nwarps;
            if (c0 < nchunks) one(c0);
        }
        __syncthreads();
        const int todo = nlong;
        for (int q = 0; q < todo; q++) {
            const int64_t c0 = longs[q][0], c1 = longs[q][1];
            const int64_t out = carry_seg ? (int64_t)carry_seg[c0] : (int64_t)carry_row[c0];
            for (int cb = 0; cb < CB; cb++) {
                TA s[8];
#pragma unroll
                for (int k = 0; k < 8; k++) s[k] = TA(0);
                int64_t m = c0 + 1 + w;
                for (; m + 7 * nw <= c1; m += 8 * nw) {
                    TA v[8];
#pragma unroll
                    for (int k = 0; k < 8; k++) v[k] = carry_first[(m + k * nw) * (32 * CB) + 32 * cb + lane];
#pragma unroll
                    for (int k = 0; k < 8; k++) s[k] += v[k];
                }
                for (; m <= c1; m += nw) s[0] += carry_first[m * (32 * CB) + 32 * cb + lane];
                wsum[w][lane] = ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
                __syncthreads();
                const int col = 32 * cb + lane;
                if (w == 0 && col < ldm) {
                    TA v = TA(0);
                    if (col < R) {
                        v = carry_last[c0 * (32 * CB) + col];
                        for (int k = 0; k < nw; k++) v += wsum[k][lane];
                    }
                    Mc[out * ldm + col] = v;
                }
                __syncthreads();
            }
        }
        __syncthreads();  // nlong is read
    }
}

}  // namespace exafac
