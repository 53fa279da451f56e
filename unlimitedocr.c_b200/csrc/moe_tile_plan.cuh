// Tile lists of the routed grouped GEMMs, written by whichever kernel has just computed the experts' row ranges.
#pragma once

#include "moe_common.cuh"

namespace uocr {

constexpr int kTileN = 192;          // tokens per tile: a tcgen05.mma costs 91 cycles up to N = 128 and 96 at N = 192 (measured),
                                     // and two accumulators of 192 columns leave 128 columns for the weight operand
constexpr uint32_t kMaxSegments = 256;

// For every segment with rows, gate/up tiles of (192 tokens, one weight-row tile) and down tiles likewise.  Entries are
// {expert, weight-row tile, first row, rows}; counts[0/1] are the list lengths.  Segment e holds the rows
// offsets[e] .. offsets[e + 1] and uses the weights of expert expert_base + e % expert_mod (single GPU: base 0, mod E;
// expert-parallel ranks receive one segment per (source rank, local expert)).
// The lists start with the segment that has the most rows (ties: lower index first): the persistent GEMM kernel deals
// tiles to its CTAs in list order, so the long segments are under way first and the short ones fill the tail.
// All threads of one CTA (at least E, a multiple of 32) call this; order [256] and first_tile [257] are shared memory, and
// offsets is readable by every thread.  The entries are written by all threads, entry i finding its segment by bisection.
__device__ __forceinline__ void write_tile_lists(const uint32_t *offsets, uint32_t E, uint32_t expert_base, uint32_t expert_mod,
                                                 const TileLists &out, uint32_t *order, uint32_t *first_tile) {
    const uint32_t tid = threadIdx.x;
    if (tid < E) {
        const uint32_t c = offsets[tid + 1] - offsets[tid];
        uint32_t rank = 0;
        for (uint32_t j = 0; j < E; ++j) {
            const uint32_t cj = offsets[j + 1] - offsets[j];
            rank += (cj > c || (cj == c && j < tid)) ? 1u : 0u;
        }
        order[rank] = tid;
    }
    __syncthreads();
    if (tid < 32) {                                        // token tiles before the segment of each rank
        const uint32_t per = (E + 31u) / 32u, k0 = min(tid * per, E), k1 = min(k0 + per, E);
        uint32_t sum = 0;
        for (uint32_t k = k0; k < k1; ++k) sum += (offsets[order[k] + 1] - offsets[order[k]] + kTileN - 1) / kTileN;
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (tid >= (uint32_t)o) incl += v;
        }
        uint32_t run = incl - sum;
        for (uint32_t k = k0; k < k1; ++k) {
            first_tile[k] = run;
            run += (offsets[order[k] + 1] - offsets[order[k]] + kTileN - 1) / kTileN;
        }
        if (tid == 31) {
            first_tile[E] = incl;
            out.counts[0] = incl * out.gu_mtiles;
            out.counts[1] = incl * out.dn_mtiles;
        }
    }
    __syncthreads();
    const uint32_t token_tiles = first_tile[E];
    for (uint32_t tt = tid; tt < token_tiles; tt += blockDim.x) {
        uint32_t lo = 0, hi = E;                           // the rank k with first_tile[k] <= tt < first_tile[k + 1]
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) / 2;
            if (first_tile[mid] <= tt) lo = mid; else hi = mid;
        }
        const uint32_t e = order[lo], t = tt - first_tile[lo];
        const uint32_t seg0 = offsets[e], cnt = offsets[e + 1] - seg0;
        uint4 entry = make_uint4(expert_base + e % expert_mod, 0u, seg0 + t * kTileN, min((uint32_t)kTileN, cnt - t * kTileN));
        for (uint32_t m = 0; m < out.gu_mtiles; ++m) { entry.y = m; out.gu[tt * out.gu_mtiles + m] = entry; }
        for (uint32_t m = 0; m < out.dn_mtiles; ++m) { entry.y = m; out.dn[tt * out.dn_mtiles + m] = entry; }
    }
}

}  // namespace uocr
