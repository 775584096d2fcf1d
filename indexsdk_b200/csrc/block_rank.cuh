// Rank search by a thread block.
#pragma once
#include <stdint.h>

namespace b200 {

constexpr int kRankBins = 1024;
struct RankScratch {
    uint32_t hist[kRankBins];
    uint32_t warp[32];
    uint32_t lo, hi, n, bin, below;
};

// r-th smallest (1-based) of the keys a block of NT threads holds; visit(f) calls f(key) for each of the
// calling thread's keys, the same ones every time.  Fewer than r keys: 0xFFFFFFFF.
// The digits are cut out of the range the keys really span, not out of the 32-bit word: the candidates of
// a query share their leading byte or two, so a digit at a fixed place sends all of them to one counter,
// whose atomics then run one after the other (22 us for the 1 500 candidates of a single query; 1 024 bins
// over the spanned range: two or three passes, almost no collisions).  After `passes` passes the upper
// edge of the bin is returned (a bound from above, 2^-20 of the range wide after two) unless the rank is
// settled before; passes = 4 always settles it.  Every thread of the block must call this.
struct RankResult {
    uint32_t lo, hi;   // the r-th smallest key lies in [lo, hi] (both 0xFFFFFFFF: fewer than r keys)
    uint32_t left;     // its rank among the keys in there
};
template <int NT, typename Visit>
__device__ __forceinline__ RankResult block_rank32(Visit visit, uint32_t r, RankScratch& s, int passes) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    constexpr int kPer = kRankBins / NT;
    if (threadIdx.x == 0) {
        s.lo = 0xFFFFFFFFu;
        s.hi = 0u;
        s.n = 0u;
    }
    __syncthreads();
    {
        uint32_t lo = 0xFFFFFFFFu, hi = 0u, n = 0u;
        visit([&](uint32_t v) {
            lo = min(lo, v);
            hi = max(hi, v);
            ++n;
        });
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        n = __reduce_add_sync(0xffffffffu, n);
        if (lane == 0 && n > 0) {
            atomicMin(&s.lo, lo);
            atomicMax(&s.hi, hi);
            atomicAdd(&s.n, n);
        }
    }
    __syncthreads();
    uint32_t lo = s.lo, hi = s.hi;
    if (s.n < r) return RankResult{0xFFFFFFFFu, 0xFFFFFFFFu, 0u};
    for (int pass = 0; pass < passes && lo != hi; ++pass) {
        const int shift = max(0, 22 - __clz(hi - lo));
        for (int b = threadIdx.x; b < kRankBins; b += NT) s.hist[b] = 0u;
        __syncthreads();
        visit([&](uint32_t v) {
            if (v >= lo && v <= hi) atomicAdd(&s.hist[(v - lo) >> shift], 1u);
        });
        __syncthreads();
        uint32_t mine[kPer], sum = 0;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            mine[j] = s.hist[threadIdx.x * kPer + j];
            sum += mine[j];
        }
        uint32_t incl = sum;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += u;
        }
        if (lane == 31) s.warp[w] = incl;
        __syncthreads();
        uint32_t before = incl - sum;
        for (int i = 0; i < w; ++i) before += s.warp[i];
        if (before < r && r <= before + sum) {
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                if (before < r && r <= before + mine[j]) {
                    s.bin = threadIdx.x * kPer + j;
                    s.below = before;
                }
                before += mine[j];
            }
        }
        __syncthreads();
        lo += s.bin << shift;
        const uint32_t top = lo + ((1u << shift) - 1u);
        hi = top < hi && top >= lo ? top : hi;
        r -= s.below;
    }
    __syncthreads();   // the scratch may be reused
    return RankResult{lo, hi, r};
}
template <int NT, typename Visit>
__device__ __forceinline__ uint32_t block_kth32(Visit visit, uint32_t r, RankScratch& s, int passes) {
    return block_rank32<NT>(visit, r, s, passes).hi;
}

}  // namespace b200
