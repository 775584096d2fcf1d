#include "select.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include "block_rank.cuh"
#include "cos16.cuh"

#include "common.cuh"
#include "dist_gemm.cuh"
#include "smem_limit.h"

namespace b200 {
namespace {

constexpr int kSelThreads = 256;
constexpr int kSmallSet = 512;   // candidate sets up to this size are sorted in shared memory

// Three bf16 terms whose sum reproduces v to 24 significant bits (an infinite v stays in the
// first term).
__device__ __forceinline__ void split3_bf16(float v, __nv_bfloat16* out) {
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    float r = isfinite(v) ? v - __bfloat162float(h) : 0.f;
    const __nv_bfloat16 m = __float2bfloat16_rn(r);
    r -= __bfloat162float(m);
    out[0] = h;
    out[1] = m;
    out[2] = __float2bfloat16_rn(r);
}

// Writes the threshold of candidate row q and what else becomes known with it, so that no launch of
// its own is spent on either (a launch in the chain of a single query costs about 3.5 us):
//   fold.counts : the row's candidate counter starts at zero
//   fold.q_bf16 / fold.bias : the threshold in the form the folded GEMM tests, c = tau / 2 (L2) or tau
//     (inner product), as three bf16 terms of the query operand or, for a segmented base, as one float
//     per candidate row.  c is first raised by a margin for the fp32 accumulation inside the tensor core:
//     d + 16 additions of terms whose partial sums stay below M = |q||y|max + |y|max^2 / 2 + |tau| perturb
//     a key by less than 2^-14.8 M in either pass, and 2^-12 M covers the sample pass, the full pass and
//     the threshold's own term together, so no key <= tau is missed.
__device__ __forceinline__ void store_tau(int q, uint32_t ord, uint32_t* tau, const TauFold& fold) {
    tau[q] = ord;
    if (fold.counts) fold.counts[q] = 0u;
    if (!fold.qnorm) return;
    const float t = ord_to_float(ord);
    const float qn = fold.qnorm[fold.q_mod > 0 ? q % fold.q_mod : q];
    const float reach = sqrtf(qn) * fold.ymax + 0.5f * fold.ymax * fold.ymax;
    float c = t + 0.000244140625f * (reach + fabsf(t));
    if (fold.metric == kMetricL2) c *= 0.5f;
    if (fold.bias) {
        fold.bias[q] = c;
    } else {
        // A query whose terms may leave the range of a float (0 x infinity included): with a threshold among
        // them a sum may be NaN where the key is a number.  Nothing passes, and the row counts as overflowed: the
        // caller searches for it without a threshold.
        if (!(reach <= 1e38f)) {
            c = __int_as_float(0xff800000);
            if (fold.counts) fold.counts[q] = 0x80000000u;
        }
        const int dp = fold.d + kFoldCols;
        // columns d + 3 .. d + 5 lie in one 8-column group (d is a multiple of 16), so they are
        // consecutive in the packed layout as well
        split3_bf16(c, static_cast<__nv_bfloat16*>(fold.q_bf16) +
                           operand_elem(packed_operands(kKindBF16, dp), q, fold.d + 3, dp, kTileQ));
    }
}

// Copies the entries of row[0..n) that are in use (not kCandInvalid) to out[0..limit); returns their number,
// which may exceed the limit (out is then incomplete).  Eight loads per thread are in flight: with one the
// copy is a chain of memory latencies.  fill: shared counter.  Every thread of the block must call this.
template <int NT>
__device__ __forceinline__ uint32_t block_compact(const uint64_t* row, uint32_t n, uint64_t* out, uint32_t limit, uint32_t* fill) {
    const int lane = threadIdx.x & 31;
    constexpr int U = 8;
    if (threadIdx.x == 0) *fill = 0u;
    __syncthreads();
    for (uint32_t i0 = threadIdx.x - lane; i0 < n; i0 += U * NT) {
        uint64_t v[U];
        uint32_t have = 0;
#pragma unroll
        for (int j = 0; j < U; ++j) {
            const uint32_t i = i0 + j * NT + lane;
            v[j] = i < n ? row[i] : kCandInvalid;
            have += v[j] != kCandInvalid ? 1u : 0u;
        }
        uint32_t before = have;   // exclusive prefix over the lanes
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, before, off);
            if (lane >= off) before += u;
        }
        const uint32_t all = __shfl_sync(0xffffffffu, before, 31);
        uint32_t slot = 0;
        if (lane == 0 && all) slot = atomicAdd(fill, all);
        slot = __shfl_sync(0xffffffffu, slot, 0) + before - have;
#pragma unroll
        for (int j = 0; j < U; ++j)
            if (v[j] != kCandInvalid) {
                if (slot < limit) out[slot] = v[j];
                ++slot;
            }
    }
    __syncthreads();
    return *fill;
}

constexpr uint32_t kKthStage = 8192;   // burst minima staged in shared memory

// A threshold may be any bound from above: two passes of the rank search (2^-20 of the range) do.
__global__ void __launch_bounds__(kSelThreads)
kth_threshold_kernel(const uint32_t* mins, int stride, int n, int k, const float* eps, uint32_t tau_all,
                     uint32_t* tau, const TauFold fold) {
    extern __shared__ uint32_t kth_keys[];   // min(n, kKthStage)
    __shared__ RankScratch rank;
    const int q = blockIdx.x;
    if (n < k) {
        if (threadIdx.x == 0) store_tau(q, tau_all, tau, fold);
        return;
    }
    const uint32_t* row = mins + static_cast<int64_t>(q) * stride;
    const bool staged = n <= static_cast<int>(kKthStage);
    if (staged) {
        for (int i = threadIdx.x; i < n; i += kSelThreads) kth_keys[i] = row[i];
        __syncthreads();
    }
    const uint32_t* keys = staged ? kth_keys : row;
    uint32_t kth = block_kth32<kSelThreads>(
        [&](auto&& f) {
            for (int i = threadIdx.x; i < n; i += kSelThreads)
                if (keys[i] != 0xFFFFFFFFu) f(keys[i]);   // bursts that were not visited do not widen the range
        },
        static_cast<uint32_t>(k), rank, 2);
    if (threadIdx.x == 0) {
        if (eps) {
            float f = ord_to_float(kth);
            f = f + 2.f * eps[fold.q_mod > 0 ? q % fold.q_mod : q];
            f = f + fabsf(f) * 9.5367431640625e-07f;  // one part in 2^20 against the rounding of the adds
            kth = (f != f) ? tau_all : float_to_ord(f);
        }
        store_tau(q, kth > tau_all ? tau_all : kth, tau, fold);
    }
}

// Drops candidates that cannot reach the exact top-k before the (costly) exact refinement.  The
// keys in the list are approximate, |approx - exact| <= eps for every candidate.  With A_k the k-th
// smallest approximate key, k candidates have exact keys <= A_k + eps, so the exact k-th key is
// <= A_k + eps and every member of the exact top-k has an approximate key <= A_k + 2 eps; all
// others are overwritten with the "invalid" marker.  A constant offset common to a row's keys
// cancels out of this argument.
constexpr uint32_t kPruneKeys = 4096;    // entries staged in shared memory for the rank search
constexpr int kPruneKeep = 2048;         // survivors staged for the in-place compaction

// Limit on the approximate key for a row whose k-th smallest (or a bound on it) is kth; false: no limit.
__device__ __forceinline__ bool prune_limit(uint32_t kth, float eps, uint32_t* lim) {
    if (kth == 0xFFFFFFFFu) return false;   // fewer than k real candidates
    float f = ord_to_float(kth);
    f = f + 2.f * eps;
    f = f + fabsf(f) * 9.5367431640625e-07f + eps * 0.125f;   // slack for the adds and the accumulation
    if (f != f) return false;
    *lim = float_to_ord(f);
    return true;
}

// Tightens a threshold part-way through the full pass: the candidates found so far (in the tiles
// already visited) contain k keys <= their k-th smallest key A_k, so A_k bounds the final k-th key
// from above and the remaining tiles need only admit keys <= min(tau, A_k (+ 2 eps where keys are
// approximate)).  Rows whose list overflowed or holds fewer than k candidates keep their threshold.
__global__ void __launch_bounds__(kSelThreads)
tighten_tau_kernel(const uint64_t* cand, const uint32_t* counts, uint32_t cap, int k, const float* eps,
                   uint32_t* tau, const TauFold fold) {
    __shared__ RankScratch rank;
    __shared__ uint32_t keys[kPruneKeys];
    const int q = blockIdx.x;
    const uint64_t* row = cand + static_cast<int64_t>(q) * cap;
    const uint32_t n = counts[q];
    if (n > cap || n < static_cast<uint32_t>(k)) return;
    const bool staged = n <= kPruneKeys;
    if (staged) {
        for (uint32_t i = threadIdx.x; i < n; i += kSelThreads) keys[i] = static_cast<uint32_t>(row[i] >> 32);
        __syncthreads();
    }
    uint32_t kth = block_kth32<kSelThreads>(
        [&](auto&& f) {
            for (uint32_t i = threadIdx.x; i < n; i += kSelThreads) {
                const uint32_t v = staged ? keys[i] : static_cast<uint32_t>(row[i] >> 32);
                if (v != 0xFFFFFFFFu) f(v);   // unused slots
            }
        },
        static_cast<uint32_t>(k), rank, 2);
    if (kth == 0xFFFFFFFFu) return;   // fewer than k real candidates
    if (threadIdx.x == 0) {
        if (eps) {
            float f = ord_to_float(kth);
            f = f + 2.f * eps[q] + eps[q] * 0.125f;
            f = f + fabsf(f) * 9.5367431640625e-07f;
            if (f != f) return;
            kth = float_to_ord(f);
        }
        if (kth < tau[q]) store_tau(q, kth, tau, fold);
    }
}

__global__ void __launch_bounds__(kSelThreads)
prune_candidates_kernel(uint64_t* cand, uint32_t* counts, uint32_t cap, int k, const float* eps) {
    __shared__ RankScratch rank;
    __shared__ uint32_t sh_fill;
    __shared__ uint32_t keys[kPruneKeys];
    __shared__ uint64_t keep[kPruneKeep];
    const int q = blockIdx.x;
    uint64_t* row = cand + static_cast<int64_t>(q) * cap;
    const uint32_t n = counts[q];
    if (n > cap) return;   // overflowed row: left as it is for the selection kernel to flag
    if (n <= static_cast<uint32_t>(k)) return;
    const bool staged = n <= kPruneKeys;
    if (staged) {
        for (uint32_t i = threadIdx.x; i < n; i += kSelThreads) keys[i] = static_cast<uint32_t>(row[i] >> 32);
        __syncthreads();
    }
    const uint32_t kth = block_kth32<kSelThreads>(
        [&](auto&& f) {
            for (uint32_t i = threadIdx.x; i < n; i += kSelThreads) {
                const uint32_t v = staged ? keys[i] : static_cast<uint32_t>(row[i] >> 32);
                if (v != 0xFFFFFFFFu) f(v);
            }
        },
        static_cast<uint32_t>(k), rank, 2);
    uint32_t lim_ord;
    if (!prune_limit(kth, eps[q], &lim_ord)) return;
    if (threadIdx.x == 0) sh_fill = 0;
    __syncthreads();
    // survivors go to shared memory first: the row is compacted in place
    for (uint32_t i = threadIdx.x; i < n; i += kSelThreads) {
        const uint64_t v = row[i];
        if (v != kCandInvalid && static_cast<uint32_t>(v >> 32) <= lim_ord) {
            const uint32_t slot = atomicAdd(&sh_fill, 1u);
            if (slot < static_cast<uint32_t>(kPruneKeep)) keep[slot] = v;
        }
    }
    __syncthreads();
    const uint32_t m = sh_fill;
    if (m <= static_cast<uint32_t>(kPruneKeep)) {
        for (uint32_t i = threadIdx.x; i < m; i += kSelThreads) row[i] = keep[i];
        if (threadIdx.x == 0) counts[q] = m;
    } else {
        // too many to stage: invalidate the losers where they are
        for (uint32_t i = threadIdx.x; i < n; i += kSelThreads) {
            const uint64_t v = row[i];
            if (v != kCandInvalid && static_cast<uint32_t>(v >> 32) > lim_ord) row[i] = kCandInvalid;
        }
    }
}

// The same threshold for short rows (n <= 32 * NPL), one WARP per query: the minima sit in
// registers, NPL per lane, and the k-th smallest is found bit by bit -- per bit every lane counts
// its values that agree with the bits fixed so far and have a 0 there, one warp reduction adds the
// counts.  The bits above the highest one in which the minima differ need no search, and 16 bits below
// it are enough: a threshold may be any bound from above (65 536 steps over the spanned range).
template <int NPL>
__global__ void __launch_bounds__(128)
kth_threshold_warp_kernel(const uint32_t* mins, int stride, int n, int nq, int k, const float* eps, uint32_t tau_all,
                          uint32_t* tau, const TauFold fold) {
    const int lane = threadIdx.x & 31;
    const int q = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (q >= nq) return;
    if (n < k) {
        if (lane == 0) store_tau(q, tau_all, tau, fold);
        return;
    }
    uint32_t v[NPL];
    const uint32_t* row = mins + static_cast<int64_t>(q) * stride;
    uint32_t all_and = 0xFFFFFFFFu, all_or = 0u, real = 0u;
#pragma unroll
    for (int j = 0; j < NPL; ++j) {
        const int i = j * 32 + lane;
        v[j] = i < n ? row[i] : 0xFFFFFFFFu;
        if (v[j] != 0xFFFFFFFFu) {   // (bursts that were not visited do not widen the range)
            all_and &= v[j];
            all_or |= v[j];
            ++real;
        }
    }
    real = __reduce_add_sync(0xffffffffu, real);
    if (real < static_cast<uint32_t>(k)) {
        if (lane == 0) store_tau(q, tau_all, tau, fold);
        return;
    }
    all_and = __reduce_and_sync(0xffffffffu, all_and);
    all_or = __reduce_or_sync(0xffffffffu, all_or);
    const uint32_t differ = all_and ^ all_or;
    const int top = 31 - __clz(differ);              // -1: all equal
    uint32_t mask = top >= 31 ? 0u : ~((2u << top) - 1u), prefix = all_and & mask, r = static_cast<uint32_t>(k);
    if (top < 0) {
        mask = 0xFFFFFFFFu;
        prefix = all_and;
    }
    for (int bit = top; bit >= 0 && bit > top - 16; --bit) {
        const uint32_t b = 1u << bit;
        uint32_t c = 0;
#pragma unroll
        for (int j = 0; j < NPL; ++j) c += ((v[j] & (mask | b)) == prefix) ? 1u : 0u;   // agrees so far, bit is 0
        c = __reduce_add_sync(0xffffffffu, c);
        if (r > c) {   // the k-th smallest has a 1 at this bit
            prefix |= b;
            r -= c;
        }
        mask |= b;
    }
    if (lane == 0) {
        uint32_t kth = prefix | ~mask;
        if (eps) {
            float f = ord_to_float(kth);
            f = f + 2.f * eps[fold.q_mod > 0 ? q % fold.q_mod : q];
            f = f + fabsf(f) * 9.5367431640625e-07f;  // one part in 2^20 against the rounding of the adds
            kth = (f != f) ? tau_all : float_to_ord(f);
        }
        store_tau(q, kth > tau_all ? tau_all : kth, tau, fold);
    }
}

__device__ __forceinline__ uint64_t shfl_xor_u64(uint64_t v, int m) {
    const uint32_t lo = __shfl_xor_sync(0xffffffffu, static_cast<uint32_t>(v), m);
    const uint32_t hi = __shfl_xor_sync(0xffffffffu, static_cast<uint32_t>(v >> 32), m);
    return static_cast<uint64_t>(hi) << 32 | lo;
}

// Ascending bitonic sort of P (a power of two, at least 64) values in shared memory by a block of NT threads.
// A warp holds 64 neighbouring values, two per lane, and does every step of stride 32 and less on them in
// registers: at P = 1 024, 10 steps and 5 visits go through shared memory and a barrier instead of 55 steps
// (4 096 selections of k = 1 000: 507 -> 360 us).
template <int NT>
__device__ __forceinline__ void bitonic_sort_u64(uint64_t* s, int P) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto in_registers = [&](int size_first, int size_last) {
        for (int seg = warp; seg < P / 64; seg += NT / 32) {
            const int e = seg * 64 + 2 * lane;
            uint64_t x0 = s[e], x1 = s[e + 1];
            for (int size = size_first; size <= size_last; size <<= 1) {
                const bool up = (e & size) == 0;   // (size >= 2: the same for both values)
                for (int stride = size >> 1 < 32 ? size >> 1 : 32; stride > 1; stride >>= 1) {
                    const int m = stride >> 1;
                    const uint64_t o0 = shfl_xor_u64(x0, m), o1 = shfl_xor_u64(x1, m);
                    const bool keep_min = ((lane & m) == 0) == up;
                    x0 = keep_min == (o0 < x0) ? o0 : x0;
                    x1 = keep_min == (o1 < x1) ? o1 : x1;
                }
                if ((x0 > x1) == up) {
                    const uint64_t t = x0;
                    x0 = x1;
                    x1 = t;
                }
            }
            s[e] = x0;
            s[e + 1] = x1;
        }
        __syncthreads();
    };
    in_registers(2, 64);
    for (int size = 128; size <= P; size <<= 1) {
        for (int stride = size >> 1; stride >= 64; stride >>= 1) {
            for (int i = threadIdx.x; i < P / 2; i += NT) {
                const int lo = 2 * i - (i & (stride - 1));
                const int hi = lo + stride;
                const bool up = (lo & size) == 0;
                const uint64_t a = s[lo], b = s[hi];
                if ((a > b) == up) {
                    s[lo] = b;
                    s[hi] = a;
                }
            }
            __syncthreads();
        }
        in_registers(size, size);
    }
}

__device__ __forceinline__ void report_error(const EmitArgs& e) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && e.err_host && *e.err) *e.err_host = *e.err;
}

// Result j of query row q: the selected candidate's distance and label.
__device__ __forceinline__ void emit_one(const EmitArgs& e, int q, int j, uint64_t c) {
    const int orow = e.qmap ? e.qmap[q] : q;
    float dist;
    int64_t label;
    if (c == kCandInvalid) {
        dist = 3.402823466e+38f;  // FLT_MAX padding, label -1
        label = -1;
    } else {
        const int qn = e.q_mod > 0 ? q % e.q_mod : q;   // row of the query norms
        const uint32_t ok = static_cast<uint32_t>(c >> 32), pos = static_cast<uint32_t>(c);
        if (e.members) {
            const MemberView& mv = e.members[q / e.q_mod];
            label = mv.labels[static_cast<int64_t>(pos) - mv.first];
        } else {
            label = e.labels ? e.labels[pos] : static_cast<int64_t>(pos);
        }
        if (e.mode == 2) {
            int32_t kv = ord_to_int(ok);
            if (e.metric == kMetricL2) dist = static_cast<float>(kv + static_cast<const int32_t*>(e.qnorm)[qn]);
            else if (e.metric == kMetricCos) dist = cos16_value(-kv);
            else dist = static_cast<float>(-kv);
        } else {
            float kv = ord_to_float(ok);
            if (e.metric == kMetricL2) {
                if (e.mode == 0) {
                    kv += static_cast<const float*>(e.qnorm)[qn];
                    kv = kv < 0.f ? 0.f : kv;
                }
                dist = kv;
            } else {
                dist = -kv;
            }
        }
    }
    e.D[static_cast<int64_t>(orow) * e.ldk + j] = dist;
    e.I[static_cast<int64_t>(orow) * e.ldk + j] = label;
}

// The k smallest of a query's candidates, in order, straight to the results.
//   up to 512 candidates : every one is placed by its rank, counted against all others (candidates are
//                          distinct: positions are unique).
//   more                 : one pass of the rank search puts the k-th key into one of 1 024 bins.  What lies below
//                          the bin is in, the few in the bin are ranked among themselves, then k are sorted.  (A
//                          full rank search went over the list eight times: 4 096 queries, k = 1000, 7 500
//                          candidates each: 652 -> 507 us.)  A crowded bin (ties) takes the full search: the k-th
//                          key, then ties with it by position.
// The row is read once when its candidates fit `stage` entries of shared memory; longer ones are read
// from memory in every step.
template <int NT>
__global__ void __launch_bounds__(NT)
select_emit_kernel(const uint64_t* cand, const uint32_t* counts, uint32_t n_fixed, uint32_t cap, int P,
                   uint32_t stage, uint8_t* overflow, uint32_t* any_overflow, const EmitArgs e) {
    extern __shared__ uint64_t sel_sm[];   // P sorted entries, then the staged ones
    __shared__ RankScratch rank;
    __shared__ uint32_t sh_fill, sh_ties;
    __shared__ uint64_t in_bin[kSmallSet];
    const int q = blockIdx.x;
    const uint64_t* row = cand + static_cast<int64_t>(q) * cap;
    const uint32_t k = static_cast<uint32_t>(e.k);
    uint32_t n = counts ? counts[q] : n_fixed;
    report_error(e);
    if (n > cap) {
        if (threadIdx.x == 0) {
            if (overflow) overflow[q] = 1;
            if (any_overflow) *any_overflow = 1u;
        }
        for (uint32_t i = threadIdx.x; i < k; i += NT) emit_one(e, q, static_cast<int>(i), kCandInvalid);
        return;
    }
    uint64_t* sorted = sel_sm;
    uint64_t* held = sel_sm + P;
    const uint64_t* src = row;
    if (n <= 4 * stage) {   // (beyond that hardly any list fits)
        const uint32_t m = block_compact<NT>(row, n, held, stage, &sh_fill);
        if (m <= stage) {
            n = m;
            src = held;
        }
        if (m <= static_cast<uint32_t>(kSmallSet)) {
            for (uint32_t i = threadIdx.x; i < m; i += NT) {
                const uint64_t v = held[i];
                uint32_t r = 0;
#pragma unroll 8
                for (uint32_t j = 0; j < m; ++j) r += held[j] < v ? 1u : 0u;
                if (r < k) sorted[r] = v;
            }
            __syncthreads();   // results leave in order: consecutive stores
            for (uint32_t i = threadIdx.x; i < k; i += NT) emit_one(e, q, static_cast<int>(i), i < m ? sorted[i] : kCandInvalid);
            return;
        }
    }
    for (int i = threadIdx.x; i < P; i += NT) sorted[i] = kCandInvalid;
    auto each = [&](auto&& f) {
        for (uint32_t i = threadIdx.x; i < n; i += NT) {
            const uint64_t v = src[i];
            if (v != kCandInvalid) f(v);
        }
    };
    const RankResult bin = block_rank32<NT>([&](auto&& f) { each([&](uint64_t v) { f(static_cast<uint32_t>(v >> 32)); }); },
                                            k, rank, 1);
    if (rank.n >= k) {
        if (threadIdx.x == 0) {
            sh_fill = 0u;
            sh_ties = 0u;
        }
        __syncthreads();
        const int lane = threadIdx.x & 31;
        const uint32_t lt = (1u << lane) - 1u;
        for (uint32_t i0 = threadIdx.x - lane; i0 < n; i0 += NT) {
            const uint64_t v = i0 + lane < n ? src[i0 + lane] : kCandInvalid;
            const uint32_t key = static_cast<uint32_t>(v >> 32);
            const bool below = v != kCandInvalid && key < bin.lo, in = v != kCandInvalid && !below && key <= bin.hi;
            const unsigned bb = __ballot_sync(0xffffffffu, below), bi = __ballot_sync(0xffffffffu, in);
            uint32_t sb = 0, si = 0;
            if (lane == 0) {
                if (bb) sb = atomicAdd(&sh_fill, static_cast<uint32_t>(__popc(bb)));
                if (bi) si = atomicAdd(&sh_ties, static_cast<uint32_t>(__popc(bi)));
            }
            sb = __shfl_sync(0xffffffffu, sb, 0) + __popc(bb & lt);
            si = __shfl_sync(0xffffffffu, si, 0) + __popc(bi & lt);
            if (below) sorted[sb] = v;   // fewer than k
            if (in && si < static_cast<uint32_t>(kSmallSet)) in_bin[si] = v;
        }
        __syncthreads();
        const uint32_t ties = sh_ties, first = sh_fill;
        if (ties <= static_cast<uint32_t>(kSmallSet)) {
            for (uint32_t i = threadIdx.x; i < ties; i += NT) {
                const uint64_t v = in_bin[i];
                uint32_t r = 0;
#pragma unroll 4
                for (uint32_t j = 0; j < ties; ++j) r += in_bin[j] < v ? 1u : 0u;
                if (r < bin.left) sorted[first + r] = v;
            }
            __syncthreads();
            bitonic_sort_u64<NT>(sorted, P);
            for (int i = threadIdx.x; i < e.k; i += NT) emit_one(e, q, i, sorted[i]);
            return;
        }
        for (int i = threadIdx.x; i < P; i += NT) sorted[i] = kCandInvalid;
        __syncthreads();
    }
    // bounds of what is kept: everything unless there are more than k
    uint32_t kth = 0xFFFFFFFFu, pos_max = 0xFFFFFFFFu;
    const uint32_t found = block_kth32<NT>([&](auto&& f) { each([&](uint64_t v) { f(static_cast<uint32_t>(v >> 32)); }); },
                                           k, rank, 4);
    const bool enough = rank.n >= k;   // else all of them (rank.n is left as it was set)
    if (enough) {
        kth = found;
        if (threadIdx.x == 0) {
            sh_fill = 0u;
            sh_ties = 0u;
        }
        __syncthreads();
        uint32_t less = 0, ties = 0;
        each([&](uint64_t v) {
            less += static_cast<uint32_t>(v >> 32) < kth ? 1u : 0u;
            ties += static_cast<uint32_t>(v >> 32) == kth ? 1u : 0u;
        });
        less = __reduce_add_sync(0xffffffffu, less);
        ties = __reduce_add_sync(0xffffffffu, ties);
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(&sh_fill, less);
            atomicAdd(&sh_ties, ties);
        }
        __syncthreads();
        const uint32_t need = k - sh_fill;   // ties with the k-th key that belong to the result: the lowest positions
        if (need < sh_ties)
            pos_max = block_kth32<NT>(
                [&](auto&& f) { each([&](uint64_t v) { if (static_cast<uint32_t>(v >> 32) == kth) f(static_cast<uint32_t>(v)); }); },
                need, rank, 4);
    }
    __syncthreads();
    if (threadIdx.x == 0) sh_fill = 0u;
    __syncthreads();
    each([&](uint64_t v) {
        const uint32_t key = static_cast<uint32_t>(v >> 32);
        if (key < kth || (key == kth && static_cast<uint32_t>(v) <= pos_max)) {
            const uint32_t slot = atomicAdd(&sh_fill, 1u);
            if (slot < static_cast<uint32_t>(P)) sorted[slot] = v;
        }
    });
    __syncthreads();
    bitonic_sort_u64<NT>(sorted, P);
    for (int i = threadIdx.x; i < e.k; i += NT) emit_one(e, q, i, sorted[i]);
}

// ---- canonical fp32 distances of candidates ----
// Sequential fmaf over the dimensions, the arithmetic of the CPU oracle.  The chain of one candidate
// cannot be split over lanes, so a lane owns a candidate -- but the rows are fetched co-operatively: a warp
// reads the rows of its 32 candidates kRefChunk floats at a time, each row as one contiguous 128-byte
// piece spread over consecutive lanes (four cache lines per load instruction instead of 32), parks them
// in shared memory and every lane then walks its own row there.  Rows are padded by 4 floats: 8
// consecutive lanes reading one float4 each fall into 8 different 16-byte bank groups.
constexpr int kRefChunk = 32;     // small, so that many warps fit an SM: the kernel lives on memory-level parallelism
constexpr int kRefPitch = kRefChunk + 4;
constexpr uint32_t kRefWindow = 512;   // candidate slots compacted at a time

// Distance of this lane's candidate (row `pos` of xb) to the query qs (shared memory); lanes without
// one pass live = false.  rows: the warp's [32][kRefPitch] floats of shared memory.  Warp-collective.
__device__ __forceinline__ float refine_lane(const float* xb, const float* qs, float* rows, uint32_t pos, bool live, int d,
                                             int metric, int lane) {
    const uint32_t live_mask = __ballot_sync(0xffffffffu, live);
    float acc = 0.f;
    if (d % kRefChunk == 0) {
        // Whole chunks only: a lane stages the same 8 rows in every chunk, so their addresses are
        // formed once per pass, and the loads of the next chunk are in flight while the current
        // one is accumulated from shared memory.
        const int j = lane & 7;
        const float4* src[8];
        uint32_t okm = 0;
#pragma unroll
        for (int it = 0; it < 8; ++it) {
            const int r = it * 4 + (lane >> 3);
            const uint32_t pr = __shfl_sync(0xffffffffu, pos, r);
            src[it] = reinterpret_cast<const float4*>(xb + static_cast<int64_t>(pr) * d) + j;
            okm |= ((live_mask >> r) & 1u) << it;   // rows of unused slots are neither fetched nor read
        }
        float4* dst = reinterpret_cast<float4*>(rows + (lane >> 3) * kRefPitch + 4 * j);
        const float4* mine = reinterpret_cast<const float4*>(rows + lane * kRefPitch);
        float4 v[8];
#pragma unroll
        for (int it = 0; it < 8; ++it)
            if ((okm >> it) & 1u) v[it] = __ldg(src[it]);
        for (int ch0 = 0; ch0 < d; ch0 += kRefChunk) {
#pragma unroll
            for (int it = 0; it < 8; ++it)
                if ((okm >> it) & 1u) dst[it * kRefPitch] = v[it];   // 4 rows further per step
            __syncwarp();
            if (ch0 + kRefChunk < d) {
#pragma unroll
                for (int it = 0; it < 8; ++it)
                    if ((okm >> it) & 1u) v[it] = __ldg(src[it] + (ch0 + kRefChunk) / 4);
            }
            const float4* qv = reinterpret_cast<const float4*>(qs + ch0);
            if (live) {
                if (metric == kMetricL2) {
#pragma unroll
                    for (int jj = 0; jj < kRefChunk / 4; ++jj) {
                        const float4 a = qv[jj], b = mine[jj];
                        float t;
                        t = a.x - b.x; acc = fmaf(t, t, acc);
                        t = a.y - b.y; acc = fmaf(t, t, acc);
                        t = a.z - b.z; acc = fmaf(t, t, acc);
                        t = a.w - b.w; acc = fmaf(t, t, acc);
                    }
                } else {
#pragma unroll
                    for (int jj = 0; jj < kRefChunk / 4; ++jj) {
                        const float4 a = qv[jj], b = mine[jj];
                        acc = fmaf(a.x, b.x, acc);
                        acc = fmaf(a.y, b.y, acc);
                        acc = fmaf(a.z, b.z, acc);
                        acc = fmaf(a.w, b.w, acc);
                    }
                }
            }
            __syncwarp();
        }
    } else {
        for (int ch0 = 0; ch0 < d; ch0 += kRefChunk) {
            const int w = d - ch0 < kRefChunk ? d - ch0 : kRefChunk;
            const int lpr = w >> 2;                                  // float4 pieces per row
            if (lpr == kRefChunk / 4) {
#pragma unroll
                for (int it = 0; it < 8; ++it) {                     // four of the 32 rows per load instruction
                    const int r = it * 4 + (lane >> 3), j = lane & 7;
                    const uint32_t pr = __shfl_sync(0xffffffffu, pos, r);
                    if ((live_mask >> r) & 1u)
                        *reinterpret_cast<float4*>(rows + r * kRefPitch + 4 * j) =
                            __ldg(reinterpret_cast<const float4*>(xb + static_cast<int64_t>(pr) * d + ch0) + j);
                }
            } else {
                for (int idx = lane; idx < 32 * lpr; idx += 32) {
                    const int r = idx / lpr, j = idx - r * lpr;
                    const uint32_t pr = __shfl_sync(0xffffffffu, pos, r);
                    if ((live_mask >> r) & 1u)
                        *reinterpret_cast<float4*>(rows + r * kRefPitch + 4 * j) =
                            __ldg(reinterpret_cast<const float4*>(xb + static_cast<int64_t>(pr) * d + ch0) + j);
                }
            }
            __syncwarp();
            const float4* mine = reinterpret_cast<const float4*>(rows + lane * kRefPitch);
            const float4* qv = reinterpret_cast<const float4*>(qs + ch0);
            if (live) {
                for (int j = 0; j < lpr; ++j) {
                    const float4 a = qv[j], b = mine[j];
                    if (metric == kMetricL2) {
                        float t;
                        t = a.x - b.x; acc = fmaf(t, t, acc);
                        t = a.y - b.y; acc = fmaf(t, t, acc);
                        t = a.z - b.z; acc = fmaf(t, t, acc);
                        t = a.w - b.w; acc = fmaf(t, t, acc);
                    } else {
                        acc = fmaf(a.x, b.x, acc);
                        acc = fmaf(a.y, b.y, acc);
                        acc = fmaf(a.z, b.z, acc);
                        acc = fmaf(a.w, b.w, acc);
                    }
                }
            }
            __syncwarp();
        }
    }
    return metric == kMetricL2 ? acc : -acc;
}

__global__ void __launch_bounds__(128)
refine_f32_kernel(uint64_t* cand, const uint32_t* counts, uint32_t n_fixed, uint32_t cap, int d, int metric,
                  const float* xq, const float* xb, int q_first, int q_mod, const MemberView* members) {
    extern __shared__ __align__(16) float ref_sm[];
    float* qs = ref_sm;                                              // [d]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* rows = ref_sm + d + warp * (32 * kRefPitch);              // [32][kRefPitch] per warp
    const int q = blockIdx.y;
    // candidate row q_first + q holds the candidates of query (q_first + q) % q_mod (several indexes
    // searched with the same queries) or of query q_first + q (q_mod = 0)
    const int qrow = q_mod > 0 ? (q_first + q) % q_mod : q_first + q;
    const uint32_t n = counts ? counts[q] : n_fixed;
    if (n > cap) return;   // overflowed: what its slots hold is not looked at
    if (blockIdx.x * kRefWindow >= n) return;
    uint32_t pos_first = 0;   // position of xb's first row
    if (members) {
        const MemberView& mv = members[(q_first + q) / q_mod];
        xb = mv.rows_f32;
        pos_first = static_cast<uint32_t>(mv.first);
    }
    for (int i = threadIdx.x; i < d / 4; i += 128)
        reinterpret_cast<float4*>(qs)[i] = __ldg(reinterpret_cast<const float4*>(xq + static_cast<int64_t>(qrow) * d) + i);
    __syncthreads();
    uint64_t* row = cand + static_cast<int64_t>(q) * cap;
    // The list is sparse (reserved but unused slots, see the GEMM's block reservation): a window of
    // slots is compacted into shared memory first, so that every warp pass works on 32 live
    // candidates.  The result goes back to the candidate's own slot: the order of compaction is free.
    __shared__ uint32_t s_slot[kRefWindow];
    __shared__ uint32_t s_pos[kRefWindow];
    __shared__ uint32_t s_cnt;
    for (uint32_t win0 = blockIdx.x * kRefWindow; win0 < n; win0 += gridDim.x * kRefWindow) {
        if (threadIdx.x == 0) s_cnt = 0u;
        __syncthreads();
        const uint32_t win1 = win0 + kRefWindow < n ? win0 + kRefWindow : n;
        for (uint32_t i = win0 + threadIdx.x; i < win1; i += 128) {
            const uint64_t c = row[i];
            if (c != kCandInvalid) {
                const uint32_t j = atomicAdd(&s_cnt, 1u);
                s_slot[j] = i;
                s_pos[j] = static_cast<uint32_t>(c) - pos_first;
            }
        }
        __syncthreads();
        const uint32_t cnt = s_cnt;
        for (uint32_t i0 = warp * 32; i0 < cnt; i0 += 128) {
            const bool live = i0 + lane < cnt;
            const uint32_t i = live ? s_slot[i0 + lane] : 0u;
            const uint32_t pos = live ? s_pos[i0 + lane] : 0u;
            const float key = refine_lane(xb, qs, rows, pos, live, d, metric, lane);
            if (live) row[i] = pack_cand(float_to_ord(key), pos + pos_first);
        }
        __syncthreads();   // the window's lists are reused
    }
}

// ---- short candidate lists of fp32 indexes: pruning, exact distances, order and results in one block ----
// What prune_candidates_kernel, refine_f32_kernel and select_emit_kernel do one after the other, for lists
// of at most `stage` candidates of which at most kFinKeep survive the pruning; the row is read once, survivors
// and exact keys stay in shared memory.  Others are left alone and marked 2 in `status` (1: the row
// overflowed, as in select_emit_kernel): the caller runs the three kernels for them.
// One query against 100 003 x 128, k = 10: 38 us in four launches -> 10; 10 000
// queries against 16 384 centroids, k = 64: 117 -> 110.
constexpr int kFinThreads = 128;
constexpr uint32_t kFinKeep = 1024;
constexpr uint32_t kFinStage = 4096;
__global__ void __launch_bounds__(kFinThreads, 6)
finish_f32_kernel(const uint64_t* cand, const uint32_t* counts, uint32_t cap, uint32_t stage, int d, const float* eps,
                  const float* xq, const float* xb, uint8_t* status, uint32_t* any_status, const EmitArgs e) {
    extern __shared__ __align__(16) uint64_t fin_sm[];
    uint64_t* keep = fin_sm;                                             // [kFinKeep]
    float* qs = reinterpret_cast<float*>(fin_sm + kFinKeep);             // [d]
    float* rows = qs + d;                                                // 4 x [32][kRefPitch], after ...
    uint64_t* held = reinterpret_cast<uint64_t*>(rows);                  // ... [stage] entries have been pruned
    uint64_t* order = held;                                              // [k] results, after the last row was read
    __shared__ RankScratch rank;
    __shared__ uint32_t sh_fill;
    const int q = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int qrow = e.q_mod > 0 ? q % e.q_mod : q;
    const uint32_t n = counts[q], k = static_cast<uint32_t>(e.k);
    report_error(e);
    auto leave = [&](uint8_t why) {
        if (threadIdx.x == 0) {
            if (status) status[q] = why;
            if (any_status) any_status[why - 1] = 1u;
        }
        // (a caller that goes on before it looks at the status finds no results, not stale ones)
        for (uint32_t i = threadIdx.x; i < k; i += kFinThreads) emit_one(e, q, static_cast<int>(i), kCandInvalid);
    };
    if (n > cap) {
        leave(1);
        return;
    }
    uint32_t pos_first = 0;
    if (e.members) {
        const MemberView& mv = e.members[q / e.q_mod];
        xb = mv.rows_f32;
        pos_first = static_cast<uint32_t>(mv.first);
    }
    for (int i = threadIdx.x; i < d / 4; i += kFinThreads)
        reinterpret_cast<float4*>(qs)[i] = __ldg(reinterpret_cast<const float4*>(xq + static_cast<int64_t>(qrow) * d) + i);
    uint32_t m = block_compact<kFinThreads>(cand + static_cast<int64_t>(q) * cap, n, held, stage, &sh_fill);
    if (m > stage) {
        leave(2);
        return;
    }
    uint32_t lim = 0xFFFFFFFFu;
    if (m > 2 * k || m > kFinKeep) {   // fewer are refined as they are
        const uint32_t kth = block_kth32<kFinThreads>(
            [&](auto&& f) {
                for (uint32_t i = threadIdx.x; i < m; i += kFinThreads) {
                    const uint32_t v = static_cast<uint32_t>(held[i] >> 32);
                    if (v != 0xFFFFFFFFu) f(v);
                }
            },
            k, rank, 2);
        if (!prune_limit(kth, eps[qrow], &lim)) lim = 0xFFFFFFFFu;
    }
    __syncthreads();
    if (threadIdx.x == 0) sh_fill = 0u;
    __syncthreads();
    for (uint32_t i0 = warp * 32; i0 < m; i0 += kFinThreads) {
        const uint64_t v = i0 + lane < m ? held[i0 + lane] : kCandInvalid;
        const bool in = i0 + lane < m && static_cast<uint32_t>(v >> 32) <= lim;
        const unsigned bal = __ballot_sync(0xffffffffu, in);
        if (!bal) continue;
        uint32_t slot = 0;
        if (lane == 0) slot = atomicAdd(&sh_fill, static_cast<uint32_t>(__popc(bal)));
        slot = __shfl_sync(0xffffffffu, slot, 0) + __popc(bal & ((1u << lane) - 1u));
        if (in && slot < kFinKeep) keep[slot] = v;
    }
    __syncthreads();
    m = sh_fill;
    if (m > kFinKeep) {
        leave(2);
        return;
    }
    for (uint32_t i0 = warp * 32; i0 < m; i0 += kFinThreads) {
        const bool live = i0 + lane < m;
        const uint32_t pos = live ? static_cast<uint32_t>(keep[i0 + lane]) - pos_first : 0u;
        const float key = refine_lane(xb, qs, rows + warp * (32 * kRefPitch), pos, live, d, e.metric, lane);
        if (live) keep[i0 + lane] = pack_cand(float_to_ord(key), pos + pos_first);
    }
    __syncthreads();
    if (m <= static_cast<uint32_t>(kSmallSet)) {
        for (uint32_t i = threadIdx.x; i < m; i += kFinThreads) {
            const uint64_t v = keep[i];
            uint32_t r = 0;
#pragma unroll 8
            for (uint32_t j = 0; j < m; ++j) r += keep[j] < v ? 1u : 0u;
            if (r < k) order[r] = v;
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < min(k, m); i += kFinThreads) emit_one(e, q, static_cast<int>(i), order[i]);
    } else {
        int P = kSmallSet;
        while (P < static_cast<int>(m)) P <<= 1;
        for (int i = static_cast<int>(m) + threadIdx.x; i < P; i += kFinThreads) keep[i] = kCandInvalid;
        __syncthreads();
        bitonic_sort_u64<kFinThreads>(keep, P);
        for (uint32_t i = threadIdx.x; i < min(k, m); i += kFinThreads) emit_one(e, q, static_cast<int>(i), keep[i]);
    }
    for (uint32_t i = m + threadIdx.x; i < k; i += kFinThreads) emit_one(e, q, static_cast<int>(i), kCandInvalid);
}

// The same for small k and lists of a few dozen: one WARP per query.  The candidates are taken 32 at a
// time (a lane each), refined, sorted across the lanes and merged with the best 32 so far, so no list is
// too long for it and a block serves four queries without a block-wide barrier.  Assigning 300 000
// vectors (d 128) to 256 centroids, two or three candidates each: 0.50 ms.
__global__ void __launch_bounds__(kFinThreads, 5)
finish_warp_f32_kernel(const uint64_t* cand, const uint32_t* counts, uint32_t cap, int d, const float* xq, const float* xb,
                       uint8_t* status, const EmitArgs e) {
    extern __shared__ __align__(16) float finw_sm[];
    __shared__ uint64_t queue[kFinThreads / 32][64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q = blockIdx.x * (kFinThreads / 32) + warp;
    if (q >= e.nq) return;
    float* qs = finw_sm + warp * (d + 32 * kRefPitch);
    float* rows = qs + d;
    uint64_t* que = queue[warp];
    const uint32_t n = counts[q];
    report_error(e);
    if (n > cap) {
        if (lane == 0) status[q] = 1;
        if (lane < e.k) emit_one(e, q, lane, kCandInvalid);
        return;
    }
    for (int i = lane; i < d / 4; i += 32)
        reinterpret_cast<float4*>(qs)[i] = __ldg(reinterpret_cast<const float4*>(xq + static_cast<int64_t>(q) * d) + i);
    const uint64_t* row = cand + static_cast<int64_t>(q) * cap;
    uint64_t best = kCandInvalid;   // ascending over the lanes
    uint32_t fill = 0;
    for (uint32_t i0 = 0;; i0 += 32) {
        const bool last = i0 + 32 >= n;
        const uint64_t v = i0 + lane < n ? row[i0 + lane] : kCandInvalid;
        const unsigned bal = __ballot_sync(0xffffffffu, v != kCandInvalid);
        if (v != kCandInvalid) que[fill + __popc(bal & ((1u << lane) - 1u))] = v;
        fill += __popc(bal);
        __syncwarp();
        while (fill >= 32 || (last && fill > 0)) {
            const bool live = static_cast<uint32_t>(lane) < fill;
            const uint32_t pos = live ? static_cast<uint32_t>(que[lane]) : 0u;
            const float key = refine_lane(xb, qs, rows, pos, live, d, e.metric, lane);
            uint64_t x = live ? pack_cand(float_to_ord(key), pos) : kCandInvalid;
#pragma unroll
            for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
                for (int stride = size >> 1; stride > 0; stride >>= 1) {
                    const uint64_t o = shfl_xor_u64(x, stride);
                    const bool keep_min = ((lane & stride) == 0) == ((lane & size) == 0);
                    x = keep_min == (o < x) ? o : x;
                }
            // the lower half of two ascending lists, one of them reversed, is a bitonic sequence
            const uint64_t o = shfl_xor_u64(x, 31);
            best = o < best ? o : best;
#pragma unroll
            for (int stride = 16; stride > 0; stride >>= 1) {
                const uint64_t b = shfl_xor_u64(best, stride);
                best = ((lane & stride) == 0) == (b < best) ? b : best;
            }
            __syncwarp();
            const uint64_t rest = que[32 + lane];
            __syncwarp();
            que[lane] = rest;
            fill = fill > 32 ? fill - 32 : 0;
            __syncwarp();
        }
        if (last) break;
    }
    if (lane < e.k) emit_one(e, q, lane, best);
}

// One warp per query; heads[] in shared memory.
__global__ void __launch_bounds__(32)
merge_topk_kernel(int nsrc, int64_t nq, int k, int descending, const float* Din, const int64_t* Iin,
                  int64_t src_stride_d, int64_t src_stride_i, float* D, int64_t* I) {
    extern __shared__ int heads[];
    const int64_t q = blockIdx.x;
    const int lane = threadIdx.x;
    for (int s = lane; s < nsrc; s += 32) heads[s] = 0;
    __syncwarp();
    for (int j = 0; j < k; ++j) {
        float bk = 0.f;
        int64_t bl = -1;
        int bs = -1;
        for (int s = lane; s < nsrc; s += 32) {
            const int h = heads[s];
            if (h >= k) continue;
            const int64_t off = q * k + h;
            const int64_t l = Iin[s * src_stride_i + off];
            if (l < 0) {
                heads[s] = k;
                continue;
            }
            const float dv = Din[s * src_stride_d + off];
            const float key = descending ? -dv : dv;
            if (bs < 0 || key < bk || (key == bk && l < bl)) {
                bk = key;
                bl = l;
                bs = s;
            }
        }
        for (int off = 16; off > 0; off >>= 1) {
            const float ok = __shfl_xor_sync(0xffffffffu, bk, off);
            const int64_t ol = __shfl_xor_sync(0xffffffffu, bl, off);
            const int os = __shfl_xor_sync(0xffffffffu, bs, off);
            if (os >= 0 && (bs < 0 || ok < bk || (ok == bk && ol < bl))) {
                bk = ok;
                bl = ol;
                bs = os;
            }
        }
        if (lane == 0) {
            if (bs >= 0) {
                D[q * k + j] = descending ? -bk : bk;
                I[q * k + j] = bl;
                heads[bs] += 1;
            } else {
                D[q * k + j] = 3.402823466e+38f;
                I[q * k + j] = -1;
            }
        }
        __syncwarp();
    }
}

// ---- preparation kernels: one warp per row ----
__device__ __forceinline__ float warp_sum(float v) {
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}
__device__ __forceinline__ int warp_sum_i(int v) {
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// Query operand rows of d + kFoldCols bf16: the query, three ones (they pick up the base row's
// folded norm), three zeros (the threshold terms, written by store_tau once the threshold is
// known) and zero padding.
__global__ void prep_queries_f32_kernel(const float* xq, int nq, int d, int metric, float ymax,
                                        __nv_bfloat16* qb, float* qnorm, float* eps) {
    const int q = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (q >= nq) return;
    const int dp = d + kFoldCols;
    const bool packed = packed_operands(kKindBF16, dp);
    float s = 0.f;
    for (int i = lane; i < d; i += 32) {
        const float v = xq[static_cast<int64_t>(q) * d + i];
        s = fmaf(v, v, s);
        qb[operand_elem(packed, q, i, dp, kTileQ)] = __float2bfloat16_rn(v);
    }
    if (lane < kFoldCols) qb[operand_elem(packed, q, d + lane, dp, kTileQ)] = __float2bfloat16_rn(lane < 3 ? 1.f : 0.f);
    s = warp_sum(s);
    if (lane == 0) {
        qnorm[q] = s;
        // Filter slack.  bf16 rounding of both operands perturbs every product by at most
        // 2^-8 (1 + 2^-10) relatively, so |dot~ - dot| <= c |q||y| with the accumulation slack
        // folded into c; the second term covers the fp32 rounding of norms and of the canonical
        // distance itself.
        const float qn = sqrtf(s + kNormFloor) * 1.0001f;
        const float c = 0.00390625f * 1.01f + static_cast<float>(d) * 4.76837158203125e-07f;
        const float g = static_cast<float>(d + 4) * 2.384185791015625e-07f;
        float e;
        if (metric == kMetricL2) e = 2.f * c * qn * ymax + g * (qn + ymax) * (qn + ymax);
        else e = c * qn * ymax + g * qn * ymax;
        eps[q] = e;
    }
}

__global__ void prep_queries_f16_kernel(const __half* xq, int nq, int d, float* qnorm) {
    const int q = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (q >= nq) return;
    float s = 0.f;
    for (int i = lane; i < d; i += 32) {
        const float v = __half2float(xq[static_cast<int64_t>(q) * d + i]);
        s = fmaf(v, v, s);
    }
    s = warp_sum(s);
    if (lane == 0) qnorm[q] = s;
}

__global__ void prep_queries_i8_kernel(const int8_t* xq, int nq, int d, int32_t* qnorm) {
    const int q = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (q >= nq) return;
    int s = 0;
    for (int i = lane; i < d; i += 32) {
        const int v = xq[static_cast<int64_t>(q) * d + i];
        s += v * v;
    }
    s = warp_sum_i(s);
    if (lane == 0) qnorm[q] = s;
}

// Base operand rows of d + kFoldCols bf16: the vector, -|y|^2 / 2 in three terms (zeros for inner
// product), three ones (they pick up the query's threshold terms) and zero padding.
// x, norms: the n rows being added; xb: the whole operand buffer, whose row row0 + r belongs to x's row r.
__global__ void base_prep_f32_kernel(const float* x, int64_t n, int d, int metric, __nv_bfloat16* xb, int64_t row0,
                                     float* norms, float* max_norm_sq) {
    const int64_t r = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (r >= n) return;
    const int dp = d + kFoldCols;
    const bool packed = packed_operands(kKindBF16, dp);
    const int64_t ro = row0 + r;
    float s = 0.f;
    for (int i = lane; i < d; i += 32) {
        const float v = x[r * d + i];
        s = fmaf(v, v, s);
        xb[operand_elem(packed, ro, i, dp, kTileB)] = __float2bfloat16_rn(v);
    }
    s = warp_sum(s);
    if (lane >= 3 && lane < kFoldCols) xb[operand_elem(packed, ro, d + lane, dp, kTileB)] = __float2bfloat16_rn(lane < 6 ? 1.f : 0.f);
    if (lane == 0) {
        split3_bf16(metric == kMetricL2 ? -0.5f * s : 0.f, xb + operand_elem(packed, ro, d, dp, kTileB));
        norms[r] = s;
        atomicMax(reinterpret_cast<unsigned int*>(max_norm_sq), __float_as_uint(s));
    }
}

__global__ void base_prep_f16_kernel(const __half* x, int64_t n, int d, float* norms) {
    const int64_t r = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (r >= n) return;
    float s = 0.f;
    for (int i = lane; i < d; i += 32) {
        const float v = __half2float(x[r * d + i]);
        s = fmaf(v, v, s);
    }
    s = warp_sum(s);
    if (lane == 0) norms[r] = s;
}

__global__ void base_prep_i8_kernel(const int8_t* x, int64_t n, int d, int32_t* norms) {
    const int64_t r = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (r >= n) return;
    int s = 0;
    for (int i = lane; i < d; i += 32) {
        const int v = x[r * d + i];
        s += v * v;
    }
    s = warp_sum_i(s);
    if (lane == 0) norms[r] = s;
}

__global__ void f32_to_f16_kernel(const float* x, int64_t count, __half* out) {
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        out[i] = __float2half_rn(x[i]);
}
__global__ void f16_to_f32_kernel(const __half* x, int64_t count, float* out) {
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        out[i] = __half2float(x[i]);
}

__global__ void fill_u32_kernel(uint32_t* p, int64_t count, uint32_t value) {
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        p[i] = value;
}
__global__ void iota_i64_kernel(int64_t* p, int64_t count, int64_t start) {
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        p[i] = start + i;
}
__global__ void gather_rows_kernel(const uint32_t* src, const int32_t* idx, int n, int row_words, uint32_t* dst) {
    const int r = blockIdx.x;
    if (r >= n) return;
    const uint32_t* s = src + static_cast<int64_t>(idx[r]) * row_words;
    uint32_t* d = dst + static_cast<int64_t>(r) * row_words;
    for (int i = threadIdx.x; i < row_words; i += blockDim.x) d[i] = s[i];
}

__global__ void scatter_rows_kernel(const uint32_t* src, const int32_t* idx, int n, int row_words, uint32_t* dst) {
    const int r = blockIdx.x;
    if (r >= n) return;
    const uint32_t* s = src + static_cast<int64_t>(r) * row_words;
    uint32_t* d = dst + static_cast<int64_t>(idx[r]) * row_words;
    for (int i = threadIdx.x; i < row_words; i += blockDim.x) d[i] = s[i];
}

inline int next_pow2(int v) {
    int p = 1;
    while (p < v) p <<= 1;
    return p;
}

}  // namespace

cudaError_t launch_kth_threshold(const uint32_t* mins, int stride, int n, int nq, int k, const float* eps,
                                 uint32_t tau_all, uint32_t* tau, const TauFold& fold, cudaStream_t stream) {
    if (nq <= 0) return cudaSuccess;
    if (n <= 32)
        kth_threshold_warp_kernel<1><<<(nq + 3) / 4, 128, 0, stream>>>(mins, stride, n, nq, k, eps, tau_all, tau, fold);
    else if (n <= 128)
        kth_threshold_warp_kernel<4><<<(nq + 3) / 4, 128, 0, stream>>>(mins, stride, n, nq, k, eps, tau_all, tau, fold);
    else if (n <= 512)
        kth_threshold_warp_kernel<16><<<(nq + 3) / 4, 128, 0, stream>>>(mins, stride, n, nq, k, eps, tau_all, tau, fold);
    else if (n <= 1024)
        kth_threshold_warp_kernel<32><<<(nq + 3) / 4, 128, 0, stream>>>(mins, stride, n, nq, k, eps, tau_all, tau, fold);
    else
        kth_threshold_kernel<<<nq, kSelThreads, n <= static_cast<int>(kKthStage) ? n * 4 : 0, stream>>>(mins, stride, n, k, eps, tau_all, tau, fold);
    return cudaGetLastError();
}

cudaError_t launch_select_emit(const uint64_t* cand, const uint32_t* counts, uint32_t n_fixed, uint32_t cap,
                               uint8_t* overflow, uint32_t* any_overflow, const EmitArgs& e, cudaStream_t stream) {
    if (e.nq <= 0 || e.k <= 0) return cudaSuccess;
    const int P = next_pow2(e.k < 64 ? 64 : e.k);
    // Room for about as many candidates as a threshold for that k lets through (two stretches: 7 - 8 k).
    // Blocks of 512 where two of them fill an SM's shared memory.
    const bool large = e.k > 128;
    const uint32_t stage = large ? 12288u : 2048u;
    const size_t smem = (static_cast<size_t>(P) + stage) * sizeof(uint64_t);
    auto kern = large ? select_emit_kernel<512> : select_emit_kernel<kSelThreads>;
    cudaError_t err = allow_max_smem(kern);
    if (err != cudaSuccess) return err;
    kern<<<e.nq, large ? 512 : kSelThreads, smem, stream>>>(cand, counts, n_fixed, cap, P, stage, overflow, any_overflow, e);
    return cudaGetLastError();
}

cudaError_t launch_finish_f32(const uint64_t* cand, const uint32_t* counts, uint32_t cap, int d, const float* eps,
                              const float* xq, const float* xb, uint8_t* status, uint32_t* any_status, const EmitArgs& e,
                              bool few, cudaStream_t stream) {
    if (e.nq <= 0 || e.k <= 0) return cudaSuccess;
    if (few && e.k <= 32 && !e.members && status) {
        const size_t smem = (kFinThreads / 32) * (static_cast<size_t>(d) + 32 * kRefPitch) * sizeof(float);
        cudaError_t err = allow_max_smem(finish_warp_f32_kernel);
        if (err != cudaSuccess) return err;
        finish_warp_f32_kernel<<<(e.nq + kFinThreads / 32 - 1) / (kFinThreads / 32), kFinThreads, smem, stream>>>(
            cand, counts, cap, d, xq, xb, status, e);
        return cudaGetLastError();
    }
    const uint32_t stage = cap < kFinStage ? cap : kFinStage;
    const size_t rows = 4 * 32 * kRefPitch * sizeof(float), held = stage * sizeof(uint64_t);
    const size_t smem = kFinKeep * sizeof(uint64_t) + static_cast<size_t>(d) * 4 + (rows > held ? rows : held);
    cudaError_t err = allow_max_smem(finish_f32_kernel);
    if (err != cudaSuccess) return err;
    finish_f32_kernel<<<e.nq, kFinThreads, smem, stream>>>(cand, counts, cap, stage, d, eps, xq, xb, status, any_status, e);
    return cudaGetLastError();
}

cudaError_t launch_tighten_tau(const uint64_t* cand, const uint32_t* counts, uint32_t cap, int nq, int k,
                               const float* eps, uint32_t* tau, const TauFold& fold, cudaStream_t stream) {
    if (nq <= 0) return cudaSuccess;
    tighten_tau_kernel<<<nq, kSelThreads, 0, stream>>>(cand, counts, cap, k, eps, tau, fold);
    return cudaGetLastError();
}

cudaError_t launch_prune_candidates(uint64_t* cand, uint32_t* counts, uint32_t cap, int nq, int k,
                                    const float* eps, cudaStream_t stream) {
    if (nq <= 0) return cudaSuccess;
    prune_candidates_kernel<<<nq, kSelThreads, 0, stream>>>(cand, counts, cap, k, eps);
    return cudaGetLastError();
}

cudaError_t launch_refine_f32(uint64_t* cand, const uint32_t* counts, uint32_t n_fixed, uint32_t cap, int nq, int d,
                              int metric, const float* xq, const float* xb, cudaStream_t stream, int q_mod,
                              const MemberView* members) {
    if (nq <= 0) return cudaSuccess;
    uint32_t per_row = counts ? cap : (n_fixed < cap ? n_fixed : cap);
    // Blocks stride over a row's candidates, so a few thousand blocks in total keep the machine
    // busy; one block per 128 candidate SLOTS would mostly launch blocks that find nothing to do.
    int gx = static_cast<int>((per_row + kRefWindow - 1) / kRefWindow);
    const int want = (2048 + nq - 1) / nq;
    if (gx > want) gx = want;
    if (gx > 64) gx = 64;
    if (gx < 1) gx = 1;
    const size_t smem = (static_cast<size_t>(d) + 4 * 32 * kRefPitch) * sizeof(float);   // (34 KB at d = 4096)
    for (int q0 = 0; q0 < nq; q0 += 65535) {
        const int nqq = nq - q0 < 65535 ? nq - q0 : 65535;
        refine_f32_kernel<<<dim3(gx, nqq), 128, smem, stream>>>(cand + static_cast<int64_t>(q0) * cap,
                                                            counts ? counts + q0 : nullptr, n_fixed, cap, d, metric,
                                                            xq, xb, q0, q_mod, members);
    }
    return cudaGetLastError();
}

cudaError_t launch_merge_topk(int nsrc, int64_t nq, int k, int descending, const float* Din, const int64_t* Iin,
                              float* D, int64_t* I, cudaStream_t stream, int64_t src_stride_d, int64_t src_stride_i) {
    if (nq <= 0 || k <= 0) return cudaSuccess;
    if (src_stride_d <= 0) src_stride_d = nq * k;
    if (src_stride_i <= 0) src_stride_i = nq * k;
    merge_topk_kernel<<<static_cast<unsigned>(nq), 32, static_cast<size_t>(nsrc) * sizeof(int), stream>>>(
        nsrc, nq, k, descending, Din, Iin, src_stride_d, src_stride_i, D, I);
    return cudaGetLastError();
}

cudaError_t launch_prep_queries_f32(const float* xq, int nq, int d, int metric, float base_max_norm, void* q_bf16,
                                    float* qnorm, float* eps, cudaStream_t stream) {
    if (nq <= 0) return cudaSuccess;
    prep_queries_f32_kernel<<<(nq + 7) / 8, 256, 0, stream>>>(xq, nq, d, metric, base_max_norm,
                                                              static_cast<__nv_bfloat16*>(q_bf16), qnorm, eps);
    return cudaGetLastError();
}
cudaError_t launch_prep_queries_f16(const void* xq, int nq, int d, float* qnorm, cudaStream_t stream) {
    if (nq <= 0) return cudaSuccess;
    prep_queries_f16_kernel<<<(nq + 7) / 8, 256, 0, stream>>>(static_cast<const __half*>(xq), nq, d, qnorm);
    return cudaGetLastError();
}
cudaError_t launch_prep_queries_i8(const int8_t* xq, int nq, int d, int32_t* qnorm, cudaStream_t stream) {
    if (nq <= 0) return cudaSuccess;
    prep_queries_i8_kernel<<<(nq + 7) / 8, 256, 0, stream>>>(xq, nq, d, qnorm);
    return cudaGetLastError();
}
cudaError_t launch_base_prep_f32(const float* x, int64_t n, int d, int metric, void* x_bf16, int64_t row0,
                                 float* norms, float* max_norm_sq, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    base_prep_f32_kernel<<<static_cast<unsigned>((n + 7) / 8), 256, 0, stream>>>(
        x, n, d, metric, static_cast<__nv_bfloat16*>(x_bf16), row0, norms, max_norm_sq);
    return cudaGetLastError();
}
cudaError_t launch_base_prep_f16(const void* x, int64_t n, int d, float* norms, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    base_prep_f16_kernel<<<static_cast<unsigned>((n + 7) / 8), 256, 0, stream>>>(static_cast<const __half*>(x), n, d,
                                                                                 norms);
    return cudaGetLastError();
}
cudaError_t launch_base_prep_i8(const int8_t* x, int64_t n, int d, int32_t* norms, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    base_prep_i8_kernel<<<static_cast<unsigned>((n + 7) / 8), 256, 0, stream>>>(x, n, d, norms);
    return cudaGetLastError();
}
cudaError_t launch_f32_to_f16(const float* x, int64_t count, void* out, cudaStream_t stream) {
    if (count <= 0) return cudaSuccess;
    int grid = static_cast<int>((count + 255) / 256 < 65535 ? (count + 255) / 256 : 65535);
    f32_to_f16_kernel<<<grid, 256, 0, stream>>>(x, count, static_cast<__half*>(out));
    return cudaGetLastError();
}
cudaError_t launch_f16_to_f32(const void* x, int64_t count, float* out, cudaStream_t stream) {
    if (count <= 0) return cudaSuccess;
    int grid = static_cast<int>((count + 255) / 256 < 65535 ? (count + 255) / 256 : 65535);
    f16_to_f32_kernel<<<grid, 256, 0, stream>>>(static_cast<const __half*>(x), count, static_cast<float*>(out));
    return cudaGetLastError();
}

namespace {
// flag |= 1 when x holds a NaN or an infinity
__global__ void check_finite_kernel(const float* x, int64_t count, int* flag) {
    bool bad = false;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        bad |= (__float_as_uint(x[i]) & 0x7f800000u) == 0x7f800000u;
    if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(flag, 1);
}
// flag |= 2 when a value lies outside [0, bound)
__global__ void check_range_i32_kernel(const int32_t* v, int64_t count, int32_t bound, int* flag) {
    bool bad = false;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        bad |= v[i] < 0 || v[i] >= bound;
    if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(flag, 2);
}
}  // namespace
cudaError_t launch_check_finite(const float* x, int64_t count, int* flag, cudaStream_t stream) {
    if (count <= 0) return cudaSuccess;
    int grid = static_cast<int>((count + 255) / 256 < 2048 ? (count + 255) / 256 : 2048);
    check_finite_kernel<<<grid, 256, 0, stream>>>(x, count, flag);
    return cudaGetLastError();
}
cudaError_t launch_check_range_i32(const int32_t* v, int64_t count, int32_t bound, int* flag, cudaStream_t stream) {
    if (count <= 0) return cudaSuccess;
    int grid = static_cast<int>((count + 255) / 256 < 2048 ? (count + 255) / 256 : 2048);
    check_range_i32_kernel<<<grid, 256, 0, stream>>>(v, count, bound, flag);
    return cudaGetLastError();
}

cudaError_t launch_fill_u32(uint32_t* p, int64_t count, uint32_t value, cudaStream_t stream) {
    if (count <= 0) return cudaSuccess;
    int grid = static_cast<int>((count + 255) / 256 < 4096 ? (count + 255) / 256 : 4096);
    fill_u32_kernel<<<grid, 256, 0, stream>>>(p, count, value);
    return cudaGetLastError();
}
cudaError_t launch_iota_i64(int64_t* p, int64_t count, int64_t start, cudaStream_t stream) {
    if (count <= 0) return cudaSuccess;
    int grid = static_cast<int>((count + 255) / 256 < 4096 ? (count + 255) / 256 : 4096);
    iota_i64_kernel<<<grid, 256, 0, stream>>>(p, count, start);
    return cudaGetLastError();
}
cudaError_t launch_gather_rows(const void* src, const int32_t* idx, int n, int row_bytes, void* dst,
                               cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    gather_rows_kernel<<<n, 128, 0, stream>>>(static_cast<const uint32_t*>(src), idx, n, row_bytes / 4,
                                              static_cast<uint32_t*>(dst));
    return cudaGetLastError();
}
cudaError_t launch_scatter_rows(const void* src, const int32_t* idx, int n, int row_bytes, void* dst,
                                cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    scatter_rows_kernel<<<n, 128, 0, stream>>>(static_cast<const uint32_t*>(src), idx, n, row_bytes / 4,
                                               static_cast<uint32_t*>(dst));
    return cudaGetLastError();
}

}  // namespace b200
