// IVFPQ scan with a bound: short codes (M = 4 or 8 bytes a vector), and wide ones (M = 16, 32, 48, 64, whose
// groups of 16 bytes are stored rotated by the position) where sorted lists are the slower filter.
//
// The lookups of a short code are few (4 or 8), so neither the 16-column tables of the wide-code scan
// nor its sorted lists in registers pay: with k = 300 the insertions into a warp's list of 512 pairs
// are a chain that costs far more than the lookups.  Instead the k-th distance is bounded first and
// everything under the bound is collected:
//   1  short_bound_kernel : one block per query.  Builds the query's table, scans the nearest lists (a
//        sixteenth of the probed vectors, at least 4 k) into a histogram of distances and takes the
//        upper edge of the bin of the k-th smallest: k vectors lie at or below it, so the k-th distance
//        of the whole query does too.  Raw codes of clustered data are equal by the thousand; then the
//        labels of the equal ones are ranked as well and bound what is collected at that distance.
//   2  short_scan_kernel  : persistent blocks over (query, share of its vectors).  The table is
//        replicated in shared memory, 32 columns (M = 4) or 16 (M = 8), so that a warp's 32 lookups
//        with 32 different codes take one or two wavefronts instead of about 3.5; a lane takes 16 bytes
//        of codes per load (4 or 2 vectors), four loads in flight.  Vectors under the bound go to the
//        query's candidate row.
//   3  short_select_kernel: one block per query, exact order by (distance, label).
// Raw encoding: the table holds the canonical |q_m - cb|^2 and they are added in ascending m, so the
// scanned distances ARE the canonical ones.  Residual encoding scans |q-c|^2 + t2 - 2 q.cb, and wide codes add
// in the order of their rotation: there the bound is widened by twice the error, and the collected vectors
// within twice the error of the k-th get their canonical distance.
// Wide codes: wide_scan_kernel takes the place of short_scan_kernel, with the table rows of the wide-code filter
// (ivfpq_index.cu); what they measured stands at use_bounded_scan.
// A query with more than `cap` vectors under its bound is flagged, and the caller searches for it with a longer
// row or another scan.
// What bounds it (64 queries, 10 M vectors, M = 4, 64 of 1024 lists, k = 300; the exact scan this
// replaces took 2.14 ms): the bound takes 41 us (64 blocks, one step
// after the other inside), the scan 65 (issue slots: about 40 instructions a vector, and two table fills per
// block), the order 20; the whole call 2.77 -> 0.23 ms.
#include "ivfpq_short_scan.cuh"

#include <algorithm>

#include "block_rank.cuh"
#include "common.cuh"
#include "ivfpq_exact.cuh"
#include "smem_limit.h"

namespace b200 {
namespace {

constexpr int kKsub = 256;
constexpr int kBins = 4096;
constexpr int kScanThreadsShort = 1024;
constexpr int kWideThreads = 384;
constexpr int kSelThreadsShort = 256;
constexpr int kSortMax = 2048;           // pairs sorted in shared memory
constexpr float kPadDist = 3.402823466e+38f;
constexpr int64_t kNoLabel = 0x7fffffffffffffffll;
constexpr uint32_t kInfBits = 0x7f800000u;

template <int M>
__host__ __device__ constexpr int replicas() { return M == 4 ? 32 : 16; }   // 128 KB either way
template <int M>
__host__ __device__ constexpr int unit_vectors() { return 4 * 512 / M; }     // four 16-byte loads per lane

struct Probe {
    uint32_t begin, len;
    float base;
};
__device__ __forceinline__ Probe load_probe(const ShortScanArgs& a, int64_t q, int p) {
    Probe r{0u, 0u, 0.f};
    const int64_t list = a.cI[q * a.nprobe + p];
    if (list >= 0 && list < a.nlist) {
        r.begin = static_cast<uint32_t>(a.offsets[list]);
        r.len = static_cast<uint32_t>(a.lens[list]);
        if (a.by_residual) r.base = a.cD[q * a.nprobe + p];
    }
    return r;
}

// Exclusive prefix sums of one value per thread (all blockDim.x threads take part); the total comes
// back through *total.  warp_tot: 32 words of shared memory.
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t* warp_tot, uint32_t* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    __syncthreads();   // warp_tot may still be read from an earlier call
    if (lane == 31) warp_tot[w] = incl;
    __syncthreads();
    uint32_t below = 0, all = 0;
    for (int i = 0; i < nw; ++i) {
        if (i == w) below = all;
        all += warp_tot[i];
    }
    *total = all;
    return below + incl - v;
}

// ---- 1. table and bound ----
template <int M>
__host__ __device__ constexpr bool wide() { return M % 16 == 0; }   // rotated codes, 16 columns per table row
// Threads of the bound's block: wide codes need 44 registers and up to 110 KB, so two blocks of 512 share an SM
// where one of 1 024 would have it alone (1 000 queries, M = 48: 121 -> 103 us).
template <int M>
__host__ __device__ constexpr int bound_threads() { return wide<M>() ? 512 : 1024; }

template <int M>
__global__ void __launch_bounds__(bound_threads<M>())
short_bound_kernel(const ShortScanArgs a) {
    constexpr int kBoundThreads = bound_threads<M>();
    extern __shared__ __align__(16) float bound_sm[];
    float* tab = bound_sm;                                                  // [M][256]
    uint32_t* hist = reinterpret_cast<uint32_t*>(tab + M * kKsub);          // [kBins]
    uint32_t* pre = hist + kBins;                                           // [nprobe + 1] vectors before the probe
    uint32_t* beg = pre + kShortMaxProbe + 1;
    float* base = reinterpret_cast<float*>(beg + kShortMaxProbe);
    float* qs = base + kShortMaxProbe;                                      // [d]
    uint32_t* dist = reinterpret_cast<uint32_t*>(qs + a.d);                 // [a.n1_max] bits of the distances
    __shared__ uint32_t s_warp[32], s_lo, s_hi, s_bin, s_below, s_in, s_base;
    __shared__ unsigned long long s_llo, s_lhi;
    __shared__ float s_qn2;
    const int64_t q = blockIdx.x;
    const int tid = threadIdx.x;
    if (tid == 0) {
        s_lo = kInfBits;
        s_hi = 0u;
        s_base = 0u;
        a.count[q] = 0u;
    }
    for (int t = tid; t < a.d; t += kBoundThreads) qs[t] = a.xq[q * a.d + t];
    for (int i = tid; i < kBins; i += kBoundThreads) hist[i] = 0u;
    uint32_t total = 0;
    for (int p0 = 0; p0 < a.nprobe; p0 += kBoundThreads) {
        const int p = p0 + tid;
        Probe pr{0u, 0u, 0.f};
        if (p < a.nprobe) pr = load_probe(a, q, p);
        uint32_t sum;
        const uint32_t ex = block_exclusive(pr.len, s_warp, &sum);
        if (a.by_residual) {   // largest magnitude (a NaN is larger still)
            const uint32_t far = __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(pr.base)));
            if ((tid & 31) == 0) atomicMax(&s_base, far);
        }
        if (p < a.nprobe) {
            pre[p] = total + ex;
            beg[p] = pr.begin;
            base[p] = pr.base;
        }
        total += sum;
    }
    if (tid == 0) {
        pre[a.nprobe] = total;
        if (a.scanned) atomicAdd(a.scanned, static_cast<unsigned long long>(total));
    }
    __syncthreads();
    for (int i = tid; i < M * kKsub; i += kBoundThreads) {
        // entry i of the table: sub-quantizer m, its codeword (rotated codes: [M / 16][256][16])
        const int m = wide<M>() ? (i >> 12) * 16 + (i & 15) : i / kKsub;
        const float* cw = (wide<M>() ? a.cbT : a.codebooks) + static_cast<int64_t>(i) * a.dsub;
        float e = 0.f;
        auto term = [&](int t, float c) {
            const float v = qs[m * a.dsub + t];
            if (a.by_residual) {
                e = fmaf(v, c, e);
            } else {
                const float df = v - c;
                e = fmaf(df, df, e);
            }
        };
        if ((a.dsub & 3) == 0) {
#pragma unroll 4
            for (int t = 0; t < a.dsub; t += 4) {
                const float4 c = __ldg(reinterpret_cast<const float4*>(cw + t));
                term(t, c.x);
                term(t + 1, c.y);
                term(t + 2, c.z);
                term(t + 3, c.w);
            }
        } else {
            for (int t = 0; t < a.dsub; ++t) term(t, __ldg(cw + t));
        }
        if (a.by_residual) e = -2.f * e;
        tab[i] = e;
        a.lut[q * (M * kKsub) + i] = e;
    }
    if (tid < 32) {
        float s = 0.f;
        if (a.by_residual)
            for (int t = tid; t < a.d; t += 32) s = fmaf(qs[t], qs[t], s);
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (tid == 0) s_qn2 = s;
    }
    __syncthreads();
    // The nearest `n1` vectors: a sixteenth of what is probed, 4 k at least.  Their distances are computed
    // once and ranked in shared memory.
    const uint32_t n1 = min(a.n1_max, min(total, max(max(total / 16u, 4u * static_cast<uint32_t>(a.k)), 2048u)));
    const uint32_t lane = tid & 31;
    {
        int p = 0;
        uint32_t lo = kInfBits, hi = 0u;
        if constexpr (!wide<M>()) {
            for (uint32_t i0 = tid; i0 < n1; i0 += 4 * kBoundThreads) {
                uint32_t w[4][M / 4];
                float t[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {   // four vectors' loads in flight
                    const uint32_t i = i0 + j * kBoundThreads;
                    t[j] = 0.f;
#pragma unroll
                    for (int g = 0; g < M / 4; ++g) w[j][g] = 0u;
                    if (i < n1) {
                        while (pre[p + 1] <= i) ++p;
                        const uint32_t pos = beg[p] + (i - pre[p]);
                        if (a.by_residual) t[j] = base[p] + __ldg(a.t2 + pos);
                        if (M == 4) {
                            w[j][0] = __ldg(reinterpret_cast<const uint32_t*>(a.codes) + pos);
                        } else {
                            const uint2 c = __ldg(reinterpret_cast<const uint2*>(a.codes) + pos);
                            w[j][0] = c.x;
                            w[j][M / 4 - 1] = c.y;
                        }
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t i = i0 + j * kBoundThreads;
                    if (i >= n1) break;
                    float acc = t[j];
#pragma unroll
                    for (int m = 0; m < M; ++m) acc = acc + tab[m * kKsub + ((w[j][m >> 2] >> (8 * (m & 3))) & 255u)];
                    // (NaN becomes 0: a query that holds one collects nothing in the scan)
                    const uint32_t b = __float_as_uint(fmaxf(acc, 0.f));
                    dist[i] = b;
                    lo = min(lo, b);
                    hi = max(hi, b);
                }
            }
        } else {
            constexpr int U = M <= 16 ? 4 : (M <= 32 ? 2 : 1);   // vectors whose codes are in flight
            for (uint32_t i0 = tid; i0 < n1; i0 += U * kBoundThreads) {
                uint4 c[U][M / 16 > 0 ? M / 16 : 1];
                float acc[U];
                uint32_t pos[U];
#pragma unroll
                for (int j = 0; j < U; ++j) {
                    const uint32_t i = i0 + j * kBoundThreads;
                    acc[j] = 0.f;
                    pos[j] = 0u;
                    if (i < n1) {
                        while (pre[p + 1] <= i) ++p;
                        pos[j] = beg[p] + (i - pre[p]);
                        if (a.by_residual) acc[j] = base[p] + __ldg(a.t2 + pos[j]);
                    }
#pragma unroll
                    for (int g = 0; g < M / 16; ++g)
                        c[j][g] = i < n1 ? __ldg(reinterpret_cast<const uint4*>(a.codes + static_cast<size_t>(pos[j]) * M) + g)
                                         : make_uint4(0u, 0u, 0u, 0u);
                }
#pragma unroll
                for (int j = 0; j < U; ++j) {
                    const uint32_t i = i0 + j * kBoundThreads;
                    if (i >= n1) break;
#pragma unroll
                    for (int g = 0; g < M / 16; ++g) {
                        const uint32_t w[4] = {c[j][g].x, c[j][g].y, c[j][g].z, c[j][g].w};
#pragma unroll
                        for (int e = 0; e < 16; ++e)
                            acc[j] += tab[(g * kKsub + ((w[e >> 2] >> (8 * (e & 3))) & 255u)) * 16 + ((e + pos[j]) & 15u)];
                    }
                    const uint32_t b = __float_as_uint(fmaxf(acc[j], 0.f));
                    dist[i] = b;
                    lo = min(lo, b);
                    hi = max(hi, b);
                }
            }
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if (lane == 0) {
            atomicMin(&s_lo, lo);
            atomicMax(&s_hi, hi);
        }
    }
    __syncthreads();
    // visit(f): f(bits of the distance, index, in) over the stretch, whole warps at a time
    auto visit = [&](auto&& f) {
        for (uint32_t i0 = tid - lane; i0 < n1; i0 += kBoundThreads) {
            const uint32_t i = i0 + lane;
            f(i < n1 ? dist[i] : 0u, i, i < n1);
        }
    };
    // Adds the block's vectors with bin < kBins to the histogram; one lane adds for all when they agree
    // (lists of equal codes).  Warp-collective.
    auto count = [&](uint32_t bin) {
        int same;
        __match_all_sync(0xffffffffu, bin, &same);
        if (bin < static_cast<uint32_t>(kBins)) {
            if (!same) atomicAdd(&hist[bin], 1u);
            else if (lane == 0) atomicAdd(&hist[bin], 32u);
        }
    };
    // Bin that holds rank r: s_bin (kBins: fewer than r), s_below, s_in (its size).  Clears the histogram.
    auto find_bin = [&](uint32_t r) {
        constexpr int kPer = kBins / kBoundThreads;
        __syncthreads();
        if (tid == 0) s_bin = kBins;
        uint32_t mine[kPer], sum = 0, all;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            mine[j] = hist[tid * kPer + j];
            hist[tid * kPer + j] = 0u;
            sum += mine[j];
        }
        uint32_t run = block_exclusive(sum, s_warp, &all);
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            if (run < r && run + mine[j] >= r) {
                s_bin = tid * kPer + j;
                s_below = run;
                s_in = mine[j];
            }
            run += mine[j];
        }
        __syncthreads();
    };
    // Bins are steps of the float's bits, i.e. about equal ratios: never coarser than 1 part in 256 (eight
    // octaves in 4095 bins and their rounding to a power of two).  Bin 0 takes the smaller values.
    const uint32_t hi_b = s_hi;
    uint32_t lo_b = max(s_lo, __float_as_uint(__uint_as_float(hi_b) * 0.00390625f));
    int shift = 0;
    while (((hi_b - min(lo_b, hi_b)) >> shift) >= static_cast<uint32_t>(kBins - 1)) ++shift;
    visit([&](uint32_t b, uint32_t, bool in) { count(!in ? 0xFFFFFFFFu : b < lo_b ? 0u : 1u + ((b - lo_b) >> shift)); });
    find_bin(static_cast<uint32_t>(a.k));
    uint32_t tb = kInfBits;             // fewer than k vectors in the bins: no bound
    uint64_t label_max = ~0ull;
    if (s_bin == 0u) {
        tb = lo_b - 1u;
    } else if (s_bin < static_cast<uint32_t>(kBins)) {
        uint32_t r = static_cast<uint32_t>(a.k) - s_below, in = s_in;
        lo_b += (s_bin - 1u) << shift;
        // a crowded bin is looked at more closely: down to one value if need be
        while (shift > 0 && in > 128u) {
            const int finer = max(0, shift - 12);
            const uint32_t last = (1u << shift) - 1u;
            visit([&](uint32_t b, uint32_t, bool ok) { count(ok && b >= lo_b && b - lo_b <= last ? (b - lo_b) >> finer : 0xFFFFFFFFu); });
            find_bin(r);
            r -= s_below;
            in = s_in;
            lo_b += s_bin << finer;
            shift = finer;
        }
        tb = min(kInfBits, lo_b + ((1u << shift) - 1u));   // (both below 2^31)
        // Thousands of vectors with one distance (equal codes): the ones with the smallest labels count, so
        // the r-th smallest label among those seen here bounds theirs.
        if (!wide<M>() && !a.by_residual && shift == 0 && in > 1024u) {
            if (tid == 0) {
                s_llo = ~0ull;
                s_lhi = 0ull;
            }
            __syncthreads();
            int p = 0;
            auto label_of = [&](uint32_t i) {   // (i grows within a visit)
                while (pre[p + 1] <= i) ++p;
                return static_cast<unsigned long long>(__ldg(a.ids + beg[p] + (i - pre[p]))) ^ (1ull << 63);
            };
            unsigned long long l0 = ~0ull, l1 = 0ull;
            visit([&](uint32_t b, uint32_t i, bool ok) {
                if (ok && b == tb) {
                    const unsigned long long v = label_of(i);
                    l0 = min(l0, v);
                    l1 = max(l1, v);
                }
            });
            for (int o = 16; o > 0; o >>= 1) {
                l0 = min(l0, __shfl_xor_sync(0xffffffffu, l0, o));
                l1 = max(l1, __shfl_xor_sync(0xffffffffu, l1, o));
            }
            if (lane == 0) {
                atomicMin(&s_llo, l0);
                atomicMax(&s_lhi, l1);
            }
            __syncthreads();
            unsigned long long lo = s_llo, hi = s_lhi;
            while (lo < hi && in > 128u) {
                const int sh = max(0, 52 - __clzll(static_cast<long long>(hi - lo)));   // 4096 bins over [lo, hi]
                p = 0;
                visit([&](uint32_t b, uint32_t i, bool ok) {
                    uint32_t bin = 0xFFFFFFFFu;
                    if (ok && b == tb) {
                        const unsigned long long v = label_of(i);
                        if (v >= lo && v <= hi) bin = static_cast<uint32_t>((v - lo) >> sh);
                    }
                    count(bin);
                });
                find_bin(r);
                r -= s_below;
                in = s_in;
                lo += static_cast<unsigned long long>(s_bin) << sh;
                const unsigned long long top = lo + ((1ull << sh) - 1ull);
                hi = top < hi ? top : hi;
            }
            label_max = hi;
        }
    }
    if (tid == 0) {
        float thr = __uint_as_float(tb);
        // scanned distances of raw short codes are the canonical ones; the others are off by eps at most
        float eps = 0.f;
        if (a.by_residual) {
            const float mag = __uint_as_float(s_base) + a.t2_bound + 2.f * sqrtf(s_qn2) * a.cb_bound;
            if (tb != kInfBits) eps = a.err_rel * (mag + thr);
            // A query whose terms leave the range of a float (or hold a NaN): their sum may be NaN where the
            // canonical distance is a number.  It collects nothing and is left to the exact scan.
            if (!(mag < kPadDist)) {
                thr = __int_as_float(0x7fc00000);
                a.count[q] = kShortExact;
            }
        } else if (wide<M>() && tb != kInfBits) {
            eps = a.err_rel * thr;
        }
        thr = thr + 2.f * eps;
        a.eps[q] = eps;
        a.thr[q] = thr;
        a.label_max[q] = label_max;
    }
}

// ---- 2. scan ----
template <int M, bool RESID>
__global__ void __launch_bounds__(kScanThreadsShort, 1)
short_scan_kernel(const ShortScanArgs a, int S) {
    constexpr int R = replicas<M>(), U = unit_vectors<M>(), VPL = 16 / M;
    extern __shared__ __align__(16) float scan_sm[];
    float* lut = scan_sm;                                                   // [M][256][R]
    uint32_t* upre = reinterpret_cast<uint32_t*>(lut + M * kKsub * R);      // [nprobe + 1] units before the probe
    uint32_t* beg = upre + kShortMaxProbe + 1;
    uint32_t* len = beg + kShortMaxProbe;
    float* base = reinterpret_cast<float*>(len + kShortMaxProbe);
    __shared__ uint32_t s_warp[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float* lut_col = lut + lane % R;
    const int64_t items = a.nq * S;
    const int64_t it0 = items * blockIdx.x / gridDim.x, it1 = items * (blockIdx.x + 1) / gridDim.x;
    int64_t cur_q = -1;
    uint32_t units = 0;
    float thr = 0.f;
    uint64_t label_max = ~0ull;
    for (int64_t it = it0; it < it1; ++it) {
        const int64_t q = it / S;
        const uint32_t split = static_cast<uint32_t>(it - q * S);
        if (q != cur_q) {
            __syncthreads();   // the previous query's table and probes are still read
            cur_q = q;
            for (int i = threadIdx.x; i < M * kKsub * R / 4; i += kScanThreadsShort) {
                const float v = __ldg(a.lut + q * (M * kKsub) + i / (R / 4));
                reinterpret_cast<float4*>(lut)[i] = make_float4(v, v, v, v);
            }
            Probe pr{0u, 0u, 0.f};
            const int p = threadIdx.x;
            if (p < a.nprobe) pr = load_probe(a, q, p);
            const uint32_t ex = block_exclusive((pr.len + U - 1) / U, s_warp, &units);
            if (p < a.nprobe) {
                upre[p] = ex;
                beg[p] = pr.begin;
                len[p] = pr.len;
                base[p] = pr.base;
            }
            thr = a.thr[q];
            if (!RESID) label_max = a.label_max[q];
            __syncthreads();
        }
        const uint32_t u0 = static_cast<uint32_t>(static_cast<uint64_t>(units) * split / S);
        const uint32_t u1 = static_cast<uint32_t>(static_cast<uint64_t>(units) * (split + 1) / S);
        for (uint32_t u = u0 + warp; u < u1; u += kScanThreadsShort / 32) {
            int l = 0, h = a.nprobe;   // last probe with upre[p] <= u: the one that holds unit u
            while (h - l > 1) {
                const int mid = (l + h) >> 1;
                if (upre[mid] <= u) l = mid;
                else h = mid;
            }
            const uint32_t first = (u - upre[l]) * U;
            const uint32_t n = len[l], pos0 = beg[l];
            const float bias = RESID ? base[l] : 0.f;
            // lists are stored padded to 32 vectors: the 16 bytes behind a real vector are the list's own
            uint4 c[4];
            float t[4][VPL];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t i = first + j * (32 * VPL) + lane * VPL;
                c[j] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                for (int e = 0; e < VPL; ++e) t[j][e] = 0.f;
                if (i < n) {
                    c[j] = __ldg(reinterpret_cast<const uint4*>(a.codes + static_cast<size_t>(pos0 + i) * M));
                    if (RESID) {
                        if (VPL == 4) {
                            const float4 v = __ldg(reinterpret_cast<const float4*>(a.t2 + pos0 + i));
                            t[j][0] = v.x; t[j][1] = v.y; t[j][VPL - 2] = v.z; t[j][VPL - 1] = v.w;
                        } else {
                            const float2 v = __ldg(reinterpret_cast<const float2*>(a.t2 + pos0 + i));
                            t[j][0] = v.x; t[j][1] = v.y;
                        }
                    }
                }
            }
            float acc[4][VPL];
            bool any = false;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t w[4] = {c[j].x, c[j].y, c[j].z, c[j].w};
#pragma unroll
                for (int e = 0; e < VPL; ++e) {
                    float s = RESID ? bias + t[j][e] : 0.f;
#pragma unroll
                    for (int m = 0; m < M; ++m) {
                        const uint32_t byte = __byte_perm(w[e * (M / 4) + (m >> 2)], 0u, 0x4440u + (m & 3));
                        s = s + lut_col[m * kKsub * R + byte * R];
                    }
                    if (first + j * (32 * VPL) + lane * VPL + e >= n) s = __int_as_float(0x7fc00000);
                    acc[j][e] = s;
                    any |= s <= thr;
                }
            }
            if (!__any_sync(0xffffffffu, any)) continue;
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < VPL; ++e) {
                    const uint32_t pos = pos0 + first + j * (32 * VPL) + lane * VPL + e;
                    bool pass = acc[j][e] <= thr;
                    if (!RESID && label_max != ~0ull && acc[j][e] == thr)
                        pass = (static_cast<uint64_t>(__ldg(a.ids + pos)) ^ (1ull << 63)) <= label_max;
                    const unsigned bal = __ballot_sync(0xffffffffu, pass);
                    if (!bal) continue;
                    uint32_t slot = 0;
                    if (lane == 0) slot = atomicAdd(a.count + q, static_cast<uint32_t>(__popc(bal)));
                    slot = __shfl_sync(0xffffffffu, slot, 0) + __popc(bal & ((1u << lane) - 1u));
                    if (pass && slot < a.cap) {
                        a.cand[q * a.cap + slot] = make_uint2(pos, __float_as_uint(acc[j][e]));
                        if (RESID) a.probe[q * a.cap + slot] = static_cast<uint16_t>(l);
                    }
                }
        }
    }
}

// ---- 2'. scan of wide codes ----
// The table of the wide-code filter (see ivfpq_index.cu): rows of 32 columns, the 16 sub-quantizers of a
// group twice, lane l at sub-quantizer (s + l) mod 16 in step s, so that 32 lanes read 32 banks.  A lane
// holds one vector; the codes of the next 32 vectors are on their way while 32 are looked up.
template <int MT, bool RESID>
__global__ void __launch_bounds__(kWideThreads, MT <= 3 ? 2 : 1)
wide_scan_kernel(const ShortScanArgs a, int S) {
    constexpr uint32_t U = 128;    // vectors of a unit
    extern __shared__ __align__(16) float wide_sm[];
    float* lut = wide_sm;                                                   // [MT][256][32]
    uint32_t* upre = reinterpret_cast<uint32_t*>(lut + MT * kKsub * 32);    // [nprobe + 1] units before the probe
    uint32_t* beg = upre + a.nprobe + 1;
    uint32_t* len = beg + a.nprobe;
    float* base = reinterpret_cast<float*>(len + a.nprobe);
    __shared__ uint32_t s_warp[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lut_base = static_cast<uint32_t>(__cvta_generic_to_shared(lut));
    uint32_t col[16];
#pragma unroll
    for (int s = 0; s < 16; ++s) col[s] = lut_base + 4u * (((s + lane) & 15) + (lane & 16));
    const int64_t items = a.nq * S;
    const int64_t it0 = items * blockIdx.x / gridDim.x, it1 = items * (blockIdx.x + 1) / gridDim.x;
    int64_t cur_q = -1;
    uint32_t units = 0;
    float thr = 0.f;
    const uint4* codes4 = reinterpret_cast<const uint4*>(a.codes);
    for (int64_t it = it0; it < it1; ++it) {
        const int64_t q = it / S;
        const uint32_t split = static_cast<uint32_t>(it - q * S);
        if (q != cur_q) {
            __syncthreads();   // the previous query's table and probes are still read
            cur_q = q;
            const float4* src = reinterpret_cast<const float4*>(a.lut + q * (MT * 16 * kKsub));
            for (int i = threadIdx.x; i < MT * kKsub * 4; i += kWideThreads) {
                const float4 v = __ldg(src + i);
                float4* row = reinterpret_cast<float4*>(lut) + (i >> 2) * 8 + (i & 3);
                row[0] = v;
                row[4] = v;
            }
            units = 0;
            for (int p0 = 0; p0 < a.nprobe; p0 += kWideThreads) {
                const int p = p0 + threadIdx.x;
                Probe pr{0u, 0u, 0.f};
                if (p < a.nprobe) pr = load_probe(a, q, p);
                uint32_t sum;
                const uint32_t ex = block_exclusive((pr.len + U - 1) / U, s_warp, &sum);
                if (p < a.nprobe) {
                    upre[p] = units + ex;
                    beg[p] = pr.begin;
                    len[p] = pr.len;
                    base[p] = pr.base;
                }
                units += sum;
            }
            thr = a.thr[q];
            __syncthreads();
        }
        const uint32_t u0 = static_cast<uint32_t>(static_cast<uint64_t>(units) * split / S);
        const uint32_t u1 = static_cast<uint32_t>(static_cast<uint64_t>(units) * (split + 1) / S);
        for (uint32_t u = u0 + warp; u < u1; u += kWideThreads / 32) {
            int l = 0, h = a.nprobe;   // last probe with upre[p] <= u: the one that holds unit u
            while (h - l > 1) {
                const int mid = (l + h) >> 1;
                if (upre[mid] <= u) l = mid;
                else h = mid;
            }
            const uint32_t first = (u - upre[l]) * U, n = len[l], pos0 = beg[l];
            const float bias = RESID ? base[l] : 0.f;
            const uint32_t last = min(first + U, n);
            uint4 c[MT], d[MT];
            float t = 0.f, tn = 0.f;
            // (lists are stored padded to 32 vectors: the loads stay inside the list)
            auto fetch = [&](uint32_t i, uint4 (&dst)[MT], float& t2) {
                const size_t v = pos0 + i + lane;
#pragma unroll
                for (int g = 0; g < MT; ++g) dst[g] = __ldg(codes4 + v * MT + g);
                if (RESID) t2 = __ldg(a.t2 + v);
            };
            auto process = [&](uint32_t i, const uint4 (&cc)[MT], float t2) {
                float acc = RESID ? bias + t2 : 0.f;
#pragma unroll
                for (int g = 0; g < MT; ++g) {
                    const uint32_t w[4] = {cc[g].x, cc[g].y, cc[g].z, cc[g].w};
#pragma unroll
                    for (int s = 0; s < 16; ++s) {
                        const uint32_t addr = __byte_perm(w[s >> 2], 0u, 0x4440u + (s & 3)) * 128u + col[s];
                        float val;
                        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(val) : "r"(addr + static_cast<uint32_t>(g) * (kKsub * 32 * 4)));
                        acc = acc + val;
                    }
                }
                const bool pass = i + lane < n && acc <= thr;
                const unsigned bal = __ballot_sync(0xffffffffu, pass);
                if (!bal) return;
                uint32_t slot = 0;
                if (lane == 0) slot = atomicAdd(a.count + q, static_cast<uint32_t>(__popc(bal)));
                slot = __shfl_sync(0xffffffffu, slot, 0) + __popc(bal & ((1u << lane) - 1u));
                if (pass && slot < a.cap) {
                    a.cand[q * a.cap + slot] = make_uint2(pos0 + i + lane, __float_as_uint(acc));
                    if (RESID) a.probe[q * a.cap + slot] = static_cast<uint16_t>(l);
                }
            };
            fetch(first, c, t);
            for (uint32_t i = first; i < last; i += 64) {
                if (i + 32 < last) fetch(i + 32, d, tn);
                process(i, c, t);
                if (i + 64 < last) fetch(i + 64, c, t);
                if (i + 32 < last) process(i + 32, d, tn);
            }
        }
    }
}

// ---- 3. exact order ----
// Rank search over unsigned keys of `bits` bits, eight at a time; key(i, &v) says whether entry i takes
// part.  Returns the r-th smallest (1-based); *left = rank among the entries equal to it.
template <typename KeyT, typename F>
__device__ KeyT block_kth(F key, uint32_t n, uint32_t r, uint32_t* hist, uint32_t* s_warp, uint32_t* s_out, uint32_t* left) {
    KeyT prefix = 0, mask = 0;
    for (int shift = static_cast<int>(sizeof(KeyT)) * 8 - 8; shift >= 0; shift -= 8) {
        if (threadIdx.x < 256) hist[threadIdx.x] = 0u;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < n; i += kSelThreadsShort) {
            KeyT v;
            if (key(i, v) && (v & mask) == prefix) atomicAdd(&hist[static_cast<uint32_t>(v >> shift) & 255u], 1u);
        }
        __syncthreads();
        const uint32_t h = threadIdx.x < 256 ? hist[threadIdx.x] : 0u;
        uint32_t all;
        const uint32_t ex = block_exclusive(h, s_warp, &all);
        if (ex < r && ex + h >= r) {
            s_out[0] = threadIdx.x;
            s_out[1] = ex;
        }
        __syncthreads();
        prefix |= static_cast<KeyT>(s_out[0]) << shift;
        mask |= static_cast<KeyT>(255) << shift;
        r -= s_out[1];
        __syncthreads();
    }
    *left = r;
    return prefix;
}

__global__ void __launch_bounds__(kSelThreadsShort, 3)
short_select_kernel(const ShortScanArgs a) {
    __shared__ __align__(16) int64_t sl[kSortMax];
    __shared__ float sd[kSortMax];
    __shared__ uint32_t hist[256], s_warp[32], s_out[2], s_fill, s_eq;
    const int64_t q = blockIdx.x;
    const uint32_t n = a.count[q];
    if (n > a.cap) {
        if (threadIdx.x == 0) a.flag[q] = n == kShortExact ? 3 : n > kShortMaxCap ? 2 : 1;
        return;
    }
    uint2* row = a.cand + q * a.cap;
    const uint32_t k = static_cast<uint32_t>(a.k);
    if (a.by_residual || a.rotated) {
        // Scanned distances are off by eps at most: k of them lie at or below their k-th smallest, so whatever
        // exceeds that by more than 2 eps is out (marked 0xFFFFFFFF); the others get their canonical distance.
        __shared__ RankScratch rank;
        const uint32_t kth_scan = block_kth32<kSelThreadsShort>(
            [&](auto&& f) { for (uint32_t i = threadIdx.x; i < n; i += kSelThreadsShort) f(float_to_ord(__uint_as_float(row[i].y))); },
            k, rank, 2);
        float lim = __uint_as_float(kInfBits);   // fewer than k: all of them
        if (kth_scan != 0xFFFFFFFFu) {
            lim = ord_to_float(kth_scan) + 2.f * a.eps[q];
            lim = lim + fabsf(lim) * 9.5367431640625e-07f;   // the rounding of the sum
            if (!(lim <= __uint_as_float(kInfBits))) lim = __uint_as_float(kInfBits);
        }
        // survivors first, so that full warps work on them (sl doubles as their list)
        uint32_t* live = reinterpret_cast<uint32_t*>(sl);
        if (threadIdx.x == 0) s_fill = 0u;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < n; i += kSelThreadsShort) {
            if (__uint_as_float(row[i].y) <= lim) {
                const uint32_t slot = atomicAdd(&s_fill, 1u);
                if (slot < 2u * kSortMax) live[slot] = i;
            }
        }
        __syncthreads();
        const uint32_t nl = s_fill;
        const bool listed = nl <= 2u * kSortMax;
        auto refine = [&](uint32_t i) {
            const uint2 c = row[i];
            const int64_t list = a.by_residual ? a.cI[q * a.nprobe + a.probe[q * a.cap + i]] : 0;
            return __float_as_uint(exact_distance(a, q, c.x, list));
        };
        if (listed) {
            uint32_t* val = reinterpret_cast<uint32_t*>(sd);   // [kSortMax]: results wait there until the others are marked
            for (uint32_t j0 = 0; j0 < nl; j0 += kSortMax) {
                const uint32_t j1 = min(nl, j0 + kSortMax);
                for (uint32_t j = j0 + threadIdx.x; j < j1; j += kSelThreadsShort) val[j - j0] = refine(live[j]);
                __syncthreads();
                if (j0 == 0)
                    for (uint32_t i = threadIdx.x; i < n; i += kSelThreadsShort)
                        if (!(__uint_as_float(row[i].y) <= lim)) row[i].y = 0xFFFFFFFFu;
                __syncthreads();
                for (uint32_t j = j0 + threadIdx.x; j < j1; j += kSelThreadsShort) row[live[j]].y = val[j - j0];
                __syncthreads();
            }
        } else {
            for (uint32_t i = threadIdx.x; i < n; i += kSelThreadsShort)
                row[i].y = __uint_as_float(row[i].y) <= lim ? refine(i) : 0xFFFFFFFFu;
            __syncthreads();
        }
    }
    auto dist_key = [&](uint32_t i, uint32_t& v) { v = row[i].y; return v != 0xFFFFFFFFu; };
    // Distances are >= 0: their bits order like the values.  All candidates when they fit the sort, else
    // those below the k-th distance and as many of the ties with it as there is room for -- the ones with
    // the smallest labels when there are more.
    uint32_t kth = 0xFFFFFFFFu;
    uint64_t label_max = ~0ull;         // ties up to this label (sign bit flipped) ...
    uint32_t eq_take = 0xFFFFFFFFu;     // ... and so many that have exactly this one
    if (n > static_cast<uint32_t>(kSortMax)) {
        uint32_t need;                  // ties that belong to the result
        kth = block_kth<uint32_t>(dist_key, n, k, hist, s_warp, s_out, &need);
        if (threadIdx.x == 0) s_fill = 0u;
        __syncthreads();
        uint32_t ties = 0;
        for (uint32_t i = threadIdx.x; i < n; i += kSelThreadsShort) ties += row[i].y == kth ? 1u : 0u;
        atomicAdd(&s_fill, ties);
        __syncthreads();
        ties = s_fill;
        if (k - need + ties > static_cast<uint32_t>(kSortMax)) {
            auto label_key = [&](uint32_t i, uint64_t& v) {
                const uint2 c = row[i];
                if (c.y != kth) return false;
                v = static_cast<uint64_t>(a.ids[c.x]) ^ (1ull << 63);
                return true;
            };
            label_max = block_kth<uint64_t>(label_key, n, need, hist, s_warp, s_out, &eq_take);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        s_fill = 0u;
        s_eq = 0u;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += kSelThreadsShort) {
        const uint2 c = row[i];
        if (c.y > kth || c.y == 0xFFFFFFFFu) continue;
        const int64_t label = a.ids[c.x];
        if (c.y == kth) {
            const uint64_t u = static_cast<uint64_t>(label) ^ (1ull << 63);
            if (u > label_max) continue;
            if (u == label_max && atomicAdd(&s_eq, 1u) >= eq_take) continue;
        }
        const uint32_t slot = atomicAdd(&s_fill, 1u);
        if (slot < static_cast<uint32_t>(kSortMax)) {
            sd[slot] = __uint_as_float(c.y);
            sl[slot] = label;
        }
    }
    __syncthreads();
    const uint32_t m = min(s_fill, static_cast<uint32_t>(kSortMax));
    uint32_t P = 32;
    while (P < m) P <<= 1;
    for (uint32_t i = m + threadIdx.x; i < P; i += kSelThreadsShort) {
        sd[i] = __uint_as_float(kInfBits);
        sl[i] = kNoLabel;
    }
    __syncthreads();
    for (uint32_t size = 2; size <= P; size <<= 1)
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
            for (uint32_t i = threadIdx.x; i < P / 2; i += kSelThreadsShort) {
                const uint32_t lo = 2 * i - (i & (stride - 1)), hi = lo + stride;
                const bool up = (lo & size) == 0;
                const float d1 = sd[lo], d2 = sd[hi];
                const int64_t l1 = sl[lo], l2 = sl[hi];
                const bool less21 = d2 < d1 || (d2 == d1 && l2 < l1);
                if (less21 == up) {
                    sd[lo] = d2; sd[hi] = d1;
                    sl[lo] = l2; sl[hi] = l1;
                }
            }
            __syncthreads();
        }
    for (uint32_t i = threadIdx.x; i < k; i += kSelThreadsShort) {
        const bool real = i < m;
        a.outD[q * a.k + i] = real ? sd[i] : kPadDist;
        a.outI[q * a.k + i] = real ? sl[i] : -1;
    }
}

template <int M>
cudaError_t launch_m(const ShortScanArgs& a, int num_sms, cudaStream_t st) {
    const size_t bound_smem = static_cast<size_t>(M * kKsub + kBins + 3 * kShortMaxProbe + 1 + a.d + a.n1_max) * 4;
    cudaError_t e = allow_max_smem(short_bound_kernel<M>);
    if (e != cudaSuccess) return e;
    short_bound_kernel<M><<<static_cast<unsigned>(a.nq), bound_threads<M>(), bound_smem, st>>>(a);
    // About eight shares per block: the blocks' loads differ by one share at most, and a block
    // changes queries (128 KB of table to fill) as seldom as the batch allows.
    const int S = static_cast<int>(std::max<int64_t>(1, (8LL * num_sms + a.nq - 1) / a.nq));
    const int grid = static_cast<int>(std::min<int64_t>(num_sms, a.nq * S));
    const size_t scan_smem = static_cast<size_t>(M * kKsub * replicas<M>() + 4 * kShortMaxProbe + 1) * 4;
    auto kern = a.by_residual ? short_scan_kernel<M, true> : short_scan_kernel<M, false>;
    e = allow_max_smem(kern);
    if (e != cudaSuccess) return e;
    kern<<<grid, kScanThreadsShort, scan_smem, st>>>(a, S);
    short_select_kernel<<<static_cast<unsigned>(a.nq), kSelThreadsShort, 0, st>>>(a);
    return cudaGetLastError();
}

template <int M>
cudaError_t launch_wide(const ShortScanArgs& a, int num_sms, cudaStream_t st) {
    constexpr int MT = M / 16;
    const size_t bound_smem = static_cast<size_t>(M * kKsub + kBins + 3 * kShortMaxProbe + 1 + a.d + a.n1_max) * 4;
    cudaError_t e = allow_max_smem(short_bound_kernel<M>);
    if (e != cudaSuccess) return e;
    short_bound_kernel<M><<<static_cast<unsigned>(a.nq), bound_threads<M>(), bound_smem, st>>>(a);
    const size_t smem = static_cast<size_t>(MT * kKsub * 32 + 4 * a.nprobe + 1) * 4;
    auto kern = a.by_residual ? wide_scan_kernel<MT, true> : wide_scan_kernel<MT, false>;
    e = allow_max_smem(kern);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kWideThreads, smem);
    if (e != cudaSuccess) return e;
    const int64_t blocks = static_cast<int64_t>(num_sms) * std::max(1, per_sm);
    // shares as in launch_m
    const int S = static_cast<int>(std::max<int64_t>(1, (4LL * blocks + a.nq - 1) / a.nq));
    kern<<<static_cast<unsigned>(std::min<int64_t>(blocks, a.nq * S)), kWideThreads, smem, st>>>(a, S);
    short_select_kernel<<<static_cast<unsigned>(a.nq), kSelThreadsShort, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_short_scan(const ShortScanArgs& a, int num_sms, cudaStream_t st) {
    switch (a.M) {
        case 4: return launch_m<4>(a, num_sms, st);
        case 8: return launch_m<8>(a, num_sms, st);
        case 16: return launch_wide<16>(a, num_sms, st);
        case 32: return launch_wide<32>(a, num_sms, st);
        case 48: return launch_wide<48>(a, num_sms, st);
        case 64: return launch_wide<64>(a, num_sms, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace b200
