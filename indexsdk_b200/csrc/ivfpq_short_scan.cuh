// IVFPQ scan for short codes (M = 4 or 8 bytes), see ivfpq_short_scan.cu.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

constexpr int kShortMaxProbe = 1024;     // probes whose metadata a block stages in shared memory
constexpr uint32_t kShortMaxBound = 32768;   // vectors the bound is taken from
constexpr uint32_t kShortMaxCap = 32768; // candidates a query may collect; more take the exact scan

struct ShortScanArgs {
    const int64_t* cI;       // [nq][nprobe] probed list ids (-1 = none), nearest first
    const float* cD;         // [nq][nprobe] coarse distances
    int nprobe, nlist, k, M, d, dsub;
    int64_t nq;
    const int64_t* offsets;  // [nlist + 1] first position of every list (multiples of 32)
    const int64_t* lens;     // [nlist]
    const uint8_t* codes;    // [positions][M], not rotated
    const int64_t* ids;
    const float* t2;         // residual encoding: the per-vector term
    int by_residual;
    const float* xq;         // [nq][d]
    const float* centroids;  // [nlist][d]
    const float* codebooks;  // [M][256][dsub]
    float err_rel, t2_bound, cb_bound;   // filter error bound of residual encoding (see IvfpqIndex::search_stages)
    // scratch
    float* lut;              // [nq][M][256]
    float* thr;              // [nq] collect below ...
    uint64_t* label_max;     // [nq] ... and at it the labels up to this one (sign bit flipped; raw encoding)
    uint32_t* count;         // [nq]
    uint2* cand;             // [nq][cap] (position, distance bits | probe)
    uint32_t cap;
    uint32_t n1_max;         // most vectors a query's bound is taken from (shared memory of that kernel)
    // results
    float* outD;             // [nq][k]
    int64_t* outI;
    uint8_t* flag;           // [nq] 1 = more than cap candidates, the query needs the exact scan
    unsigned long long* scanned;
};

// Whether this scan takes a search, and takes less time than the exact one.  visited: vectors a query's
// lists hold on average.  Its three kernels and the 128 KB table cost a query as much as the exact scan
// needs for about 32 000 lookups (d 128, 1 024 queries, k = 10: M = 4, 3 900 vectors 319 us against 275,
// 15 600 321 against 327, 62 500 474 against 642; M = 8, 780 vectors 217 against 195, 3 100 256 against 272), or
// fewer when k is large (k = 100: 265 against 355 at 3 100 vectors).  The exact scan of residual codes
// builds a table per list: two lists are enough (4 lists of 50 vectors, M = 8: 231 us against 353).
inline bool use_short_scan(int M, bool residual, double visited, int nprobe, int k) {
    if ((M != 4 && M != 8) || nprobe > kShortMaxProbe || k > 1024) return false;
    if (residual && nprobe > 1) return true;
    return visited * M >= (residual || k > 64 ? 4096.0 : 32768.0);
}
cudaError_t launch_short_scan(const ShortScanArgs& a, int num_sms, cudaStream_t st);

}  // namespace b200
