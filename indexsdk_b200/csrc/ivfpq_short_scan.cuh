// IVFPQ scan with a bound, for short codes (M = 4 or 8 bytes) and for large k, see ivfpq_short_scan.cu.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

constexpr int kShortMaxProbe = 1024;     // probes whose metadata a block stages in shared memory
constexpr uint32_t kShortMaxBound = 16384;   // vectors the bound is taken from (wide codes: half as many)
constexpr uint32_t kShortMaxCap = 32768; // most candidates a query may collect; more take another scan
constexpr uint32_t kShortExact = 0xFFFFFFFFu;   // count of a query that needs the exact scan

struct ShortScanArgs {
    const int64_t* cI;       // [nq][nprobe] probed list ids (-1 = none), nearest first
    const float* cD;         // [nq][nprobe] coarse distances
    int nprobe, nlist, k, M, d, dsub;
    int64_t nq;
    const int64_t* offsets;  // [nlist + 1] first position of every list (multiples of 32)
    const int64_t* lens;     // [nlist]
    const uint8_t* codes;    // [positions][M]
    int rotated;             // M = 16, 32, 48, 64: bytes of a 16-byte group rotated by the position
    const int64_t* ids;
    const float* t2;         // residual encoding: the per-vector term
    int by_residual;
    const float* xq;         // [nq][d]
    const float* centroids;  // [nlist][d]
    const float* codebooks;  // [M][256][dsub]
    const float* cbT;        // rotated codes: regrouped [M / 16][256][16][dsub]
    float err_rel, t2_bound, cb_bound;   // filter error bound of residual encoding (see IvfpqIndex::search_stages)
    // scratch
    float* lut;              // [nq][M][256], rotated codes [nq][M / 16][256][16]
    float* eps;              // [nq] error of a scanned distance that matters
    float* thr;              // [nq] collect below ...
    uint64_t* label_max;     // [nq] ... and at it the labels up to this one (sign bit flipped; raw encoding)
    uint32_t* count;         // [nq]
    uint2* cand;             // [nq][cap] (position, distance bits)
    uint16_t* probe;         // [nq][cap] which probe (residual encoding)
    uint32_t cap;
    uint32_t n1_max;         // most vectors a query's bound is taken from (shared memory of that kernel)
    // results
    float* outD;             // [nq][k]
    int64_t* outI;
    uint8_t* flag;           // [nq] written when the query has more than cap candidates: 1, or 2 for more than kShortMaxCap;
                             // 3 = exact scan
    unsigned long long* scanned;
};

// Whether this scan takes a search, and takes less time than the exact one.  visited: vectors a query's
// lists hold on average.  Its three kernels and the 128 KB table cost a query as much as the exact scan
// needs for about 32 000 lookups (d 128, 1 024 queries, k = 10: M = 4, 3 900 vectors 319 us against 275,
// 15 600 321 against 327, 62 500 474 against 642; M = 8, 780 vectors 217 against 195, 3 100 256 against 272), or
// fewer when k is large (k = 100: 265 against 355 at 3 100 vectors).  The exact scan of residual codes
// builds a table per list: two lists are enough (4 lists of 50 vectors, M = 8: 231 us against 353).
// There is no line above: in clustered data the exact scan is ten times slower at any size (M = 4, 512 queries of
// 1 M vectors, k = 900: 8.1 ms against 0.84), and where lists are no better than one another and most queries of a
// large k end up with it after all, bound and scan come on top of it (23.3 ms against 28.3).
inline bool use_short_scan(int M, bool residual, double visited, int nprobe, int k) {
    if ((M != 4 && M != 8) || nprobe > kShortMaxProbe || k > 1024) return false;
    if (residual && nprobe > 1) return true;
    return visited * M >= (residual || k > 64 ? 4096.0 : 32768.0);
}
// Wide codes (M = 16, 32, 48, 64): sorted lists in registers are a good filter while they are short (k' = 32 or
// 64, k <= 48) and the batch is large; otherwise the insertions, or the one block per query and split, cost
// more than the bound does.  nq queries, us before / this way (1 M vectors, residual codes):
//   k = 100, 3 900 vectors visited, 512 queries: M = 16 230 / 168, M = 64 424 / 246; k = 300: 1 149 / 199, 1 661 / 280
//   k = 100, 31 000, 2 048 queries: M = 16 861 / 650, M = 32 1 471 / 894, M = 48 1 795 / 1 209, M = 64 3 333 / 1 653
//   k = 10,  3 900, 64 queries: M = 32 108 / 106, M = 64 123 / 112;   512 queries: M = 32 148 / 179, M = 64 220 / 246
//   k = 10,  31 000, 512 queries: M = 32 427 / 307, M = 48 497 / 414, M = 64 831 / 501
//   k = 10,  31 000, 2 048 queries: M = 16 375 / 645, M = 32 859 / 886, M = 48 1 036 / 1 202, M = 64 2 020 / 1 646
// Below about 2 000 vectors a query the bound is not worth its launch.  16-byte codes with k <= 48 stay with the
// lists: their tables are small, and the persistent kernel takes over from 1 184 queries on.
// The other way round, once the lists are full, hardly a vector gets past them, and the filter's loop is the
// faster one (4 M vectors, 1 024 lists, us before / this way; vectors near their centroids, and without structure):
//   k = 10,  M = 48, 64 queries of 1.0 M: 1 324 / 1 045 and 4 491 / 2 140;  of 3.0 M: 2 537 / 2 903 and 5 922 / 3 613
//   k = 10,  M = 48, 512 queries of 102 k: 1 032 / 863 and 5 377 / 3 074;   of 500 k: 2 969 / 3 565 and 11 385 / 9 881
//   k = 100, M = 16, 512 queries of 500 k: 1 805 / 1 452 and 5 147 / 4 234; of 1.0 M: 2 778 / 2 950, of 3.0 M: 6 773 / 8 526
//   k = 100, M = 48, 512 queries of 500 k: 3 736 / 3 577 and 12 869 / 9 909; of 1.0 M: 5 809 / 7 191
//   k = 100, M = 48, 10 000 queries of 781 k (100 M vectors, 16 384 lists): 20.9 ms / 26.9
// so the product of queries and vectors has a limit.  Longer lists (k > 112: k' of 256 and more) never catch up
// in that range (k = 300, M = 48, 512 queries of 102 k: 10 692 / 905 and 24 182 / 4 029).
inline bool use_bounded_scan(int M, double visited, int nprobe, int k, int64_t nq) {
    if (M % 16 != 0 || M > 64 || k > 1024 || nprobe > kShortMaxProbe || visited < 2048.0) return false;
    const double all = visited * static_cast<double>(nq);
    if (k > 48) return k > 112 || all <= 3e8;
    if (M == 16 || all > 1.3e8) return false;
    if (nq <= 64) return true;
    return visited >= 16384.0 && (nq <= 1024 || M == 64);
}
// Given probes may name a list as often as they like, and a query's vectors are counted in 32 bits.
inline bool counts_fit(int64_t longest_list, int nprobe) { return longest_list * nprobe <= 0xFFFFFFFFll; }
cudaError_t launch_short_scan(const ShortScanArgs& a, int num_sms, cudaStream_t st);

}  // namespace b200
