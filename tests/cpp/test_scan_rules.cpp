// Which scan an IVFPQ search takes (host code only): on both sides of every line of the rules.
#include "../../indexsdk_b200/csrc/ivfpq_short_scan.cuh"

#include <cstdio>

static int failed = 0;
static void wide(bool want, int M, double visited, int nprobe, int k, int64_t nq) {
    if (b200::use_bounded_scan(M, visited, nprobe, k, nq) == want) return;
    std::printf("FAILED: M = %d, %.0f vectors, %d probes, k = %d, %lld queries\n", M, visited, nprobe, k, static_cast<long long>(nq));
    ++failed;
}
static void small(bool want, int M, bool residual, double visited, int nprobe, int k) {
    if (b200::use_short_scan(M, residual, visited, nprobe, k) == want) return;
    std::printf("FAILED: M = %d, residual %d, %.0f vectors, %d probes, k = %d\n", M, residual, visited, nprobe, k);
    ++failed;
}

int main() {
    // sorted lists in registers: short ones for large batches, any once they are full
    wide(true, 48, 39000, 128, 100, 1000);
    wide(true, 16, 500e3, 128, 100, 512);
    wide(false, 16, 1e6, 256, 100, 512);
    wide(false, 48, 781e3, 128, 100, 10000);
    wide(true, 48, 1e6, 256, 300, 512);
    wide(true, 48, 1e6, 256, 10, 64);
    wide(false, 48, 3e6, 768, 10, 64);
    wide(true, 48, 102e3, 26, 10, 512);
    wide(false, 48, 500e3, 128, 10, 512);
    wide(false, 16, 39000, 64, 10, 100);
    wide(false, 48, 15000, 64, 10, 512);
    wide(true, 64, 31000, 64, 10, 2048);
    wide(false, 48, 31000, 64, 10, 2048);
    // where the bound is not worth its launch, and beyond what its kernels hold
    wide(false, 48, 2000, 64, 100, 64);
    wide(false, 48, 39000, 1025, 100, 64);
    wide(false, 24, 39000, 64, 100, 64);
    small(true, 4, false, 8192, 8, 10);
    small(false, 4, false, 8191, 8, 10);
    small(true, 4, false, 1024, 8, 65);
    small(true, 8, true, 1, 2, 10);
    small(false, 8, true, 511, 1, 10);
    small(false, 8, true, 1e6, 1025, 10);
    small(false, 8, true, 1e6, 8, 1025);
    small(false, 12, true, 1e6, 8, 10);
    // given probes that all name one list of 2^22 vectors
    if (!b200::counts_fit(1 << 22, 1023) || b200::counts_fit(1 << 22, 1024) || b200::counts_fit(int64_t(1) << 30, 1024)) {
        std::printf("FAILED: counts of repeated lists\n");
        ++failed;
    }
    std::printf("%d failed\n", failed);
    return failed != 0;
}
