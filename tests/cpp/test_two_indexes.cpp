// Two host threads, each searching an index of its own on one GPU.  The indexes go through the same kernels with
// different amounts of shared memory; every search has to succeed and to find what it found alone.
#include <b200idx.h>

#include <atomic>
#include <cstdio>
#include <cstring>
#include <random>
#include <string>
#include <thread>
#include <vector>

struct Job {
    b200idx_t* ix = nullptr;
    int n = 1, k = 1;
    std::vector<float> xq;
    std::vector<signed char> xq8;
    std::vector<float> D;
    std::vector<int64_t> I;
    const void* queries() const { return xq8.empty() ? static_cast<const void*>(xq.data()) : xq8.data(); }
};

static std::atomic<int> failed{0};
static void must(int rc, const b200idx_t* ix, const char* what) {
    if (rc == B200IDX_OK) return;
    if (++failed <= 5) std::printf("FAILED %s: %d %s\n", what, rc, b200idx_last_error(ix));
}
static std::vector<float> gaussian(size_t n, unsigned seed) {
    std::mt19937 g(seed);
    std::normal_distribution<float> f;
    std::vector<float> x(n);
    for (float& v : x) v = f(g);
    return x;
}

static Job int8_index(int k) {
    Job j;
    const int d = 32, n = 4000;
    must(b200idx_create_int8flat(d, B200IDX_METRIC_L2, 0, &j.ix), nullptr, "create");
    std::mt19937 g(static_cast<unsigned>(k));
    std::vector<signed char> x(static_cast<size_t>(n) * d);
    for (signed char& v : x) v = static_cast<signed char>(static_cast<int>(g() % 256) - 128);
    must(b200idx_add(j.ix, n, x.data(), nullptr), j.ix, "add");
    j.xq8.assign(x.begin(), x.begin() + d);
    j.k = k;
    return j;
}
static Job fp32_index(int d) {
    Job j;
    must(b200idx_create_flat(d, B200IDX_METRIC_L2, B200IDX_F32, 0, &j.ix), nullptr, "create");
    must(b200idx_add(j.ix, 9000, gaussian(static_cast<size_t>(9000) * d, 1).data(), nullptr), j.ix, "add");
    j.xq = gaussian(static_cast<size_t>(d), 2);
    j.k = 10;
    return j;
}
static Job ivfpq_index(int k) {
    Job j;
    const int d = 16, M = 16, nlist = 8, n = 4000;
    must(b200idx_create_ivfpq(d, B200IDX_METRIC_L2, nlist, M, 8, 0, 0, &j.ix), nullptr, "create");
    must(b200idx_ivfpq_set_centroids(j.ix, gaussian(nlist * d, 1).data()), j.ix, "centroids");
    must(b200idx_ivfpq_set_codebooks(j.ix, gaussian(256 * d, 2).data()), j.ix, "codebooks");
    must(b200idx_add(j.ix, n, gaussian(static_cast<size_t>(n) * d, 3).data(), nullptr), j.ix, "add");
    must(b200idx_ivfpq_set_nprobe(j.ix, nlist), j.ix, "nprobe");
    j.xq = gaussian(d, 4);
    j.k = k;
    return j;
}

static void search(Job& j, std::vector<float>& D, std::vector<int64_t>& I) {
    D.assign(static_cast<size_t>(j.n) * j.k, 0.f);
    I.assign(static_cast<size_t>(j.n) * j.k, -2);
    must(b200idx_search(j.ix, j.n, j.queries(), j.k, D.data(), I.data()), j.ix, "search");
}

int main(int argc, char** argv) {
    const std::string which = argc > 1 ? argv[1] : "";
    std::vector<Job> jobs;
    if (which == "select") {           // sorted entries beside the staged ones
        jobs.push_back(int8_index(1000));
        jobs.push_back(int8_index(129));
    } else if (which == "finish") {    // fp32 lists of one query, rows of 4 096 and of 64 floats
        jobs.push_back(fp32_index(4096));
        jobs.push_back(fp32_index(64));
    } else {                           // the bound of 16-byte codes
        jobs.push_back(ivfpq_index(900));
        jobs.push_back(ivfpq_index(60));
    }
    for (Job& j : jobs) search(j, j.D, j.I);
    std::vector<std::thread> threads;
    for (Job& j : jobs)
        threads.emplace_back([&j] {
            std::vector<float> D;
            std::vector<int64_t> I;
            for (int r = 0; r < 20000 && failed < 5; ++r) {
                search(j, D, I);
                if (std::memcmp(D.data(), j.D.data(), D.size() * 4) != 0 || I != j.I)
                    if (++failed <= 5) std::printf("FAILED: another result in round %d\n", r);
            }
        });
    for (std::thread& t : threads) t.join();
    for (Job& j : jobs) b200idx_destroy(j.ix);
    std::printf("%d failed\n", failed.load());
    return failed != 0;
}
