#include "multi_flat.h"

#include <algorithm>
#include <limits>
#include <stdexcept>
#include <string>

#include "select.cuh"

namespace b200 {
namespace {

constexpr int64_t kMaxMemberRows = 65536;                 // larger members use the thresholded pipeline of their own
constexpr size_t kGroupCandBytes = size_t(2) << 30;       // candidate scratch per pass
constexpr size_t kGroupBaseBytes = size_t(8) << 30;       // operand, norms and exact rows of all members
inline int64_t pad_tile(int64_t n) { return (n + kTileB - 1) / kTileB * kTileB; }
inline size_t op_elem(int dtype) { return dtype == kI8 ? 1 : 2; }

// Operand rows and norms of one tile, a block each; rows past the member's end are zeros (their keys
// are never read: the epilogue stops at the end of the member).  packed: a tile is one image, copied whole.
__global__ void gather_members_kernel(const MemberView* members, const int32_t* seg_index, int row_bytes, int packed,
                                      uint4* xop, uint32_t* norms) {
    const int64_t t = blockIdx.x;
    const MemberView v = members[seg_index[t]];
    const int64_t row0 = t * kTileB - v.first;
    const int rows = static_cast<int>(v.n - row0 < kTileB ? v.n - row0 : kTileB);
    const int row_words = row_bytes / 16, words = kTileB * row_words, real = packed ? words : rows * row_words;
    const uint4* src = reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(v.operand) + row0 * row_bytes);
    uint4* dst = xop + t * words;
    for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = i < real ? __ldg(src + i) : make_uint4(0u, 0u, 0u, 0u);
    for (int i = threadIdx.x; i < kTileB; i += blockDim.x)
        norms[t * kTileB + i] = i < rows ? __ldg(static_cast<const uint32_t*>(v.norms) + row0 + i) : 0u;
}

}  // namespace

bool FlatGroup::eligible(const std::vector<FlatIndex*>& m, int64_t nq, int k) {
    if (m.size() < 2 || nq <= 0 || nq > 0x7FFFFFFF / static_cast<int64_t>(m.size())) return false;
    int64_t cap = 0, total = 0;
    for (const FlatIndex* ix : m) {
        if (ix->ntotal() <= 0 || ix->ntotal() > kMaxMemberRows) return false;
        cap = std::max(cap, pad_tile(ix->ntotal()));
        total += pad_tile(ix->ntotal());
    }
    if (k > cap) return false;   // (short results are padded by the per-index path)
    const size_t row = static_cast<size_t>(m[0]->op_cols()) * op_elem(m[0]->dtype()) +
                       (m[0]->dtype() == kF32 ? static_cast<size_t>(m[0]->d()) * 4 : 0) + 12;
    if (static_cast<size_t>(total) * row > kGroupBaseBytes) return false;
    // one member's candidate rows must fit a pass (members are paged, queries are not)
    return static_cast<size_t>(nq) * static_cast<size_t>(cap) * 8 <= kGroupCandBytes;
}

void FlatGroup::refresh(const std::vector<FlatIndex*>& members, cudaStream_t st) {
    bool same = cur_.size() == members.size();
    for (size_t i = 0; same && i < members.size(); ++i)
        same = cur_[i] == members[i] && cur_gen_[i] == members[i]->generation();
    if (same) return;
    cur_.clear();
    const FlatIndex* f0 = members[0];
    d_ = f0->d();
    metric_ = f0->metric();
    dtype_ = f0->dtype();
    op_cols_ = f0->op_cols();
    kind_ = f0->gemm_kind_public();
    const FlatIndex::RawView v0 = f0->raw_view();
    num_sms_ = v0.num_sms;
    use_simt_ = v0.use_simt;
    seg_start_.assign(members.size() + 1, 0);
    cap_ = 0;
    max_norm_ = 0.f;
    for (size_t i = 0; i < members.size(); ++i) {
        const int64_t p = pad_tile(members[i]->ntotal());
        seg_start_[i + 1] = seg_start_[i] + p;
        cap_ = std::max<uint32_t>(cap_, static_cast<uint32_t>(p));
        const float norm = members[i]->raw_view().max_norm;
        // (a member with rows whose norm is not a number has no error bound: infinity keeps every key)
        max_norm_ = norm == norm ? std::max(max_norm_, norm) : std::numeric_limits<float>::infinity();
    }
    total_rows_ = seg_start_.back();
    // Everything a pass needs to know about its members travels in one copy.  Their data is not
    // moved: exact distances and labels are read through the member table, and so are packed operand
    // tiles.  Row-major operands are gathered by one kernel, since one tensor map has to cover them.
    // (One copy call per member and array, as this was at first, cost 0.8 ms for 32 members of
    // 20 000 x 128 whenever the set of members changed: such a call took 1.03 ms, now 0.23 like a repeated one.)
    const size_t nm = members.size(), n_tiles = static_cast<size_t>(total_rows_ / kTileB);
    in_place_ = packed_operands(kind_, op_cols_) && !use_simt_;
    const size_t row_op = static_cast<size_t>(op_cols_) * op_elem(dtype_);
    const size_t bytes = nm * sizeof(MemberView) + n_tiles * (8 + 8 + 8 + 4);
    uint8_t* dev = static_cast<uint8_t*>(tables_.ensure(bytes));
    B200_CUDA_CHECK(cudaStreamSynchronize(st));   // an earlier copy out of h_tables_ may still be under way
    uint8_t* host = static_cast<uint8_t*>(h_tables_.ensure(bytes));
    MemberView* mv = reinterpret_cast<MemberView*>(host);
    const void** tile = reinterpret_cast<const void**>(mv + nm);
    int64_t* col0 = reinterpret_cast<int64_t*>(tile + n_tiles);
    int64_t* end = col0 + n_tiles;
    int32_t* idx = reinterpret_cast<int32_t*>(end + n_tiles);
    for (size_t i = 0; i < nm; ++i) {
        const FlatIndex::RawView v = members[i]->raw_view();
        mv[i] = MemberView{v.rows_f32, v.labels, v.operand, v.norms, seg_start_[i], v.n};
        for (int64_t t = seg_start_[i] / kTileB; t < seg_start_[i + 1] / kTileB; ++t) {
            const int64_t row0 = t * kTileB - seg_start_[i];
            tile[t] = static_cast<const uint8_t*>(v.operand) + static_cast<size_t>(row0) * row_op;
            col0[t] = seg_start_[i];
            end[t] = seg_start_[i] + v.n;
            idx[t] = static_cast<int32_t>(i);
        }
    }
    auto on_device = [&](const void* p) { return dev + (static_cast<const uint8_t*>(p) - host); };
    members_ = reinterpret_cast<const MemberView*>(dev);
    seg_tile_ = reinterpret_cast<const void* const*>(on_device(tile));
    seg_col0_ = reinterpret_cast<const int64_t*>(on_device(col0));
    seg_end_ = reinterpret_cast<const int64_t*>(on_device(end));
    seg_index_ = reinterpret_cast<const int32_t*>(on_device(idx));
    B200_CUDA_CHECK(cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st));
    if (!in_place_) {
        void* xop = xop_.ensure(static_cast<size_t>(total_rows_) * row_op);
        void* nrm = norms_.ensure(static_cast<size_t>(total_rows_) * 4);
        gather_members_kernel<<<static_cast<unsigned>(n_tiles), 256, 0, st>>>(
            members_, seg_index_, static_cast<int>(row_op), packed_operands(kind_, op_cols_) ? 1 : 0,
            static_cast<uint4*>(xop), static_cast<uint32_t*>(nrm));
        B200_CUDA_CHECK(cudaGetLastError());
        if (!use_simt_ && encode_operand_map(&map_b_, kind_, xop, total_rows_, op_cols_, kTileB) != 0)
            throw std::runtime_error("cuTensorMapEncodeTiled failed for the gathered operand rows");
    }
    if (!w_err_.get()) {
        w_err_.ensure(sizeof(int));
        B200_CUDA_CHECK(cudaMemsetAsync(w_err_.get(), 0, sizeof(int), st));
    }
    cur_.assign(members.begin(), members.end());
    cur_gen_.resize(members.size());
    for (size_t i = 0; i < members.size(); ++i) cur_gen_[i] = members[i]->generation();
    ++rebuilds_;
}

void FlatGroup::search_device(const std::vector<FlatIndex*>& members, int64_t nq64, const void* xq, int k, float* D,
                              int64_t* I, cudaStream_t st, const std::function<void()>& then) {
    DeviceGuard g(device_);
    refresh(members, st);
    const int nq = static_cast<int>(nq64);
    // query preparation, once for all members
    void* qnorm = w_qnorm_.ensure(static_cast<size_t>(nq) * 4);
    const void* xq_op = xq;
    if (dtype_ == kF32) {
        void* qop = w_qop_.ensure(static_cast<size_t>((nq + kTileQ - 1) / kTileQ * kTileQ) * op_cols_ * 2);   // whole tiles
        float* eps = static_cast<float*>(w_eps_.ensure(static_cast<size_t>(nq) * 4));
        B200_CUDA_CHECK(launch_prep_queries_f32(static_cast<const float*>(xq), nq, d_, metric_, max_norm_, qop,
                                                static_cast<float*>(qnorm), eps, st));
        xq_op = qop;
    } else if (dtype_ == kF16) {
        void* qop = w_qop_.ensure(static_cast<size_t>(nq) * d_ * 2);
        B200_CUDA_CHECK(launch_f32_to_f16(static_cast<const float*>(xq), static_cast<int64_t>(nq) * d_, qop, st));
        B200_CUDA_CHECK(launch_prep_queries_f16(qop, nq, d_, static_cast<float*>(qnorm), st));
        xq_op = qop;
        ++launches_;
    } else {
        B200_CUDA_CHECK(launch_prep_queries_i8(static_cast<const int8_t*>(xq), nq, d_, static_cast<int32_t*>(qnorm), st));
    }
    ++launches_;
    CUtensorMap map_a;
    if (!use_simt_ && encode_operand_map(&map_a, kind_, xq_op, nq, op_cols_, kTileQ) != 0)
        throw std::runtime_error("cuTensorMapEncodeTiled failed for the query operand");

    // Members large enough against k are searched with a threshold per (member, query), like a small
    // index on its own: a first GEMM pass takes the minimum of every burst of 32 (or 8) rows, the k-th
    // smallest minimum of a member bounds its k-th key, and the second pass keeps the few keys below it.
    // Writing every key instead (what remains for tiny members and as the re-run when a row overflows)
    // costs 8 bytes and, for fp32 members, an exact distance per (query, row): 32 members of 20 000 x 128,
    // 64 queries, k = 10: 3.5 ms of kernels against 0.15 ms.  The line: with bursts of 8 and at least 4 k
    // of them in the largest member, about 1.2 k keys pass there; members too small for the bound to
    // help pass at most 9 k (the k-th of B minima admits B ln(1 / (1 - k / B)) keys, and B < 1.1 k
    // means fewer than 9 k rows), which the candidate rows have room for.
    const bool thresholded = static_cast<int64_t>(cap_) / 8 >= 4LL * k;
    // [0] error word, [1] a candidate row overflowed, [2] a list was too long for the fused tail: pinned,
    // written by the kernels
    volatile uint32_t* h = static_cast<uint32_t*>(h_flags_.ensure(12));
    for (Pass pass = thresholded ? kPassThresholds : kPassEveryKey;;) {
        h[0] = h[1] = h[2] = 0u;
        run_passes(pass, nq, xq, xq_op, map_a, qnorm, k, D, I, st);
        if (then) then();
        B200_CUDA_CHECK(cudaStreamSynchronize(st));
        if (h[0]) {
            const uint32_t err = h[0];
            B200_CUDA_CHECK(cudaMemsetAsync(w_err_.get(), 0, sizeof(int), st));
            throw std::runtime_error("device pipeline reported error word " + std::to_string(err) + " (bounded wait ran out)");
        }
        if (h[1]) pass = kPassEveryKey;
        else if (h[2]) pass = kPassLongLists;
        else return;
    }
}

void FlatGroup::run_passes(Pass pass, int nq, const void* xq, const void* xq_op, const CUtensorMap& map_a,
                           const void* qnorm, int k, float* D, int64_t* I, cudaStream_t st) {
    const bool is_int = dtype_ == kI8, with_tau = pass != kPassEveryKey;
    const uint32_t tau_all = is_int ? 0xFFFFFFFFu : 0xFF800000u;
    const size_t nm = cur_.size();
    const int n_qb = (nq + kTileQ - 1) / kTileQ;
    uint32_t cap = cap_;
    int burst = 32, step = 1;
    if (with_tau) {
        int64_t least = cap_;
        for (size_t i = 0; i < nm; ++i) least = std::min(least, seg_start_[i + 1] - seg_start_[i]);
        // The minima of every fourth tile are enough where each member has many bursts of 8 in them: four
        // times the candidates (k of every 4 k rows pass), but the first pass reads a quarter of the
        // rows, and with few queries it is bound by that (32 members of 20 000 x 128, 64 queries, k = 10:
        // 38 -> 14 us, the end 26 -> 34).  How many depends on the queries, whose candidates all have to be
        // refined.  us with every tile / every fourth, 32 members, by bursts / k:
        //   1 query:     8: 136 / 129 (5 000 rows: 100 / 104), 16: 124 / 114, 30: 160 / 138, 61: 152 / 131
        //   64 queries:  8: 177 / 188, 16: 158 / 167, 30: 189 / 188, 61: 181 / 166;  of 16 members: 62: 175 / 160;
        //                74 of 59 members of 5 400 x 256: 32: 312 / 298
        //   512 queries: 16: 402 / 516, 32: 368 / 404, 61: 480 / 497;  of 16 members: 62: 431 / 423, 125: 404 / 387
        const int64_t per_k = std::max(8, std::min(64, nq / 3));
        if ((least / kTileB) / 4 * (kTileB / 8) >= per_k * k) step = 4;
        if (least / kTileB / step * (kTileB / 32) < 8LL * k) burst = 8;
        // Room for 9 k keys, and for the slots the epilogue's threads reserve in blocks of 8 and leave
        // unused: four threads per row in each CTA that walks the member, an open and a reserved block each.
        const double ctas = static_cast<double>(cap_ / kTileB) * num_sms_ / (static_cast<double>(n_qb) * (total_rows_ / kTileB));
        const uint64_t want = (step > 1 ? 12ull : 10ull) * k + 64ull * (static_cast<uint64_t>(std::min<double>(ctas, cap_ / kTileB)) + 2);
        cap = 512;
        while (cap < want) cap <<= 1;
    }
    const int mins_stride = static_cast<int>(cap_) / burst;
    // members per pass: their [member][query] candidate rows of cap slots share the scratch
    const size_t per_member = static_cast<size_t>(nq) * (static_cast<size_t>(cap) * 8 + (with_tau ? static_cast<size_t>(mins_stride) * 4 : 0));
    const size_t per_pass = std::max<size_t>(1, kGroupCandBytes / per_member);
    const size_t max_rows = std::min(nm, per_pass) * static_cast<size_t>(nq);
    uint64_t* cand = static_cast<uint64_t*>(w_cand_.ensure(max_rows * cap * 8));
    uint32_t* tau = static_cast<uint32_t*>(w_tau_.ensure(max_rows * 12));   // thresholds, counters, folded thresholds
    uint32_t* counts = tau + max_rows;
    float* bias = reinterpret_cast<float*>(counts + max_rows);
    uint32_t* mins = with_tau ? static_cast<uint32_t*>(w_mins_.ensure(max_rows * mins_stride * 4)) : nullptr;
    if (!with_tau) {
        B200_CUDA_CHECK(launch_fill_u32(tau, static_cast<int64_t>(max_rows), tau_all, st));
        ++launches_;
    }
    for (size_t m0 = 0; m0 < nm; m0 += per_pass) {
        const size_t m1 = std::min(nm, m0 + per_pass);
        const int rows = static_cast<int>((m1 - m0) * static_cast<size_t>(nq));
        GemmArgs a{};
        a.A = xq_op;
        a.B = xop_.get();
        a.seg_tile = in_place_ ? seg_tile_ : nullptr;
        a.d = op_cols_;
        a.nq = nq;
        a.N = total_rows_;
        a.n_tiles_total = static_cast<int>(total_rows_ / kTileB);
        a.tile_first = static_cast<int>(seg_start_[m0] / kTileB);
        a.n_tiles_sel = static_cast<int>((seg_start_[m1] - seg_start_[m0]) / kTileB);
        a.metric = metric_;
        a.bnorm = norms_.get();
        a.qnorm_i32 = dtype_ == kI8 ? static_cast<const int32_t*>(qnorm) : nullptr;
        a.tau = tau;
        a.cand = cand;
        a.cap = cap;
        a.seg_index = seg_index_;
        a.seg_first = static_cast<int>(m0);
        a.seg_col0 = seg_col0_;
        a.seg_end = seg_end_;
        a.err = w_err_.as<int>();
        GemmLaunch L{};
        L.kind = kind_;
        L.simt = use_simt_ ? 1 : 0;
        L.num_sms = num_sms_;
        // Lists that turned out too long for the fused tail are still there when one pass covers all members.
        const bool listed = pass == kPassLongLists && nm <= per_pass;
        a.counts = counts;
        if (listed) {
            // nothing to find
        } else if (with_tau) {
            // bursts that a shorter member does not have never win
            B200_CUDA_CHECK(cudaMemsetAsync(mins, 0xFF, static_cast<size_t>(rows) * mins_stride * 4, st));
            a.mins = mins;
            a.mins_stride = mins_stride;
            L.mode = kModeBurstMin;
            L.burst = burst;
            GemmArgs sample = a;
            sample.tile_step = step;
            sample.n_tiles_sel = (a.n_tiles_sel + step - 1) / step;
            B200_CUDA_CHECK(launch_dist_gemm(L, sample, &map_a, &map_b_, st));
            TauFold fold;
            fold.counts = counts;
            fold.q_mod = nq;
            if (dtype_ == kF32) {
                fold.qnorm = static_cast<const float*>(qnorm);
                fold.ymax = max_norm_;
                fold.metric = metric_;
                fold.bias = bias;
                a.seg_bias = bias;
            }
            B200_CUDA_CHECK(launch_kth_threshold(mins, mins_stride, mins_stride, rows, k, dtype_ == kF32 ? w_eps_.as<float>() : nullptr,
                                                 tau_all, tau, fold, st));
            launches_ += 2;
        } else {
            B200_CUDA_CHECK(cudaMemsetAsync(cand, 0xFF, static_cast<size_t>(rows) * cap * 8, st));
            a.direct = 1;
        }
        L.mode = kModeAppend;
        L.burst = 32;
        if (!listed) {
            B200_CUDA_CHECK(launch_dist_gemm(L, a, &map_a, &map_b_, st));
            ++launches_;
        }
        EmitArgs e{};
        e.nq = rows;
        e.k = k;
        e.metric = metric_;
        e.mode = is_int ? 2 : (dtype_ == kF32 ? 1 : 0);
        e.qnorm = qnorm;
        e.D = D + m0 * static_cast<size_t>(nq) * k;
        e.I = I + m0 * static_cast<size_t>(nq) * k;
        e.ldk = k;
        e.q_mod = nq;
        e.members = members_ + m0;
        uint32_t* any_left = h_flags_.as<uint32_t>() + 1;
        e.err = w_err_.as<int>();
        e.err_host = h_flags_.as<int>();
        ++launches_;
        if (pass == kPassThresholds && dtype_ == kF32 && k <= kFinishMaxK) {
            B200_CUDA_CHECK(launch_finish_f32(cand, counts, cap, d_, w_eps_.as<float>(), static_cast<const float*>(xq), nullptr,
                                              nullptr, any_left, e, false, st));
            continue;
        }
        const uint32_t* n_cand = with_tau ? counts : nullptr;
        if (dtype_ == kF32) {
            B200_CUDA_CHECK(launch_refine_f32(cand, n_cand, cap, cap, rows, d_, metric_, static_cast<const float*>(xq),
                                              nullptr, st, nq, members_ + m0));
            ++launches_;
        }
        B200_CUDA_CHECK(launch_select_emit(cand, n_cand, cap, cap, nullptr, any_left, e, st));
    }
}

}  // namespace b200
