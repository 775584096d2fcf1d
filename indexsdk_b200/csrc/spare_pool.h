// Device blocks between two uses, shared by the indexes of a device.
#pragma once
#include <map>
#include <memory>
#include <mutex>
#include <vector>

#include "device_mem.h"

namespace b200 {

// Merging vectors into an index takes a dozen arrays: work arrays, and new list arrays that change places with
// the old ones.  Allocating and freeing them was 12 of the 22 ms that adding 300 000 vectors took, so they go
// through here.  At most kSpareTotal bytes of a device lie here, whatever the number of its indexes, and none
// once the last index is gone or when an allocation fails.  A block that is given must have no work left on it:
// it may be taken by another thread for another stream.
class SparePool {
public:
    static constexpr size_t kSpareBlock = size_t(64) << 20, kSpareTotal = size_t(128) << 20;

    static SparePool& of(int device) {
        static std::mutex mu;
        static std::map<int, SparePool*>& pools = *new std::map<int, SparePool*>;   // outlives every index
        std::lock_guard<std::mutex> l(mu);
        SparePool*& p = pools[device];
        if (!p) p = new SparePool;
        return *p;
    }
    // Held by every index that merges.
    class User {
    public:
        User() = default;
        User(const User&) = delete;
        User& operator=(const User&) = delete;
        ~User() {
            if (!pool_) return;
            std::lock_guard<std::mutex> l(pool_->mu_);
            if (--pool_->users_ == 0) pool_->clear();
        }
        void join(int device) {
            pool_ = &of(device);
            std::lock_guard<std::mutex> l(pool_->mu_);
            ++pool_->users_;
        }

    private:
        SparePool* pool_ = nullptr;
    };
    // An empty buffer gets at least `bytes`.  A spare block may be half as large again: it may become an index's
    // own storage.
    void* take(DeviceBuffer& b, size_t bytes) {
        {
            std::lock_guard<std::mutex> l(mu_);
            size_t best = blocks_.size();
            for (size_t i = 0; i < blocks_.size(); ++i)
                if (blocks_[i]->bytes() >= bytes && blocks_[i]->bytes() <= bytes + bytes / 2 + 65536 &&
                    (best == blocks_.size() || blocks_[i]->bytes() < blocks_[best]->bytes()))
                    best = i;
            if (best < blocks_.size()) {
                b.swap(*blocks_[best]);
                total_ -= b.bytes();
                blocks_.erase(blocks_.begin() + static_cast<std::ptrdiff_t>(best));
                return b.get();
            }
        }
        try {
            return b.ensure(bytes);
        } catch (const CudaError&) {
            cudaGetLastError();
            std::lock_guard<std::mutex> l(mu_);
            if (blocks_.empty()) throw;
            clear();
        }
        return b.ensure(bytes);
    }
    void give(DeviceBuffer& b) {
        if (!b.get()) return;
        if (b.bytes() > kSpareBlock) {
            b.release();
            return;
        }
        std::lock_guard<std::mutex> l(mu_);
        while (total_ + b.bytes() > kSpareTotal) {   // the oldest go first
            total_ -= blocks_.front()->bytes();
            blocks_.erase(blocks_.begin());
        }
        blocks_.emplace_back(new DeviceBuffer);
        blocks_.back()->swap(b);
        total_ += blocks_.back()->bytes();
    }

private:
    void clear() {
        blocks_.clear();
        total_ = 0;
    }
    std::mutex mu_;
    std::vector<std::unique_ptr<DeviceBuffer>> blocks_;   // oldest first
    size_t total_ = 0;
    int users_ = 0;
};

}  // namespace b200
