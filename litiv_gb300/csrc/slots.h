// A fixed set of places (counters in device memory, say) that calls take in turn.
#pragma once
#include <condition_variable>
#include <mutex>
#include <vector>

namespace lvbgs {

// The places 0 .. n-1. More calls at once than places wait for one another. A place whose work may not be over, or did
// not end as it should, is retired: the next call on it would meet what is left there.
class SlotPool {
public:
    explicit SlotPool(int n) : left_(n) {
        for (int i = n - 1; i >= 0; --i) free_.push_back(i);
    }
    // -1 once every place has been retired
    int take() {
        std::unique_lock<std::mutex> lk(mu_);
        cv_.wait(lk, [this] { return !free_.empty() || left_ == 0; });
        if (free_.empty()) return -1;
        const int slot = free_.back();
        free_.pop_back();
        return slot;
    }
    void give(int slot) {
        {
            std::lock_guard<std::mutex> lk(mu_);
            free_.push_back(slot);
        }
        cv_.notify_one();
    }
    void retire() {
        {
            std::lock_guard<std::mutex> lk(mu_);
            --left_;
        }
        cv_.notify_all();
    }

private:
    std::mutex mu_;
    std::condition_variable cv_;
    std::vector<int> free_;
    int left_;  // places that are not retired
};

// One call's place: done() gives it back, a call that ends without done() retires it.
class SlotLease {
public:
    explicit SlotLease(SlotPool& pool) : pool_(pool), slot_(pool.take()) {}
    SlotLease(const SlotLease&) = delete;
    SlotLease& operator=(const SlotLease&) = delete;
    ~SlotLease() {
        if (slot_ >= 0 && !done_) pool_.retire();
    }
    int slot() const { return slot_; }
    void done() {
        if (slot_ >= 0 && !done_) pool_.give(slot_);
        done_ = true;
    }

private:
    SlotPool& pool_;
    const int slot_;
    bool done_ = false;
};

}  // namespace lvbgs
