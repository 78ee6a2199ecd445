// Sets of words for measurements of ranges that run at the same time.  Host code of its own: what it calls is declared in front of it.
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <mutex>

namespace zkds {

constexpr int kRangeSets = 8;
// mapped host words of the current device, four a set, as the host and as the device see them; false where there are none
bool range_words(uint64_t** host, uint64_t** dev);

// The words that one measurement works in and is answered in: one of eight sets of a device, the caller's until it has its answer.
struct RangeAnswer {
    static constexpr int kSets = kRangeSets;
    uint64_t* partial = nullptr;
    unsigned* arrived = nullptr;
    volatile uint64_t *host = nullptr, *dev = nullptr;
    uint64_t ticket = 0;

    bool claim()
    {
        if (cudaGetDevice(&device_) != cudaSuccess || device_ < 0 || device_ >= 64) return false;
        Pool& p = pool(device_);
        std::lock_guard<std::mutex> lk(p.mu);
        while (set_ < kSets && (p.taken >> set_ & 1)) ++set_;
        if (set_ == kSets) return false;
        const size_t each = 256 + (size_t)sm_count() * 8 * 2 * sizeof(uint64_t);
        size_t fresh = 0;
        uint8_t* ws = (uint8_t*)workspace_fresh(each * kSets, 7, &fresh);
        if (fresh) p.cleared = false;
        uint64_t *words, *words_dev;
        if (!ws || !range_words(&words, &words_dev)) return false;
        // the kernel leaves its counter at zero.  New words whose clearing fails (a first call under capture) are cleared by a later call
        if (!p.cleared && (cudaMemset(ws, 0, each * kSets) != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess)) {
            cudaGetLastError();
            return false;
        }
        p.cleared = true;
        p.taken |= 1u << set_;
        held_ = true;
        arrived = (unsigned*)(ws + each * set_);
        partial = (uint64_t*)(ws + each * set_ + 256);
        host = words + 4 * set_;
        dev = words_dev + 4 * set_;
        ticket = ++p.tickets;
        return true;
    }
    ~RangeAnswer()
    {
        if (!held_) return;
        Pool& p = pool(device_);
        std::lock_guard<std::mutex> lk(p.mu);
        p.taken &= ~(1u << set_);
    }

  private:
    struct Pool {
        std::mutex mu;
        unsigned taken = 0;
        uint64_t tickets = 0;
        bool cleared = false;
    };
    static Pool& pool(int device)
    {
        static Pool pools[64];
        return pools[device];
    }
    int device_ = 0, set_ = 0;
    bool held_ = false;
};

}  // namespace zkds
