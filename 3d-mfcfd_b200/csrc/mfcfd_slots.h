/*
 * mfcfd_slots.h - the slots of a device that chain sweeps running at once
 * share (host code only, no CUDA calls).
 *
 * Every wait of a chain sweep is for a point of the same sweep, so all blocks
 * of the sweeps running at once have to be resident together.  They are
 * counted in slots of a sixth of an SM (see k_sweep_chain).
 */
#pragma once

#include <algorithm>
#include <condition_variable>
#include <mutex>
#include <utility>

#include "../../include/mfcfd.h"

namespace mfcfd {

// Warps per block of the chain sweep kernels.
constexpr int CH_WPB = 4;

// Launch shape of a chain sweep: the warps that walk a chain together (1, 2 or
// 4), the FP64 build for three blocks per SM instead of two, one block per SM
// (mfcfd_params.chain_spread).
struct ChainShape {
    int team, dense, spread;
};
inline bool operator==(const ChainShape &a, const ChainShape &b) {
    return a.team == b.team && a.dense == b.dense && a.spread == b.spread;
}

// Blocks and slots of a chain sweep.
inline int chain_blocks(int chains, const ChainShape &c) { return (chains * c.team + CH_WPB - 1) / CH_WPB; }
inline int chain_slots(int chains, const ChainShape &c, int precision) {
    const int each = c.spread ? 6 : (precision != MFCFD_PRECISION_FP64 || c.dense ? 2 : 3);
    return chain_blocks(chains, c) * each;
}

// The largest teams with which the sweeps of these chain counts fit `slots`
// together; teams of one (which fit their budgets) if none does.
inline ChainShape chain_fit(const int *chains, int count, int precision, int spread, int slots) {
    ChainShape c{};
    c.spread = spread;
    c.team = spread ? 1 : CH_WPB;
    for (;; c.team /= 2) {
        for (c.dense = 0; c.dense < 2; ++c.dense) {
            int sum = 0;
            for (int i = 0; i < count; ++i) sum += chain_slots(chains[i], c, precision);
            if (sum <= slots) return c;
            if (precision != MFCFD_PRECISION_FP64) break;
        }
        if (c.team == 1) break;
    }
    c.dense = 0;
    return c;
}

// A run's claim: its handles' chain counts, the slots of their budgets, and the
// slots it would use if they were free.
struct SlotAsk {
    const int *chains;
    int count, precision, spread, budget, want;
};

// Slots of a device's chain sweeps in use (chain_slot_capacity), over every
// handle and thread of the process.  A run holds at least its handles'
// budgets (mfcfd_info.chain_slots), whose sum over concurrent runs is the
// callers' to bound; a run of mfcfd_run, mfcfd_run_batch, mfcfd_run_group or
// the request server may hold more while nobody needs it, for one chunk of
// iterations at a time, and whoever does not find room for its budget beside
// such a run waits for that chunk.
class SlotPool {
public:
    // Slots taken, given back when the object goes: on every path, so with an
    // exception too.  The sweeps that use them have to have ended by then.
    class Lease {
    public:
        Lease() = default;
        Lease(Lease &&o) noexcept { swap(o); }
        Lease &operator=(Lease &&o) noexcept {
            Lease old(std::move(*this));
            swap(o);
            return *this;
        }
        ~Lease() {
            if (pool_) pool_->give(budget_, slots_);
        }
        explicit operator bool() const { return pool_ != nullptr; }
        int slots() const { return slots_; }
        bool lent() const { return slots_ > budget_; }       // beyond the budget
        const ChainShape &shape() const { return shape_; }

    private:
        friend class SlotPool;
        void swap(Lease &o) noexcept {
            std::swap(pool_, o.pool_);
            std::swap(budget_, o.budget_);
            std::swap(slots_, o.slots_);
            std::swap(shape_, o.shape_);
        }
        SlotPool *pool_ = nullptr;
        int budget_ = 0, slots_ = 0;
        ChainShape shape_{};
    };

    // The largest teams within max(budget, min(want, what is free)); empty, with
    // `wait` false, instead of waiting (for a caller that itself holds more
    // than its budgets).
    Lease take(int capacity, const SlotAsk &a, bool wait) {
        std::unique_lock<std::mutex> lock(mu_);
        auto room = [&] { return used_ + a.budget <= capacity || excess_ == 0; };
        Lease l;
        if (!wait && !room()) return l;
        freed_.wait(lock, room);
        l.shape_ = chain_fit(a.chains, a.count, a.precision, a.spread, std::max(a.budget, std::min(a.want, capacity - used_)));
        for (int i = 0; i < a.count; ++i) l.slots_ += chain_slots(a.chains[i], l.shape_, a.precision);
        l.slots_ = std::max(l.slots_, a.budget);
        l.budget_ = a.budget;
        l.pool_ = this;
        used_ += l.slots_;
        excess_ += l.slots_ - l.budget_;
        return l;
    }

    // Slots held now.
    int held() {
        std::lock_guard<std::mutex> lock(mu_);
        return used_;
    }

private:
    void give(int budget, int slots) {
        {
            std::lock_guard<std::mutex> lock(mu_);
            used_ -= slots;
            excess_ -= slots - budget;
        }
        freed_.notify_all();
    }
    std::mutex mu_;
    std::condition_variable freed_;
    int used_ = 0, excess_ = 0;
};

}  // namespace mfcfd
