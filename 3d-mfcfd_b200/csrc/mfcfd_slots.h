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
#include <vector>

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
// slots it would use if they were free (SLOTS_EVEN: an even share with the runs
// that hold slots).
struct SlotAsk {
    const int *chains;
    int count, precision, spread, budget, want;
};
constexpr int SLOTS_EVEN = -1;

// Slots of a device's chain sweeps in use (chain_slot_capacity), over every
// handle and thread of the process.  A run takes slots for one chunk of
// iterations at a time: its handles' budgets (mfcfd_info.chain_slots) at once,
// and more while they are free.  Where its budget does not fit beside the
// chunks that hold slots, its own chunk waits on the device for some of them
// to end (those that hold more than their budgets first, the oldest first): a
// host thread waits for another's launch calls at most, never for its
// iterations.  What a run holds counts from the moment it asks, so the others'
// next chunks leave it room.
//
// The sweeps on the device at any time fit it together: of those running, the
// one that asked last had, when it asked, room beside all others that it did
// not wait for.
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
            if (pool_) pool_->give(id_);
        }
        explicit operator bool() const { return pool_ != nullptr; }
        int slots() const { return slots_; }
        bool lent() const { return lent_; }                  // beyond the budget
        const ChainShape &shape() const { return shape_; }
        // The chunk is launched; `end` is recorded behind it, and stays
        // recorded until the slots are given back.
        void launched(void *end) {
            if (pool_) pool_->mark(id_, end);
        }

    private:
        friend class SlotPool;
        void swap(Lease &o) noexcept {
            std::swap(pool_, o.pool_);
            std::swap(id_, o.id_);
            std::swap(slots_, o.slots_);
            std::swap(lent_, o.lent_);
            std::swap(shape_, o.shape_);
        }
        SlotPool *pool_ = nullptr;
        long id_ = 0;
        int slots_ = 0;
        bool lent_ = false;
        ChainShape shape_{};
    };

    // Slots with the largest teams within max(budget, min(want, what is free)).
    // after(end): has the chunk about to be launched wait for another's; false
    // if that fails.  Empty if it failed or, with `wait` false, instead of any
    // such wait (for a caller with chunks of its own to attend to).
    template <typename After>
    Lease take(int capacity, const SlotAsk &a, bool wait, After after) {
        Lease l;
        std::unique_lock<std::mutex> lock(mu_);
        int used = 0;
        for (const Held &h : held_) used += h.slots;
        const int want = a.want == SLOTS_EVEN ? capacity / ((int)held_.size() + 1) : a.want;
        l.shape_ = chain_fit(a.chains, a.count, a.precision, a.spread, std::max(a.budget, std::min(want, capacity - used)));
        for (int i = 0; i < a.count; ++i) l.slots_ += chain_slots(a.chains[i], l.shape_, a.precision);
        l.slots_ = std::max(l.slots_, a.budget);
        l.lent_ = l.slots_ > a.budget;
        std::vector<long> ids;
        for (int lent = 1; lent >= 0; --lent)
            for (const Held &h : held_)
                if (h.lent == (lent != 0) && used + l.slots_ > capacity) {
                    used -= h.slots;
                    ids.push_back(h.id);
                }
        if (!ids.empty() && !wait) return Lease();
        held_.push_back({next_, l.slots_, l.lent_, false, nullptr});
        l.id_ = next_++;
        l.pool_ = this;
        // each was taken before this one, so no two wait for each other
        for (const long id : ids) {
            const Held *h;
            launched_.wait(lock, [&] { return !(h = find(id)) || h->launched; });
            if (h && !after(h->end)) return Lease();         // and l goes back
        }
        return l;
    }

    // Slots held now.
    int held() {
        std::lock_guard<std::mutex> lock(mu_);
        int used = 0;
        for (const Held &h : held_) used += h.slots;
        return used;
    }

private:
    struct Held {
        long id;
        int slots;
        bool lent, launched;
        void *end;
    };
    Held *find(long id) {
        for (Held &h : held_)
            if (h.id == id) return &h;
        return nullptr;
    }
    void mark(long id, void *end) {
        {
            std::lock_guard<std::mutex> lock(mu_);
            Held *h = find(id);
            h->launched = true;
            h->end = end;
        }
        launched_.notify_all();
    }
    void give(long id) {
        {
            std::lock_guard<std::mutex> lock(mu_);
            held_.erase(held_.begin() + (find(id) - held_.data()));
        }
        launched_.notify_all();
    }
    std::mutex mu_;
    std::condition_variable launched_;
    std::vector<Held> held_;                                 // by age
    long next_ = 0;
};

}  // namespace mfcfd
