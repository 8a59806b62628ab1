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

// Blocks of a chain sweep, the slots of one, and of all.
inline int chain_blocks(int chains, const ChainShape &c) { return (chains * c.team + CH_WPB - 1) / CH_WPB; }
inline int chain_block_slots(const ChainShape &c, int precision) {
    return c.spread ? 6 : (precision != MFCFD_PRECISION_FP64 || c.dense ? 2 : 3);
}
inline int chain_slots(int chains, const ChainShape &c, int precision) {
    return chain_blocks(chains, c) * chain_block_slots(c, precision);
}

// A run's claim: its handles' chain counts, the slots of their budgets, and the
// slots it would use if they were free (SLOTS_ALL: any).
struct SlotAsk {
    const int *chains;
    int count, precision, spread, budget, want;
};
constexpr int SLOTS_ALL = 1 << 20;
// Iterations that a chunk lasts at most beyond its run's budget, so that whoever
// asks next does not wait for it long, or beside others, so that their room is
// taken up soon after they have ended; fewer where that would be more than
// LENT_POINTS iterations of a point (0.6 s with 260,000 points, 0.35 s with 1.1M).
constexpr int LENT_CHUNK = 64;
constexpr long LENT_POINTS = 1 << 24;

// Slots of a device's chain sweeps in use (chain_slot_capacity), over every
// handle and thread of the process.  A run takes slots for one chunk of
// iterations at a time: the most that it wants and that are free, at least its
// handles' budgets (mfcfd_info.chain_slots).  Where these do not fit beside the
// chunks that hold slots, its own chunk waits on the device for as few of them
// as it must (those that hold more than their budgets first, the oldest first)
// and takes what they leave: a host thread waits for another's launch calls at
// most, never for its iterations.  What a run holds counts from the moment it
// asks, so the others' next chunks leave it room or queue behind it, and runs
// that each want the whole device alternate (sharing it would leave each with
// teams of one: 62,400 points 10.7 ms an iteration against 5.0 with teams of
// four; two groups of converging clouds 0.421 solves/s alternating, 0.389 with
// the second beside the first).
//
// The sweeps on the device at any time fit it together: of those running, the
// one that asked last had, when it asked, room beside all others that it did
// not wait for.
//
// Blocks of one size fill SMs without a remainder.  Where sizes differ, two
// blocks of any size may leave no room for one more (two blocks of two slots
// none for one of three, or for a spread one, which needs half of the SM's
// shared memory), but never fewer: a block then counts as half an SM at least,
// so some SM always has room for the next.  A handle in FP64 has a build of
// either size and takes the one that fits.
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
        // Iterations of the next chunk, of `iters` to run on clouds of `points` in all
        // (an even number: the U/q buffers alternate, and a graph is kept for either).
        int chunk(int iters, long points) const {
            if (!lent_ && !beside_) return iters;
            const long most = LENT_POINTS / std::max(points, 1l) & ~1l;
            return (int)std::min<long>(iters, std::min<long>(std::max(most, 2l), LENT_CHUNK));
        }
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
            std::swap(beside_, o.beside_);
            std::swap(shape_, o.shape_);
        }
        SlotPool *pool_ = nullptr;
        long id_ = 0;
        int slots_ = 0;
        bool lent_ = false, beside_ = false;
        ChainShape shape_{};
    };

    // Slots with the shape within max(budget, want) that waits for the fewest
    // chunks, and of these the one with the largest teams.
    // after(end): has the chunk about to be launched wait for another's; false
    // if that fails.  Empty if it failed or, with `wait` false, instead of any
    // such wait (for a caller with chunks of its own to attend to).
    template <typename After>
    Lease take(int capacity, const SlotAsk &a, bool wait, After after) {
        Lease l;
        std::unique_lock<std::mutex> lock(mu_);
        // the order in which chunks are waited for
        std::vector<const Held *> order;
        for (int lent = 1; lent >= 0; --lent)
            for (const Held &h : held_)
                if (h.lent == (lent != 0)) order.push_back(&h);
        size_t waits = order.size() + 1;
        int block = 0, halves = 0;
        for (ChainShape c{a.spread ? 1 : CH_WPB, 0, a.spread};;) {
            const int each = chain_block_slots(c, a.precision);
            int blocks = 0;
            for (int i = 0; i < a.count; ++i) blocks += chain_blocks(a.chains[i], c);
            const int slots = std::max(blocks * each, a.budget), half = std::max(slots, blocks * 3);
            const bool last = c.team == 1 && (c.dense || c.spread || a.precision != MFCFD_PRECISION_FP64);
            const size_t w = waits_for(order, capacity, slots, half, each);
            const bool own = slots <= a.budget || (c.team == 1 && !c.dense);   // (teams of one fit their budget)
            if (w < waits && (own || slots <= std::min(a.want, capacity))) {
                waits = w;
                block = each;
                halves = half;
                l.shape_ = c;
                l.slots_ = slots;
            }
            if (waits == 0 || last) break;
            if (a.precision != MFCFD_PRECISION_FP64 || c.dense) c.team /= 2, c.dense = 0;
            else c.dense = 1;
        }
        if (waits > 0 && !wait) return Lease();
        l.lent_ = l.slots_ > a.budget;
        l.beside_ = !held_.empty();
        std::vector<long> ids;
        for (size_t k = 0; k < waits; ++k) ids.push_back(order[k]->id);
        held_.push_back({next_, l.slots_, halves, block, l.lent_, false, nullptr});
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
        int slots, halves, block;                            // slots beside blocks of other sizes; of a block
        bool lent, launched;
        void *end;
    };
    // How many of the chunks in `order` have to end before `slots` in blocks of
    // `block` (beside other sizes: `halves`) have room beside the others.
    static size_t waits_for(const std::vector<const Held *> &order, int capacity, int slots, int halves, int block) {
        for (size_t w = 0; w < order.size(); ++w) {
            int sum = slots, apart = halves;
            bool same = true;
            for (size_t k = w; k < order.size(); ++k) {
                sum += order[k]->slots;
                apart += order[k]->halves;
                same = same && order[k]->block == block;
            }
            if ((same ? sum : apart) <= capacity) return w;
        }
        return order.size();
    }
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
