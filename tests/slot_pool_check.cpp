// Checks of the slot pool (csrc/mfcfd_slots.h) that need no GPU.  Prints "ok"
// and exits 0, or prints the first violation and exits 1.  Built and run by
// tests/test_slots.py, one check per argument.
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstring>
#include <functional>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

#include "mfcfd_slots.h"

using namespace mfcfd;

namespace {

#define REQUIRE(cond)                                                \
    do {                                                             \
        if (!(cond)) {                                               \
            std::printf("line %d: %s\n", __LINE__, #cond);           \
            return 1;                                                \
        }                                                            \
    } while (0)

constexpr int CAP = 792;                  // 132 SMs

// take's argument where nothing has to be waited for
bool no_wait(void *) { return false; }

SlotAsk ask(const int &chains, int precision, int budget, int want) { return {&chains, 1, precision, 0, budget, want}; }

// A chunk that ends in an exception, with slots beyond its budget.
void throwing_chunk(SlotPool &p, const int &chains) {
    const SlotPool::Lease l = p.take(CAP, ask(chains, MFCFD_PRECISION_FP64, 90, CAP), true, no_wait);
    if (!l.lent()) return;
    throw std::bad_alloc();
}

// Slots return on every path, and a later run does not wait for lost ones.
int leases() {
    SlotPool p;
    const int chains = 120;
    {
        SlotPool::Lease a = p.take(CAP, ask(chains, MFCFD_PRECISION_FP64, 90, CAP), true, no_wait);
        REQUIRE(a && a.lent() && p.held() == a.slots() && a.slots() == chain_slots(chains, a.shape(), MFCFD_PRECISION_FP64));
        SlotPool::Lease b(std::move(a));
        REQUIRE(!a && b && p.held() == b.slots());
        a = p.take(CAP, ask(chains, MFCFD_PRECISION_FP64, 90, 0), true, no_wait);   // its budget beside b
        REQUIRE(a && !a.lent() && a.slots() == 90 && p.held() == b.slots() + 90);
        b = std::move(a);                                                  // b's first slots return
        REQUIRE(!a && b.slots() == 90 && p.held() == 90);
        b = SlotPool::Lease();
        REQUIRE(!b && p.held() == 0);
    }
    bool thrown = false;
    try {
        throwing_chunk(p, chains);
    } catch (const std::bad_alloc &) {
        thrown = true;
    }
    REQUIRE(thrown && p.held() == 0);
    const SlotPool::Lease all = p.take(CAP, ask(chains, MFCFD_PRECISION_MIXED, CAP, CAP), false, no_wait);
    REQUIRE(all && all.slots() == CAP);
    return 0;
}

// A stand-in for the device: a chunk starts when the chunks that it waits for
// have ended, and ends when its work has.
struct Chunk {
    std::vector<Chunk *> after;
    std::mutex mu;
    std::condition_variable cv;
    bool done = false;
    void wait() {
        std::unique_lock<std::mutex> lock(mu);
        cv.wait(lock, [&] { return done; });
    }
    void run(const std::function<void()> &work) {
        for (Chunk *c : after) c->wait();
        work();
        std::lock_guard<std::mutex> lock(mu);
        done = true;
        cv.notify_all();
    }
};

// A launch beside a run that holds every slot asks for its budget and is back
// at once: its chunk waits on the device, and the run's next chunk leaves it
// room.
int launch_beside_a_run() {
    SlotPool p;
    const int chains = 264;
    int end = 0;
    std::vector<void *> waited;
    auto after = [&](void *e) { return waited.push_back(e), true; };
    SlotPool::Lease run = p.take(CAP, ask(chains, MFCFD_PRECISION_FP64, 198, SLOTS_ALL), true, no_wait);
    REQUIRE(run.lent() && run.slots() == CAP);
    run.launched(&end);
    REQUIRE(!p.take(CAP, ask(chains, MFCFD_PRECISION_FP64, 300, 0), false, after) && waited.empty());
    SlotPool::Lease launch = p.take(CAP, ask(chains, MFCFD_PRECISION_FP64, 300, 0), true, after);
    REQUIRE(run.chunk(1000, 60000) == LENT_CHUNK && run.chunk(10, 60000) == 10);   // not kept waiting for long
    REQUIRE(launch.chunk(1000, 600) == LENT_CHUNK);                       // nor at its budget once there is room
    REQUIRE(launch && !launch.lent() && launch.slots() == 300 && waited == std::vector<void *>{&end});
    run = SlotPool::Lease();
    run = p.take(CAP, ask(chains, MFCFD_PRECISION_FP64, 198, SLOTS_ALL), true, no_wait);
    REQUIRE(run && run.slots() <= CAP - 300);
    // a chunk whose wait cannot be queued does not run, and holds nothing
    REQUIRE(run.chunk(1000, 1104000) == 14 && run.chunk(1000, 100000000) == 2 && run.chunk(1, 100000000) == 1);
    const int before = p.held();
    run.launched(&end);
    launch.launched(&end);
    REQUIRE(!p.take(CAP, ask(chains, MFCFD_PRECISION_FP64, CAP, 0), true, no_wait) && p.held() == before);
    run = SlotPool::Lease();
    launch = SlotPool::Lease();
    launch = p.take(CAP, ask(chains, MFCFD_PRECISION_FP64, 300, 0), true, no_wait);
    REQUIRE(launch.chunk(1000, 1104000) == 1000);                             // alone, within its budget
    return 0;
}

// Threads that run chunk after chunk, each alone able to fill the device: all
// of them advance, their sweeps fit it at every moment, and the budgets of
// those that fit together run side by side.
int threads_share() {
    for (const int threads : {2, 3, 5}) {
        SlotPool p;
        std::atomic<int> on_device{0}, most{0}, over{0};
        std::vector<int> chunks(threads, 0);
        std::atomic<bool> stop{false};
        std::vector<std::vector<std::unique_ptr<Chunk>>> all(threads);   // others may wait for them to the end
        std::vector<std::thread> pool;
        for (int k = 0; k < threads; ++k)
            pool.emplace_back([&, k] {
                const int chains = 240, budget = 180;      // 4 of 5 fit
                while (!stop) {
                    all[k].emplace_back(new Chunk());
                    Chunk *c = all[k].back().get();
                    SlotPool::Lease l = p.take(CAP, ask(chains, MFCFD_PRECISION_FP64, budget, SLOTS_ALL), true, [&](void *e) {
                        c->after.push_back((Chunk *)e);
                        return true;
                    });
                    l.launched(c);
                    c->run([&] {
                        const int now = on_device += l.slots();
                        if (now > CAP) ++over;
                        for (int m = most; now > m && !most.compare_exchange_weak(m, now);) {}
                        std::this_thread::sleep_for(std::chrono::milliseconds(2));
                        on_device -= l.slots();
                    });
                    ++chunks[k];
                }
            });
        std::this_thread::sleep_for(std::chrono::milliseconds(1000));
        stop = true;
        for (std::thread &t : pool) t.join();
        int least = chunks[0], top = chunks[0];
        for (const int c : chunks) least = std::min(least, c), top = std::max(top, c);
        REQUIRE(!over && p.held() == 0 && most > 2 * 180);
        REQUIRE(4 * least >= top);
    }
    return 0;
}

// Shapes of a block, and an SM's room for them: registers (168 a thread where
// three blocks share an SM, else 256) and kilobytes of shared memory.
struct Block {
    int slots, regs, smem;
};
constexpr Block BLOCKS[] = {{2, 168 * 128, 76}, {3, 256 * 128, 76}, {6, 256 * 128, 117}, {6, 168 * 128, 117}};
bool fits_sm(const int n[4]) {
    int regs = 0, smem = 0;
    for (int b = 0; b < 4; ++b) regs += n[b] * BLOCKS[b].regs, smem += n[b] * BLOCKS[b].smem;
    return regs <= 65536 && smem <= 228;
}

// Whether an SM that holds n has no room for another block of kind b.
bool full_for(const int n[4], int b) {
    int m[4] = {n[0], n[1], n[2], n[3]};
    ++m[b];
    return fits_sm(n) && !fits_sm(m);
}

// The most SMs that `blocks` (of each kind) can leave without room for one more
// of kind b, bounded by duality: with weights of which every SM without room
// holds 1 or more, the weight of all blocks.  In sixtieths.
int most_without_room(const int blocks[4], int b) {
    static std::vector<std::vector<int>> weights[16][4];
    int have = 0;
    for (int k = 0; k < 4; ++k) have |= blocks[k] > 0 ? 1 << k : 0;
    auto &ws = weights[have][b];
    if (ws.empty()) {
        const int W[] = {0, 10, 15, 20, 30, 40, 60};
        int n[4];
        std::vector<std::vector<int>> full;
        for (n[0] = 0; n[0] <= (have & 1 ? 3 : 0); ++n[0])
            for (n[1] = 0; n[1] <= (have & 2 ? 3 : 0); ++n[1])
                for (n[2] = 0; n[2] <= (have & 4 ? 2 : 0); ++n[2])
                    for (n[3] = 0; n[3] <= (have & 8 ? 2 : 0); ++n[3])
                        if (full_for(n, b)) full.push_back({n[0], n[1], n[2], n[3]});
        for (int i = 0; i < 7 * 7 * 7 * 7; ++i) {
            const int w[4] = {W[i % 7], W[i / 7 % 7], W[i / 49 % 7], W[i / 343]};
            bool valid = true;
            for (const auto &f : full) valid = valid && f[0] * w[0] + f[1] * w[1] + f[2] * w[2] + f[3] * w[3] >= 60;
            if (valid) ws.push_back({w[0], w[1], w[2], w[3]});
        }
    }
    int least = 1 << 30;
    for (const auto &w : ws) least = std::min(least, blocks[0] * w[0] + blocks[1] * w[1] + blocks[2] * w[2] + blocks[3] * w[3]);
    return least / 60;
}

// Blocks of different sizes leave parts of SMs that no other block fits, so
// counting slots is not enough: the sweeps that the pool lets run at once are
// all resident together, in whatever order their blocks were placed, since
// every block finds an SM with room whatever the others hold.
int block_sizes() {
    unsigned seed = 1;
    auto rnd = [&](int n) { return (int)((seed = seed * 1664525u + 1013904223u) >> 8) % n; };
    int mixed_sizes = 0;
    for (int round = 0; round < 20000; ++round) {
        SlotPool p;
        std::vector<SlotPool::Lease> running;
        int blocks[4] = {0, 0, 0, 0};
        const int share = rnd(3) ? 1 + rnd(CAP) : SLOTS_ALL;
        for (int k = 0; k < 12; ++k) {
            const int precision = rnd(2) ? MFCFD_PRECISION_FP64 : MFCFD_PRECISION_MIXED, spread = rnd(8) == 0;
            const int chains = 1 + rnd(spread ? 130 : rnd(3) ? 264 : 1000);
            const int budget = (chains + 3) / 4 * (spread ? 6 : precision == MFCFD_PRECISION_FP64 ? 3 : 2);
            const SlotAsk a{&chains, 1, precision, spread, budget, share};
            if (budget > CAP) continue;
            SlotPool::Lease l = p.take(CAP, a, false, no_wait);
            if (!l) continue;
            REQUIRE(p.held() <= CAP);
            const ChainShape c = l.shape();
            blocks[spread ? (precision == MFCFD_PRECISION_FP64 ? 2 : 3)
                          : (precision == MFCFD_PRECISION_FP64 && !c.dense ? 1 : 0)] += chain_blocks(chains, c);
            REQUIRE(l.slots() >= chain_slots(chains, c, precision) && (l.lent() || l.slots() == budget));
            running.push_back(std::move(l));
        }
        mixed_sizes += (blocks[0] > 0) + (blocks[1] > 0) + (blocks[2] + blocks[3] > 0) > 1;
        for (int b = 0; b < 4; ++b) {
            if (!blocks[b]) continue;
            --blocks[b];
            const int without = most_without_room(blocks, b);
            ++blocks[b];
            if (without >= 148) {
                std::printf("%d, %d, %d and %d blocks: one of kind %d may have room on none of 148 SMs\n", blocks[0], blocks[1],
                            blocks[2], blocks[3], b);
                return 1;
            }
        }
    }
    REQUIRE(mixed_sizes > 1000);
    return 0;
}

// What the pool gives sweeps that differ in block size: the FP64 build of the
// size that is running, and the device to one size after the other where
// neither fits beside the other.
int block_size_choice() {
    SlotPool p;
    {
        // alone, too many chains for teams of four in either build but one
        const int many = 396, more = 528;
        const SlotPool::Lease l = p.take(CAP, ask(many, MFCFD_PRECISION_FP64, 297, SLOTS_ALL), true, no_wait);
        REQUIRE(l.shape().team == 4 && l.shape().dense == 1 && l.slots() == CAP);
        SlotPool q;
        const SlotPool::Lease m = q.take(CAP, ask(more, MFCFD_PRECISION_FP64, 396, SLOTS_ALL), true, no_wait);
        REQUIRE(m.shape().team == 2 && m.shape().dense == 0 && m.slots() == CAP);
    }
    const int few = 88, many = 264;
    int end = 0;
    std::vector<void *> waited;
    auto after = [&](void *e) { return waited.push_back(e), true; };
    SlotPool::Lease mixed = p.take(CAP, ask(many, MFCFD_PRECISION_MIXED, 132, 528), true, no_wait);
    REQUIRE(mixed.slots() == 528 && mixed.shape().team == 4);
    mixed.launched(&end);
    // (blocks of three slots would count the running ones as half an SM each)
    SlotPool::Lease f64 = p.take(CAP, ask(few, MFCFD_PRECISION_FP64, 66, 264), true, no_wait);
    REQUIRE(f64 && f64.shape().dense == 1 && f64.shape().team == 4 && f64.slots() == 176);
    f64 = SlotPool::Lease();
    mixed = SlotPool::Lease();
    f64 = p.take(CAP, ask(many, MFCFD_PRECISION_FP64, 198, CAP), true, no_wait);
    REQUIRE(f64.shape().dense == 0 && f64.slots() == CAP);
    f64.launched(&end);
    mixed = p.take(CAP, ask(many, MFCFD_PRECISION_MIXED, 132, 0), true, after);
    REQUIRE(mixed && !mixed.lent() && waited == std::vector<void *>{&end});
    return 0;
}

}  // namespace

int main(int argc, char **argv) {
    int bad = argc < 2;
    for (int i = 1; i < argc && !bad; ++i) {
        if (!std::strcmp(argv[i], "leases")) bad = leases();
        else if (!std::strcmp(argv[i], "launch_beside_a_run")) bad = launch_beside_a_run();
        else if (!std::strcmp(argv[i], "threads_share")) bad = threads_share();
        else if (!std::strcmp(argv[i], "block_sizes")) bad = block_sizes();
        else if (!std::strcmp(argv[i], "block_size_choice")) bad = block_size_choice();
        else bad = 1;
    }
    if (!bad) std::printf("ok\n");
    return bad;
}
