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
    const int chains = 396;
    int end = 0;
    std::vector<void *> waited;
    auto after = [&](void *e) { return waited.push_back(e), true; };
    SlotPool::Lease run = p.take(CAP, ask(chains, MFCFD_PRECISION_FP64, 180, SLOTS_EVEN), true, no_wait);
    REQUIRE(run.lent() && run.slots() == CAP);
    run.launched(&end);
    REQUIRE(!p.take(CAP, ask(chains, MFCFD_PRECISION_FP64, 300, 0), false, after) && waited.empty());
    SlotPool::Lease launch = p.take(CAP, ask(chains, MFCFD_PRECISION_FP64, 300, 0), true, after);
    REQUIRE(launch && !launch.lent() && launch.slots() == 300 && waited == std::vector<void *>{&end});
    run = SlotPool::Lease();
    run = p.take(CAP, ask(chains, MFCFD_PRECISION_FP64, 180, SLOTS_EVEN), true, no_wait);
    REQUIRE(run && run.slots() <= CAP - 300);
    // a chunk whose wait cannot be queued does not run, and holds nothing
    const int before = p.held();
    run.launched(&end);
    launch.launched(&end);
    REQUIRE(!p.take(CAP, ask(chains, MFCFD_PRECISION_FP64, CAP, 0), true, no_wait) && p.held() == before);
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
                const int chains = 396, budget = 180;      // 4 of 5 fit
                while (!stop) {
                    all[k].emplace_back(new Chunk());
                    Chunk *c = all[k].back().get();
                    SlotPool::Lease l = p.take(CAP, ask(chains, MFCFD_PRECISION_FP64, budget, SLOTS_EVEN), true, [&](void *e) {
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

}  // namespace

int main(int argc, char **argv) {
    int bad = argc < 2;
    for (int i = 1; i < argc && !bad; ++i) {
        if (!std::strcmp(argv[i], "leases")) bad = leases();
        else if (!std::strcmp(argv[i], "launch_beside_a_run")) bad = launch_beside_a_run();
        else if (!std::strcmp(argv[i], "threads_share")) bad = threads_share();
        else bad = 1;
    }
    if (!bad) std::printf("ok\n");
    return bad;
}
