// Checks of the slot pool (csrc/mfcfd_slots.h) that need no GPU.  Prints "ok"
// and exits 0, or prints the first violation and exits 1.  Built and run by
// tests/test_slots.py, one check per argument.
#include <cstdio>
#include <cstring>
#include <new>

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

SlotAsk ask(const int &chains, int precision, int budget, int want) { return {&chains, 1, precision, 0, budget, want}; }

// A chunk that ends in an exception, with slots beyond its budget.
void throwing_chunk(SlotPool &p, const int &chains) {
    const SlotPool::Lease l = p.take(CAP, ask(chains, MFCFD_PRECISION_FP64, 90, CAP), true);
    if (!l.lent()) return;
    throw std::bad_alloc();
}

// Slots return on every path, and a later run does not wait for lost ones.
int leases() {
    SlotPool p;
    const int chains = 120;
    {
        SlotPool::Lease a = p.take(CAP, ask(chains, MFCFD_PRECISION_FP64, 90, CAP), true);
        REQUIRE(a && a.lent() && p.held() == a.slots() && a.slots() == chain_slots(chains, a.shape(), MFCFD_PRECISION_FP64));
        SlotPool::Lease b(std::move(a));
        REQUIRE(!a && b && p.held() == b.slots());
        a = p.take(CAP, ask(chains, MFCFD_PRECISION_FP64, 90, 0), true);   // its budget beside b
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
    const SlotPool::Lease all = p.take(CAP, ask(chains, MFCFD_PRECISION_MIXED, CAP, CAP), false);
    REQUIRE(all && all.slots() == CAP);
    return 0;
}

}  // namespace

int main(int argc, char **argv) {
    int bad = argc < 2;
    for (int i = 1; i < argc && !bad; ++i) {
        if (!std::strcmp(argv[i], "leases")) bad = leases();
        else bad = 1;
    }
    if (!bad) std::printf("ok\n");
    return bad;
}
