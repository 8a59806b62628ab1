/*
 * mfcfd_chain.cuh - the chain schedule's LU-SGS sweep (included by
 * mfcfd_kernels.cu; the other schedules' sweep_point and the hand-off words
 * are described there).
 *
 * A chain is a list of points in topological order, fixed at set-up, in which
 * a point usually follows its deepest dependency.  A team of warps of one
 * block walks it, warp s taking positions s, s + team, ...: while one warp
 * computes a point, the others have the following points' inputs staged,
 * their terms gathered and their sums advanced, and wait for the team's own
 * increments in shared memory.  So a level of the sweep takes the dependent
 * arithmetic of one point (remaining sums, solve, own flux) and a
 * shared-memory hand-off, not the fetches around it.  Measured (B200, FP64,
 * both sweeps of an iteration; before: one warp per chain, which did all of a
 * point's work in turn): 62,400 points 13.6 -> 4.6 ms (1.25 us per level),
 * 1.1M points 49.6 -> 19.4 ms, mixed precision at 62,400 11.4 -> 3.5 ms.  On
 * the critical path of the 62,400-point sweep seven hops in ten are from a
 * chain's point to its next (0.86 us: its own flux about 855 cycles, the sums
 * after the ring term 150, the solve 150, the rest of dU 165), one in four to
 * another chain through L2 (1.9 us), one in thirteen at a wall point (3.5 us).
 *
 * Ring.  The team's last increments lie in a shared ring of TEAM_RING slots of
 * 32 words (lane l's component), one per position (a team of one warp:
 * CHAIN_RING slots, and no marks or waits).  A word is DU_PENDING
 * until its point's warp writes it; lane l of a consumer polls the word that
 * lane l of the producer writes.  Position i marks slot i + CHAIN_RING
 * pending when it starts, and starts when positions up to i - CHAIN_RING are
 * done.  A consumer of position j is at most at j + CHAIN_RING, so (a) when
 * j or a consumer of j starts, position j - CHAIN_RING has marked j's slot,
 * and (b) the position whose increment that mark replaced (j - TEAM_RING) has
 * no consumer left, since TEAM_RING >= 3 * CHAIN_RING.
 * Waits are for earlier positions of the same chain or for producers on
 * earlier levels only, so they end; each is bounded anyway.
 */
#pragma once

namespace mfcfd {

constexpr int TEAM_RING = 24;
static_assert(TEAM_RING >= 3 * CHAIN_RING, "ring slots outlive their readers");
constexpr int GATHER = 16;               // terms of a list gathered at a time
// ring slots of a team: a warp alone reads a slot before it writes it again
__host__ __device__ constexpr int ring_slots(int team) { return team == 1 ? CHAIN_RING : TEAM_RING; }
constexpr int CHAIN_WARP_BYTES = SW_T_DOUBLES * 8 + 2 * (int)sizeof(SweepStage);
static_assert(GATHER * 32 * 8 <= SW_T_DOUBLES * 8, "gathered terms fit the T buffer");
static_assert(CHAIN_WARP_BYTES % 16 == 0, "stage alignment");

struct Team {
    double *ring;        // `slots` x 32 words
    int *at;             // position each warp of the team is at
    int size, sub, slots;
};

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ double lds_relaxed(unsigned a) {
    double v;
    asm volatile("ld.relaxed.cta.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts_relaxed(unsigned a, double v) {
    asm volatile("st.relaxed.cta.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
// the word of a term that has landed (no memory clobber, so that the loads of
// a list's terms overlap)
__device__ __forceinline__ double lds_term(unsigned a) {
    double v;
    asm volatile("ld.relaxed.cta.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ int lds_acquire(unsigned a) {
    int v;
    asm volatile("ld.acquire.cta.shared.s32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts_release(unsigned a, int v) {
    asm volatile("st.release.cta.shared.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// Waits inside a block outlast the bounded waits on global memory (a warp may
// wait here for one that waits there): the same limit in rounds of 32 polls.
__device__ __forceinline__ bool team_spin_continue(int &polls, const DevCloud &d) {
    if (++polls & 31) return true;
    int rounds = (polls >> 5) - 1;
    return spin_continue(rounds, d);
}

// Start of position `pos`: see the ring's rule above.
__device__ __forceinline__ void team_enter(const DevCloud &d, const Team &t, int pos, int lane) {
    if (t.size == 1) return;
    const unsigned a = smem_addr(t.at + (lane < t.size ? lane : 0));
    int spins = 0;
    bool wait;
    do {
        wait = lds_acquire(a) <= pos - CHAIN_RING;
        if (wait && !team_spin_continue(spins, d)) wait = false;
    } while (__any_sync(FULL, wait));
    __syncwarp();
    sts_relaxed(smem_addr(t.ring + ((pos + CHAIN_RING) % TEAM_RING) * 32 + lane),
                __longlong_as_double((long long)DU_PENDING));
}

// End of position `pos`: its ring reads and its own word are done.
__device__ __forceinline__ void team_leave(const Team &t, int pos, int lane) {
    __syncwarp();
    if (lane == 0) sts_release(smem_addr(t.at + t.sub), pos + t.size);
}

// Sum of the six 5-bit counts of ChainItem::cnt (or of those a mask leaves).
__device__ __forceinline__ int count_sum(uint32_t cnt) {
    const uint32_t m = 0x01f07c1fu;                       // every other field
    const uint32_t a = (cnt & m) + ((cnt >> 5) & m);
    return (int)((a & 1023u) + ((a >> 10) & 1023u) + (a >> 20));
}

// A lane's fixed part in staging a point (stage_issue without its branches):
// one 8-byte copy (U, base, frame or D_inv) and two 16-byte ones (geometry
// and flux rows) besides the terms.
struct StageLane {
    const char *src8, *src16;
    unsigned step8, step16;        // bytes per point
    unsigned dst8, dst16;          // offsets in the stage; lanes without a copy: none
};
__device__ __forceinline__ StageLane stage_lane(const DevCloud &d, bool forward, int lane) {
    StageLane L;
    const double *a = d.U + lane;
    L.step8 = 40;
    L.dst8 = offsetof(SweepStage, U) + 8 * lane;
    if (lane >= 5) {
        a = (forward ? d.flux_res : d.dUp) + (lane - 5);
        L.dst8 = offsetof(SweepStage, base) + 8 * (lane - 5);
    }
    if (lane >= 10) {
        a = d.frame + (lane - 10);
        L.step8 = 72;
        L.dst8 = offsetof(SweepStage, frame) + 8 * (lane - 10);
    }
    if (lane >= 19) {
        a = d.dinv;
        L.step8 = 8;
        L.dst8 = offsetof(SweepStage, dinv);
    }
    L.src8 = reinterpret_cast<const char *>(a);
    const bool geo = lane < GEO_STRIDE / 2;
    L.src16 = geo ? reinterpret_cast<const char *>(d.geo) + 16 * lane
                  : reinterpret_cast<const char *>(d.gold) + 16 * (lane - GEO_STRIDE / 2);
    L.step16 = geo ? GEO_STRIDE * 8 : 240;
    L.dst16 = geo ? offsetof(SweepStage, geo) + 16 * lane : offsetof(SweepStage, gold) + 16 * (lane - GEO_STRIDE / 2);
    return L;
}
__device__ __forceinline__ void chain_stage(const DevCloud &d, const StageLane &L, const ChainItem &it, bool forward,
                                            int lane, SweepStage *st) {
    char *sb = reinterpret_cast<char *>(st);
    const size_t p = (size_t)it.p;
    const int chunks = 2 * count_sum(it.cnt);
    const char *es = reinterpret_cast<const char *>((forward ? d.fwd_ent : d.bwd_ent) + it.off) + 16 * lane;
    char *ed = reinterpret_cast<char *>(st->ent) + 16 * lane;
    for (int j = lane; j < chunks; j += 32, es += 512, ed += 512) cp_async16(ed, es);
    cp_async16(sb + L.dst16, L.src16 + p * L.step16);
    if (lane < 7) cp_async16(st->gold + 16 + 2 * lane, d.gold + 30 * p + 16 + 2 * lane);
    if (lane < 20) cp_async8(sb + L.dst8, L.src8 + p * L.step8);
    if (!(it.info & CI_SHARED)) {
        if (lane < 8) cp_async16(st->slot_nbr + 4 * lane, d.slot_nbr + p * MAX_SLOTS + 4 * lane);
        else if (lane < 10) cp_async16(st->slot_mask + 16 * (lane - 8), d.sweep_slot_mask + p * MAX_SLOTS + 16 * (lane - 8));
        else if (lane == 10) cp_async4(&st->need, (forward ? d.fwd_need : d.bwd_need) + p);
        else if (lane == 11) cp_async4(&st->old, (forward ? d.fwd_old : d.bwd_old) + p);
    }
}

// Ring slot of the position `dist` (0 .. CHAIN_RING) before `pos`.
__device__ __forceinline__ int ring_slot(const Team &t, int pos, int dist) {
    if (t.slots == CHAIN_RING) return (pos - dist) & (CHAIN_RING - 1);
    const int s = pos % TEAM_RING - dist;
    return s < 0 ? s + TEAM_RING : s;
}

// v = the word at p when `take` (a predicated load: no branch, and loads of
// several terms overlap)
__device__ __forceinline__ void ldg_if(unsigned long long &v, const double *p, bool take) {
    asm volatile("{\n\t.reg .pred %%p;\n\tsetp.ne.s32 %%p, %2, 0;\n\t@%%p ld.relaxed.gpu.global.b64 %0, [%1];\n\t}"
                 : "+l"(v)
                 : "l"(p), "r"((int)take));
}
__device__ __forceinline__ void lds_if(unsigned long long &v, unsigned a, bool take) {
    asm volatile("{\n\t.reg .pred %%p;\n\tsetp.ne.s32 %%p, %2, 0;\n\t@%%p ld.relaxed.cta.shared.b64 %0, [%1];\n\t}"
                 : "+l"(v)
                 : "r"(a), "r"((int)take));
}
__device__ __forceinline__ bool pending_word(unsigned long long v) {
    // no increment, flux or D_inv has this upper half (a signalling NaN)
    return (unsigned)(v >> 32) == (unsigned)(DU_PENDING >> 32);
}
// The ring word at `a` once its position has written it (every lane calls; a
// lane without `need` does not wait).
__device__ __forceinline__ double ring_word(const DevCloud &d, unsigned a, bool need) {
    int spins = 0;
    double t;
    bool wait;
    do {
        t = lds_relaxed(a);
        wait = need && pending_word((unsigned long long)__double_as_longlong(t));
        if (wait && !team_spin_continue(spins, d)) wait = false;
    } while (__any_sync(FULL, wait));
    return t;
}

// s += term x weight, in the list's order; a no-op unless `in`.
template <bool FOLD>
struct Sums {
    double x = 0.0, y = 0.0, z = 0.0;
    __device__ __forceinline__ void add(bool in, double px, double py, double pz) {
        if (in) {
            x = x + px;
            if constexpr (!FOLD) {
                y = y + py;
                z = z + pz;
            }
        }
    }
    __device__ __forceinline__ void term(bool in, double t, const SweepEntry &E) {
        if constexpr (FOLD) add(in, t * E.w[0], 0.0, 0.0);
        else add(in, t * E.w[0], t * E.w[1], t * E.w[2]);
    }
};

// List sums of a point in the shared frame: lane (list dd, component c) adds
// its list's terms in list order.  The terms' increments are read together
// (up to GATHER of each list in flight) and re-read while pending; terms from
// the team's ring join them when their words are there.  The newest position
// among the point's ring terms is the one most likely still to be computed:
// the terms before it are added, and the products of the AFTER terms after
// it formed, before the wait for its word.  Straight-line code with predicated
// loads and sums: a divergent branch per term costs more than the term.
// (GATHER, AFTER) measured at 62,400 points, ms per iteration: (16, 8) 4.99,
// (12, 8) 5.25, (8, 8) 6.40, (20, 8) 5.13, (16, 6) 5.11, (16, 10) 4.99 (1.1M
// points: 25.9 against 25.4).
constexpr int AFTER = 8;
template <bool FOLD>
__device__ __forceinline__ void shared_sums(const DevCloud &d, const SweepEntry *E, int n, const double *src,
                                            unsigned tl, unsigned rl, const Team &team, int pos, Sums<FOLD> &s) {
    const int nmax = (int)__reduce_max_sync(FULL, (unsigned)n);
    for (int base = 0; base < nmax; base += GATHER, E += GATHER) {
        const int m = min(n - base, GATHER);
        unsigned rm = 0;               // this list's ring terms
        int k[GATHER];
        unsigned long long v[GATHER];
#pragma unroll
        for (int q = 0; q < GATHER; ++q) {
            const int2 kp = *reinterpret_cast<const int2 *>(&E[q]);
            const bool in = q < m, ring = (kp.y & ENT_RING) != 0;
            k[q] = in ? kp.x : 0;
            rm |= in && ring ? 1u << q : 0u;
            v[q] = 0;
            ldg_if(v[q], src + DG_STRIDE * (long long)k[q], in && !ring);
        }
        // each ring term's distance; the newest position of all lists
        int hot = GATHER, near = CHAIN_RING + 1;
        for (unsigned r = rm; r; r &= r - 1u) {
            const int q = __ffs(r) - 1;
            const int dist = ((pos - 1 - (E[q].pad >> ENT_RING_SHIFT)) & (CHAIN_RING - 1)) + 1;
            if (dist < near) {
                near = dist;
                hot = q;
            }
        }
        const int newest = (int)__reduce_min_sync(FULL, (unsigned)near);
        if (near != newest) hot = GATHER;
        unsigned early = hot < GATHER ? rm & ~(1u << hot) : rm;
        int spins = 0;
        for (;;) {
            bool pend = false;
#pragma unroll
            for (int q = 0; q < GATHER; ++q) pend = pend || pending_word(v[q]);
            if (!__any_sync(FULL, pend)) break;
            if (pend && !spin_continue(spins, d)) {
                // the wait ran out (d.err is set): the terms stay unset
#pragma unroll
                for (int q = 0; q < GATHER; ++q) v[q] = pending_word(v[q]) ? 0 : v[q];
            }
#pragma unroll
            for (int q = 0; q < GATHER; ++q) ldg_if(v[q], src + DG_STRIDE * (long long)k[q], pending_word(v[q]));
        }
        if (newest <= CHAIN_RING) {
#pragma unroll
            for (int q = 0; q < GATHER; ++q) sts_relaxed(tl + q * 256, __longlong_as_double((long long)v[q]));
            if (__any_sync(FULL, early != 0)) {
                const unsigned er = early;
                while (__any_sync(FULL, early != 0)) {
                    const int q = early ? __ffs(early) - 1 : 0;
                    const int dist = ((pos - 1 - (E[q].pad >> ENT_RING_SHIFT)) & (CHAIN_RING - 1)) + 1;
                    const double t = ring_word(d, rl + ring_slot(team, pos, dist) * 256, early != 0);
                    if (early) sts_relaxed(tl + q * 256, t);
                    early &= early - 1u;
                }
#pragma unroll
                for (int q = 0; q < GATHER; ++q) lds_if(v[q], tl + q * 256, (er >> q) & 1u);
            }
        }
        const int lim = min(hot, m);
#pragma unroll
        for (int q = 0; q < GATHER; ++q) s.term(q < lim, __longlong_as_double((long long)v[q]), E[q]);
        if (newest > CHAIN_RING) continue;
        // the newest ring term and what follows it
        const SweepEntry *H = E + (hot < GATHER ? hot : 0);
        const unsigned hl = tl + (hot < GATHER ? hot : 0) * 256;
        const int after = hot < GATHER ? m - hot - 1 : 0;
        const double hx = H->w[0], hy = H->w[1], hz = H->w[2];
        double px[AFTER], py[AFTER], pz[AFTER];
#pragma unroll
        for (int q = 0; q < AFTER; ++q) {
            const double t = lds_term(hl + (q + 1) * 256);
            px[q] = t * H[q + 1].w[0];
            py[q] = t * H[q + 1].w[1];
            pz[q] = t * H[q + 1].w[2];
        }
        const bool more = __any_sync(FULL, after > AFTER);
        const double t = ring_word(d, rl + ring_slot(team, pos, newest) * 256, true);
        s.add(hot < GATHER, t * hx, t * hy, t * hz);
#pragma unroll
        for (int q = 0; q < AFTER; ++q) s.add(q < after, px[q], py[q], pz[q]);
        if (more) {
            for (int q = AFTER; __any_sync(FULL, q < after); ++q)
                if (q < after) s.term(true, lds_term(hl + (q + 1) * 256), H[q + 1]);
        }
    }
}

// The same for the backup driver, whose terms may be from before the sweep
// (ENT_OLD: from `old`): OLD_GATHER terms of each list are read together, then
// the ring's.  Most of its terms are old, so what counts is how many reads are
// in flight (62,400 points: 3.4 ms an iteration, 6.4 with a poll per term).
constexpr int OLD_GATHER = 8;
template <bool FOLD>
__device__ __forceinline__ void old_sums(const DevCloud &d, const SweepEntry *E, int n, const double *src, const double *old,
                                         unsigned rl, const Team &team, int pos, Sums<FOLD> &s) {
    const int nmax = (int)__reduce_max_sync(FULL, (unsigned)n);
    for (int base = 0; base < nmax; base += OLD_GATHER, E += OLD_GATHER) {
        const int m = min(n - base, OLD_GATHER);
        const double *at[OLD_GATHER];
        unsigned long long v[OLD_GATHER];
        unsigned rm = 0;               // this list's ring terms
#pragma unroll
        for (int q = 0; q < OLD_GATHER; ++q) {
            const int2 kp = *reinterpret_cast<const int2 *>(&E[q]);
            const bool in = q < m, ring = (kp.y & ENT_RING) != 0;
            at[q] = ((kp.y & ENT_OLD) ? old : src) + DG_STRIDE * (long long)(in ? kp.x : 0);
            rm |= in && ring ? 1u << q : 0u;
            v[q] = 0;
            ldg_if(v[q], at[q], in && !ring);
        }
        int spins = 0;
        for (;;) {
            bool pend = false;
#pragma unroll
            for (int q = 0; q < OLD_GATHER; ++q) pend = pend || pending_word(v[q]);
            if (!__any_sync(FULL, pend)) break;
            if (pend && !spin_continue(spins, d)) {
                // the wait ran out (d.err is set): the terms stay unset
#pragma unroll
                for (int q = 0; q < OLD_GATHER; ++q) v[q] = pending_word(v[q]) ? 0 : v[q];
            }
#pragma unroll
            for (int q = 0; q < OLD_GATHER; ++q) ldg_if(v[q], at[q], pending_word(v[q]));
        }
#pragma unroll
        for (int q = 0; q < OLD_GATHER; ++q) {
            const bool ring = (rm >> q) & 1u;
            if (__any_sync(FULL, ring)) {
                const int dist = ring ? ((pos - 1 - (E[q].pad >> ENT_RING_SHIFT)) & (CHAIN_RING - 1)) + 1 : 1;
                const double t = ring_word(d, rl + ring_slot(team, pos, dist) * 256, ring);
                if (ring) v[q] = (unsigned long long)__double_as_longlong(t);
            }
            s.term(q < m, __longlong_as_double((long long)v[q]), E[q]);
        }
    }
}

// A wall or interior point's slot: its fluxes along the three axes, less what T
// holds, into T.  The sign of each axis's list is selected, not branched on.
template <typename R>
__device__ __forceinline__ void slot_fluxes(bool wall, int mask, const FluxPreT<R> &P, const AxisTermsT<R> A[3], int lane,
                                            double *T) {
    for (; __any_sync(FULL, mask != 0); mask = mask_rest(mask)) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int both = (mask >> (2 * a)) & 3;
            const bool pos = (both & 1) != 0;
            R f[5];
            axis_flux(wall && a < 2, a, pos, P, A[a], A[2].An, -A[2].B, f);
            double *t = T + ((2 * a + (pos ? 0 : 1)) * MAX_SLOTS + lane) * 5;
            if (both) {
#pragma unroll
                for (int c = 0; c < 5; ++c) t[c] = (double)(f[c] - (R)t[c]);
            }
        }
    }
}

// The state of a slot's neighbour (conserved U in frame Fk) in the point's
// frame with the operators, where it left the range of the straight-line code.
template <typename R>
__device__ __noinline__ void slot_state_general(const R U[5], const FrameT<R> &Fk, const FrameT<R> &Fp, FluxPreT<R> &P,
                                                AxisTermsT<R> A[3]) {
    R pn[5];
    conserved_to_primitive(U, Fk, pn);
    flux_pre(pn, Fp, P);
    for (int a = 0; a < 3; ++a) axis_terms(P, a, A[a]);
}

// Term fluxes of a point outside the shared frame, lane per neighbour slot,
// into T[(list * MAX_SLOTS + slot) * 5 + component] (phases A and B of
// sweep_point).
template <typename R>
__device__ __noinline__ void unshared_terms(const DevCloud &d, ChainItem it, const SweepStage *st, int cls, bool forward,
                                            int lane, double *T, bool g0_newer) {
    const bool mine = (st->need >> lane) & 1u;
    const bool g0 = (it.info & CI_G0) != 0;
    const int k_slot = mine ? st->slot_nbr[lane] : it.p;
    const int mask_slot = mine ? st->slot_mask[lane] : 0;
    // the slot's state before the wait for its increment
    double Uk[5];
#pragma unroll
    for (int r = 0; r < 5; ++r) Uk[r] = d.U[5 * (size_t)k_slot + r];
    FrameT<R> Fk, Fp;
    load_frame(d.frame + 9 * (size_t)k_slot, Fk);
    load_frame(st->frame, Fp);
    if (mine && !g0) neighbour_fluxes<R>(d, cls, Fp, k_slot, mask_slot, lane, T);
    unsigned long long v[5] = {0, 0, 0, 0, 0};
    {
        const bool old = mine && ((st->old >> lane) & 1u);   // backup driver: from before the sweep
        const double *dsrc = (old ? d.dU_old : (forward ? d.dUp : d.dUn)) + 5 * (size_t)k_slot;
        int spins = 0;
        bool wait = mine;
        while (__any_sync(FULL, wait)) {
#pragma unroll
            for (int r = 0; r < 5; ++r) ldg_if(v[r], dsrc + r, wait);
            wait = wait && !ready5(v);
            if (wait && !spin_continue(spins, d)) wait = false;
        }
    }
    R U[5];
#pragma unroll
    for (int r = 0; r < 5; ++r) U[r] = (R)(__longlong_as_double((long long)v[r]) + Uk[r]);
    FluxPreT<R> P;
    AxisTermsT<R> A[3];
    bool ok = true;
    R yspb;
    state_core(U, Fk, Fp, P, yspb, ok);
    axes_core(P, yspb, A, ok);
    if (!__all_sync(FULL, ok || !mine)) {
        R Uc[5] = {U[0], U[1], U[2], U[3], U[4]};
        FrameT<R> Fkc = Fk, Fpc = Fp;
        FluxPreT<R> Pc;
        AxisTermsT<R> Ac[3];
        slot_state_general<R>(Uc, Fkc, Fpc, Pc, Ac);
        P = Pc;
#pragma unroll
        for (int a = 0; a < 3; ++a) A[a] = Ac[a];
    }
    if (g0) {
        // the copied phase-A fluxes: every lane's copies have landed
        if (g0_newer) cp_async_wait_one();
        else cp_async_wait_all();
        __syncwarp();
    }
    if (cls != CLS_OUTER) {
        slot_fluxes<R>(cls == CLS_WALL, mask_slot, P, A, lane, T);
    } else if (mine) {
        for (int e = 0; e < NDIR; ++e) {
            if (!(mask_slot & (1 << e))) continue;
            const int kind = flux_kind(cls, e);
#pragma unroll
            for (int cc = 0; cc < 5; ++cc) {
                double *t = &T[(e * MAX_SLOTS + lane) * 5 + cc];
                *t = (double)(flux_component(kind, cc, P, A) - (R)*t);
            }
        }
    }
    __syncwarp();
}

// The operators' form of a point whose arguments were out of the range of the
// branch-free ones: dU and the point's flux in the shared frame (component c of
// list dd) from its list sums.
struct PointOut {
    double dnew, flux;
};
__device__ __forceinline__ double list_total(bool wall, const double gd[NDIR]) {
    const double x = gd[0] + gd[1] + gd[2] + gd[3] + (wall ? gd[5] : gd[4]);
    return wall ? 2.0 * x : x + gd[5];
}
template <typename R, bool FOLD>
__device__ __noinline__ PointOut point_general(const double *frame0, const SweepStage *st, bool wall, bool forward, int dd,
                                               int c, double sx, double sy, double sz, double dinv, double base5) {
    double G = sx;
    if constexpr (!FOLD) {
        const double *g = st->geo + dd * 8;
        G = cramer_select(dd >> 1, g, sx, sy, sz) / g[6];
    }
    double gd[NDIR];
#pragma unroll
    for (int e = 0; e < NDIR; ++e) gd[e] = __shfl_sync(FULL, G, e * 5 + c);
    const double lu = list_total(wall, gd);
    PointOut o;
    o.dnew = forward ? -(dinv * (base5 + lu)) : base5 - dinv * lu;
    R U[5];
#pragma unroll
    for (int r = 0; r < 5; ++r) U[r] = (R)(__shfl_sync(FULL, o.dnew, r) + st->U[r]);
    FrameT<R> F0, F;
    load_frame(frame0, F0);
    load_frame(st->frame, F);
    o.flux = (double)state_flux_general<R>(dd, c, U, F, F0);
    return o;
}

// A point's own flux where the shared frame is not the global axes: component c
// of list dd at the conserved state U in frame F.  A kernel of its own (AXES
// false), since the launch knows the frame: one kernel with both forms had up to
// 5% slower sweeps in the axes.  62,400 points with a turned frame, ms per
// iteration: FP64 5.1 (9.0 with the operators after a straight-line form that
// such a frame always left), mixed precision 4.0 (6.1).
template <typename R>
__device__ __forceinline__ R turned_flux(int dd, int c, const R U[5], const FrameT<R> &F, const FrameT<R> &F0, bool &ok) {
    FluxPreT<R> P;
    R yspb, e, er;
    state_core(U, F, F0, P, yspb, ok);
    const int a = dd >> 1;
    const bool pos = (dd & 1) == 0;
    const R ua = pick3(a, P.ut1, P.ut2, P.un);
    gauss_core(ua * P.sb, e, er, ok);
    const R B = quot_nz(R(0.5) * e, P.spb, yspb), A = R(0.5) * (R(1.0) + (pos ? er : -er));
    return split_component(pos, c == a + 1, c, P.rho, P.pr, ua, pick3(c - 1, P.ut1, P.ut2, P.un), P.usq, A, B);
}

// A point in the shared frame, or a wall point, of a cloud with a shared frame
// under the alias driver: the sweep's common cases, kept apart from the others
// so that their code is short, free of the others' branches and, beyond the
// sums, the same for both (a wall point's own code is seldom in the
// instruction cache).  AXES: the shared frame is the global axes, and the driver
// the alias one.
template <typename R, bool FOLD, bool AXES>
__device__ __forceinline__ void common_point(const DevCloud &d, const ChainItem &it, const SweepStage *st, bool forward,
                                             int lane, int word, int dd, int c, double *T, const Team &team, int pos,
                                             bool g0_newer) {
    const int p = it.p;
    const bool hold = p + 1 == d.withhold1;           // failure-detection hook: publish nothing
    const bool wall = (it.info & CI_WALL) != 0;
    const double gold = st->gold[word], dinv = st->dinv[0], base5 = st->base[c];
    const double Uc = st->U[c];
    const int lo = count_sum(it.cnt & ((1u << (5 * dd)) - 1u)), n = item_count(it.cnt, dd);
    double g[7] = {0, 0, 0, 0, 0, 0, 1.0};
    double ydet = 0.0;
    bool ok = !AXES || d.frame0_axes != 0;
    if constexpr (!FOLD) {
#pragma unroll
        for (int r = 0; r < 7; ++r) g[r] = st->geo[dd * 8 + r];
        if (wall && dd == 4) g[6] = 1.0;              // a list walls do not have
        ok &= ieee_ok(fabs(g[6]));
        ydet = rcp_rn(g[6]);
    }
    double *out = (forward ? d.dgf : d.dgb) + (DG_LIST * dd + c);
    Sums<FOLD> s;
    const SweepEntry *E = st->ent + lo;
    if (wall) {
        unshared_terms<R>(d, it, st, CLS_WALL, forward, lane, T, g0_newer);
        const double *Tl = T + dd * MAX_SLOTS * 5 + c;
        const int nmax = (int)__reduce_max_sync(FULL, (unsigned)n);
        for (int j = 0; j < nmax; j += 4) {
            // past the list's end: its first terms, unused
            double t[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) t[q] = Tl[((E[j + q < n ? j + q : 0].pad >> 8) & (MAX_SLOTS - 1)) * 5];
#pragma unroll
            for (int q = 0; q < 4; ++q) s.term(j + q < n, t[q], E[j + q < n ? j + q : 0]);
        }
    } else {
        shared_sums<FOLD>(d, E, n, out, smem_addr(T + lane), smem_addr(team.ring + word), team, pos, s);
    }
    double G = s.x;
    if constexpr (!FOLD) {
        const double num = cramer_select(dd >> 1, g, s.x, s.y, s.z);
        ok &= ieee_num_ok(num);
        G = quot_rn(num, g[6], ydet);
    }
    double gd[NDIR];
#pragma unroll
    for (int e = 0; e < NDIR; ++e) gd[e] = __shfl_sync(FULL, G, e * 5 + c);
    const double lu = list_total(wall, gd);
    double dnew = forward ? -(dinv * (base5 + lu)) : base5 - dinv * lu;
    const double un = dnew + Uc;
    R Un[5];
#pragma unroll
    for (int r = 0; r < 5; ++r) Un[r] = (R)__shfl_sync(FULL, un, r);
    double flux;
    if constexpr (AXES) {
        if (wall) {
            // back from the point's frame (conserved_to_primitive)
            FrameT<R> F;
            load_frame(st->frame, F);
            const R m1 = Un[1], m2 = Un[2], m3 = Un[3];
#pragma unroll
            for (int r = 0; r < 3; ++r) Un[1 + r] = F.t1[r] * m1 + F.t2[r] * m2 + F.n[r] * m3;
        }
        flux = (double)state_flux(dd, c, Un, ok);
    } else {
        FrameT<R> F, F0;
        load_frame(st->frame, F);
        load_frame(d.frame0, F0);
        flux = (double)turned_flux(dd, c, Un, F, F0, ok);
    }
    if (!__all_sync(FULL, ok)) {
        const PointOut o = point_general<R, FOLD>(d.frame0, st, wall, forward, dd, c, s.x, s.y, s.z, dinv, base5);
        dnew = o.dnew;
        flux = o.flux;
    }
    const double v = sizeof(R) == 8 ? flux - gold : (double)((R)flux - (R)gold);
    sts_relaxed(smem_addr(team.ring + ring_slot(team, pos, 0) * 32 + lane), v);
    if (lane < 30 && (it.info & CI_PUBLISH) && !hold) st_relaxed_f64(out + DG_STRIDE * (size_t)p, v);
    if (lane < 5 && !hold) st_relaxed_f64((forward ? d.dUp : d.dUn) + 5 * (size_t)p + lane, dnew);
    team_leave(team, pos, lane);
}

// One point of the forward (LdelU) or backward (UdelU) sweep by one warp of
// its chain's team (implicit_forward_and_reverse_sweeps.f90:30-37 / :61-68),
// from its stage in shared memory: any class of point.  Lane (list dd,
// component c); lanes 30 and 31 repeat lanes 25 and 26 and store nothing.
//
// R: the type of the flux evaluations (float in mixed precision); the list
// sums, 3x3 solves, D_inv and the increments themselves are double.
// FOLD (mixed precision): each term's weight carries its list's 3x3 solve
// (folded when the handle is attached), so the sums are the derivatives;
// otherwise the three weighted moments are summed in FP64 and solved, as the
// reference does.
// OLD: points of the backup driver in the shared frame are among them.
template <typename R, bool FOLD, bool OLD>
__device__ __noinline__ void general_point(const DevCloud &d, ChainItem it, const SweepStage *st, bool forward, int lane,
                                           double *T, Team team, int pos, bool g0_newer) {
    const int p = it.p;
    const bool wall = (it.info & CI_WALL) != 0;
    const bool copy = (it.info & CI_COPY) != 0;       // supersonic point
    const bool outer = (it.info & CI_OUTER) != 0;     // backup driver
    const bool hold = p + 1 == d.withhold1;           // failure-detection hook: publish nothing
    const int word = lane < 30 ? lane : lane - 5;
    const int dd = word / 5, c = word - 5 * dd;
    double *dU = (forward ? d.dUp : d.dUn) + 5 * (size_t)p;
    FrameT<R> Fp;
    load_frame(st->frame, Fp);
    const double gold = st->gold[word];
    double dnew = 0.0;
    if (copy) {
        // implicit_forward_and_reverse_sweeps.f90:38-51 / :69-82: the
        // nearest neighbour's increment, updated earlier in this sweep or
        // from before it
        const int q = st->ent[0].k;
        if (q >= 0)
            dnew = (st->ent[0].pad & ENT_COPY_NEW) ? poll_word((forward ? d.dUp : d.dUn) + 5 * (size_t)q + c, d)
                                                   : d.dU_old[5 * (size_t)q + c];
    } else {
        const double dinv = st->dinv[0], base5 = st->base[c];
        int lo = 0, n = 0;
#pragma unroll
        for (int e = 0; e < NDIR; ++e) {
            const int ce = item_count(it.cnt, e);
            if (e < dd) lo += ce;
            if (e == dd) n = ce;
        }
        const SweepEntry *E = st->ent + lo;
        const bool shared = OLD && (it.info & CI_SHARED) != 0;
        if (!shared) {
            const int cls = wall ? CLS_WALL : (outer ? CLS_OUTER : CLS_INTERIOR);
            unshared_terms<R>(d, it, st, cls, forward, lane, T, g0_newer);
        }
        Sums<FOLD> s;
        if (OLD && shared) {
            const double *src = (forward ? d.dgf : d.dgb) + (DG_LIST * dd + c);
            old_sums<FOLD>(d, E, n, src, d.dg_old + (DG_LIST * dd + c), smem_addr(team.ring + word), team, pos, s);
        } else {
            const double *Tl = T + dd * MAX_SLOTS * 5 + c;
            const int nmax = (int)__reduce_max_sync(FULL, (unsigned)n);
            for (int j = 0; j < nmax; j += 2) {
                // past the list's end: its first terms, unused
                double t[2];
#pragma unroll
                for (int q = 0; q < 2; ++q) t[q] = Tl[((E[j + q < n ? j + q : 0].pad >> 8) & (MAX_SLOTS - 1)) * 5];
#pragma unroll
                for (int q = 0; q < 2; ++q) s.term(j + q < n, t[q], E[j + q < n ? j + q : 0]);
            }
        }
        __syncwarp();
        double G = s.x;
        if constexpr (!FOLD) {
            const double *g = st->geo + ((outer && dd == 4) ? 5 : dd) * 8;   // outer z+ over conn: row 5
            G = cramer_select(dd >> 1, g, s.x, s.y, s.z) / g[6];
        }
        double gd[NDIR];
#pragma unroll
        for (int e = 0; e < NDIR; ++e) gd[e] = __shfl_sync(FULL, G, e * 5 + c);
        double lu;
        if (wall) lu = 2.0 * (gd[0] + gd[1] + gd[2] + gd[3] + gd[5]);
        else if (outer) lu = gd[0] + gd[1] + gd[2] + gd[3] + gd[4];   // *_sweep_outer.f90:406
        else lu = gd[0] + gd[1] + gd[2] + gd[3] + gd[4] + gd[5];
        dnew = forward ? -(dinv * (base5 + lu)) : base5 - dinv * lu;
    }
    if (lane < 5 && !hold) st_relaxed_f64(dU + lane, dnew);
    if (d.shared_frame) {
        // publish this point's increment for the consumers in the shared frame
        R U[5];
#pragma unroll
        for (int r = 0; r < 5; ++r) U[r] = (R)(__shfl_sync(FULL, dnew, r) + st->U[r]);
        FrameT<R> F0;
        load_frame(d.frame0, F0);
        const double v = (double)(state_flux_general<R>(dd, c, U, Fp, F0) - (R)gold);
        sts_relaxed(smem_addr(team.ring + ring_slot(team, pos, 0) * 32 + lane), v);
        if (lane < 30 && (it.info & CI_PUBLISH) && !hold)
            st_relaxed_f64((forward ? d.dgf : d.dgb) + DG_STRIDE * (size_t)p + DG_LIST * dd + c, v);
    }
    team_leave(team, pos, lane);
}

// Shared memory of one block: each warp's T buffer and two stages, then each
// team's ring and positions.
__host__ __device__ constexpr int chain_smem_bytes(int team) {
    return CH_WPB * CHAIN_WARP_BYTES + CH_WPB / team * ring_slots(team) * 256 + CH_WPB * 4;
}

// One block of a cloud's chain sweep: block `block` of the cloud's
// chain_blocks(ch_chains, ch_shape).
template <typename R, bool FOLD, bool AXES>
__device__ __forceinline__ void chain_sweep(const DevCloud &d, int forward, int block) {
    extern __shared__ double smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int size = d.ch_shape.team, teams = CH_WPB / size, mine = warp / size;
    char *sm = reinterpret_cast<char *>(smem);
    double *T = reinterpret_cast<double *>(sm + warp * CHAIN_WARP_BYTES);
    SweepStage *stg = reinterpret_cast<SweepStage *>(T + SW_T_DOUBLES);
    char *shared = sm + CH_WPB * CHAIN_WARP_BYTES;
    Team team;
    team.size = size;
    team.sub = warp - mine * size;
    team.slots = ring_slots(size);
    team.ring = reinterpret_cast<double *>(shared) + mine * team.slots * 32;
    team.at = reinterpret_cast<int *>(shared + teams * team.slots * 256) + mine * size;
    for (int j = team.sub; j < team.slots; j += size)
        team.ring[j * 32 + lane] = __longlong_as_double((long long)DU_PENDING);
    if (lane == 0) team.at[team.sub] = team.sub;
    __syncthreads();
    const int me = block * teams + mine;
    if (me >= d.ch_chains) return;
    const int dir = forward ? 0 : 1;
    const int a = d.ch_ptr[dir][me], len = d.ch_ptr[dir][me + 1] - a;
    const ChainItem *items = d.ch_items[dir] + a;
    // lanes 30 and 31 repeat lanes 25 and 26 and store nothing
    const int word = lane < 30 ? lane : lane - 5;
    const int dd = word / 5, c = word - 5 * dd;
    int pos = team.sub;
    if (pos < len) {
        ChainItem cur = items[pos];
        const StageLane L = stage_lane(d, forward != 0, lane);
        chain_stage(d, L, cur, forward != 0, lane, &stg[0]);
        cp_async_commit();
        ChainItem nxt = pos + size < len ? items[pos + size] : cur;
        int s = 0;
        for (; pos < len; pos += size) {
            const bool more = pos + size < len;
            cp_async_wait_all();
            __syncwarp();
            if (cur.info & CI_G0) {
                // phase A of this point, computed before the sweep (k_g0): into T,
                // which the previous point no longer uses
                const char *src = reinterpret_cast<const char *>(d.g0 + (size_t)(cur.info >> CI_G0_SHIFT) * G0_DOUBLES);
                char *dst = reinterpret_cast<char *>(T);
                for (int j = lane; j < G0_DOUBLES / 2; j += 32) cp_async16(dst + 16 * j, src + 16 * j);
                cp_async_commit();
            }
            if (more) {
                chain_stage(d, L, nxt, forward != 0, lane, &stg[s ^ 1]);
                cp_async_commit();
            }
            const ChainItem after = pos + 2 * size < len ? items[pos + 2 * size] : nxt;
            team_enter(d, team, pos, lane);
            if ((cur.info & (CI_SHARED | CI_WALL)) && d.shared_frame && !d.dg_old)
                common_point<R, FOLD, AXES>(d, cur, &stg[s], forward != 0, lane, word, dd, c, T, team, pos, more);
            else
                general_point<R, FOLD, !AXES>(d, cur, &stg[s], forward != 0, lane, T, team, pos, more);
            cur = nxt;
            nxt = after;
            s ^= 1;
        }
    }
    // the chain's end: the others need not wait for this warp
    __syncwarp();
    if (lane == 0) sts_release(smem_addr(team.at + team.sub), 0x7fffffff);
}

}  // namespace mfcfd
