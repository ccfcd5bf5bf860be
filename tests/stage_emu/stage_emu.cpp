// stage_emu.cpp - CPU emulation of the staged passes, for tests.
//
// Runs a gate list on a host state the way qs_gates_apply does with k_stage
// (qpanda_b200/csrc/qs_stage.cu): the library's own planner (passes, stages,
// parameter blocks), the tile bases, the load and store offsets, the slots of
// every stage change and the per-thread arithmetic (qs_stage.h, the functions
// the kernel calls), in the state's own precision.  Checks that every
// amplitude is loaded once and stored once, every shared-memory slot written
// and read once per stage change, all of them in range, and counts the bank
// conflicts of the stage changes.
//
//   g++ -O2 -std=c++17 -shared -fPIC stage_emu.cpp -I<csrc> -I<include> -L<lib> -lqsb200
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <vector>

#include "qs_stage.h"

using namespace qs_stg;

namespace {

char g_err[256];

int fail(const char *msg, long long a = 0, long long b = 0)
{
    snprintf(g_err, sizeof(g_err), msg, a, b);
    return 1;
}

struct Stats {
    long long passes, stages, conflicts, ops, small;
};

template <typename T>
struct V2 {
    T x, y;
};

// extra wavefronts of one access instruction: a phase is the lanes that fill
// one 128-byte row
long long conflicts(const std::vector<uint32_t> &slots, int per_row)
{
    long long extra = 0;
    for (size_t p = 0; p + per_row <= slots.size(); p += per_row) {
        std::vector<int> hit(per_row, 0);
        int worst = 0;
        for (int l = 0; l < per_row; ++l) worst = std::max(worst, ++hit[slots[p + l] % per_row]);
        extra += worst - 1;
    }
    return extra;
}

template <typename T, typename R>
int run_pass(std::vector<V2<T>> &a, int n, const R &P, Stats &st)
{
    constexpr int RB = Traits<T>::RB, NR = 1 << RB;
    const uint32_t threads = 1u << (P.K - RB);
    if (P.nstages < 1 || P.nstages > R::NST || P.nladders > R::NLAD) return fail("stages %lld", P.nstages);
    std::vector<uint8_t> seen(a.size(), 0), stored(a.size(), 0);
    const uint32_t slots_n = tile_slots<T>(P.K);
    std::vector<V2<T>> tile(slots_n), out(a);
    std::vector<Regs<T, RB>> v(threads);
    for (uint64_t tl = 0; tl < a.size() >> P.K; ++tl) {
        const uint64_t base = tile_base(P, tl);
        auto offset = [&](uint32_t t, int r, const uint32_t *gt, const uint32_t (&gr)[4]) {
            constexpr int LOW = Traits<T>::LOW;
            uint64_t u = reg_sum<RB>(r, gr);
            for (int j = LOW; j < kMaxThreadBits; ++j) u += (t >> j & 1) * gt[j];
            return base + (t & ((1u << LOW) - 1)) + (u << LOW);
        };
        for (uint32_t t = 0; t < threads; ++t)
            for (int r = 0; r < NR; ++r) {
                const uint64_t o = offset(t, r, P.gin_t, P.gin_r);
                if (o >= a.size() || seen[o]++) return fail("amplitude %lld loaded twice or out of range", (long long)o);
                v[t].r[r] = a[o].x;
                v[t].i[r] = a[o].y;
            }
        std::vector<uint32_t> tt(threads, 0);
        for (int s = 0; s < P.nstages; ++s) {
            const Stage &sg = P.st[s];
            std::vector<uint32_t> prev(tt);
            for (uint32_t t = 0; t < threads; ++t) {
                tt[t] = 0;
                for (int j = 0; j < kMaxThreadBits; ++j) tt[t] += (t >> j & 1) * sg.tb[j];
            }
            if (s) {
                std::vector<uint8_t> wr(slots_n, 0), rd(slots_n, 0);
                for (int write = 1; write >= 0; --write) {
                    uint32_t pr[4];
                    for (int j = 0; j < 4; ++j) pr[j] = write ? P.st[s - 1].pr[j] : sg.pr[j];
                    for (int r = 0; r < NR; ++r) {
                        std::vector<uint32_t> slots(threads);
                        for (uint32_t t = 0; t < threads; ++t) {
                            const uint32_t sl = ((write ? prev[t] : tt[t]) >> 16) + reg_sum<RB>(r, pr);
                            if (sl >= slots_n || (write ? wr : rd)[sl]++) return fail("slot %lld used twice", sl);
                            if (write) tile[sl] = {v[t].r[r], v[t].i[r]};
                            else { v[t].r[r] = tile[sl].x; v[t].i[r] = tile[sl].y; }
                            slots[t] = sl;
                        }
                        st.conflicts += conflicts(slots, 1 << Traits<T>::LB);
                    }
                }
            }
            for (int o = sg.first; o < sg.first + sg.count; ++o) {
                if (o >= R::NOP) return fail("op %lld past the block", o);
                const Op<T> &op = P.op[o];
                if (((op.kind >= K_LADR && op.kind <= K_LAD0) || op.kind >= K_LADH) && (int)op.ladder >= P.nladders) return fail("ladder %lld", op.ladder);
                if (!op.cond && (op.need || op.cthr)) return fail("op %lld hides its condition", o);
                if ((base & op.need) != op.need) continue;
                for (uint32_t t = 0; t < threads; ++t) {
                    if ((tt[t] & op.cthr) != op.cthr) continue;
                    apply_op<T, RB>(v[t], op, [&](uint32_t l, T &fr, T &fi) {
                        double lr, li, wr, wi;
                        ladder_lane(P, l, t & 31, lr, li);
                        ladder_warp(P, l, t >> 5, base, wr, wi);
                        fr = (T)lr;
                        fi = (T)li;
                        cmul(fr, fi, (T)wr, (T)wi);
                    });
                }
            }
        }
        for (uint32_t t = 0; t < threads; ++t)
            for (int r = 0; r < NR; ++r) {
                if (P.scale_kind == 1) { v[t].r[r] *= P.scale[0]; v[t].i[r] *= P.scale[0]; }
                if (P.scale_kind == 2) cmul(v[t].r[r], v[t].i[r], P.scale[0], P.scale[1]);
                const uint64_t o = offset(t, r, P.gout_t, P.gout_r);
                if (o >= a.size() || stored[o]++) return fail("amplitude %lld stored twice or out of range", (long long)o);
                if (P.nstages == 1 && o != offset(t, r, P.gin_t, P.gin_r))
                    return fail("one stage alone stores elsewhere than it loads (thread %lld)", t);
                // in place: what one tile stores, that tile alone has loaded
                if (!seen[o]) return fail("amplitude %lld stored before its load", (long long)o);
                out[o] = {v[t].r[r], v[t].i[r]};
            }
    }
    for (size_t i = 0; i < a.size(); ++i)
        if (seen[i] != 1 || stored[i] != 1) return fail("amplitude %lld missed", (long long)i);
    a.swap(out);
    ++st.passes;
    st.stages += P.nstages;
    st.ops += P.st[P.nstages - 1].first + P.st[P.nstages - 1].count;
    return 0;
}

template <typename T>
int run_permute(std::vector<V2<T>> &a, const Permute &P, Stats &st)
{
    constexpr int RB = Traits<T>::RB, NR = 1 << RB, LOW = Traits<T>::LOW;
    constexpr uint32_t slots_n = tile_slots<T>(RB + 8);
    const uint32_t threads = 1u << (P.K - RB);
    if (P.K != RB + 8 && P.K != RB + 7) return fail("permute tile %lld", P.K);
    std::vector<uint8_t> seen(a.size(), 0), stored(a.size(), 0);
    std::vector<V2<T>> out(a), tile(2 * slots_n);
    for (uint64_t tl = 0; tl < a.size() >> P.K; ++tl) {
        const uint64_t base = tile_base(P, tl), other = permute_partner(P, base);
        if (permute_partner(P, other) != base) return fail("tile %lld has no partner", (long long)tl);
        if (base > other) continue;
        const int two = other != base;
        std::vector<uint8_t> wr(2 * slots_n, 0), rd(2 * slots_n, 0);
        for (int store = 0; store < 2; ++store)
            for (int side = 0; side <= two; ++side)
                for (int k = 0; k < NR; ++k) {
                    std::vector<uint32_t> slots(threads);
                    for (uint32_t t = 0; t < threads; ++t) {
                        uint32_t u = 0, w = 0;
                        for (int j = 0; j < 8; ++j) {
                            u += (t >> j & 1) * P.g_t[j];
                            w += (t >> j & 1) * (store ? P.r_t[j] : P.w_t[j]);
                        }
                        const uint32_t sl = side * slots_n + w + reg_sum<RB>(k, store ? P.r_r : P.w_r);
                        const uint64_t at = ((store ? !side : side) && two ? other : base) + (t & ((1u << LOW) - 1)) +
                                            ((uint64_t)(u + reg_sum<RB>(k, P.g_r)) << LOW);
                        if (at >= a.size() || sl >= 2 * slots_n || (store ? stored : seen)[at]++ || (store ? rd : wr)[sl]++)
                            return fail("amplitude %lld or slot %lld used twice", (long long)at, sl);
                        if (store && (!seen[at] || !wr[sl])) return fail("amplitude %lld stored before its load", (long long)at);
                        if (store) out[at] = tile[sl];
                        else tile[sl] = a[at];
                        slots[t] = sl;
                    }
                    st.conflicts += conflicts(slots, 1 << Traits<T>::LB);
                }
    }
    for (size_t i = 0; i < a.size(); ++i)
        if (seen[i] != 1 || stored[i] != 1) return fail("amplitude %lld missed", (long long)i);
    a.swap(out);
    ++st.passes;
    return 0;
}

template <typename T>
int run(double *amp, int n, const std::vector<qs_prim> &prims, int dtype, bool execute, Stats &st)
{
    std::vector<V2<T>> a(execute ? (size_t)1 << n : 0);
    for (size_t i = 0; i < a.size(); ++i) a[i] = {(T)amp[2 * i], (T)amp[2 * i + 1]};
    Planner P(prims, n, dtype);
    uint64_t qmask;
    std::vector<int> pass, rest;
    auto S = new RunSmall<T>();
    auto L = new RunLarge<T>();
    int r = 0;
    Permute perm;
    while (!r) {
        if (plan_permute<T>(P, &perm)) {
            if (execute) r = run_permute<T>(a, perm, st);
            else ++st.passes;
            break;
        }
        if (!P.next(&qmask, &pass)) break;
        bool done = false;
        if ((int)pass.size() < RunSmall<T>::NOP - 1) {
            plan_pass<RunSmall<T>, T>(P, qmask, pass, S, &rest);
            if ((done = rest.empty())) {
                ++st.small;
                if (execute) r = run_pass<T>(a, n, *S, st);
                else { ++st.passes; st.stages += S->nstages; }
            }
        }
        if (!done) {
            plan_pass<RunLarge<T>, T>(P, qmask, pass, L, &rest);
            if (rest.size() == pass.size()) r = fail("a pass of %lld ops takes none", (long long)pass.size());
            P.give_back(rest);
            if (execute) r = r ? r : run_pass<T>(a, n, *L, st);
            else { ++st.passes; st.stages += L->nstages; }
        }
    }
    delete S;
    delete L;
    for (size_t i = 0; i < a.size(); ++i) {
        amp[2 * i] = a[i].x;
        amp[2 * i + 1] = a[i].y;
    }
    return r;
}

}  // namespace

extern "C" const char *stage_emu_error(void) { return g_err; }

// amp: 2^n complex128, in place (NULL: plan only).  stats[5]: passes, stages,
// bank conflicts, ops, passes in the small parameter block.
extern "C" int stage_emu_apply(double *amp, int n, const void *gates, int count, int dtype, long long *stats)
{
    g_err[0] = 0;
    const qs_gate *g = static_cast<const qs_gate *>(gates);
    std::vector<qs_prim> prims(count);
    for (int i = 0; i < count; ++i)
        if (qs_lower_gate(n, &g[i], &prims[i])) return fail("gate %lld does not lower", i);
    Stats st = {0, 0, 0, 0, 0};
    const int r = dtype == QS_C64 ? run<float>(amp, n, prims, dtype, amp != nullptr, st)
                                  : run<double>(amp, n, prims, dtype, amp != nullptr, st);
    stats[0] = st.passes;
    stats[1] = st.stages;
    stats[2] = st.conflicts;
    stats[3] = st.ops;
    stats[4] = st.small;
    return r;
}
