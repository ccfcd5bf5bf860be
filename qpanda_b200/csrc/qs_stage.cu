// qs_stage.cu - the kernel of the staged passes (plan and arithmetic: qs_stage.h).
#include <atomic>
#include <vector>

#include "qs_common.cuh"
#include "qs_stage.h"

namespace {

using namespace qs_stg;

// Five CTAs per SM in FP32 (48 registers, a few words spilled): an op is a chain
// of record loads, a jump and multiply-adds, and more warps cover it.  28-qubit
// depth-16 list on a dense state: three CTAs 37.1 ms, four 32.6, five 27.4, six
// (40 registers) 31.3; 28-qubit QFT 6.25, 5.63, 5.29, 7.2 (5.04 since).  FP64: two CTAs of 512
// threads, three (40 registers) 15.6 against 13.2 ms (26 qubits, depth 16).
template <typename T, typename R>
__global__ void __launch_bounds__(1 << (kMaxTile - Traits<T>::RB), sizeof(T) == 4 ? 5 : 2)
k_stage(T *__restrict__ a, const __grid_constant__ R P)
{
    constexpr int RB = Traits<T>::RB, NR = 1 << RB;
    typedef typename vec2<T>::type V;
    extern __shared__ __align__(16) unsigned char stage_smem[];
    V *tile = reinterpret_cast<V *>(stage_smem);
    V *pa = reinterpret_cast<V *>(a);
    constexpr int LOW = Traits<T>::LOW;
    const uint32_t t = threadIdx.x;
    qs_let_next_start();
    const uint64_t base = tile_base(P, blockIdx.x);
    Regs<T, RB> v;
    // the state address of a thread's register r: thread part + register part
    // (the same for all threads), both in units of 2^LOW amplitudes
    auto thread_at = [&](const uint32_t *gt) {
        uint32_t u = 0;
#pragma unroll
        for (int j = LOW; j < kMaxThreadBits; ++j) u += (t >> j & 1) * gt[j];
        return pa + base + (t & ((1u << LOW) - 1)) + ((uint64_t)u << LOW);
    };
    auto reg_at = [&](V *p, int r, const uint32_t (&gr)[4]) { return p + ((uint64_t)reg_sum<RB>(r, gr) << LOW); };
    {
        V *p = thread_at(P.gin_t);
        qs_wait_previous();
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const V x = *reg_at(p, r, P.gin_r);
            v.r[r] = x.x;
            v.i[r] = x.y;
        }
    }
    // The first passes after |0...0> meet tiles of zeros only (a qubit outside
    // the tile is still in |0> and set in the tile's base).  Gates are linear:
    // such a tile stays as it is, neither computed nor stored.
    if (P.zeros) {
        bool any = false;
#pragma unroll
        for (int r = 0; r < NR; ++r) any = any || !(v.r[r] == 0) || !(v.i[r] == 0);
        if (!__syncthreads_or(any)) return;
    }
    // the ladders' factors, while the loads are in flight
    V *lane_f = tile + tile_slots<T>(P.K), *warp_f = lane_f + 32 * P.nladders;
    const uint32_t lw = warp_bits<T>(P.K);
    if (P.nladders) {
        for (uint32_t i = t; i < 32u * P.nladders; i += blockDim.x) {
            double fr, fi;
            ladder_lane(P, i >> 5, i & 31, fr, fi);
            lane_f[i] = V{(T)fr, (T)fi};
        }
        for (uint32_t i = t; i < (uint32_t)P.nladders << lw; i += blockDim.x) {
            double fr, fi;
            ladder_warp(P, i >> lw, i & ((1u << lw) - 1), base, fr, fi);
            warp_f[i] = V{(T)fr, (T)fi};
        }
        __syncthreads();
    }
    auto factor = [&](uint32_t l, T &fr, T &fi) {
        const V x = lane_f[32 * l + (t & 31)], y = warp_f[(l << lw) + (t >> 5)];
        fr = x.x;
        fi = x.y;
        cmul(fr, fi, y.x, y.y);
    };
    uint32_t slot = 0;
    for (int s = 0; s < P.nstages; ++s) {
        const Stage &st = P.st[s];
        uint32_t tt = 0;
#pragma unroll
        for (int j = 0; j < kMaxThreadBits; ++j) tt += (t >> j & 1) * st.tb[j];
        if (s) {
            // to the new stage's registers through shared memory.  The slots
            // written are the ones this thread read at the stage before, so
            // one barrier is enough.
            const Stage &sp = P.st[s - 1];
            uint32_t pr[4];
#pragma unroll
            for (int j = 0; j < RB; ++j) pr[j] = sp.pr[j];
            V *w = tile + slot;
#pragma unroll
            for (int r = 0; r < NR; ++r) w[reg_sum<RB>(r, pr)] = V{v.r[r], v.i[r]};
            __syncthreads();
#pragma unroll
            for (int j = 0; j < RB; ++j) pr[j] = st.pr[j];
            w = tile + (tt >> 16);
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const V x = w[reg_sum<RB>(r, pr)];
                v.r[r] = x.x;
                v.i[r] = x.y;
            }
        }
        slot = tt >> 16;
        const uint32_t ti = tt & 0xffffu;
        const int end = st.first + st.count;
        for (int o = st.first; o < end; ++o) {
            const Op<T> &op = P.op[o];
            if (op.cond) {
                if ((base & op.need) != op.need) continue;     // the same for the whole CTA
                if ((ti & op.cthr) != op.cthr) continue;
            }
            apply_op<T, RB>(v, op, factor);
        }
    }
    {
        if (P.scale_kind == 1) {
#pragma unroll
            for (int r = 0; r < NR; ++r) { v.r[r] *= P.scale[0]; v.i[r] *= P.scale[0]; }
        } else if (P.scale_kind == 2) {
#pragma unroll
            for (int r = 0; r < NR; ++r) cmul(v.r[r], v.i[r], P.scale[0], P.scale[1]);
        }
        V *p = thread_at(P.gout_t);
#pragma unroll
        for (int r = 0; r < NR; ++r) *reg_at(p, r, P.gout_r) = V{v.r[r], v.i[r]};
    }
}

// Exchange amplitudes in place: see Permute (qs_stage.h).  Bound by HBM: one
// read and one write of the state, in rows of at least 128 bytes on both
// sides, however many pairs (the ten pairs that a 28-qubit QFT's last gate
// pass leaves took three staged passes).
template <typename T>
__global__ void __launch_bounds__(256, 2) k_permute(T *__restrict__ a, const __grid_constant__ Permute P)
{
    constexpr int RB = Traits<T>::RB, NR = 1 << RB, LOW = Traits<T>::LOW;
    typedef typename vec2<T>::type V;
    extern __shared__ __align__(16) unsigned char stage_smem[];
    V *tile = reinterpret_cast<V *>(stage_smem);
    const uint32_t t = threadIdx.x;
    qs_let_next_start();
    const uint64_t base = tile_base(P, blockIdx.x), other = permute_partner(P, base);
    if (base > other) return;                                  // the partner's CTA does both
    uint32_t u = 0, w = 0, r = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        u += (t >> j & 1) * P.g_t[j];
        w += (t >> j & 1) * P.w_t[j];
        r += (t >> j & 1) * P.r_t[j];
    }
    V *here = reinterpret_cast<V *>(a) + base + (t & ((1u << LOW) - 1)) + ((uint64_t)u << LOW);
    V *there = here + (other - base);
    constexpr uint32_t kSlots = tile_slots<T>(RB + 8);
    const bool two = other != base;
    V x[NR], y[NR];
    qs_wait_previous();
#pragma unroll
    for (int k = 0; k < NR; ++k) x[k] = here[(uint64_t)reg_sum<RB>(k, P.g_r) << LOW];
    if (two) {
#pragma unroll
        for (int k = 0; k < NR; ++k) y[k] = there[(uint64_t)reg_sum<RB>(k, P.g_r) << LOW];
    }
#pragma unroll
    for (int k = 0; k < NR; ++k) tile[w + reg_sum<RB>(k, P.w_r)] = x[k];
    if (two) {
#pragma unroll
        for (int k = 0; k < NR; ++k) tile[kSlots + w + reg_sum<RB>(k, P.w_r)] = y[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NR; ++k) there[(uint64_t)reg_sum<RB>(k, P.g_r) << LOW] = tile[r + reg_sum<RB>(k, P.r_r)];
    if (two) {
#pragma unroll
        for (int k = 0; k < NR; ++k) here[(uint64_t)reg_sum<RB>(k, P.g_r) << LOW] = tile[kSlots + r + reg_sum<RB>(k, P.r_r)];
    }
}

template <typename T>
int launch_permute(qs_state *s, const Permute &P)
{
    constexpr size_t smem = 2 * 2 * sizeof(T) * tile_slots<T>(Traits<T>::RB + 8);
    QS_CUDA_TRY(cudaFuncSetAttribute(k_permute<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    QS_CUDA_TRY(qs_launch_overlapped(k_permute<T>, (unsigned)(s->N >> P.K), 1u << (P.K - Traits<T>::RB), smem,
                                     s->stream, static_cast<T *>(s->amp), P));
    QS_LAUNCH_CHECK("k_permute");
    return QS_OK;
}

template <typename T, typename R>
int launch(qs_state *s, const R &P)
{
    const size_t amps = tile_slots<T>(P.K) + (size_t)P.nladders * (32 + (1u << warp_bits<T>(P.K)));
    const size_t smem = 2 * sizeof(T) * amps;
    if (smem > 48 * 1024) {
        // once per device and kernel: the largest a pass can need
        static std::atomic<uint64_t> done{0};
        const uint64_t bit = 1ull << (s->device & 63);
        if (!(done.load() & bit)) {
            const int most = (int)(2 * sizeof(T) * (tile_slots<T>(kMaxTile) + R::NLAD * (32 + (1u << warp_bits<T>(kMaxTile)))));
            QS_CUDA_TRY(cudaFuncSetAttribute(k_stage<T, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
            done.fetch_or(bit);
        }
    }
    QS_CUDA_TRY(qs_launch_overlapped(k_stage<T, R>, (unsigned)(s->N >> P.K), 1u << (P.K - Traits<T>::RB), smem,
                                     s->stream, static_cast<T *>(s->amp), P));
    return QS_OK;
}

// one op on the per-gate kernels
int launch_op(qs_state *s, const Planner &P, const GOp &g)
{
    int r = QS_OK;
    if (g.type == G_U || (g.type == G_DIAG && g.ctrl == 0)) {
        const uint64_t t = g.type == G_U ? g.tgt : g.off1;
        return launch_pair(s, t, 0, 0, t, g.m);
    }
    if (g.type == G_DIAG) {
        for (int k = g.first; !r && k < g.first + g.count; ++k) {
            const Term &t = P.terms[(size_t)k];
            r = launch_phase(s, g.ctrl | (t.q >= 0 ? 1ull << t.q : 0), t.re, t.im);
        }
        return r;
    }
    if (g.type == G_CU) return launch_pair(s, g.tgt | g.ctrl, g.ctrl, 0, g.tgt, g.m);
    return launch_pair(s, g.tgt | g.ctrl, g.ctrl, g.off0, g.off1, g.m);
}

// HBM traffic of an op on the per-gate kernels, in passes over the state,
// in whole 32-byte sectors: each control or phase bit above the sector halves
// it, and so does an exchange whose higher bit is.
double op_traffic(const Planner &P, const GOp &g)
{
    const int sb = P.dtype == QS_C64 ? 2 : 1;
    auto part = [&](uint64_t bits) { return std::ldexp(1.0, -__builtin_popcountll(bits >> sb)); };
    if (g.type == G_U || (g.type == G_DIAG && g.ctrl == 0)) return 1.0;
    if (g.type == G_DIAG) {
        double sum = 0;
        for (int k = g.first; k < g.first + g.count; ++k) {
            const Term &t = P.terms[(size_t)k];
            sum += part(g.ctrl | (t.q >= 0 ? 1ull << t.q : 0));
        }
        return sum;
    }
    const double c = part(g.ctrl);
    return g.type == G_CU || !((g.off0 | g.off1) >> sb) ? c : c / 2;
}

template <typename T>
int apply_t(qs_state *s, const std::vector<qs_prim> &prims)
{
    Planner P(prims, s->n, s->dtype);
    uint64_t qmask;
    std::vector<int> pass, rest;
    RunSmall<T> small;
    static thread_local RunLarge<T> large;
    bool finite = true;                          // zero times infinity would not stay zero
    for (const qs_prim &p : prims)
        for (int k = 0; s->untouched && k < 8; ++k) finite = finite && std::isfinite(p.m[k]);
    Permute perm;
    while (true) {
        if (plan_permute<T>(P, &perm)) {
            s->untouched = 0;
            return launch_permute<T>(s, perm);
        }
        if (!P.next(&qmask, &pass)) break;
        // a pass that would move more than its gates one by one stays with them,
        // and so does a lone one (a ladder is as many launches as it has phases: 23
        // phases of 24 qubits complex128 1063 us so, 96 in a pass)
        double traffic = 0;
        int launches = 0;
        for (int i : pass) {
            const GOp &g = P.ops[(size_t)i];
            traffic += op_traffic(P, g);
            launches += g.type == G_DIAG ? g.count : 1;
        }
        int r = QS_OK;
        const bool zeros = finite && (s->untouched & ~qmask) != 0;
        auto one_by_one = [&]() {
            for (size_t k = 0; !r && k < pass.size(); ++k) r = launch_op(s, P, P.ops[(size_t)pass[k]]);
            return r;
        };
        if (launches == 1 || (traffic <= 1.0 && s->amp_bytes() >= (64ull << 20))) {
            if (one_by_one()) return r;
            continue;
        }
        bool done = false;
        if ((int)pass.size() < RunSmall<T>::NOP - 1) {
            plan_pass<RunSmall<T>, T>(P, qmask, pass, &small, &rest);
            done = rest.empty();
            small.zeros = zeros;
            if (done) r = launch<T>(s, small);
        }
        if (!done) {
            plan_pass<RunLarge<T>, T>(P, qmask, pass, &large, &rest);
            if (rest.size() == pass.size()) {        // none fits a parameter block: planned again, none would
                if (one_by_one()) return r;
                continue;
            }
            if (!rest.empty()) P.give_back(rest);
            large.zeros = zeros;
            r = launch<T>(s, large);
        }
        for (int i : pass) s->untouched &= ~P.ops[(size_t)i].tgt;
        if (r) return r;
    }
    return QS_OK;
}

}  // namespace

// Apply a lowered gate list with staged passes (states of kMinTile qubits and
// more); asynchronous on the state's stream.
int qs_stage_apply(qs_state *s, const std::vector<qs_prim> &prims)
{
    return s->dtype == QS_C64 ? apply_t<float>(s, prims) : apply_t<double>(s, prims);
}

int qs_stage_min_qubits() { return kMinTile; }
