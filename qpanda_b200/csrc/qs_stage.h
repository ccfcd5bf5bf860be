// qs_stage.h - staged passes: the plan and the per-thread arithmetic.
//
// A staged pass applies many gates in one read and one write of the state
// (k_stage, qs_stage.cu).  A tile is the 2^K amplitudes that agree on every
// qubit outside a set Q of K qubits; a CTA loads a tile straight into
// registers, 2^RB amplitudes per thread, and stores it straight from
// registers.  Which RB tile bits index a thread's registers is a *stage*:
// within a stage every gate whose targets are register bits runs on registers
// alone; between two stages the tile goes through shared memory once.  Gates
// need only their targets in the tile: controls and phase masks may lie on
// any qubits (a tile-uniform test on the tile's base, a per-thread test on
// the thread's tile bits, or a choice of registers).
//
// What the planner (qs_stage_plan.cpp) does to the gate list, all of it exact
// algebra on the gates:
//  - 1-qubit gates that follow each other on a qubit are multiplied in FP64;
//  - a real or RX-like 1-qubit matrix is taken as p * [[1, r], [q, +-1]] with
//    its largest row entry p pulled out: 4 multiply-adds per amplitude pair
//    instead of 16; the p's of a pass are collected (FP64, on the host) and
//    applied once, when the tile is stored;
//  - controlled phases that share a qubit (a QFT's CR ladder) become one
//    diagonal factor per amplitude, a product of per-qubit phases;
//  - a SWAP of two tile qubits renames tile bits and costs nothing;
//  - gates that commute (no shared qubit, or diagonal on every shared one)
//    may be taken out of order when that fills a pass or a stage.
//
// Shared memory is XOR-swizzled by a linear map: tile bit b >= LB adds the
// LB-bit vector kVec[b] to the slot's low LB bits (LB = log2 of the
// amplitudes per 128-byte row: 4 for complex64, 3 for complex128).  Any 4
// register bits leave thread bits whose LB-bit images span all LB dimensions
// (the images of the K <= 13 bits are distinct nonzero vectors for LB = 4,
// each used at most twice for LB = 3: a code of distance > 4), and each stage
// orders its lane bits so that the first LB are independent: every access
// phase hits distinct banks.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "qs_prim.h"

#ifdef __CUDACC__
#define QS_HD __host__ __device__ __forceinline__
#define QS_UNROLL _Pragma("unroll")
#else
#define QS_HD inline
#define QS_UNROLL
#endif

namespace qs_stg {

constexpr int kMaxTile = 12;         // tile qubits
constexpr int kMinTile = 9;          // narrower states stay on k_lowstage
constexpr int kMaxThreadBits = 9;
constexpr int kMaxSeg = kMaxTile + 1;

template <typename T> struct Traits;
// RB: register bits (2^RB amplitudes per thread); LB: amplitudes per 128-byte
// row; LOW: the qubits 0..LOW-1 that every tile holds and whose tile bits are
// the lowest lane bits of the load and the store: 128-byte runs
template <> struct Traits<float> { static constexpr int RB = 4, LB = 4, LOW = 4; };
template <> struct Traits<double> { static constexpr int RB = 3, LB = 3, LOW = 3; };

// op kinds.  (x, y): the amplitudes of a pair, register bit j clear and set;
// a kind's value is its base + j.
enum Kind : uint8_t {
    K_RAP = 0,       // x + r y,        y + q x           real matrices, diagonal pivot
    K_RAM = 4,       // x + r y,        q x - y
    K_RBP = 8,       // r x + y,        x + q y           off-diagonal pivot
    K_RBM = 12,      // r x + y,        q y - x
    K_IA = 16,       // x + i r y,      y + i q x         RX: real diagonal, imaginary off it
    K_IB = 20,       // r x + i y,      q y + i x
    K_GEN = 24,      // dense 2x2
    K_GENR = 28,     // dense 2x2 where the register bits creg are set
    K_X = 32,        // exchange x and y
    K_XR = 36,       // the same where the register bits creg are set
    K_PH = 40,       // y *= m
    K_PH0 = 44,      // every register *= m
    K_PHR = 45,      // the registers with every bit of creg *= m
    K_SCALE = 46,    // every register *= m[0] (real)
    K_LADR = 47,     // ladder on the registers with every bit of creg
    K_LAD = 48,      // ladder on the registers with bit j set
    K_LAD0 = 52,     // ladder on every register
    K_EX = 53        // dense 2x2 on (r | bit ja, r | bit jb), ja < jb, where creg is set: 53 + pair index
};

template <typename T>
struct Op {
    uint8_t kind;
    uint8_t creg;                // register-index bits that must be set
    uint16_t cthr;               // tile-index bits (thread bits of the stage) that must be set
    uint32_t ladder;             // K_LAD*: index of its tables
    uint64_t need;               // state-index bits outside the tile that must be set
    T m[8];                      // dense: 2x2 row-major complex; pivot kinds: r, q; phase: one complex;
                                 // ladder: one complex per register bit
};

struct Stage {
    uint16_t first, count;                 // its ops
    uint16_t pr[4];                        // slot offset of register bit j
    uint32_t tb[kMaxThreadBits];           // thread bit j: tile offset | slot offset << 16
};

// One ladder: the phases w of its entries multiply where the entry's bit is
// set.  Entries [first, first + nthr): thread bits (where = thread bit index);
// the next nout: qubits outside the tile (where = qubit).  Entries on
// register bits are in the op.
struct Ladder {
    uint16_t first, nthr, nout, pad;
};
struct Entry {
    double re, im;
    int32_t where, pad;
};

// What a launch needs, passed by value.  Two sizes: a pass of a few gates
// should not pay for copying the largest parameter block.
template <typename T, int NOP_, int NST_, int NLAD_, int NENT_>
struct Run {
    static constexpr int NOP = NOP_, NST = NST_, NLAD = NLAD_, NENT = NENT_;
    int32_t K, nstages, nladders, nseg;
    T scale[2];                            // applied at the store
    int32_t scale_kind;                    // 0: none, 1: real, 2: complex
    int32_t pad;
    uint64_t seg_mask[kMaxSeg];            // the tile index's bits, segment by segment ...
    uint64_t gin_t[kMaxThreadBits], gin_r[4];      // state offsets of the load's thread and register bits
    uint64_t gout_t[kMaxThreadBits], gout_r[4];    // ... and of the store's
    uint8_t seg_shift[kMaxSeg + 3];        // ... shifted left by this
    Stage st[NST_];
    Ladder lad[NLAD_];
    Entry ent[NENT_];
    Op<T> op[NOP_];
};
template <typename T> using RunSmall = Run<T, 40, 12, 2, 24>;
template <typename T> using RunLarge = Run<T, 208, 56, 16, 256>;
static_assert(sizeof(RunLarge<double>) <= 32764, "kernel parameters are at most 32764 bytes");

// ------------------------------------------------------------------ index maps
template <typename T>
constexpr uint32_t bit_image(int b)
{
    // the vectors of tile bits >= LB (bits below LB: their own)
    constexpr uint8_t v4[12] = {3, 5, 6, 9, 10, 12, 7, 11, 13, 14, 15, 15};
    constexpr uint8_t v3[12] = {3, 5, 6, 7, 1, 2, 4, 3, 5, 6, 7, 7};
    return b < Traits<T>::LB ? 1u << b : Traits<T>::LB == 4 ? v4[b - 4] : v3[b - 3];
}

// the shared-memory slot of tile index 2^b
template <typename T>
constexpr uint32_t bit_slot(int b)
{
    return b < Traits<T>::LB ? 1u << b : (1u << b) | bit_image<T>(b);
}

template <typename R>
QS_HD uint64_t tile_base(const R &P, uint64_t tl)
{
    uint64_t b = 0;
    for (int j = 0; j < P.nseg; ++j) b |= (tl & P.seg_mask[j]) << P.seg_shift[j];
    return b;
}

template <int RB>
QS_HD uint32_t reg_xor(int r, const uint32_t (&b)[4])
{
    uint32_t o = 0;
    for (int j = 0; j < RB; ++j) o ^= (r >> j & 1) ? b[j] : 0u;
    return o;
}

// ------------------------------------------------------------------ arithmetic on one thread's registers
template <typename T, int RB>
struct Regs {
    T r[1 << RB], i[1 << RB];
};

QS_HD float f_ma(float a, float b, float c) { return fmaf(a, b, c); }
QS_HD double f_ma(double a, double b, double c) { return fma(a, b, c); }

template <typename T>
QS_HD void cmul(T &xr, T &xi, T pr, T pi)
{
    const T x = xr, y = xi;
    xr = f_ma(x, pr, -(y * pi));
    xi = f_ma(x, pi, y * pr);
}

template <typename T>
QS_HD void dense2(T &ar, T &ai, T &br, T &bi, const T *m)
{
    const T xr = ar, xi = ai, yr = br, yi = bi;
    ar = f_ma(-m[3], yi, f_ma(m[2], yr, f_ma(-m[1], xi, m[0] * xr)));
    ai = f_ma(m[3], yr, f_ma(m[2], yi, f_ma(m[1], xr, m[0] * xi)));
    br = f_ma(-m[7], yi, f_ma(m[6], yr, f_ma(-m[5], xi, m[4] * xr)));
    bi = f_ma(m[7], yr, f_ma(m[6], yi, f_ma(m[5], xr, m[4] * xi)));
}

template <typename T, int RB, int J, int KIND>
QS_HD void op_pair(Regs<T, RB> &v, const T *m, uint32_t creg)
{
    if constexpr (J < RB) {
        const T r = m[0], q = m[1];
QS_UNROLL
        for (int a = 0; a < (1 << RB); ++a) {
            if (a >> J & 1) continue;
            const int b = a | 1 << J;
            T xr = v.r[a], xi = v.i[a], yr = v.r[b], yi = v.i[b];
            if constexpr (KIND == K_RAP) {
                v.r[a] = f_ma(r, yr, xr); v.i[a] = f_ma(r, yi, xi);
                v.r[b] = f_ma(q, xr, yr); v.i[b] = f_ma(q, xi, yi);
            } else if constexpr (KIND == K_RAM) {
                v.r[a] = f_ma(r, yr, xr); v.i[a] = f_ma(r, yi, xi);
                v.r[b] = f_ma(q, xr, -yr); v.i[b] = f_ma(q, xi, -yi);
            } else if constexpr (KIND == K_RBP) {
                v.r[a] = f_ma(r, xr, yr); v.i[a] = f_ma(r, xi, yi);
                v.r[b] = f_ma(q, yr, xr); v.i[b] = f_ma(q, yi, xi);
            } else if constexpr (KIND == K_RBM) {
                v.r[a] = f_ma(r, xr, yr); v.i[a] = f_ma(r, xi, yi);
                v.r[b] = f_ma(q, yr, -xr); v.i[b] = f_ma(q, yi, -xi);
            } else if constexpr (KIND == K_IA) {
                v.r[a] = f_ma(-r, yi, xr); v.i[a] = f_ma(r, yr, xi);
                v.r[b] = f_ma(-q, xi, yr); v.i[b] = f_ma(q, xr, yi);
            } else if constexpr (KIND == K_IB) {
                v.r[a] = f_ma(r, xr, -yi); v.i[a] = f_ma(r, xi, yr);
                v.r[b] = f_ma(q, yr, -xi); v.i[b] = f_ma(q, yi, xr);
            } else if constexpr (KIND == K_GEN) {
                dense2(v.r[a], v.i[a], v.r[b], v.i[b], m);
            } else if constexpr (KIND == K_GENR) {
                if ((a & creg) == creg) dense2(v.r[a], v.i[a], v.r[b], v.i[b], m);
            } else if constexpr (KIND == K_X) {
                v.r[a] = yr; v.i[a] = yi;
                v.r[b] = xr; v.i[b] = xi;
            } else if constexpr (KIND == K_XR) {
                const bool on = (a & creg) == creg;
                v.r[a] = on ? yr : xr; v.i[a] = on ? yi : xi;
                v.r[b] = on ? xr : yr; v.i[b] = on ? xi : yi;
            } else {                                        // K_PH
                cmul(v.r[b], v.i[b], m[0], m[1]);
            }
        }
    }
}

template <typename T, int RB, int JA, int JB>
QS_HD void op_exchange(Regs<T, RB> &v, const T *m, uint32_t creg)
{
    if constexpr (JB < RB) {
QS_UNROLL
        for (int a = 0; a < (1 << RB); ++a) {
            if ((a >> JA & 1) || (a >> JB & 1)) continue;
            if ((a & creg) != creg) continue;
            dense2(v.r[a | 1 << JA], v.i[a | 1 << JA], v.r[a | 1 << JB], v.i[a | 1 << JB], m);
        }
    }
}

// every register whose index has bit HUB (HUB < 0: every register; HUB ==
// RB: every bit of creg) times f and the phases of its set register bits,
// depth first: two factors live per level
template <typename T, int RB, int HUB, int LEVEL, int IDX>
QS_HD void ladder_walk(Regs<T, RB> &v, T fr, T fi, const T *m, uint32_t creg)
{
    if constexpr (LEVEL < 0) {
        if (HUB == RB && (IDX & creg) != creg) return;
        cmul(v.r[IDX], v.i[IDX], fr, fi);
    } else if constexpr (LEVEL == HUB) {
        // the hub's own phase (a term on the hub alone) is its register entry
        T gr = fr, gi = fi;
        cmul(gr, gi, m[2 * LEVEL], m[2 * LEVEL + 1]);
        ladder_walk<T, RB, HUB, LEVEL - 1, (IDX | 1 << LEVEL)>(v, gr, gi, m, creg);
    } else {
        ladder_walk<T, RB, HUB, LEVEL - 1, IDX>(v, fr, fi, m, creg);
        T gr = fr, gi = fi;
        cmul(gr, gi, m[2 * LEVEL], m[2 * LEVEL + 1]);
        ladder_walk<T, RB, HUB, LEVEL - 1, (IDX | 1 << LEVEL)>(v, gr, gi, m, creg);
    }
}

// One op on a thread's registers (its need and cthr hold).  fr + i fi: a
// ladder's factor for this thread.
template <typename T, int RB>
QS_HD void apply_op(Regs<T, RB> &v, const Op<T> &op, T fr, T fi)
{
    const T *m = op.m;
    const uint32_t creg = op.creg;
    switch (op.kind) {
#define QS_STG_J(KIND)                                             \
    case KIND + 0: op_pair<T, RB, 0, KIND>(v, m, creg); break;     \
    case KIND + 1: op_pair<T, RB, 1, KIND>(v, m, creg); break;     \
    case KIND + 2: op_pair<T, RB, 2, KIND>(v, m, creg); break;     \
    case KIND + 3: op_pair<T, RB, 3, KIND>(v, m, creg); break;
    QS_STG_J(K_RAP)
    QS_STG_J(K_RAM)
    QS_STG_J(K_RBP)
    QS_STG_J(K_RBM)
    QS_STG_J(K_IA)
    QS_STG_J(K_IB)
    QS_STG_J(K_GEN)
    QS_STG_J(K_GENR)
    QS_STG_J(K_X)
    QS_STG_J(K_XR)
    QS_STG_J(K_PH)
#undef QS_STG_J
    case K_PH0:
QS_UNROLL
        for (int a = 0; a < (1 << RB); ++a) cmul(v.r[a], v.i[a], m[0], m[1]);
        break;
    case K_PHR:
QS_UNROLL
        for (int a = 0; a < (1 << RB); ++a)
            if ((a & creg) == creg) cmul(v.r[a], v.i[a], m[0], m[1]);
        break;
    case K_SCALE:
QS_UNROLL
        for (int a = 0; a < (1 << RB); ++a) { v.r[a] *= m[0]; v.i[a] *= m[0]; }
        break;
    case K_LADR: ladder_walk<T, RB, RB, RB - 1, 0>(v, fr, fi, m, creg); break;
    case K_LAD + 0: ladder_walk<T, RB, 0, RB - 1, 0>(v, fr, fi, m, creg); break;
    case K_LAD + 1: ladder_walk<T, RB, 1, RB - 1, 0>(v, fr, fi, m, creg); break;
    case K_LAD + 2: ladder_walk<T, RB, 2, RB - 1, 0>(v, fr, fi, m, creg); break;
    case K_LAD + 3:
        if constexpr (RB > 3) ladder_walk<T, RB, 3, RB - 1, 0>(v, fr, fi, m, creg);
        break;
    case K_LAD0: ladder_walk<T, RB, -2, RB - 1, 0>(v, fr, fi, m, creg); break;
    case K_EX + 0: op_exchange<T, RB, 0, 1>(v, m, creg); break;
    case K_EX + 1: op_exchange<T, RB, 0, 2>(v, m, creg); break;
    case K_EX + 2: op_exchange<T, RB, 1, 2>(v, m, creg); break;
    case K_EX + 3: op_exchange<T, RB, 0, 3>(v, m, creg); break;
    case K_EX + 4: op_exchange<T, RB, 1, 3>(v, m, creg); break;
    case K_EX + 5: op_exchange<T, RB, 2, 3>(v, m, creg); break;
    default: break;
    }
}

// A ladder's factors, in FP64: of a lane (thread bits 0..4), and of a warp of
// a tile (the other thread bits and the qubits outside the tile).
template <typename R>
QS_HD void ladder_lane(const R &P, int l, uint32_t lane, double &fr, double &fi)
{
    fr = 1; fi = 0;
    const Ladder L = P.lad[l];
    for (int e = L.first; e < L.first + L.nthr; ++e)
        if (P.ent[e].where < 5 && (lane >> P.ent[e].where & 1)) cmul(fr, fi, P.ent[e].re, P.ent[e].im);
}

template <typename R>
QS_HD void ladder_warp(const R &P, int l, uint32_t warp, uint64_t base, double &fr, double &fi)
{
    fr = 1; fi = 0;
    const Ladder L = P.lad[l];
    for (int e = L.first; e < L.first + L.nthr; ++e)
        if (P.ent[e].where >= 5 && (warp >> (P.ent[e].where - 5) & 1)) cmul(fr, fi, P.ent[e].re, P.ent[e].im);
    for (int e = L.first + L.nthr; e < L.first + L.nthr + L.nout; ++e)
        if (base >> P.ent[e].where & 1) cmul(fr, fi, P.ent[e].re, P.ent[e].im);
}

// ------------------------------------------------------------------ planner (qs_stage_plan.cpp)
// One operation of the simplified gate list.
enum GType : uint8_t { G_U, G_CU, G_EX, G_SWAP, G_DIAG };
struct GOp {
    uint8_t type;
    uint64_t tgt;                // qubits it mixes: they must be tile qubits
    uint64_t diag;               // qubits it is diagonal on (controls, phase masks)
    uint64_t ctrl;               // G_CU, G_EX: controls; G_DIAG: the hub (bits every term shares)
    uint64_t off0, off1;         // G_EX: the exchanged qubits
    double m[8];                 // G_U, G_CU, G_EX: 2x2; G_DIAG: m[0] + i m[1] a factor of every amplitude
    int first, count;            // G_DIAG: its terms [first, first + count) in Planner::terms
    int prim, nprims;            // the gates it stands for, when they are nprims = 1: prims[prim]
};
struct Term {
    int q;                       // the phase applies where the hub and this qubit are set (-1: the hub alone)
    double re, im;
};

// The passes of a gate list on an n-qubit state, one at a time, so that the
// device works on a pass while the host plans the next.
struct Planner {
    Planner(const std::vector<qs_prim> &prims, int n, int dtype);
    // The next pass: its tile qubits and the ops that run in it (indices into
    // ops, in an order that respects the gate list).  False when none are left.
    bool next(uint64_t *qmask, std::vector<int> *pass_ops);
    // ops that a pass could not take after all (its parameter block was full)
    void give_back(const std::vector<int> &rest);
    int n, dtype, K, low;
    std::vector<GOp> ops;
    std::vector<Term> terms;
    std::vector<int> left;       // ops not yet in a pass, in order
private:
    int scan(uint64_t q, std::vector<uint64_t> *wants, std::vector<int> *taken) const;
};

// The stages of a pass (a RunSmall or RunLarge): fills R from pass_ops on the
// tile of qmask; ops that do not fit R come back in *rest, in order.
template <typename R, typename T>
void plan_pass(const Planner &P, uint64_t qmask, const std::vector<int> &pass_ops, R *out, std::vector<int> *rest);

}  // namespace qs_stg
