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
//  - 1-qubit gates that follow each other on a qubit are multiplied in FP64
//    where the product keeps their form, or three or more follow;
//  - a real or RX-like 1-qubit matrix is taken as p * [[1, r], [q, +-1]] with
//    its largest row entry p pulled out: 4 multiply-adds per amplitude pair
//    instead of 16; the p's of a pass are collected (in extended precision, on the
//    host) and applied once, when the tile is stored;
//  - controlled phases that share a qubit (a QFT's CR ladder) become one
//    diagonal factor per amplitude, a product of per-qubit phases;
//  - a SWAP of two tile qubits renames tile bits and costs nothing;
//  - gates that commute (no shared qubit, or diagonal on every shared one)
//    may be taken out of order when that fills a pass or a stage.
//
// Shared memory is padded, and additive: tile bit b weighs slot_weight(b)
// slots, 2^b for the bits of one 128-byte row and, row digit by row digit, a
// number that is 2^(b mod LB) modulo the row (LB = log2 of the amplitudes per
// 128-byte row: 4 for complex64, 3 for complex128).  An amplitude's slot is
// then the sum of a thread's part and a register's part, the second the same
// for all threads: no instruction per access goes into addresses (an XOR
// swizzle took one, on the pipe that was full).  Lanes whose LB first bits
// differ modulo LB hit distinct banks; a stage orders its lane bits so,
// which fails only when the registers take all of a residue class (3 or 4
// tile bits), and then costs a second wavefront.
#pragma once

#include <cmath>
#include <complex>
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
// Narrower states stay on k_lowstage (48 gates of 8 qubits: 54 us there, 42
// here; of 6 and 7 qubits 47 and 49 on both).
constexpr int kMinTile = 8;
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
    K_EX = 53,       // dense 2x2 on (r | bit ja, r | bit jb), ja < jb, where creg is set: 53 + pair index
    K_XC = 60,       // exchange x and y of register bit j where register bit c is set: 60 + 4 c + j
    K_LADH = 76      // ladder on the registers with bit j set, then x + y, x - y on the pairs of bit j
};

template <typename T>
struct Op {
    uint8_t kind;
    uint8_t creg;                // register-index bits that must be set
    uint16_t cthr;               // tile-index bits (thread bits of the stage) that must be set
    uint16_t cond;               // need or cthr is not empty
    uint16_t ladder;             // K_LAD*: index of its tables
    uint64_t need;               // state-index bits outside the tile that must be set
    T m[8];                      // dense: 2x2 row-major complex; pivot kinds: r, q; phase: one complex;
                                 // ladder: one complex per register bit
};

struct Stage {
    uint16_t first, count;                 // its ops
    uint16_t pr[4];                        // slot weight of register bit j
    uint32_t tb[kMaxThreadBits];           // thread bit j: tile offset | slot weight << 16
};

// One ladder: the phases w of its entries multiply where the entry's bit is
// set.  Entries [first, first + nthr): thread bits (where = thread bit index);
// the next nout: qubits outside the tile (where = qubit) and terms on the hub
// alone (where < 0).  Entries on register bits are in the op.
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
    int32_t zeros;                         // tiles of zeros are likely: they stay as they are
    uint64_t seg_mask[kMaxSeg];            // the tile index's bits, segment by segment ...
    // state offsets, in units of 2^LOW amplitudes, of the load's and the store's
    // thread bits from LOW up (the first LOW are qubits 0..LOW-1) and register bits
    uint32_t gin_t[kMaxThreadBits], gin_r[4];
    uint32_t gout_t[kMaxThreadBits], gout_r[4];
    uint8_t seg_shift[kMaxSeg + 3];        // ... shifted left by this
    Stage st[NST_];
    Ladder lad[NLAD_];
    Entry ent[NENT_];
    Op<T> op[NOP_];
};
template <typename T> using RunSmall = Run<T, 40, 12, 2, 24>;
template <typename T> using RunLarge = Run<T, 208, 56, 16, 256>;
static_assert(sizeof(RunLarge<double>) <= 32764, "kernel parameters are at most 32764 bytes");
static_assert(RunLarge<double>::NENT > 64, "a ladder has a term per qubit and one on its hub alone: any one fits");

// ------------------------------------------------------------------ index maps
// the weight of tile bit b in shared-memory slots: digit d of base 2^LB
// strides 1, 17, 273 (complex64) or 1, 9, 73, 585 (complex128), each past the
// largest sum of the digits below it
template <typename T>
constexpr uint32_t slot_weight(int b)
{
    constexpr uint32_t stride4[3] = {1, 17, 273}, stride3[4] = {1, 9, 73, 585};
    return (Traits<T>::LB == 4 ? stride4[b / 4] : stride3[b / 3]) << (b % Traits<T>::LB);
}

// slots of a K-bit tile
template <typename T>
constexpr uint32_t tile_slots(int K)
{
    uint32_t n = 1;
    for (int b = 0; b < K; ++b) n += slot_weight<T>(b);
    return n;
}

// log2 of a CTA's warps (narrow tiles: part of one)
template <typename T>
QS_HD int warp_bits(int K)
{
    return K - Traits<T>::RB > 5 ? K - Traits<T>::RB - 5 : 0;
}

template <typename R>
QS_HD uint64_t tile_base(const R &P, uint64_t tl)
{
    uint64_t b = 0;
    for (int j = 0; j < P.nseg; ++j) b |= (tl & P.seg_mask[j]) << P.seg_shift[j];
    return b;
}

template <int RB>
QS_HD uint32_t reg_sum(int r, const uint32_t (&b)[4])
{
    uint32_t o = 0;
    for (int j = 0; j < RB; ++j) o += (r >> j & 1) ? b[j] : 0u;
    return o;
}

// ------------------------------------------------------------------ arithmetic on one thread's registers
template <typename T, int RB>
struct Regs {
    T r[1 << RB], i[1 << RB];
};

QS_HD float f_ma(float a, float b, float c) { return fmaf(a, b, c); }
QS_HD double f_ma(double a, double b, double c) { return fma(a, b, c); }

// The updates of an amplitude pair, x and y on one component or on both.  On
// the device each is one asm statement that reads its values and writes them
// back in place, so that every case of apply_op leaves all registers where it
// found them: as plain expressions the compiler kept the cases' results apart
// and copied every amplitude after each op, about 100 moves an op (12 RY
// gates, 28 qubits complex64: 1.64 ms, with the statements 1.33 ms).
#ifdef __CUDA_ARCH__
#define QS_UPD_T(NAME, T, C, S, BODY)                                                                              \
    __device__ __forceinline__ void NAME(T &x, T &y, T r, T q)                                                     \
    {                                                                                                              \
        asm volatile("{\n\t.reg ." S " t, u;\n\t" BODY(S) "mov." S " %0, t;\n\t}" : "+" C(x), "+" C(y) : C(r), C(q)); \
    }
#define QS_UPD(NAME, BODY, HOST) QS_UPD_T(NAME, float, "f", "f32", BODY) QS_UPD_T(NAME, double, "d", "f64", BODY)
#else
#define QS_UPD(NAME, BODY, HOST) \
    template <typename T> inline void NAME(T &x, T &y, T r, T q) { const T x0 = x, y0 = y; HOST; }
#endif
#define QS_B_AP(t) "fma.rn." t " t, %2, %1, %0;\n\tfma.rn." t " %1, %3, %0, %1;\n\t"
#define QS_B_AM(t) "fma.rn." t " t, %2, %1, %0;\n\tneg." t " u, %1;\n\tfma.rn." t " %1, %3, %0, u;\n\t"
#define QS_B_BP(t) "fma.rn." t " t, %2, %0, %1;\n\tfma.rn." t " %1, %3, %1, %0;\n\t"
#define QS_B_BM(t) "fma.rn." t " t, %2, %0, %1;\n\tneg." t " u, %0;\n\tfma.rn." t " %1, %3, %1, u;\n\t"
#define QS_B_BN(t) "neg." t " u, %1;\n\tfma.rn." t " t, %2, %0, u;\n\tfma.rn." t " %1, %3, %1, %0;\n\t"
#define QS_B_SWAP(t) "mov." t " t, %1;\n\tmov." t " %1, %0;\n\t"
QS_UPD(upd_ap, QS_B_AP, (x = f_ma(r, y0, x0), y = f_ma(q, x0, y0)))
QS_UPD(upd_am, QS_B_AM, (x = f_ma(r, y0, x0), y = f_ma(q, x0, -y0)))
QS_UPD(upd_bp, QS_B_BP, (x = f_ma(r, x0, y0), y = f_ma(q, y0, x0)))
QS_UPD(upd_bm, QS_B_BM, (x = f_ma(r, x0, y0), y = f_ma(q, y0, -x0)))
QS_UPD(upd_bn, QS_B_BN, (x = f_ma(r, x0, -y0), y = f_ma(q, y0, x0)))
QS_UPD(upd_swap4, QS_B_SWAP, (x = y0, y = x0, (void)r, (void)q))

template <typename T>
QS_HD void upd_swap(T &x, T &y) { upd_swap4(x, y, (T)0, (T)0); }

#ifdef __CUDA_ARCH__
#define QS_DENSE(T, C, t)                                                                                         \
    __device__ __forceinline__ void dense2(T &xr, T &xi, T &yr, T &yi, const T *m)                                \
    {                                                                                                             \
        asm volatile("{\n\t.reg ." t " a, b, c, d, n;\n\t"                                                        \
                     "mul.rn." t " a, %4, %0;\n\tmul.rn." t " b, %4, %1;\n\t"                                     \
                     "mul.rn." t " c, %8, %0;\n\tmul.rn." t " d, %8, %1;\n\t"                                     \
                     "fma.rn." t " b, %5, %0, b;\n\tfma.rn." t " d, %9, %0, d;\n\t"                               \
                     "neg." t " n, %1;\n\tfma.rn." t " a, %5, n, a;\n\tfma.rn." t " c, %9, n, c;\n\t"             \
                     "fma.rn." t " a, %6, %2, a;\n\tfma.rn." t " b, %6, %3, b;\n\t"                               \
                     "fma.rn." t " c, %10, %2, c;\n\tfma.rn." t " d, %10, %3, d;\n\t"                             \
                     "fma.rn." t " b, %7, %2, b;\n\tfma.rn." t " d, %11, %2, d;\n\t"                              \
                     "neg." t " n, %3;\n\tfma.rn." t " a, %7, n, a;\n\tfma.rn." t " c, %11, n, c;\n\t"            \
                     "mov." t " %0, a;\n\tmov." t " %1, b;\n\tmov." t " %2, c;\n\tmov." t " %3, d;\n\t}"          \
                     : "+" C(xr), "+" C(xi), "+" C(yr), "+" C(yi)                                                 \
                     : C(m[0]), C(m[1]), C(m[2]), C(m[3]), C(m[4]), C(m[5]), C(m[6]), C(m[7]));                   \
    }
QS_DENSE(float, "f", "f32")
QS_DENSE(double, "d", "f64")
#else
template <typename T>
inline void dense2(T &ar, T &ai, T &br, T &bi, const T *m)
{
    const T xr = ar, xi = ai, yr = br, yi = bi;
    ar = f_ma(m[3], -yi, f_ma(m[2], yr, f_ma(m[1], -xi, m[0] * xr)));
    ai = f_ma(m[3], yr, f_ma(m[2], yi, f_ma(m[1], xr, m[0] * xi)));
    br = f_ma(m[7], -yi, f_ma(m[6], yr, f_ma(m[5], -xi, m[4] * xr)));
    bi = f_ma(m[7], yr, f_ma(m[6], yi, f_ma(m[5], xr, m[4] * xi)));
}
#endif

// (x + iy) *= r + iq.  Without a move, and in FP32 with the closing steps packed:
// with the packed half of RX (pair_ia, pair_ib) 30-qubit depth-16 circuit 115.4
// -> 113.0 ms, 28-qubit QFT 5.39 -> 5.29 ms, 27-qubit complex128 QFT 4.57 -> 4.53
// ms, same bits.
#ifdef __CUDA_ARCH__
__device__ __forceinline__ void cmul(double &x, double &y, double r, double q)
{
    asm volatile("{\n\t.reg .f64 t, u;\n\tmul.rn.f64 t, %1, %3;\n\tmul.rn.f64 u, %0, %3;\n\tneg.f64 t, t;\n\t"
                 "fma.rn.f64 %0, %0, %2, t;\n\tfma.rn.f64 %1, %1, %2, u;\n\t}"
                 : "+d"(x), "+d"(y) : "d"(r), "d"(q));
}
__device__ __forceinline__ void cmul(float &x, float &y, float r, float q)
{
    asm volatile("{\n\t.reg .f32 t, u;\n\t.reg .b64 v, f, a;\n\tneg.f32 t, %3;\n\tmul.rn.f32 t, %1, t;\n\t"
                 "mul.rn.f32 u, %0, %3;\n\tmov.b64 a, {t, u};\n\tmov.b64 v, {%0, %1};\n\tmov.b64 f, {%2, %2};\n\t"
                 "fma.rn.f32x2 v, v, f, a;\n\tmov.b64 {%0, %1}, v;\n\t}"
                 : "+f"(x), "+f"(y) : "f"(r), "f"(q));
}
#else
template <typename T>
inline void cmul(T &x, T &y, T r, T q)
{
    const T x0 = x, y0 = y;
    x = f_ma(x0, r, -(y0 * q));
    y = f_ma(y0, r, x0 * q);
}
#endif

// The same on both components of a pair of amplitudes.  In FP32 the device has
// both in one packed multiply-add: the FMA pipe takes as long as for two (3.9
// against 4.3 clocks per pair and scheduler), but half the instructions are
// issued, and issue is what bounds the kernel (30-qubit depth-16 circuit 131.6
// -> 129.5 ms, 28-qubit QFT 5.48 -> 5.42 ms, same bits).
#define QS_PAIR(NAME, UPD)                                                     \
    template <typename T>                                                      \
    QS_HD void NAME(T &xr, T &xi, T &yr, T &yi, T r, T q)                      \
    {                                                                          \
        UPD(xr, yr, r, q);                                                     \
        UPD(xi, yi, r, q);                                                     \
    }
QS_PAIR(pair_ap, upd_ap)
QS_PAIR(pair_am, upd_am)
QS_PAIR(pair_bp, upd_bp)
QS_PAIR(pair_bm, upd_bm)
template <typename T>
QS_HD void pair_ia(T &xr, T &xi, T &yr, T &yi, T r, T q)
{
    upd_ap(xr, yi, -r, q);
    upd_ap(xi, yr, r, -q);
}
template <typename T>
QS_HD void pair_ib(T &xr, T &xi, T &yr, T &yi, T r, T q)
{
    upd_bn(xr, yi, r, q);
    upd_bm(xi, yr, r, q);
}
#ifdef __CUDA_ARCH__
#define QS_PAIR2(NAME, BODY)                                                                                      \
    __device__ __forceinline__ void NAME(float &xr, float &xi, float &yr, float &yi, float r, float q)            \
    {                                                                                                             \
        asm volatile("{\n\t.reg .b64 x, y, r, q, t;\n\t.reg .f32 a, b;\n\t"                                     \
                     "mov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\t"                                          \
                     "mov.b64 r, {%4, %4};\n\tmov.b64 q, {%5, %5};\n\t" BODY                                     \
                     "mov.b64 {%0, %1}, t;\n\tmov.b64 {%2, %3}, y;\n\t}"                                         \
                     : "+f"(xr), "+f"(xi), "+f"(yr), "+f"(yi) : "f"(r), "f"(q));                                  \
    }
QS_PAIR2(pair_ap, "fma.rn.f32x2 t, r, y, x;\n\tfma.rn.f32x2 y, q, x, y;\n\t")
QS_PAIR2(pair_bp, "fma.rn.f32x2 t, r, x, y;\n\tfma.rn.f32x2 y, q, y, x;\n\t")
QS_PAIR2(pair_am, "fma.rn.f32x2 t, r, y, x;\n\tneg.f32 a, %2;\n\tneg.f32 b, %3;\n\tmov.b64 y, {a, b};\n\t"
                  "fma.rn.f32x2 y, q, x, y;\n\t")
QS_PAIR2(pair_bm, "fma.rn.f32x2 t, r, x, y;\n\tneg.f32 a, %0;\n\tneg.f32 b, %1;\n\tmov.b64 x, {a, b};\n\t"
                  "fma.rn.f32x2 y, q, y, x;\n\t")
// RX: the components of y are one packed step on x's, exchanged before x changes
#define QS_PAIR2I(NAME, BODY)                                                                                     \
    __device__ __forceinline__ void NAME(float &xr, float &xi, float &yr, float &yi, float r, float q)            \
    {                                                                                                             \
        asm volatile("{\n\t.reg .b64 y, q, t;\n\t.reg .f32 n;\n\tmov.b64 y, {%2, %3};\n\t" BODY                   \
                     "mov.b64 {%2, %3}, y;\n\t}"                                                                  \
                     : "+f"(xr), "+f"(xi), "+f"(yr), "+f"(yi) : "f"(r), "f"(q));                                  \
    }
QS_PAIR2I(pair_ia, "mov.b64 t, {%1, %0};\n\tneg.f32 n, %5;\n\tmov.b64 q, {n, %5};\n\tneg.f32 n, %4;\n\t"
                   "fma.rn.f32 %0, n, %3, %0;\n\tfma.rn.f32 %1, %4, %2, %1;\n\tfma.rn.f32x2 y, q, t, y;\n\t")
QS_PAIR2I(pair_ib, "neg.f32 n, %1;\n\tmov.b64 t, {n, %0};\n\tmov.b64 q, {%5, %5};\n\tneg.f32 n, %3;\n\t"
                   "fma.rn.f32 %0, %4, %0, n;\n\tfma.rn.f32 %1, %4, %1, %2;\n\tfma.rn.f32x2 y, q, y, t;\n\t")
#endif

template <typename T, int RB, int J, int KIND>
QS_HD void op_pair(Regs<T, RB> &v, const T *m, uint32_t creg)
{
    if constexpr (J < RB) {
        const T r = m[0], q = m[1];
QS_UNROLL
        for (int a = 0; a < (1 << RB); ++a) {
            if (a >> J & 1) continue;
            const int b = a | 1 << J;
            T &xr = v.r[a], &xi = v.i[a], &yr = v.r[b], &yi = v.i[b];
            if constexpr (KIND == K_RAP) {
                pair_ap(xr, xi, yr, yi, r, q);
            } else if constexpr (KIND == K_RAM) {
                pair_am(xr, xi, yr, yi, r, q);
            } else if constexpr (KIND == K_RBP) {
                pair_bp(xr, xi, yr, yi, r, q);
            } else if constexpr (KIND == K_RBM) {
                pair_bm(xr, xi, yr, yi, r, q);
            } else if constexpr (KIND == K_IA) {
                pair_ia(xr, xi, yr, yi, r, q);
            } else if constexpr (KIND == K_IB) {
                pair_ib(xr, xi, yr, yi, r, q);
            } else if constexpr (KIND == K_GEN) {
                dense2(xr, xi, yr, yi, m);
            } else if constexpr (KIND == K_GENR) {
                if ((a & creg) == creg) dense2(xr, xi, yr, yi, m);
            } else if constexpr (KIND == K_X) {
                upd_swap(xr, yr); upd_swap(xi, yi);
            } else if constexpr (KIND == K_XR) {
                if ((a & creg) == creg) { upd_swap(xr, yr); upd_swap(xi, yi); }
            } else if constexpr (KIND >= K_XC) {
                if (a >> ((KIND - K_XC) / 4) & 1) { upd_swap(xr, yr); upd_swap(xi, yi); }
            } else {                                        // K_PH
                cmul(yr, yi, m[0], m[1]);
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
// RB: every bit of creg) times f and the phases of its set register bits but
// the hub, depth first: two factors live per level
template <typename T, int RB, int HUB, int LEVEL, int IDX>
QS_HD void ladder_walk(Regs<T, RB> &v, T fr, T fi, const T *m, uint32_t creg)
{
    if constexpr (LEVEL < 0) {
        if (HUB == RB && (IDX & creg) != creg) return;
        cmul(v.r[IDX], v.i[IDX], fr, fi);
    } else if constexpr (LEVEL == HUB) {
        ladder_walk<T, RB, HUB, LEVEL - 1, (IDX | 1 << LEVEL)>(v, fr, fi, m, creg);
    } else {
        ladder_walk<T, RB, HUB, LEVEL - 1, IDX>(v, fr, fi, m, creg);
        T gr = fr, gi = fi;
        cmul(gr, gi, m[2 * LEVEL], m[2 * LEVEL + 1]);
        ladder_walk<T, RB, HUB, LEVEL - 1, (IDX | 1 << LEVEL)>(v, gr, gi, m, creg);
    }
}

// x, y := x + f y, x - f y (y as 2 x - x'): a ladder and the H behind it in 6
// multiply-adds per pair instead of 8 and two walks over the registers.
#ifdef __CUDA_ARCH__
#define QS_BFLY(T, C, t)                                                                                          \
    __device__ __forceinline__ void butterfly(T &xr, T &xi, T &yr, T &yi, T fr, T fi)                             \
    {                                                                                                             \
        const T two = 2;                                                                                          \
        asm volatile("{\n\t.reg ." t " a, b, n;\n\tneg." t " n, %3;\n\t"                                    \
                     "fma.rn." t " a, %4, %2, %0;\n\tfma.rn." t " b, %4, %3, %1;\n\t"                         \
                     "fma.rn." t " a, %5, n, a;\n\tfma.rn." t " b, %5, %2, b;\n\t"                            \
                     "neg." t " n, a;\n\tfma.rn." t " %2, %6, %0, n;\n\t"                                     \
                     "neg." t " n, b;\n\tfma.rn." t " %3, %6, %1, n;\n\t"                                     \
                     "mov." t " %0, a;\n\tmov." t " %1, b;\n\t}"                                              \
                     : "+" C(xr), "+" C(xi), "+" C(yr), "+" C(yi) : C(fr), C(fi), C(two));                        \
    }
QS_BFLY(float, "f", "f32")
QS_BFLY(double, "d", "f64")
#else
template <typename T>
inline void butterfly(T &xr, T &xi, T &yr, T &yi, T fr, T fi)
{
    const T a = f_ma(fi, -yi, f_ma(fr, yr, xr)), b = f_ma(fi, yr, f_ma(fr, yi, xi));
    yr = f_ma((T)2, xr, -a);
    yi = f_ma((T)2, xi, -b);
    xr = a;
    xi = b;
}
#endif

template <typename T, int RB, int HUB, int LEVEL, int IDX>
QS_HD void ladder_h_walk(Regs<T, RB> &v, T fr, T fi, const T *m)
{
    if constexpr (LEVEL < 0) {
        constexpr int Y = IDX | 1 << HUB;
        butterfly(v.r[IDX], v.i[IDX], v.r[Y], v.i[Y], fr, fi);
    } else if constexpr (LEVEL == HUB) {
        ladder_h_walk<T, RB, HUB, LEVEL - 1, IDX>(v, fr, fi, m);
    } else {
        ladder_h_walk<T, RB, HUB, LEVEL - 1, IDX>(v, fr, fi, m);
        const T pr = m[2 * LEVEL], pi = m[2 * LEVEL + 1];
        const T gr = f_ma(fr, pr, -(fi * pi)), gi = f_ma(fi, pr, fr * pi);
        ladder_h_walk<T, RB, HUB, LEVEL - 1, (IDX | 1 << LEVEL)>(v, gr, gi, m);
    }
}

// One op on a thread's registers (its need and cthr hold).  factor(ladder,
// fr, fi) gives a ladder's factor for this thread.
template <typename T, int RB, typename F>
QS_HD void apply_op(Regs<T, RB> &v, const Op<T> &op, const F &factor)
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
#define QS_STG_LAD(KIND, HUB)                                                     \
    case KIND:                                                                    \
        if constexpr (HUB < RB || KIND == K_LADR) {                               \
            T fr, fi;                                                             \
            factor(op.ladder, fr, fi);                                            \
            ladder_walk<T, RB, HUB, RB - 1, 0>(v, fr, fi, m, creg);               \
        }                                                                         \
        break;
    QS_STG_LAD(K_LADR, RB)
    QS_STG_LAD(K_LAD + 0, 0)
    QS_STG_LAD(K_LAD + 1, 1)
    QS_STG_LAD(K_LAD + 2, 2)
    QS_STG_LAD(K_LAD + 3, 3)
    QS_STG_LAD(K_LAD0, -2)
#undef QS_STG_LAD
#define QS_STG_LADH(HUB)                                                          \
    case K_LADH + HUB:                                                            \
        if constexpr (HUB < RB) {                                                 \
            T fr, fi;                                                             \
            factor(op.ladder, fr, fi);                                            \
            ladder_h_walk<T, RB, HUB, RB - 1, 0>(v, fr, fi, m);                   \
        }                                                                         \
        break;
    QS_STG_LADH(0)
    QS_STG_LADH(1)
    QS_STG_LADH(2)
    QS_STG_LADH(3)
#undef QS_STG_LADH
#define QS_STG_XC(C)                                                              \
    QS_STG_XCJ(C, 0) QS_STG_XCJ(C, 1) QS_STG_XCJ(C, 2) QS_STG_XCJ(C, 3)
#define QS_STG_XCJ(C, J)                                                          \
    case K_XC + 4 * C + J:                                                        \
        if constexpr (C < RB && C != J) op_pair<T, RB, J, K_XC + 4 * C>(v, m, creg); \
        break;
    QS_STG_XC(0) QS_STG_XC(1) QS_STG_XC(2) QS_STG_XC(3)
#undef QS_STG_XCJ
#undef QS_STG_XC
    case K_EX + 0: op_exchange<T, RB, 0, 1>(v, m, creg); break;
    case K_EX + 1: op_exchange<T, RB, 0, 2>(v, m, creg); break;
    case K_EX + 2: op_exchange<T, RB, 1, 2>(v, m, creg); break;
    case K_EX + 3: op_exchange<T, RB, 0, 3>(v, m, creg); break;
    case K_EX + 4: op_exchange<T, RB, 1, 3>(v, m, creg); break;
    case K_EX + 5: op_exchange<T, RB, 2, 3>(v, m, creg); break;
    default: __builtin_unreachable();      // no range check before the jump table
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
        if (P.ent[e].where < 0 || (base >> P.ent[e].where & 1)) cmul(fr, fi, P.ent[e].re, P.ent[e].im);
}

// ------------------------------------------------------------------ planner (qs_stage_plan.cpp)
// One operation of the simplified gate list.
enum GType : uint8_t { G_NONE, G_U, G_CU, G_EX, G_SWAP, G_DIAG };
struct GOp {
    uint8_t type;
    uint64_t tgt;                // qubits it mixes: they must be tile qubits
    uint64_t diag;               // qubits it is diagonal on (controls, phase masks)
    uint64_t ctrl;               // G_CU, G_EX: controls; G_DIAG: the hub (bits every term shares)
    uint64_t off0, off1;         // G_EX: the exchanged qubits
    double m[8];                 // G_U, G_CU, G_EX: 2x2; G_DIAG: m[0] + i m[1] a factor of every amplitude
    long double det;             // G_U: |det| of its gates, before their product was rounded
    int first, count;            // G_DIAG: its terms [first, first + count) in Planner::terms
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
    struct Masks {
        uint64_t tgt, diag;
        int op;
    };
    int n, dtype, K, low;
    std::vector<GOp> ops;
    std::vector<Term> terms;
    // The ops not yet in a pass, in order: left[front..].  A pass looks at a
    // window of them, takes what it can and moves what it has passed over up to
    // where it stopped, so that planning is linear in the list's length
    // (complex64 layers of 10 qubits: 0.34 us a gate at 600 gates, 0.4 at
    // 60,000, where copies of the rest of the list made it 7.3; 720 gates of 30
    // qubits 0.47 ms, 0.62 with the copies).
    std::vector<Masks> left;
    size_t front = 0;
    // What the factors of the passes so far lost when they were rounded: the next
    // pass with a factor owes it.  lost: the same with the pass that plan_pass made
    // last, which runs when next() is called again.
    std::complex<long double> owed = 1, lost = 1;
private:
    int count(uint64_t q) const;
    void take(uint64_t q, std::vector<uint64_t> *wants, std::vector<int> *taken);
    std::vector<Masks> behind;
};
// What a pass looks at and takes at most.  Layers of random gates come to the
// same passes and stages without these bounds (8 to 30 qubits, up to 60,000
// gates): a scan ends where every qubit is held by an op that stays behind, well
// within the window, which bounds lists that leave a qubit idle for long; and a
// pass's parameter block holds half of what the pass is handed.
constexpr size_t kWindow = 2048, kPassOps = 2 * RunLarge<float>::NOP;

// A list that ends in SWAPs of disjoint qubits (a QFT's reversal) ends in one
// exchange of amplitudes in place, whatever the number of pairs (k_permute,
// qs_stage.cu), where staged passes rename at most the qubits of a tile each.
// A tile holds the lowest qubits, their partners and more pairs (or unpaired
// qubits); with the tile's amplitudes at one setting of the other qubits go
// those at the setting that the other pairs exchange it with.
struct Permute {
    int32_t K, nseg, npairs, pad;
    uint64_t seg_mask[kMaxSeg];            // the tile index's bits (see Run)
    uint64_t pair_a[16], pair_b[16];       // qubits outside the tile that trade places (2^q)
    uint32_t g_t[kMaxThreadBits], g_r[4];  // state offsets of thread bits from LOW up and of register bits (see Run)
    uint32_t w_t[kMaxThreadBits];          // slot weights of thread bits: written ...
    uint32_t r_t[kMaxThreadBits];          // ... and read, at the partner's tile bit
    uint32_t w_r[4], r_r[4];               // the same of register bits
    uint8_t seg_shift[kMaxSeg + 3];
};

// The setting of the qubits outside the tile that base trades with.
QS_HD uint64_t permute_partner(const Permute &P, uint64_t base)
{
    for (int j = 0; j < P.npairs; ++j) {
        const bool a = (base & P.pair_a[j]) != 0, b = (base & P.pair_b[j]) != 0;
        if (a != b) base ^= P.pair_a[j] | P.pair_b[j];
    }
    return base;
}

// True, and P, when the ops still left are SWAPs of disjoint pairs that staged
// passes would take more than one pass for.
template <typename T>
bool plan_permute(const Planner &plan, Permute *P);

// The stages of a pass (a RunSmall or RunLarge): fills R from pass_ops on the
// tile of qmask; ops that do not fit R come back in *rest, in order.
template <typename R, typename T>
void plan_pass(Planner &P, uint64_t qmask, const std::vector<int> &pass_ops, R *out, std::vector<int> *rest);

}  // namespace qs_stg
