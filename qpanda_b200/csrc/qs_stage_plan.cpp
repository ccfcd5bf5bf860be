// qs_stage_plan.cpp - planner of the staged passes (qs_stage.h): gate list ->
// simplified ops -> passes -> stages.  Host-only.
#include <algorithm>
#include <complex>

#include "qs_stage.h"

namespace qs_stg {

namespace {

typedef std::complex<double> cd;
typedef std::complex<long double> cl;

// a * b without std::complex's look at infinities
inline cl mul(const cl &a, const cl &b)
{
    return cl(a.real() * b.real() - a.imag() * b.imag(), a.real() * b.imag() + a.imag() * b.real());
}

inline int popc(uint64_t x) { return __builtin_popcountll(x); }
inline int low_bit(uint64_t x) { return __builtin_ctzll(x); }

bool is_x(const double m[8])
{
    return m[0] == 0 && m[1] == 0 && m[2] == 1 && m[3] == 0 && m[4] == 1 && m[5] == 0 && m[6] == 0 && m[7] == 0;
}

bool is_diag(const double m[8]) { return m[2] == 0 && m[3] == 0 && m[4] == 0 && m[5] == 0; }

// diagonal, real, real diagonal with imaginary rest (RX), or none of these
int form(const double m[8])
{
    if (is_diag(m)) return 0;
    if (m[1] == 0 && m[3] == 0 && m[5] == 0 && m[7] == 0) return 1;
    if (m[1] == 0 && m[7] == 0 && m[2] == 0 && m[4] == 0) return 2;
    return 3;
}

// |det| of a 2x2 row-major complex matrix: how it scales the norm, squared
template <typename T>
long double abs_det(const T m[8])
{
    const long double re = (long double)m[0] * m[6] - (long double)m[1] * m[7] - (long double)m[2] * m[4] + (long double)m[3] * m[5];
    const long double im = (long double)m[0] * m[7] + (long double)m[1] * m[6] - (long double)m[2] * m[5] - (long double)m[3] * m[4];
    return im == 0 ? std::fabs(re) : std::sqrt(re * re + im * im);
}

// a := b * a, 2x2 row-major complex
void mul2(double a[8], const double b[8])
{
    const cd a00(a[0], a[1]), a01(a[2], a[3]), a10(a[4], a[5]), a11(a[6], a[7]);
    const cd b00(b[0], b[1]), b01(b[2], b[3]), b10(b[4], b[5]), b11(b[6], b[7]);
    const cd c[4] = {b00 * a00 + b01 * a10, b00 * a01 + b01 * a11, b10 * a00 + b11 * a10, b10 * a01 + b11 * a11};
    for (int k = 0; k < 4; ++k) {
        a[2 * k] = c[k].real();
        a[2 * k + 1] = c[k].imag();
    }
}

}  // namespace

// ------------------------------------------------------------------ the simplified gate list
Planner::Planner(const std::vector<qs_prim> &prims, int n_, int dtype_) : n(n_), dtype(dtype_)
{
    K = n < kMaxTile ? n : kMaxTile;
    low = dtype == QS_C64 ? Traits<float>::LOW : Traits<double>::LOW;
    ops.reserve(prims.size());
    // the 1-qubit ops at the end of a qubit's list: the last one and, when
    // nothing else lies between, the one before it
    int open[64], before[64];
    for (int q = 0; q < 64; ++q) open[q] = before[q] = -1;
    // Gates on several qubits that touch a qubit close its last op, except
    // where that op commutes with them: a diagonal op with controls and
    // phases, an X-type op (a I + b X: RX) with the target of an X.  Only gates
    // of the same type may then still join it (in layers of random rotations
    // and CNOTs every ninth does).
    uint64_t diag_only = 0, x_only = 0;
    auto x_type = [](const double m[8]) { return m[0] == m[6] && m[1] == m[7] && m[2] == m[4] && m[3] == m[5]; };
    auto close = [&](uint64_t qs, uint64_t z, uint64_t x) {      // z, x: the qubits of qs it acts on like Z, like X
        for (; qs; qs &= qs - 1) {
            const int q = low_bit(qs), o = open[q];
            before[q] = -1;
            if (o < 0) continue;
            const uint64_t b = 1ull << q;
            if ((z & b) && is_diag(ops[o].m) && !(x_only & b)) diag_only |= b;
            else if ((x & b) && x_type(ops[o].m) && !(diag_only & b)) x_only |= b;
            else open[q] = -1;
        }
    };
    int last_diag = -1;                    // the phase op that another phase may join ...
    uint64_t since = 0;                    // ... and the qubits mixed after it
    for (size_t i = 0; i < prims.size(); ++i) {
        const qs_prim &p = prims[i];
        if (p.kind == QS_PRIM_PAIR && p.off0 == 0 && p.cmask == 0) {
            // Gates of one form multiply into one op.  Two of different forms
            // stay two ops: their product would be dense, 20 instructions per
            // pair against 6 + 5 for a rotation and a phase; three become one.
            const int q = low_bit(p.off1);
            if (((diag_only >> q & 1) && !is_diag(p.m)) || ((x_only >> q & 1) && !x_type(p.m))) open[q] = -1;
            const int o = open[q];
            if (o >= 0 && (form(ops[o].m) == form(p.m) || form(ops[o].m) == 3)) {
                mul2(ops[o].m, p.m);
                ops[o].det *= abs_det(p.m);
                continue;
            }
            if (o >= 0 && before[q] >= 0) {
                GOp &g = ops[before[q]];
                mul2(g.m, ops[o].m);
                mul2(g.m, p.m);
                g.det *= ops[o].det * abs_det(p.m);
                ops[o].type = G_NONE;
                open[q] = before[q];
                before[q] = -1;
                continue;
            }
            GOp g = {};
            g.type = G_U;
            g.tgt = p.off1;
            memcpy(g.m, p.m, sizeof(g.m));
            g.det = abs_det(p.m);
            before[q] = (diag_only | x_only) >> q & 1 ? -1 : o;
            open[q] = (int)ops.size();
            diag_only &= ~g.tgt;
            x_only &= ~g.tgt;
            since |= g.tgt;
            ops.push_back(g);
            continue;
        }
        close(p.holes, p.kind == QS_PRIM_PHASE ? p.holes : p.cmask, p.off0 == 0 && is_x(p.m) ? p.off1 : 0);
        if (p.kind == QS_PRIM_PHASE) {
            if (last_diag >= 0 && !(since & p.holes)) {
                // join the last phase op when every term then has at most one
                // qubit beside a common hub; phases on one qubit are one term, so
                // that a ladder has at most one per qubit and fits a parameter block
                // however many phases share its hub
                GOp &d = ops[last_diag];
                const uint64_t hub = d.ctrl & p.holes;
                const uint64_t mine = p.holes & ~hub, first = d.ctrl & ~hub;
                if (hub && popc(mine) <= 1 && (first == 0 || (d.count == 1 && popc(first) == 1)) &&
                    d.first + d.count == (int)terms.size()) {
                    if (first) terms[d.first].q = low_bit(first);
                    d.ctrl = hub;
                    d.diag |= p.holes;
                    const int q = mine ? low_bit(mine) : -1;
                    auto t = std::find_if(terms.begin() + d.first, terms.end(), [&](const Term &x) { return x.q == q; });
                    if (t == terms.end()) {
                        terms.push_back({q, p.m[0], p.m[1]});
                        ++d.count;
                    } else {
                        const cd w = cd(t->re, t->im) * cd(p.m[0], p.m[1]);
                        t->re = w.real();
                        t->im = w.imag();
                    }
                    continue;
                }
            }
            GOp g = {};
            g.type = G_DIAG;
            g.diag = g.ctrl = p.holes;
            g.m[0] = 1;
            g.first = (int)terms.size();
            g.count = 1;
            terms.push_back({-1, p.m[0], p.m[1]});
            last_diag = (int)ops.size();
            since = 0;
            ops.push_back(g);
            continue;
        }
        GOp g = {};
        memcpy(g.m, p.m, sizeof(g.m));
        g.ctrl = g.diag = p.cmask;
        if (p.off0 == 0) {
            g.type = G_CU;
            g.tgt = p.off1;
        } else {
            g.type = p.cmask == 0 && is_x(p.m) ? G_SWAP : G_EX;
            g.tgt = p.off0 | p.off1;
            g.off0 = p.off0;
            g.off1 = p.off1;
        }
        since |= g.tgt;
        ops.push_back(g);
    }
    // diagonal 1-qubit ops mix nothing: a factor m00 of everything (m00 on the
    // controls' subspace) and a phase m11 / m00 where the qubit is set
    for (GOp &g : ops) {
        if ((g.type != G_U && g.type != G_CU) || !is_diag(g.m)) continue;
        const cd m00(g.m[0], g.m[1]), w = cd(g.m[6], g.m[7]) / m00;
        g.first = (int)terms.size();
        g.count = 0;
        if (g.type == G_CU && !(m00 == cd(1, 0))) {
            terms.push_back({-1, m00.real(), m00.imag()});
            ++g.count;
        }
        terms.push_back({low_bit(g.tgt), w.real(), w.imag()});
        ++g.count;
        g.diag |= g.tgt;
        g.off1 = g.tgt;
        g.tgt = 0;
        g.type = G_DIAG;
    }
    // a ladder runs where its hub is mixed next (as one op with an H): it counts
    // as a gate on the hub, or it would run as soon as its qubits are ready, on
    // tiles and threads that half of the time have the hub clear
    uint64_t mixed = 0;                    // qubits that a 1-qubit op mixes next
    for (size_t i = ops.size(); i-- > 0;) {
        GOp &g = ops[i];
        if (g.type == G_NONE) continue;
        const bool ladder = g.type == G_DIAG && g.count > 1 && popc(g.ctrl) == 1;
        if (ladder && (g.ctrl & mixed)) g.tgt = g.ctrl;
        if (g.type == G_U) mixed |= g.tgt;
        else if (!ladder) mixed &= ~(g.tgt | g.diag);
    }
    left.reserve(ops.size());
    for (size_t i = 0; i < ops.size(); ++i)
        if (ops[i].type != G_NONE) left.push_back({ops[i].tgt, ops[i].diag, (int)i});
}

// The ops left that can run in a pass on the tile of q: their targets in q, and
// they commute with every earlier op that stays behind.  A scan looks at kWindow
// ops at most, and no further than where nothing can run.  count() returns how
// many there are; take() moves them into *taken (up to kPassOps), and *wants, if
// asked for, gets the target sets that alone keep an op out.
int Planner::count(uint64_t q) const
{
    const uint64_t all = n >= 64 ? ~0ull : (1ull << n) - 1;
    uint64_t skip_all = 0, skip_tgt = 0;
    int found = 0;
    const Masks *g = left.data() + front, *const end = g + std::min(left.size() - front, kWindow);
    for (; g < end; ++g) {
        if (!(g->tgt & (skip_all | ~q)) && !(g->diag & skip_tgt)) {
            ++found;
            continue;
        }
        skip_all |= g->tgt | g->diag;
        skip_tgt |= g->tgt;
        if ((skip_all & all) == all) break;
    }
    return found;
}

void Planner::take(uint64_t q, std::vector<uint64_t> *wants, std::vector<int> *taken)
{
    const uint64_t all = n >= 64 ? ~0ull : (1ull << n) - 1;
    uint64_t skip_all = 0, skip_tgt = 0;
    behind.clear();
    Masks *const from = left.data() + front, *const end = from + std::min(left.size() - front, kWindow);
    Masks *p = from;
    for (; p < end && (skip_all & all) != all && taken->size() < kPassOps; ++p) {
        const Masks g = *p;
        const bool free = !(g.tgt & skip_all) && !(g.diag & skip_tgt);
        if (free && !(g.tgt & ~q)) {
            taken->push_back(g.op);
            continue;
        }
        if (free && wants) {
            const uint64_t w = g.tgt & ~q;
            if (popc(q | w) <= K && std::find(wants->begin(), wants->end(), w) == wants->end()) wants->push_back(w);
        }
        skip_all |= g.tgt | g.diag;
        skip_tgt |= g.tgt;
        behind.push_back(g);
    }
    // what was passed over moves up to where the scan stopped
    std::copy(behind.begin(), behind.end(), p - behind.size());
    front += (size_t)(p - from) - behind.size();
}

bool Planner::next(uint64_t *qmask, std::vector<int> *pass_ops)
{
    pass_ops->clear();
    owed = lost;
    if (front == left.size()) return false;
    uint64_t q = n <= K ? (1ull << n) - 1 : (1ull << low) - 1;
    std::vector<uint64_t> wants;
    double last[64];                               // a qubit's gain when it was last looked at
    for (double &g : last) g = 1e9;
    while (true) {
        // what runs on a tile runs on every larger one, so a round looks at what
        // stays behind only
        wants.clear();
        take(q, popc(q) < K ? &wants : nullptr, pass_ops);
        if (popc(q) >= K) break;
        // grow the tile by the target set that lets the most ops per qubit in;
        // gains change little from round to round, so sets are looked at by
        // their last gain, and not those whose last gain is below half the best
        auto guess = [&](uint64_t w) { return popc(w) == 1 ? last[low_bit(w)] : 1e8; };
        std::stable_sort(wants.begin(), wants.end(), [&](uint64_t x, uint64_t y) { return guess(x) > guess(y); });
        uint64_t best = 0;
        double best_gain = -1;
        for (uint64_t w : wants) {
            if (guess(w) < best_gain * 0.5) break;
            const double gain = (double)count(q | w) / popc(w);
            if (popc(w) == 1) last[low_bit(w)] = gain;
            if (gain > best_gain) {
                best_gain = gain;
                best = w;
            }
        }
        if (best) {
            q |= best;
            continue;
        }
        for (int b = 0; b < n && popc(q) < K; ++b) q |= 1ull << b;
    }
    if (n > K) std::sort(pass_ops->begin(), pass_ops->end());      // more than one round
    *qmask = q;
    return true;
}

void Planner::give_back(const std::vector<int> &rest)
{
    if (rest.empty()) return;
    // into the places that they and the pass's ops left free, in order
    size_t end = front;
    while (end < left.size() && left[end].op < rest.back()) ++end;
    behind.assign(left.begin() + (long)front, left.begin() + (long)end);
    front -= rest.size();
    auto b = behind.begin();
    auto out = left.begin() + (long)front;
    for (int i : rest) {
        while (b != behind.end() && b->op < i) *out++ = *b++;
        *out++ = {ops[(size_t)i].tgt, ops[(size_t)i].diag, i};
    }
    std::copy(b, behind.end(), out);
}

namespace {

// The bits of a tile index in the qubits outside the tile, run by run; returns
// the number of runs.
int tile_segments(uint64_t qmask, int n, uint64_t *mask, uint8_t *shift)
{
    int nseg = 0;
    for (int q = 0, from = 0; q < n;) {
        if (qmask >> q & 1) { ++q; continue; }
        int len = 0;
        while (q + len < n && !(qmask >> (q + len) & 1)) ++len;
        mask[nseg] = ((1ull << len) - 1) << from;
        shift[nseg] = (uint8_t)(q - from);
        ++nseg;
        from += len;
        q += len;
    }
    return nseg;
}

}  // namespace

// ------------------------------------------------------------------ the closing exchange
template <typename T>
bool plan_permute(const Planner &plan, Permute *P)
{
    constexpr int RB = Traits<T>::RB, LOW = Traits<T>::LOW;
    constexpr int K = RB + 8;                          // 256 threads (128 when no bit is left without its partner)
    const int n = plan.n;
    const size_t left = plan.left.size() - plan.front;
    if (n < K || left < 2 || left > 16 + K / 2) return false;
    int partner[64];
    for (int q = 0; q < n; ++q) partner[q] = q;
    uint64_t all = 0;
    for (size_t i = plan.front; i < plan.left.size(); ++i) {
        const GOp &g = plan.ops[(size_t)plan.left[i].op];
        if (g.type != G_SWAP || (all & g.tgt)) return false;
        all |= g.tgt;
        const int a = low_bit(g.tgt), b = 63 - __builtin_clzll(g.tgt);
        partner[a] = b;
        partner[b] = a;
    }
    const uint64_t low = (1ull << LOW) - 1;
    if (popc(all | low) <= plan.K) return false;       // one staged pass
    // the tile: the lowest qubits and their partners, then pairs and unpaired
    // qubits from the lowest up (rows of the state stay together)
    uint64_t q = low;
    for (int b = 0; b < LOW; ++b) q |= 1ull << partner[b];
    for (int b = 0; b < n && popc(q) < K; ++b) {
        const uint64_t add = (1ull << b | 1ull << partner[b]) & ~q;
        if (popc(q | add) <= K) q |= add;
    }
    if (popc(q) < K - 1) return false;
    memset(P, 0, sizeof(*P));
    P->K = popc(q);
    P->nseg = tile_segments(q, n, P->seg_mask, P->seg_shift);
    for (int a = 0; a < n; ++a)
        if (partner[a] > a && !(q >> a & 1)) {
            if (P->npairs == 16) return false;
            P->pair_a[P->npairs] = 1ull << a;
            P->pair_b[P->npairs++] = 1ull << partner[a];
        }
    int pos[64], k = 0;
    for (int b = 0; b < n; ++b)
        if (q >> b & 1) pos[b] = k++;
    for (int b = 0; b < n; ++b) {
        if (!(q >> b & 1)) continue;
        const int at = pos[b];
        const bool thread = at < P->K - RB;
        const int j = thread ? at : at - (P->K - RB);
        (thread ? P->w_t : P->w_r)[j] = slot_weight<T>(at);
        (thread ? P->r_t : P->r_r)[j] = slot_weight<T>(pos[partner[b]]);
        if (at >= LOW) (thread ? P->g_t : P->g_r)[j] = 1u << (b - LOW);
    }
    return true;
}

template bool plan_permute<float>(const Planner &, Permute *);
template bool plan_permute<double>(const Planner &, Permute *);

// ------------------------------------------------------------------ stages of a pass
namespace {

// p * [[.., ..], [.., ..]] with the pivot p pulled out: the kind (base + 0),
// r, q and the factor that is left.  Kinds of dense ops keep the matrix.  What is
// rounded to T turns the gate by that rounding; p makes up for what it does to
// the norm: the determinant is that of the gates in the list.
template <typename T>
uint8_t classify(const GOp &g, T *out, long double *p)
{
    const double *m = g.m;
    *p = 1;
    for (int k = 0; k < 8; ++k) out[k] = (T)m[k];
    if (is_x(m)) return K_X;
    const double tol = 9e-16;            // 4 ulp: products of a few rotations
    double r = 0, q = 0, piv = 1;
    uint8_t kind = K_GEN;
    if (m[1] == 0 && m[3] == 0 && m[5] == 0 && m[7] == 0) {
        if (std::fabs(m[0]) >= std::fabs(m[2])) {
            piv = m[0]; r = m[2] / piv; q = m[4] / piv;
            if (std::fabs(m[6] / piv - 1) < tol) kind = K_RAP;
            else if (std::fabs(m[6] / piv + 1) < tol) kind = K_RAM;
        } else {
            piv = m[2]; r = m[0] / piv; q = m[6] / piv;
            if (std::fabs(m[4] / piv - 1) < tol) kind = K_RBP;
            else if (std::fabs(m[4] / piv + 1) < tol) kind = K_RBM;
        }
    } else if (m[1] == 0 && m[7] == 0 && m[2] == 0 && m[4] == 0) {
        if (std::fabs(m[0]) >= std::fabs(m[3])) {
            piv = m[0]; r = m[3] / piv; q = m[5] / piv;
            if (std::fabs(m[6] / piv - 1) < tol) kind = K_IA;
        } else {
            piv = m[3]; r = m[0] / piv; q = m[6] / piv;
            if (std::fabs(m[5] / piv - 1) < tol) kind = K_IB;
        }
    }
    long double det;                     // of what runs
    if (kind == K_GEN) {
        piv = 1;
        det = abs_det(out);
    } else {
        out[0] = (T)r;
        out[1] = (T)q;
        const long double rq = (long double)out[0] * out[1];
        det = std::fabs(kind == K_RAP || kind == K_RBP ? 1 - rq : 1 + rq);
    }
    // sqrt(g.det / det), the gates being unitary up to rounding
    *p = piv + piv * (g.det - (long double)piv * piv * det) / 2;
    return kind;
}

int pair_index(int ja, int jb) { return jb * (jb - 1) / 2 + ja; }

}  // namespace

template <typename R, typename T>
void plan_pass(Planner &P, uint64_t qmask, const std::vector<int> &pass_ops, R *out, std::vector<int> *rest)
{
    constexpr int RB = Traits<T>::RB, LB = Traits<T>::LB, LOW = Traits<T>::LOW;
    const int K = popc(qmask), n = P.n, tbits = K - RB;
    R &S = *out;
    S.K = K;
    S.nstages = S.nladders = 0;
    S.zeros = 0;
    memset(S.gin_t, 0, sizeof(S.gin_t));
    memset(S.gin_r, 0, sizeof(S.gin_r));
    memset(S.gout_t, 0, sizeof(S.gout_t));
    memset(S.gout_r, 0, sizeof(S.gout_r));
    rest->clear();
    // tile bit of a qubit, and the qubit of a tile bit at the load
    int pos[64], qubit[kMaxTile];
    {
        int k = 0;
        for (int q = 0; q < n; ++q) {
            pos[q] = -1;
            if (qmask >> q & 1) {
                qubit[k] = q;
                pos[q] = k++;
            }
        }
    }
    S.nseg = tile_segments(qmask, n, S.seg_mask, S.seg_shift);
    auto tile_bits = [&](uint64_t qs, const int *ps) {
        uint32_t o = 0;
        for (qs &= qmask; qs; qs &= qs - 1) o |= 1u << ps[low_bit(qs)];
        return o;
    };
    // The pass's ops with their qubits as tile bits at the load: which ops may
    // pass which does not depend on where a SWAP has put a qubit since.
    struct Todo {
        uint32_t tgt, diag;
        int op;
        bool swap;
    };
    int home[64];
    memcpy(home, pos, sizeof(home));
    std::vector<Todo> todo;
    std::vector<int> take;
    bool swaps = false;
    todo.reserve(pass_ops.size());
    for (int i : pass_ops) {
        const GOp &g = P.ops[(size_t)i];
        todo.push_back({tile_bits(g.tgt, pos), tile_bits(g.diag, pos), i, g.type == G_SWAP});
        swaps = swaps || g.type == G_SWAP;
    }
    int at[kMaxTile];                              // tile bit of a qubit now, by its tile bit at the load
    for (int b = 0; b < K; ++b) at[b] = b;
    // ops of list that run in a stage with these register bits (tile bits now)
    auto scan = [&](const std::vector<Todo> &list, uint32_t regs, std::vector<uint32_t> *wants,
                    std::vector<int> *taken, std::vector<Todo> *kept) {
        const uint32_t all = (1u << K) - 1;
        uint32_t skip_all = 0, skip_tgt = 0;
        int count = 0, ps[kMaxTile];
        if (swaps) memcpy(ps, at, sizeof(ps));
        for (size_t i = 0; i < list.size(); ++i) {
            const Todo &g = list[i];
            if (!(g.tgt & skip_all) && !(g.diag & skip_tgt)) {
                if (g.swap) {
                    std::swap(ps[low_bit(g.tgt)], ps[31 - __builtin_clz(g.tgt)]);
                    if (taken) taken->push_back(g.op);
                    continue;
                }
                uint32_t t = g.tgt;
                if (swaps) {
                    t = 0;
                    for (uint32_t m = g.tgt; m; m &= m - 1) t |= 1u << ps[low_bit(m)];
                }
                if (!(t & ~regs)) {
                    count += t ? 1 : 0;            // what needs no register bit runs in any stage
                    if (taken) taken->push_back(g.op);
                    continue;
                }
                const uint32_t w = t & ~regs;
                if (wants && popc(regs | w) <= RB && std::find(wants->begin(), wants->end(), w) == wants->end())
                    wants->push_back(w);
            }
            skip_all |= g.tgt | g.diag;
            skip_tgt |= g.tgt;
            if (kept) kept->push_back(g);
            if (skip_all == all) {
                if (kept) kept->insert(kept->end(), list.begin() + (long)i + 1, list.end());
                break;
            }
        }
        return count;
    };
    cl scale(1, 0);
    double growth = 1;
    int nops = 0, nent = 0;
    const uint32_t low_tile = (1u << LOW) - 1, all_tile = (1u << K) - 1;
    std::vector<Todo> rest_of, behind;
    std::vector<uint32_t> wants;
    auto choose = [&](uint32_t allowed) {
        uint32_t regs = 0;
        rest_of = todo;
        while (popc(regs) < RB) {
            wants.clear();
            if (swaps) {
                scan(todo, regs, &wants, nullptr, nullptr);
            } else {                               // as in next(): a round looks at what stays behind only
                behind.clear();
                scan(rest_of, regs, &wants, nullptr, &behind);
                rest_of.swap(behind);
            }
            const int have = swaps ? scan(todo, regs, nullptr, nullptr, nullptr) : 0;
            uint32_t best = 0;
            double best_gain = -1;
            for (uint32_t w : wants) {
                if (w & ~allowed) continue;
                // a tie goes to the lowest bits: left to the last stage with
                // ops, they cost a stage of their own before the store
                const double gain =
                    (double)(scan(swaps ? todo : rest_of, regs | w, nullptr, nullptr, nullptr) - have) / popc(w) +
                    (w & low_tile ? 0.1 : 0);
                if (gain > best_gain) { best_gain = gain; best = w; }
            }
            if (!best) break;
            regs |= best;
        }
        for (int b = K - 1; b >= 0 && popc(regs) < RB; --b)
            if (allowed >> b & 1) regs |= 1u << b;
        return regs;
    };
    // the stage's layout; lanes: the tile bits that must come first, in order
    int thread_of[kMaxTile], reg_of[kMaxTile], reg_at[4], reg_in[4];
    auto add_stage = [&](uint32_t regs, const int *lanes, int nlanes) {
        Stage &st = S.st[S.nstages++];
        memset(&st, 0, sizeof(st));
        st.first = (uint16_t)nops;
        int order[kMaxTile], no = 0;
        uint32_t classes = 0, used = regs;
        auto independent = [&](int b) {                // another residue class of the row's banks
            if (classes >> (b % LB) & 1) return false;
            classes |= 1u << (b % LB);
            return true;
        };
        for (int j = 0; j < nlanes; ++j) {
            order[no++] = lanes[j];
            used |= 1u << lanes[j];
            independent(lanes[j]);
        }
        for (int b = 0; b < K && no < LB; ++b)
            if (!(used >> b & 1) && independent(b)) {
                order[no++] = b;
                used |= 1u << b;
            }
        for (int b = 0; b < K; ++b)
            if (!(used >> b & 1)) order[no++] = b;
        for (int b = 0; b < K; ++b) thread_of[b] = reg_of[b] = -1;
        for (int j = 0; j < tbits; ++j) {
            st.tb[j] = (1u << order[j]) | slot_weight<T>(order[j]) << 16;
            thread_of[order[j]] = j;
        }
        int j = 0;
        for (int b = 0; b < K; ++b)
            if (regs >> b & 1) {
                st.pr[j] = (uint16_t)slot_weight<T>(b);
                reg_at[j] = b;
                reg_of[b] = j++;
            }
        return &st;
    };
    const uint64_t outside = ~qmask;
    // masks of a condition on qubits, by where each lies now
    auto condition = [&](uint64_t qs, Op<T> *op) {
        op->need = qs & outside;
        op->cthr = 0;
        op->creg = 0;
        const uint32_t tb = tile_bits(qs, pos);
        for (int b = 0; b < K; ++b)
            if (tb >> b & 1) {
                if (reg_of[b] >= 0) op->creg |= 1u << reg_of[b];
                else op->cthr |= 1u << b;
            }
        op->cond = op->need || op->cthr;
    };
    auto reg_bit = [&](uint64_t qs) { return reg_of[pos[low_bit(qs)]]; };
    // one op at the current stage; false when it does not fit the parameter block
    auto emit = [&](const GOp &g) {
        if (g.type == G_SWAP) {
            const uint32_t t = tile_bits(g.tgt, home);
            std::swap(at[low_bit(t)], at[31 - __builtin_clz(t)]);
            std::swap(pos[low_bit(g.off0)], pos[low_bit(g.off1)]);
            return true;
        }
        if (nops + 2 > R::NOP) return false;
        Op<T> &op = S.op[nops];
        memset(&op, 0, sizeof(op));
        if (g.type == G_U) {
            long double p;
            const int j = reg_bit(g.tgt);
            const uint8_t kind = classify<T>(g, op.m, &p);
            scale *= p;
            growth /= (double)std::fabs(p);
            // an H right behind the ladder whose hub it mixes: one op
            Op<T> *last = nops > S.st[S.nstages - 1].first ? &S.op[nops - 1] : nullptr;
            if (kind == K_RAM && op.m[0] == 1 && op.m[1] == 1 && last && last->kind == K_LAD + j && !last->cond) {
                last->kind = (uint8_t)(K_LADH + j);
                --nops;                            // counted again below
            } else {
                op.kind = (uint8_t)(kind + j);
            }
        } else if (g.type == G_CU) {
            condition(g.ctrl, &op);
            for (int k = 0; k < 8; ++k) op.m[k] = (T)g.m[k];
            const bool x = is_x(g.m);
            const bool one = op.creg && !(op.creg & (op.creg - 1));
            op.kind = (uint8_t)((x ? (one ? K_XC + 4 * low_bit(op.creg) : op.creg ? K_XR : K_X) : op.creg ? K_GENR : K_GEN) +
                                reg_bit(g.tgt));
        } else if (g.type == G_EX) {
            condition(g.ctrl, &op);
            int ja = reg_bit(g.off0), jb = reg_bit(g.off1);
            for (int k = 0; k < 8; ++k) op.m[k] = (T)(ja < jb ? g.m[k] : g.m[6 - 2 * (k / 2) + (k & 1)]);
            if (ja > jb) std::swap(ja, jb);
            op.kind = (uint8_t)(K_EX + pair_index(ja, jb));
        } else if (g.count == 1) {
            const Term &t = P.terms[(size_t)g.first];
            condition(g.ctrl | (t.q >= 0 ? 1ull << t.q : 0), &op);
            op.m[0] = (T)t.re;
            op.m[1] = (T)t.im;
            op.kind = op.creg == 0 ? K_PH0 : (op.creg & (op.creg - 1)) ? K_PHR : K_PH + low_bit(op.creg);
        } else {
            if (S.nladders == R::NLAD || nent + g.count > R::NENT) return false;
            condition(g.ctrl, &op);
            for (int j = 0; j < RB; ++j) op.m[2 * j] = 1;
            op.ladder = (uint16_t)S.nladders;
            Ladder &L = S.lad[S.nladders++];
            L.first = (uint16_t)nent;
            L.nthr = L.nout = L.pad = 0;
            for (int side = 0; side < 2; ++side)
                for (int k = 0; k < g.count; ++k) {
                    const Term &t = P.terms[(size_t)(g.first + k)];
                    const bool alone = t.q < 0;              // on the hub alone
                    const bool out_q = alone || (outside >> t.q & 1);
                    if (!out_q && reg_of[pos[t.q]] >= 0) {
                        if (side) continue;
                        T *w = &op.m[2 * reg_of[pos[t.q]]];
                        w[0] = (T)t.re;
                        w[1] = (T)t.im;
                    } else if (out_q == (side == 1)) {
                        S.ent[nent++] = {t.re, t.im, alone ? -1 : out_q ? t.q : thread_of[pos[t.q]], 0};
                        ++(out_q ? L.nout : L.nthr);
                    }
                }
            op.kind = op.creg == 0 ? K_LAD0 : (op.creg & (op.creg - 1)) ? K_LADR : K_LAD + low_bit(op.creg);
        }
        if (g.type == G_DIAG && g.ctrl == 0) {
            // m00 and, of what w lost when it was rounded, one half (w has modulus 1):
            // the other half stays where the qubit is set
            const cl m00(g.m[0], g.m[1]), m11(g.m[6], g.m[7]), w(op.m[0], op.m[1]);
            scale = mul(scale, m00 + mul(m11 - mul(m00, w), std::conj(w) * 0.5L));
        }
        ++nops;
        if (growth > 0x1p8) {                     // the pivots' factors so far, before values grow further
            Op<T> &sc = S.op[nops++];
            memset(&sc, 0, sizeof(sc));
            sc.kind = K_SCALE;
            sc.m[0] = (T)std::abs(scale);
            scale /= (long double)sc.m[0];
            growth = 1;
        }
        return true;
    };
    bool full = false, stored = false;
    while (!stored) {
        const bool first = S.nstages == 0;
        const uint32_t regs = choose(first ? all_tile & ~low_tile : all_tile);
        take.clear();
        scan(todo, regs, nullptr, &take, nullptr);
        // the store reads the tile with the lowest qubits on the lowest lanes
        int ps[64], lanes[LOW];
        memcpy(ps, pos, sizeof(ps));
        for (int i : take) {
            const GOp &g = P.ops[(size_t)i];
            if (g.type == G_SWAP) std::swap(ps[low_bit(g.off0)], ps[low_bit(g.off1)]);
        }
        bool last = take.size() == todo.size();
        for (int q = 0; q < LOW; ++q) {
            lanes[q] = ps[q];
            last = last && !(regs >> ps[q] & 1);
        }
        static const int natural[4] = {0, 1, 2, 3};
        // one stage alone has no barrier between its loads and its stores:
        // every thread must then store where it loaded
        if (first && last) last = memcmp(ps, pos, sizeof(int) * (size_t)n) == 0;
        Stage *st = add_stage(regs, first ? natural : lanes, first || last ? LOW : 0);
        if (first) memcpy(reg_in, reg_at, sizeof(reg_in));
        size_t k = 0, t = 0;
        for (; k < take.size(); ++k)
            if (!emit(P.ops[(size_t)take[k]])) {
                full = true;
                break;
            }
        st->count = (uint16_t)(nops - st->first);
        // todo minus what was emitted
        for (size_t i = 0, e = 0; i < todo.size(); ++i) {
            if (e < k && todo[i].op == take[e]) { ++e; continue; }
            todo[t++] = todo[i];
        }
        todo.resize(t);
        if (full || S.nstages + 1 >= R::NST) {
            for (const Todo &o : todo) rest->push_back(o.op);
            todo.clear();
            full = true;
        }
        stored = last && !full;
        if (stored || todo.empty()) {
            if (!stored) {
                for (int q = 0; q < LOW; ++q) lanes[q] = pos[q];
                uint32_t low_now = 0, regs2 = 0;
                for (int q = 0; q < LOW; ++q) low_now |= 1u << lanes[q];
                for (int b = K - 1; b >= 0 && popc(regs2) < RB; --b)
                    if (!(low_now >> b & 1)) regs2 |= 1u << b;
                add_stage(regs2, lanes, LOW)->count = 0;
                stored = true;
            }
        }
    }
    // state offsets of the load (first stage) and the store (last stage)
    int stored_q[kMaxTile];                        // qubit behind a tile bit at the store
    for (int q = 0; q < n; ++q)
        if (pos[q] >= 0) stored_q[pos[q]] = q;
    auto offsets = [&](const Stage &st, const int *regs, const int *qs, uint32_t *gt, uint32_t *gr) {
        for (int j = LOW; j < tbits; ++j) gt[j] = 1u << (qs[low_bit(st.tb[j] & 0xffffu)] - LOW);
        for (int j = 0; j < RB; ++j) gr[j] = 1u << (qs[regs[j]] - LOW);
    };
    offsets(S.st[0], reg_in, qubit, S.gin_t, S.gin_r);
    offsets(S.st[S.nstages - 1], reg_at, stored_q, S.gout_t, S.gout_r);
    S.scale_kind = scale.imag() != 0 ? 2 : scale.real() != 1 ? 1 : 0;
    P.lost = P.owed;
    if (S.scale_kind) {
        // with what the passes before lost when their factors were rounded; a real
        // factor stays one
        const cl f = S.scale_kind == 2 ? P.owed : cl(P.owed.real(), 0);
        scale = mul(scale, f);
        S.scale[0] = (T)scale.real();
        S.scale[1] = (T)scale.imag();
        P.lost = P.owed / f * (scale / cl(S.scale[0], S.scale[1]));
    }
}

template void plan_pass<RunSmall<float>, float>(Planner &, uint64_t, const std::vector<int> &, RunSmall<float> *, std::vector<int> *);
template void plan_pass<RunLarge<float>, float>(Planner &, uint64_t, const std::vector<int> &, RunLarge<float> *, std::vector<int> *);
template void plan_pass<RunSmall<double>, double>(Planner &, uint64_t, const std::vector<int> &, RunSmall<double> *, std::vector<int> *);
template void plan_pass<RunLarge<double>, double>(Planner &, uint64_t, const std::vector<int> &, RunLarge<double> *, std::vector<int> *);

}  // namespace qs_stg
