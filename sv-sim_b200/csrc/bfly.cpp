// Planner of the butterfly engine (bfly.h).
//
// 1. The elementary ops are rewritten where a short form exists: CX D CX on one pair with D
//    diagonal on the target is a phase on the parity of the two qubits, H CX H a controlled
//    Z (two phases and a parity phase), three CXs a swap of labels.  Phases need no qubit
//    to be local to a tile.
// 2. select_passes cuts the ops into passes of 12 (FP64) or 13 (FP32) local qubits.
// 3. In a pass, one-qubit ops collect in a pending 2x2 matrix per qubit.  A CX whose control's
//    pending matrix is diagonal and whose target's is a I + b X passes by them; otherwise the
//    qubit's matrix is first split and its non-commuting rest applied (BF_ROT) while the
//    qubit sits in a register.  A stage is a choice of 4 register qubits; everything that can
//    go in it goes, then the tile is redistributed.  Whether a matrix is diagonal or a I + b X
//    is decided by the gates' forms and not by their values, so circuits of one structure
//    have plans of one structure.
// 4. What is pending at the end of a pass waits for the next pass that acts on the qubit.
//    Where the qubit is not local there (it is then a control or has a phase), the matrix is
//    made diagonal first; after the last one it is applied.
#include <algorithm>
#include <array>
#include <cmath>
#include <complex>
#include <cstring>

#include "bfly_core.cuh"

namespace svb {
namespace {

// 80-bit: a circuit's matrices pass through many products and splits before they are rounded
// once; in 64 bits those roundings, the same for every amplitude, outweighed the kernel's
// (n = 16, 309 gates: 3.7e-15 off the exact state, the tensor-core blocks 1.9e-15).
using real = long double;
using cplx = std::complex<real>;
using M2 = std::array<cplx, 4>;          // row-major 2x2

inline uint64_t bit(int q) { return 1ull << q; }

M2 ident2() { return M2{cplx(1), cplx(0), cplx(0), cplx(1)}; }
M2 mul2(const M2& a, const M2& b)
{
    M2 r;
    for (int i = 0; i < 2; i++)
        for (int j = 0; j < 2; j++) r[i * 2 + j] = a[i * 2] * b[j] + a[i * 2 + 1] * b[2 + j];
    return r;
}

// 2x2 matrix of an elementary op, read off the kernels' own expressions on the basis
M2 matrix_of(const EOp& e)
{
    const Coef<double> c = load_coef<double>(e.m);
    M2 u{};
    for (int col = 0; col < 2; col++) {
        double2 a0 = make_double2(col == 0 ? 1.0 : 0.0, 0.0), a1 = make_double2(col == 1 ? 1.0 : 0.0, 0.0);
        if (form_is_diag(e.form)) {
            diag_one<double>(e.form, c, a1);
            if (e.form == F_DIAG) diag_zero<double>(e.form, c, a0);
        } else {
            dense_pair<double>(e.form, c, a0, a1);
        }
        u[col] = cplx(a0.x, a0.y);
        u[2 + col] = cplx(a1.x, a1.y);
    }
    return u;
}

// What a pending matrix commutes with: DIAG with a control, XT (a I + b X) with a target.
enum Cls : uint8_t { C_ID = 0, C_DIAG, C_XT, C_GEN };
Cls cls_of(uint8_t form)
{
    if (form_is_diag(form)) return C_DIAG;
    if (form == F_X || form == F_RX || form == F_W) return C_XT;
    return C_GEN;
}
Cls cls_mul(Cls a, Cls b) { return a == C_ID ? b : (a == b ? a : C_GEN); }

// ---- 1. short forms ---------------------------------------------------------------------

enum ItemKind : uint8_t { I_ONE, I_CX, I_PP, I_SWAP, I_MAKE_DIAG, I_APPLY };

struct Item {
    ItemKind kind;
    Cls cls;                             // I_ONE
    int q, c;                            // qubit; CX control, second qubit of PP and SWAP
    uint64_t touch;
    M2 m;                                // I_ONE matrix; I_PP: m[0], m[1] = even and odd phase
};

// rewrites ops into the list that is cut into passes
std::vector<EOp> shorten(const std::vector<EOp>& in)
{
    const int N = (int)in.size();
    // next op on the same qubit, for the op's first (q) and second (c) qubit
    std::vector<int> nq(N, -1), nc(N, -1), last(64, -1);
    for (int i = N - 1; i >= 0; i--) {
        nq[i] = last[in[i].q];
        if (in[i].form == F_CX) {
            nc[i] = last[in[i].c];
            last[in[i].c] = i;
        }
        last[in[i].q] = i;
    }
    auto next_on = [&](int i, uint32_t q) { return in[i].q == q ? nq[i] : nc[i]; };
    std::vector<int> prev_q(N, -1);      // previous op on a CX's target
    std::fill(last.begin(), last.end(), -1);
    for (int i = 0; i < N; i++) {
        prev_q[i] = last[in[i].q];
        last[in[i].q] = i;
        if (in[i].form == F_CX) last[in[i].c] = i;
    }
    std::vector<char> gone(N, 0);
    std::vector<std::vector<EOp>> repl;
    std::vector<int> repl_of(N, -1);
    auto put = [&](int i, std::vector<EOp> ops) {
        repl_of[i] = (int)repl.size();
        repl.push_back(std::move(ops));
    };
    auto simple = [&](const EOp& src, uint8_t form, uint32_t q) {
        EOp e = src;
        e.form = form;
        e.q = q;
        return e;
    };
    auto parity_phase = [&](const EOp& cx, cplx d0, cplx d1) {
        EOp e = cx;
        e.form = F_PP;
        e.m[0] = (double)d0.real();
        e.m[1] = (double)d0.imag();
        e.m[2] = (double)d1.real();
        e.m[3] = (double)d1.imag();
        return e;
    };
    for (int i = 0; i < N; i++) {
        if (gone[i] || in[i].form != F_CX) continue;
        const uint32_t t = in[i].q, c = in[i].c;
        // three CXs, the middle one the other way round
        const int j = nq[i], k = j >= 0 && nc[i] == j && in[j].form == F_CX && in[j].q == c && in[j].c == t ? nq[j] : -1;
        if (k >= 0 && nc[j] == k && in[k].form == F_CX && in[k].q == t && in[k].c == c && !gone[j] && !gone[k]) {
            gone[j] = gone[k] = 1;
            put(i, {simple(in[i], F_SWAP, t)});
            continue;
        }
        // diagonal ops on the target up to the same CX again
        cplx d0 = 1, d1 = 1;
        int x = j;
        std::vector<int> diag;
        while (x >= 0 && !gone[x] && form_is_diag(in[x].form) && in[x].q == t) {
            const M2 m = matrix_of(in[x]);
            d0 *= m[0];
            d1 *= m[3];
            diag.push_back(x);
            x = nq[x];
        }
        if (x >= 0 && !gone[x] && in[x].form == F_CX && in[x].q == t && in[x].c == c) {
            // what the control meets in between must commute with being a control
            int y = nc[i];
            while (y >= 0 && y != x && ((form_is_diag(in[y].form) && in[y].q == c) || (in[y].form == F_CX && in[y].c == c)))
                y = next_on(y, c);
            if (y == x) {
                for (int z : diag) gone[z] = 1;
                gone[x] = 1;
                gone[i] = 1;
                put(i, {parity_phase(in[i], d0, d1)});
                continue;
            }
        }
        // H on the target right before and after: a controlled Z
        const int h0 = prev_q[i];
        if (h0 >= 0 && !gone[h0] && in[h0].form == F_H && in[h0].q == t && j >= 0 && !gone[j] && in[j].form == F_H &&
            in[j].q == t) {
            gone[h0] = gone[j] = 1;
            put(i, {simple(in[i], F_S, c), simple(in[i], F_S, t), parity_phase(in[i], 1, cplx(0, -1))});
        }
    }
    std::vector<EOp> out;
    out.reserve(N);
    for (int i = 0; i < N; i++) {
        if (repl_of[i] >= 0) out.insert(out.end(), repl[repl_of[i]].begin(), repl[repl_of[i]].end());
        else if (!gone[i]) out.push_back(in[i]);
    }
    return out;
}

// ---- 3. a pass --------------------------------------------------------------------------

struct Row {                             // value of a local position, see bfly.h
    uint8_t rm = 0;                      // register bits (bit 4: packed half)
    uint16_t tm = 0;                     // thread bits, named by the position each held at the stage's start
    uint64_t xm = 0;                     // global index bits of the tile
};

struct StageOp {
    BfOp op;
    uint16_t tm;                         // thread mask by position, as in Row
    uint64_t xm;                         // tile mask
};

struct St {                              // what a stage changes
    Row row[BF_MAX_POS];
    int8_t reg[BF_MAX_POS];              // register bit of the position, -1: thread bit
    uint8_t cls[64];
};

struct Split {                           // U = left . W, W = p [[1, u], [-conj u, 1]] or SROT
    M2 left;
    real p;
    cplx b;                              // p u
    real norm;                           // of U, where it is not in left: the reference's H, T and
                                         // U2 are unitary up to the rounding of sqrt(1/2) only, and
                                         // a few hundred of them show
};

// control side: left diagonal
Split split_diag(const M2& m)
{
    Split s;
    const real p = std::abs(m[0]);
    const cplx d0 = p > 0 ? m[0] / p : cplx(1);
    s.b = m[1] * std::conj(d0);
    cplx d1 = p >= std::abs(s.b) ? m[3] : -m[2] / std::conj(s.b);
    d1 /= std::abs(d1);
    s.p = p;
    s.norm = std::sqrt(std::norm(m[0]) + std::norm(m[1]));
    s.left = M2{d0, cplx(0), cplx(0), d1};
    return s;
}

// target side: left = a I + b X, chosen so that W's diagonal is real
Split split_x(const M2& m)
{
    Split s;
    const cplx g = std::sqrt(m[0] * m[3] - m[1] * m[2]);
    const cplx P = m[0] / g, Q = m[2] / g;
    const real h = std::hypot(Q.real(), P.imag());
    real ca = h > 0 ? Q.real() / h : real(1), sa = h > 0 ? P.imag() / h : real(0);
    real p = ca * P.real() + sa * Q.imag();
    if (p < 0) {
        ca = -ca;
        sa = -sa;
        p = -p;
    }
    s.p = p;
    s.norm = 1;
    s.b = -std::conj(ca * Q - cplx(0, sa) * P);
    s.left = M2{g * ca, g * cplx(0, sa), g * cplx(0, sa), g * ca};
    return s;
}

struct PassPlanner {
    BfPlan& plan;
    const int n;
    const int M;                         // local positions
    const int pack;                      // 1: position 0 is the half of a packed unit
    const bool fp32;
    M2* pend;                            // pending matrix of every qubit
    int local_q[BF_MAX_POS];
    int pos_of[64];
    std::vector<StageOp> out;            // ops of the current stage
    real scale = 1;                      // of the pass
    uint32_t coef_base = 0;
    int op_limit = 0;                    // of plan.ops, where the pass has to end
    size_t coef_limit = 0;               // of plan.coefs
    const int32_t* stage_masks = nullptr; // tile masks of the pass's finished stages
    bool ok = true;                      // false: a layout that the kernel cannot address

    int reg_of(const St& s, int p) const { return (pack && p == 0) ? BF_PACK : s.reg[p]; }

    bool column_pure(const St& s, int p) const
    {
        const int r = reg_of(s, p);
        for (int x = 0; x < M; x++)
            if (x != p && ((s.row[x].rm >> r) & 1)) return false;
        return true;
    }
    bool can_rot(const St& s, int p) const { return reg_of(s, p) >= 0 && column_pure(s, p); }

    // a phase's coefficients: doubles in either precision
    uint32_t coef_phase(cplx d0, cplx d1)
    {
        const double d[4] = {(double)d0.real(), (double)d0.imag(), (double)d1.real(), (double)d1.imag()};
        if (!fp32) return coef({d[0], d[1], d[2], d[3]});
        if ((plan.coefs.size() - coef_base) & 1) plan.coefs.push_back(0);
        const uint32_t at = (uint32_t)plan.coefs.size() - coef_base;
        plan.raw.push_back(plan.coefs.size());
        for (int i = 0; i < 4; i++) {
            plan.coefs.push_back(d[i]);      // replaced by its two halves when uploaded
            plan.coefs.push_back(0);
        }
        return at;
    }
    uint32_t coef(std::initializer_list<double> v)
    {
        const uint32_t at = (uint32_t)plan.coefs.size() - coef_base;
        plan.coefs.insert(plan.coefs.end(), v);
        return at;
    }
    BfOp blank(BfKind k) const
    {
        BfOp o;
        std::memset(&o, 0, sizeof(o));
        o.kind = k;
        o.tile_bit = BF_NO_TILE;
        return o;
    }
    void emit(const BfOp& o, uint16_t tm, uint64_t xm) { out.push_back({o, tm, xm}); }

    void set_u(BfOp& o, double re, double im) const
    {
        if (fp32) {
            o.f[0] = (float)re;
            o.f[1] = (float)im;
        } else {
            o.d[0] = re;
            o.d[1] = im;
        }
    }

    double round_to(double x) const { return fp32 ? (double)(float)x : x; }

    // applies what of pend[q] does not commute with a control (x = false) or target (x = true)
    void rot(St& s, int q, bool x, bool dry)
    {
        const int p = pos_of[q];
        s.cls[q] = x ? C_XT : C_DIAG;
        if (dry) return;
        const Split sp = x ? split_x(pend[q]) : split_diag(pend[q]);
        pend[q] = sp.left;
        BfOp o = blank(BF_ROT);
        o.tgt = (uint8_t)reg_of(s, p);
        if (o.tgt == BF_PACK) o.kind = BF_PROT;
        cplx u = sp.p > 0 ? sp.b / sp.p : cplx(0);
        const double ur = fp32 ? (float)u.real() : (double)u.real(), ui = fp32 ? (float)u.imag() : (double)u.imag();
        const real f = 1 / std::sqrt(1 + (real)ur * ur + (real)ui * ui);    // of u as rounded
        if (!(sp.p > 0 && scale * f >= (fp32 ? BF_LEAST32 : BF_LEAST64))) {
            // with the scale so far in the matrix, the pass begins anew at 1 (times what p and b
            // lost in their rounding)
            const cplx b = sp.b * scale;
            const double pr = round_to((double)(sp.p * scale)), br = round_to((double)b.real()),
                         bi = round_to((double)b.imag());
            o.kind = BF_SROT;
            o.coef = coef({pr});
            set_u(o, br, bi);
            scale *= std::sqrt((sp.p * sp.p + std::norm(sp.b)) / ((real)pr * pr + (real)br * br + (real)bi * bi));
        } else {
            scale *= f * sp.norm;
            set_u(o, ur, ui);
        }
        emit(o, s.row[p].tm, s.row[p].xm);
        plan.n_gates2++;
    }

    // register bit i's value ^= register mask m: permutes the registers, keeps the rows' meaning
    void move_regs(St& s, int p_t, uint8_t m, bool dry)
    {
        const int i = reg_of(s, p_t);
        for (int x = 0; x < M; x++)
            if (x != p_t && ((s.row[x].rm >> i) & 1)) s.row[x].rm ^= m;
        if (dry) return;
        for (int j = 0; j <= BF_PACK; j++) {
            if (!((m >> j) & 1)) continue;
            BfOp o = blank(BF_CX);
            o.tgt = (uint8_t)i;
            o.ctl = (uint8_t)j;
            emit(o, 0, 0);
            plan.n_moves++;
        }
    }

    // x_t ^= x_c; false if the layout does not allow it
    bool cx_rows(St& s, int qc, int qt, bool dry)
    {
        const int t = pos_of[qt], c = pos_of[qc];
        if (c < 0) {
            s.row[t].xm ^= bit(qc);
            return true;
        }
        const int i = reg_of(s, t);
        if (i >= 0) {
            const uint8_t m = s.row[c].rm;
            if ((m >> i) & 1) return false;
            // a position other than 0 cannot differ between the halves of a packed unit: its
            // relayout slots and offsets are the unit's.  Registers that other rows share
            // with t would make theirs differ; the next stage begins with pure rows.
            if (pack && i != BF_PACK && ((m >> BF_PACK) & 1) && !column_pure(s, t)) return false;
            if (m) move_regs(s, t, m, dry);
        } else {
            if (pack && ((s.row[c].rm >> BF_PACK) & 1)) return false;
            s.row[t].rm ^= s.row[c].rm;
        }
        s.row[t].tm ^= s.row[c].tm;
        s.row[t].xm ^= s.row[c].xm;
        return true;
    }

    bool diag_ok(const St& s, int q) const { return s.cls[q] == C_ID || s.cls[q] == C_DIAG; }

    bool make_diag(St& s, int q, bool dry)
    {
        if (diag_ok(s, q)) return true;
        if (pos_of[q] < 0 || !can_rot(s, pos_of[q])) return false;
        rot(s, q, false, dry);
        return true;
    }
    bool make_x(St& s, int q, bool dry)
    {
        if (s.cls[q] == C_ID || s.cls[q] == C_XT) return true;
        if (!can_rot(s, pos_of[q])) return false;
        rot(s, q, true, dry);
        return true;
    }

    bool phase(St& s, uint64_t qubits, cplx d0, cplx d1, bool dry)
    {
        Row r;
        for (int q = 0; q < n; q++) {
            if (!((qubits >> q) & 1)) continue;
            const int p = pos_of[q];
            if (p < 0) {
                r.xm ^= bit(q);
            } else {
                r.rm ^= s.row[p].rm;
                r.tm ^= s.row[p].tm;
                r.xm ^= s.row[p].xm;
            }
        }
        if (__builtin_popcount(r.rm & (BF_NR - 1)) > 2) return false;
        if (dry) return true;
        BfOp o = blank(BF_DIAG);
        o.rmask = r.rm;
        o.coef = coef_phase(d0, d1);
        emit(o, r.tm, r.xm);
        plan.n_diags++;
        return true;
    }

    // tile masks a pass can still take: those of finished stages, and at worst one of each op
    // of this one
    int masks_left() const
    {
        int k = 0;
        for (const StageOp& o : out) k += o.xm != 0;
        if (k + *stage_masks < BF_NO_TILE - 4) return BF_NO_TILE;    // the usual case
        std::vector<uint64_t> seen;
        for (const StageOp& o : out)
            if (o.xm && std::find(seen.begin(), seen.end(), o.xm) == seen.end()) seen.push_back(o.xm);
        return BF_NO_TILE - *stage_masks - (int)seen.size();
    }

    // one item, if the stage allows it; parts of it may be done already when it does not
    bool exec(St& s, const Item& it, bool dry)
    {
        switch (it.kind) {
        case I_ONE:
            s.cls[it.q] = cls_mul((Cls)s.cls[it.q], it.cls);
            if (!dry) pend[it.q] = mul2(it.m, pend[it.q]);
            return true;
        case I_CX: {
            // both sides, so that the one that can go goes even if the other must wait
            const bool x = make_x(s, it.q, dry), d = make_diag(s, it.c, dry);
            if (!x || !d) return false;
            return cx_rows(s, it.c, it.q, dry);
        }
        case I_PP: {
            const bool a = make_diag(s, it.q, dry), b = make_diag(s, it.c, dry);
            return a && b && phase(s, bit(it.q) | bit(it.c), it.m[0], it.m[1], dry);
        }
        case I_SWAP: {
            const int a = pos_of[it.q], b = pos_of[it.c];
            if (pack && (a == 0 || b == 0)) {
                // the packed qubit stays packed: three CXs in registers
                const int o = a == 0 ? it.c : it.q, z = a == 0 ? it.q : it.c;
                if (!can_rot(s, pos_of[o])) return false;
                cx_rows(s, z, o, dry);
                cx_rows(s, o, z, dry);
                cx_rows(s, z, o, dry);
            } else {
                std::swap(s.row[a], s.row[b]);
                std::swap(s.reg[a], s.reg[b]);
            }
            std::swap(s.cls[it.q], s.cls[it.c]);
            if (!dry) std::swap(pend[it.q], pend[it.c]);
            return true;
        }
        case I_MAKE_DIAG:
            return make_diag(s, it.q, dry);
        default:                             // I_APPLY
            if (s.cls[it.q] == C_ID) return true;
            // the part that needs a register, then the diagonal rest as a phase
            if (!make_diag(s, it.q, dry) || !phase(s, bit(it.q), pend[it.q][0], pend[it.q][3], dry)) return false;
            s.cls[it.q] = C_ID;
            if (!dry) pend[it.q] = ident2();
            return true;
        }
    }

    // runs what can go; `left` receives the items that remain.  Returns how much was done
    // (gates that needed a register weigh most).
    int run_stage(St& s, const std::vector<const Item*>& items, std::vector<const Item*>* left, bool dry)
    {
        uint64_t blocked = 0;
        const uint64_t all = n >= 64 ? ~0ull : bit(n) - 1;
        int score = 0;
        for (size_t i = 0; i < items.size(); i++) {
            const Item& it = *items[i];
            if (it.touch & blocked) {
                blocked |= it.touch;
                if (left) left->push_back(&it);
                else if (blocked == all) break;
                continue;
            }
            if (!dry && (plan.ops.size() + out.size() > (size_t)op_limit || plan.coefs.size() > coef_limit ||
                         masks_left() < 4)) {
                blocked = all;
                left->push_back(&it);
                continue;
            }
            const uint8_t cq = s.cls[it.q], cc = it.c >= 0 ? s.cls[it.c] : 0;
            if (exec(s, it, dry)) {
                if (it.kind != I_ONE) {
                    score += 1;
                    if (it.kind != I_SWAP) score += 4 * ((cq != s.cls[it.q]) + (it.c >= 0 && cc != s.cls[it.c]));
                }
            } else {
                if (it.kind == I_CX || it.kind == I_PP) score += 4 * ((cq != s.cls[it.q]) + (cc != s.cls[it.c]));
                blocked |= it.touch;
                if (left) left->push_back(&it);
            }
        }
        return score;
    }

    // positions that will have to sit in a register, in the order the items ask for them
    void needs(const St& s, const std::vector<const Item*>& items, std::vector<int>& order) const
    {
        uint8_t cls[64];
        std::memcpy(cls, s.cls, sizeof(cls));
        uint32_t seen = pack ? 1u : 0u;
        order.clear();
        auto need = [&](int q) {
            const int p = pos_of[q];
            if (p >= 0 && !((seen >> p) & 1)) {
                seen |= 1u << p;
                order.push_back(p);
            }
        };
        for (const Item* it : items) {
            auto diag = [&](int q) {
                if (cls[q] != C_ID && cls[q] != C_DIAG) {
                    need(q);
                    cls[q] = C_DIAG;
                }
            };
            switch (it->kind) {
            case I_ONE: cls[it->q] = cls_mul((Cls)cls[it->q], it->cls); break;
            case I_CX:
                if (cls[it->q] != C_ID && cls[it->q] != C_XT) {
                    need(it->q);
                    cls[it->q] = C_XT;
                }
                diag(it->c);
                if (pack && pos_of[it->c] == 0) need(it->q);
                break;
            case I_PP:
                diag(it->q);
                diag(it->c);
                break;
            case I_SWAP:
                if (pack && (pos_of[it->q] == 0 || pos_of[it->c] == 0)) {
                    need(it->q);
                    need(it->c);
                }
                std::swap(cls[it->q], cls[it->c]);
                break;
            case I_MAKE_DIAG: diag(it->q); break;
            default:
                if (cls[it->q] == C_XT || cls[it->q] == C_GEN) need(it->q);
                cls[it->q] = C_ID;
                break;
            }
        }
    }

    void set_layout(St& s, const int* regs) const
    {
        for (int p = 0; p < M; p++) s.reg[p] = -1;
        for (int i = 0; i < BF_RB; i++) s.reg[regs[i]] = (int8_t)i;
        for (int p = 0; p < M; p++) {
            Row& r = s.row[p];
            const int i = reg_of(s, p);
            r.rm = i >= 0 ? (uint8_t)(1u << i) : 0;
            r.tm = i >= 0 ? 0 : (uint16_t)(1u << p);
        }
    }

    void choose(const St& s, const std::vector<const Item*>& items, bool first, int* regs)
    {
        std::vector<int> order;
        needs(s, items, order);
        const int low = pack + BF_COAL;
        if (first) order.erase(std::remove_if(order.begin(), order.end(), [&](int p) { return p < low; }), order.end());
        int k = 0;
        uint32_t in = 0;
        for (int p : order) {
            if (k == BF_RB) break;
            regs[k++] = p;
            in |= 1u << p;
        }
        const int wanted = k;
        for (int p = M - 1; k < BF_RB; p--)
            if (!((in >> p) & 1)) {
                regs[k++] = p;
                in |= 1u << p;
            }
        if ((int)order.size() <= BF_RB || wanted < BF_RB) return;
        // one qubit at a time exchanged for a later one, where the stage gets more done; the
        // first need stays, so that every stage gets on
        auto value = [&](const int* r) {
            St t = s;
            set_layout(t, r);
            return run_stage(t, items, nullptr, true);
        };
        int best = value(regs);
        for (int slot = BF_RB - 1; slot >= 1; slot--)
            for (int p : order) {
                if ((in >> p) & 1) continue;
                int r[BF_RB];
                std::memcpy(r, regs, sizeof(r));
                r[slot] = p;
                const int v = value(r);
                if (v > best) {
                    best = v;
                    in = (in & ~(1u << regs[slot])) | (1u << p);
                    regs[slot] = p;
                }
            }
    }

    // unit slot image (swizzled) of a set of positions
    uint16_t slot(uint32_t positions) const { return (uint16_t)Swz<double>::f(positions >> pack); }
    static int rank3(uint32_t a, uint32_t b, uint32_t c)
    {
        a &= 7;
        b &= 7;
        c &= 7;
        return a && b && c && a != b && a != c && b != c && (a ^ b) != c;
    }

    // thread bits: which position sits on which at the start of the stage
    void assign(const St& s, bool loads, bool stores, bool reads, bool writes, int* bits) const
    {
        std::vector<int> thr;
        uint32_t col[BF_MAX_POS] = {0};
        for (int p = pack; p < M; p++) {
            for (int x = pack; x < M; x++)
                if ((s.row[x].tm >> p) & 1) col[p] |= 1u << x;
        }
        for (int p = pack; p < M; p++)
            if (start_reg[p] < 0) thr.push_back(p);
        const uint32_t low = ((1u << BF_COAL) - 1) << pack;
        auto in_low = [&](int p) { return col[p] && !(col[p] & ~low); };
        uint16_t rslot[BF_TB], wslot[BF_TB];
        for (int a = 0; a < BF_TB; a++) {
            rslot[a] = slot(1u << thr[a]);
            wslot[a] = slot(col[thr[a]]);
        }
        // the first choice of the highest value; no search beyond one that has all
        const int most = 16 * loads + 16 * stores + 4 * reads + 4 * writes + (loads || stores);
        int best = -1, pick[3] = {0, 1, 2};
        for (int a = 0; a < BF_TB && best < most; a++)
            for (int b = a + 1; b < BF_TB && best < most; b++)
                for (int c = 0; c < BF_TB && best < most; c++) {
                    if (c == a || c == b) continue;
                    const int A = thr[a], B = thr[b], C = thr[c];
                    int v = 0;
                    if (loads && ((1u << A | 1u << B) == low)) v += 16;
                    if (stores && in_low(A) && in_low(B) && col[A] != col[B]) v += 16;
                    if (reads && rank3(rslot[a], rslot[b], rslot[c])) v += 4;
                    if (writes && rank3(wslot[a], wslot[b], wslot[c])) v += 4;
                    // lane 2 on the next lowest qubit: 128-byte runs
                    if ((loads && C == pack + BF_COAL) || (stores && col[C] == 1u << (pack + BF_COAL))) v += 1;
                    if (v > best) {
                        best = v;
                        pick[0] = a;
                        pick[1] = b;
                        pick[2] = c;
                    }
                }
        int k = 0;
        for (int i = 0; i < 3; i++) bits[k++] = thr[pick[i]];
        for (int i = 0; i < BF_TB; i++)
            if (i != pick[0] && i != pick[1] && i != pick[2]) bits[k++] = thr[i];
    }

    // first: the layout also loads the tile, so lanes 0 and 1 are the low positions themselves
    bool storable(const St& s, bool first) const
    {
        const uint32_t low = ((1u << BF_COAL) - 1) << pack;
        uint32_t got = 0, cnt = 0;
        for (int p = pack; p < M; p++) {
            if (start_reg[p] >= 0 || (first && p >= pack + BF_COAL)) continue;
            uint32_t col = 0;
            for (int x = pack; x < M; x++)
                if ((s.row[x].tm >> p) & 1) col |= 1u << x;
            if (col && !(col & ~low)) {
                if (cnt == 0 || col != got) cnt++;
                got = col;
            }
        }
        return cnt >= 2;
    }

    int8_t start_reg[BF_MAX_POS];        // register bit of each position at the stage's start

    // phases commute: each run of them between other ops is ordered by register mask, and
    // those of one mask become one multiplication of the units
    void order_phases()
    {
        bool any = false;
        for (size_t i = 0; i < out.size();) {
            if (out[i].op.kind != BF_DIAG) {
                i++;
                continue;
            }
            any = true;
            size_t j = i;
            while (j < out.size() && out[j].op.kind == BF_DIAG) j++;
            std::stable_sort(out.begin() + i, out.begin() + j,
                             [](const StageOp& a, const StageOp& b) { return a.op.rmask < b.op.rmask; });
            for (size_t x = i; x < j; x++) {
                const bool begin = x == i || out[x - 1].op.rmask != out[x].op.rmask;
                const bool end = x + 1 == j || out[x + 1].op.rmask != out[x].op.rmask;
                out[x].op.run = (begin ? 1 : 0) | (end ? 2 : 0);
            }
            i = j;
        }
        if (any) emit(blank(BF_FLUSH), 0, 0);
    }

    // the finished stage's ops, its thread bits and its side of the relayouts around it
    void finish(const St& s, bool loads, bool stores, int rel_in, int rel_out, BfPass& P)
    {
        int bits[BF_TB];
        assign(s, loads, stores, rel_in >= 0, rel_out >= 0, bits);
        auto thr_bits = [&](uint16_t tm) {
            uint16_t r = 0;
            for (int b = 0; b < BF_TB; b++)
                if ((tm >> bits[b]) & 1) r |= (uint16_t)(1u << b);
            return r;
        };
        for (const StageOp& o : out) {
            plan.ops.push_back(o.op);
            plan.ops.back().thr_mask = (uint8_t)thr_bits(o.tm);
            if (o.xm) {
                int i = 0;
                while (i < P.n_tile_masks && P.tile_mask[i] != o.xm) i++;
                if (i == P.n_tile_masks) P.tile_mask[P.n_tile_masks++] = o.xm;
                plan.ops.back().tile_bit = (uint8_t)i;
            }
        }
        out.clear();
        uint32_t wcol[BF_TB] = {0}, wreg[BF_RB] = {0};
        for (int x = pack; x < M; x++) {
            if (s.row[x].rm >> BF_RB) ok = false;    // differs between the halves of a unit
            for (int b = 0; b < BF_TB; b++)
                if ((s.row[x].tm >> bits[b]) & 1) wcol[b] |= 1u << x;
            for (int i = 0; i < BF_RB; i++)
                if ((s.row[x].rm >> i) & 1) wreg[i] |= 1u << x;
        }
        int rpos[BF_RB] = {0};
        for (int p = pack; p < M; p++)
            if (start_reg[p] >= 0) rpos[start_reg[p]] = p;
        auto global = [&](uint32_t positions) {
            uint64_t g = 0;
            for (int p = 0; p < M; p++)
                if ((positions >> p) & 1) g |= bit(local_q[p]);
            return g;
        };
        if (loads) {
            for (int b = 0; b < BF_TB; b++) P.in_thr[b] = global(1u << bits[b]);
            for (int i = 0; i < BF_RB; i++) P.in_reg[i] = global(1u << rpos[i]);
        }
        if (rel_in >= 0) {
            BfRelayout& R = plan.rels[rel_in];
            for (int b = 0; b < BF_TB; b++) R.rthr[b] = slot(1u << bits[b]);
            for (int i = 0; i < BF_RB; i++) R.rreg[i] = slot(1u << rpos[i]);
        }
        if (rel_out >= 0) {
            BfRelayout& R = plan.rels[rel_out];
            for (int b = 0; b < BF_TB; b++) R.wthr[b] = slot(wcol[b]);
            for (int i = 0; i < BF_RB; i++) R.wreg[i] = slot(wreg[i]);
        }
        if (stores) {
            for (int b = 0; b < BF_TB; b++) P.out_thr[b] = global(wcol[b]);
            for (int i = 0; i < BF_RB; i++) P.out_reg[i] = global(wreg[i]);
            P.n_flips = 0;
            for (int p = pack; p < M; p++)
                if (s.row[p].xm) P.flips[P.n_flips++] = BfFlip{s.row[p].xm, global(1u << p)};
        }
    }

    // the packed half's thread (and tile) mask, before the units leave their threads
    void fix_pack(St& s, bool tile)
    {
        if (!pack || (!s.row[0].tm && !(tile && s.row[0].xm))) return;
        BfOp o = blank(BF_PFIX);
        emit(o, s.row[0].tm, tile ? s.row[0].xm : 0);
        s.row[0].tm = 0;
        if (tile) s.row[0].xm = 0;
    }

    // Plans one pass over `items`; returns those left for a further pass over the same
    // qubits.
    std::vector<const Item*> run(uint64_t L, std::vector<const Item*> items, uint8_t* cls)
    {
        BfPass P;
        std::memset(&P, 0, sizeof(P));
        for (int q = 0; q < 64; q++) pos_of[q] = -1;
        int nl = 0;
        for (int q = 0; q < n; q++) {
            if ((L >> q) & 1) {
                local_q[nl] = q;
                pos_of[q] = nl++;
            } else {
                P.nonlocal_q[P.n_nonlocal++] = (uint8_t)q;
            }
        }
        stage_masks = &P.n_tile_masks;
        P.op_begin = (int32_t)plan.ops.size();
        P.rel_begin = (int32_t)plan.rels.size();
        // an item emits at most 6 ops (two gates, four register moves), a stage's end four
        op_limit = P.op_begin + BF_MAX_OPS - 16 - 4 * BF_MAX_REL;
        coef_base = (uint32_t)plan.coefs.size();
        coef_limit = coef_base + BF_MAX_COEF - 32;     // an item has at most 9
        P.coef_begin = (int32_t)coef_base;
        scale = 1;
        St s;
        std::memset(s.reg, -1, sizeof(s.reg));
        std::memcpy(s.cls, cls, sizeof(s.cls));
        std::vector<const Item*> left;
        int rel_in = -1;
        bool first = true;
        for (;;) {
            int regs[BF_RB];
            choose(s, items, first, regs);
            set_layout(s, regs);
            std::memcpy(start_reg, s.reg, sizeof(start_reg));
            left.clear();
            run_stage(s, items, &left, false);
            items.swap(left);
            const bool full = (int)plan.rels.size() - P.rel_begin >= BF_MAX_REL - 1 ||
                              (int)(plan.ops.size() + out.size()) > op_limit || plan.coefs.size() > coef_limit ||
                              masks_left() < 4;
            const bool last = items.empty() || full;
            const bool stores = last && storable(s, first);
            order_phases();
            fix_pack(s, stores);
            int rel_out = -1;
            if (!stores) {
                rel_out = (int)plan.rels.size();
                plan.rels.emplace_back();
                BfOp o = blank(BF_RELAYOUT);
                o.lay = (uint8_t)(rel_out - P.rel_begin);
                emit(o, 0, 0);
            }
            finish(s, first, stores, rel_in, rel_out, P);
            first = false;
            rel_in = rel_out;
            if (stores) break;
            if (last) {                      // a layout that stores whole runs
                int r[BF_RB];
                for (int i = 0; i < BF_RB; i++) r[i] = M - 1 - i;
                set_layout(s, r);
                std::memcpy(start_reg, s.reg, sizeof(start_reg));
                fix_pack(s, true);
                finish(s, false, true, rel_in, -1, P);
                break;
            }
        }
        std::memcpy(cls, s.cls, sizeof(s.cls));
        coef({(double)scale});
        if (plan.coefs.size() & 1) coef({(double)scale});
        plan.ops.push_back(blank(BF_END));
        P.n_ops = (int32_t)plan.ops.size() - P.op_begin;
        P.n_rel = (int32_t)plan.rels.size() - P.rel_begin;
        P.n_coef = (int32_t)plan.coefs.size() - P.coef_begin;
        plan.smem_bytes = std::max(plan.smem_bytes, bfly_smem(P.n_ops, P.n_rel, P.n_coef, fp32));
        plan.passes.push_back(P);
        return items;
    }
};

}  // namespace

bool bfly_supported(const std::vector<EOp>& ops, int n, int precision)
{
    if (n < BF_UNIT_BITS + (precision == SVB_FP32 ? 1 : 0)) return false;
    for (const EOp& e : ops)
        if (e.form == F_SRN || e.form == F_M4 || e.form == F_R || e.form == F_DIAG) return false;
    return true;
}

// FP64, by the counts of the shortened circuit: the estimate is the logarithm of butterflies'
// time over the blocks', fitted to the circuits below with as many phases and swaps as CXs (off
// by 0.19, one sigma).  Where it is clear one form is planned, since a second plan takes as long
// as 1 to 4 runs up to 20 qubits (Fourier transform of 16 qubits, upload and run 440 us, with
// both plans 550) and 7% of a run at 25.  Up to 20 qubits the estimate decides alone: of 164 such
// circuits it took butterflies on 14 whose runs are 2-19% slower, 1 to 7 us, and whose planning
// is 10 to 40 us shorter, and passed over 5-14% on three; butterflies for all of them were slower
// on 37, by up to 32%.  Circuits of more CXs take 0.94 (23 qubits, depth 25) to 1.5 (12 qubits,
// depth 2) of the blocks' time below 25 qubits, and from 25 on 1.04 to 1.38 at depth 2 to 4.
// FP32: only where phases outnumber the gates that need arithmetic, FFMA2 on the CUDA cores
// against tcgen05: Fourier transform of 13 / 16 / 20 / 28 qubits 0.80 / 0.67 / 0.50 / 0.45 of
// the fused engine's time, ten layers of controlled phases 0.55 to 0.83, half of the gates phases
// 0.8 to 1.4, random circuits 0.9 to 1.6.
BfChoice bfly_choice(const std::vector<EOp>& raw, int n, int precision)
{
    if (!bfly_supported(raw, n, precision)) return BfChoice::BLOCKS;
    size_t phases = 0, swaps = 0, cx = 0, dense = 0;
    for (const EOp& e : shorten(raw)) {
        if (e.form == F_PP) phases++;
        else if (e.form == F_SWAP) swaps++;
        else if (e.form == F_CX) cx++;
        else if (!form_is_diag(e.form)) dense++;
    }
    if (precision == SVB_FP32) return phases >= 2 * (dense + cx) ? BfChoice::BUTTERFLIES : BfChoice::BLOCKS;
    if (phases + swaps == 0 || phases + swaps < cx)
        return n >= 25 && dense >= 6 * (size_t)n ? BfChoice::COMPARE : BfChoice::BLOCKS;
    const double two = (double)(phases + swaps + cx);
    const double estimate = -0.82 + (0.28 * (double)dense + 0.78 * (double)cx + 0.105 * n) / two;
    if (n <= 20) return estimate < 0 ? BfChoice::BUTTERFLIES : BfChoice::BLOCKS;
    return estimate < -0.2 ? BfChoice::BUTTERFLIES : (estimate > 0.05 ? BfChoice::BLOCKS : BfChoice::COMPARE);
}

// Time of either plan by the counts of its parts in us at 25 qubits (from 21 on there are two
// tiles an SM and more), fitted to 188 circuits of 25 to 30 qubits on one B200 (random,
// brickwork, mixed, Fourier transform; depth 2 to 30): 1-2% off a run's time.  A gate costs a
// third of a two-qubit block, but a block takes in two gates and more, so butterflies need some
// depth or phases.  At 25 qubits, of the blocks' time: random U3 + CX of depth 2 / 4 / 10 / 30
// 1.2 / 1.07 / 0.98 / 0.94, brickwork 1.38 / 1.15 / 1.05 / 0.99, half phases and swaps 1.09 /
// 0.94 / 0.85 / 0.8, Fourier transform 0.35.  Of 227 circuits of 21 to 30 qubits the comparison
// was wrong by more than 1% on three (at most 1.4%) and passed over up to 2% on three;
// butterflies for all of them were slower on 78 (up to 38%).
bool bfly_cheaper(const BfPlan& b, const PairPlan& p)
{
    // passes, relayouts, gates, scaled gates, register moves, phases, flushes; passes,
    // relayouts, blocks, exchanges (a lane permutation's share did not show)
    struct Weights {
        double b[7], p[4];
    };
    const Weights w = {{97, 32, 11.6, 17.7, 7.4, 8.9, 20}, {107, 80, 33.4, 3.2}};
    size_t kind[BF_END + 1] = {0};
    for (const BfOp& o : b.ops) kind[o.kind]++;
    const size_t nb[7] = {b.passes.size(), b.rels.size(), kind[BF_ROT], kind[BF_SROT],
                          kind[BF_CX],     kind[BF_DIAG], kind[BF_FLUSH]};
    const size_t np[4] = {p.passes.size(), p.n_relayouts, p.n_blocks, p.n_swaps};
    double tb = 0, tp = 0;
    for (int i = 0; i < 7; i++) tb += w.b[i] * (double)nb[i];
    for (int i = 0; i < 4; i++) tp += w.p[i] * (double)np[i];
    return tb < tp;
}

std::vector<float> bfly_coefs32(const BfPlan& plan)
{
    std::vector<float> f(plan.coefs.begin(), plan.coefs.end());
    for (size_t r : plan.raw)
        for (int i = 0; i < 4; i++) std::memcpy(&f[r + 2 * i], &plan.coefs[r + 2 * i], sizeof(double));
    return f;
}

bool plan_bfly(const std::vector<EOp>& raw, int n, int precision, BfPlan& plan)
{
    plan = BfPlan{};
    const bool fp32 = precision == SVB_FP32;
    const int M = BF_UNIT_BITS + (fp32 ? 1 : 0);
    plan.tile_bits = M;
    const std::vector<EOp> ops = shorten(raw);
    std::vector<Item> items(ops.size());
    for (size_t i = 0; i < ops.size(); i++) {
        const EOp& e = ops[i];
        Item& it = items[i];
        it.q = (int)e.q;
        it.c = -1;
        it.cls = C_ID;
        it.touch = bit(it.q);
        if (e.form == F_CX || e.form == F_PP || e.form == F_SWAP) {
            it.kind = e.form == F_CX ? I_CX : (e.form == F_PP ? I_PP : I_SWAP);
            it.c = (int)e.c;
            it.touch |= bit(it.c);
            it.m = M2{cplx(e.m[0], e.m[1]), cplx(e.m[2], e.m[3]), cplx(0), cplx(0)};
        } else {
            it.kind = I_ONE;
            it.cls = cls_of(e.form);
            it.m = matrix_of(e);
        }
    }
    std::vector<std::pair<uint64_t, std::vector<int>>> cuts;
    select_passes(
        ops, n, M, BF_COAL + (fp32 ? 1 : 0),
        [&](uint64_t L, const std::vector<int>& taken) {
            cuts.push_back({L, taken});
            return std::vector<int>{};
        },
        32);
    // the next cut that touches each qubit, from the last one backwards
    std::vector<std::array<int32_t, 64>> next(cuts.size());
    {
        std::array<int32_t, 64> at;
        at.fill(-1);
        for (size_t ci = cuts.size(); ci-- > 0;) {
            next[ci] = at;
            for (int i : cuts[ci].second)
                for (int q = 0; q < n; q++)
                    if ((items[i].touch >> q) & 1) at[q] = (int32_t)ci;
        }
    }
    std::vector<M2> pend(64, ident2());
    uint8_t cls[64] = {0};
    PassPlanner pp{plan, n, M, fp32 ? 1 : 0, fp32, pend.data()};
    for (size_t ci = 0; ci < cuts.size(); ci++) {
        const uint64_t L = cuts[ci].first;
        std::vector<Item> ends;
        uint64_t touched = 0;
        for (int i : cuts[ci].second) touched |= items[i].touch;
        for (int q = 0; q < n; q++) {
            if (!((touched >> q) & 1)) continue;
            const int nx = next[ci][q];
            Item it;
            it.q = q;
            it.c = -1;
            it.cls = C_ID;
            it.touch = bit(q);
            if (nx < 0) it.kind = I_APPLY;
            else if (((L >> q) & 1) && !((cuts[nx].first >> q) & 1)) it.kind = I_MAKE_DIAG;
            else continue;
            ends.push_back(it);
        }
        std::vector<const Item*> todo;
        for (int i : cuts[ci].second) todo.push_back(&items[i]);
        for (const Item& it : ends) todo.push_back(&it);
        while (!todo.empty()) {
            const size_t before = todo.size(), done = plan.n_gates2 + plan.n_diags + plan.n_moves;
            todo = pp.run(L, todo, cls);
            if (!pp.ok || (todo.size() == before && plan.n_gates2 + plan.n_diags + plan.n_moves == done)) return false;
        }
    }
    return true;
}

}  // namespace svb
