// Per-thread arithmetic and data movement of the butterfly engine (see bfly.h), shared by
// the kernel and, compiled for the host, by the tests' plan runner.
#pragma once

#include "bfly.h"
#include "staged_core.cuh"

namespace svb {

// A packed pair of FP32 values, the operand of fma.rn.f32x2 (one instruction for two FMAs:
// 126 FMA/clk per SM measured, against 108 for scalar FFMA with half the issue slots left).
struct F2 {
    uint64_t b;
};

SVB_HD F2 f2_make(float lo, float hi)
{
    F2 r;
#ifdef __CUDA_ARCH__
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.b) : "f"(lo), "f"(hi));
#else
    uint32_t w[2];
    memcpy(&w[0], &lo, 4);
    memcpy(&w[1], &hi, 4);
    r.b = (uint64_t)w[0] | ((uint64_t)w[1] << 32);
#endif
    return r;
}
SVB_HD void f2_split(F2 a, float& lo, float& hi)
{
#ifdef __CUDA_ARCH__
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.b));
#else
    const uint32_t w[2] = {(uint32_t)a.b, (uint32_t)(a.b >> 32)};
    memcpy(&lo, &w[0], 4);
    memcpy(&hi, &w[1], 4);
#endif
}

// scalar type of a unit's real and imaginary part
template <typename T> struct BfScalar;
template <> struct BfScalar<double> {
    using S = double;
    static constexpr bool packed = false;
    SVB_HD static S dup(double x) { return x; }
    SVB_HD static S fma_(S a, S b, S c) { return ::fma(a, b, c); }
    SVB_HD static S mul(S a, S b) { return a * b; }
    SVB_HD static S neg(S a) { return -a; }
    SVB_HD static S swap(S a) { return a; }
    SVB_HD static S lohi(double lo, double) { return lo; }
    SVB_HD static S mix(S a, S) { return a; }                 // low half of a, high half of b
};
template <> struct BfScalar<float> {
    using S = F2;
    static constexpr bool packed = true;
    SVB_HD static S dup(float x) { return f2_make(x, x); }
    SVB_HD static S lohi(float lo, float hi) { return f2_make(lo, hi); }
    SVB_HD static S fma_(S a, S b, S c)
    {
        S r;
#ifdef __CUDA_ARCH__
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.b) : "l"(a.b), "l"(b.b), "l"(c.b));
#else
        float a0, a1, b0, b1, c0, c1;
        f2_split(a, a0, a1);
        f2_split(b, b0, b1);
        f2_split(c, c0, c1);
        r = f2_make(::fmaf(a0, b0, c0), ::fmaf(a1, b1, c1));
#endif
        return r;
    }
    SVB_HD static S mul(S a, S b)
    {
        S r;
#ifdef __CUDA_ARCH__
        asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.b) : "l"(a.b), "l"(b.b));
#else
        float a0, a1, b0, b1;
        f2_split(a, a0, a1);
        f2_split(b, b0, b1);
        r = f2_make(a0 * b0, a1 * b1);
#endif
        return r;
    }
    SVB_HD static S neg(S a)
    {
        S r;
        r.b = a.b ^ 0x8000000080000000ull;
        return r;
    }
    SVB_HD static S swap(S a)
    {
        float lo, hi;
        f2_split(a, lo, hi);
        return f2_make(hi, lo);
    }
    SVB_HD static S mix(S a, S b)
    {
        float a0, a1, b0, b1;
        f2_split(a, a0, a1);
        f2_split(b, b0, b1);
        return f2_make(a0, b1);
    }
};

template <typename T>
struct BfUnit {                          // 16 bytes
    typename BfScalar<T>::S re, im;
};

// the 16 bytes of a unit in the state: a complex<double>, or two adjacent complex<float>
SVB_HD void bf_load(const double2& a, BfUnit<double>& u) { u.re = a.x; u.im = a.y; }
SVB_HD void bf_load(const float4& a, BfUnit<float>& u) { u.re = f2_make(a.x, a.z); u.im = f2_make(a.y, a.w); }
SVB_HD void bf_store(const BfUnit<double>& u, double2& a) { a.x = u.re; a.y = u.im; }
SVB_HD void bf_store(const BfUnit<float>& u, float4& a)
{
    f2_split(u.re, a.x, a.z);
    f2_split(u.im, a.y, a.w);
}
template <typename T> struct BfWord;
template <> struct BfWord<double> { using type = double2; };
template <> struct BfWord<float> { using type = float4; };

// ---- in-place arithmetic -----------------------------------------------------------------
//
// Every change of a thread's units below is inline PTX on read-write operands, so that each
// case of the dispatch leaves every unit in the registers it found it in.  Written as plain
// expressions the compiler moved the 16 units around after every op (7,000 instructions a
// tile and warp where the gates themselves take 1,400).  SVB_BF_ASM gives a body its two
// forms: f64 on "d" operands, f32x2 on "l".

#ifdef __CUDA_ARCH__
#define SVB_BF_ASM(BODY)                                                                  \
    if constexpr (sizeof(T) == 8) { SVB_BF_EMIT(BODY, "f64", "f64", "d", ) }              \
    else { SVB_BF_EMIT(BODY, "b64", "f32x2", "l", .b) }
#endif

// x <-> y
template <typename T>
SVB_HD void bf_exchange(BfUnit<T>& x, BfUnit<T>& y)
{
#ifdef __CUDA_ARCH__
#define SVB_BF_EMIT(B, R, F, C, M)                                                        \
    asm("{\n\t.reg ." R " t, u;\n\tmov." R " t, %0;\n\tmov." R " u, %1;\n\t"              \
        "mov." R " %0, %2;\n\tmov." R " %1, %3;\n\tmov." R " %2, t;\n\tmov." R " %3, u;\n\t}" \
        : "+" C(x.re M), "+" C(x.im M), "+" C(y.re M), "+" C(y.im M));
    SVB_BF_ASM()
#undef SVB_BF_EMIT
#else
    const BfUnit<T> t = x;
    x = y;
    y = t;
#endif
}

// halves of a packed unit exchanged
SVB_HD void bf_swap_halves(BfUnit<double>&) {}
SVB_HD void bf_swap_halves(BfUnit<float>& u)
{
#ifdef __CUDA_ARCH__
    asm("{\n\t.reg .b32 l, h;\n\tmov.b64 {l, h}, %0;\n\tmov.b64 %0, {h, l};\n\t"
        "mov.b64 {l, h}, %1;\n\tmov.b64 %1, {h, l};\n\t}" : "+l"(u.re.b), "+l"(u.im.b));
#else
    u.re = BfScalar<float>::swap(u.re);
    u.im = BfScalar<float>::swap(u.im);
#endif
}

// high halves of two packed units exchanged (a CX controlled by the packed qubit)
SVB_HD void bf_swap_high(BfUnit<double>&, BfUnit<double>&) {}
SVB_HD void bf_swap_high(BfUnit<float>& x, BfUnit<float>& y)
{
#ifdef __CUDA_ARCH__
    asm("{\n\t.reg .b32 l, h, m, i;\n\t"
        "mov.b64 {l, h}, %0;\n\tmov.b64 {m, i}, %2;\n\tmov.b64 %0, {l, i};\n\tmov.b64 %2, {m, h};\n\t"
        "mov.b64 {l, h}, %1;\n\tmov.b64 {m, i}, %3;\n\tmov.b64 %1, {l, i};\n\tmov.b64 %3, {m, h};\n\t}"
        : "+l"(x.re.b), "+l"(x.im.b), "+l"(y.re.b), "+l"(y.im.b));
#else
    using B = BfScalar<float>;
    const BfUnit<float> a = x, b = y;
    x = BfUnit<float>{B::mix(a.re, b.re), B::mix(a.im, b.im)};
    y = BfUnit<float>{B::mix(b.re, a.re), B::mix(b.im, a.im)};
#endif
}

// u *= c + i s (ns = -s)
template <typename T>
SVB_HD void bf_scale_unit(BfUnit<T>& u, typename BfScalar<T>::S c, typename BfScalar<T>::S s,
                          typename BfScalar<T>::S ns)
{
#ifdef __CUDA_ARCH__
#define SVB_BF_EMIT(B, R, F, C, M)                                                        \
    asm("{\n\t.reg ." R " t;\n\tmul.rn." F " t, %3, %0;\n\tmul.rn." F " %0, %2, %0;\n\t"  \
        "fma.rn." F " %0, %4, %1, %0;\n\tfma.rn." F " %1, %2, %1, t;\n\t}"                \
        : "+" C(u.re M), "+" C(u.im M) : C(c M), C(s M), C(ns M));
    SVB_BF_ASM()
#undef SVB_BF_EMIT
#else
    using B = BfScalar<T>;
    const typename B::S t = B::mul(s, u.re);
    u.re = B::fma_(ns, u.im, B::mul(c, u.re));
    u.im = B::fma_(c, u.im, t);
#endif
}

// a, b <- a + w b, b - conj(w) a, w = r + i s, nr = -r, ns = -s
template <typename T>
SVB_HD void bf_rot_pair(BfUnit<T>& a, BfUnit<T>& b, typename BfScalar<T>::S r, typename BfScalar<T>::S nr,
                        typename BfScalar<T>::S s, typename BfScalar<T>::S ns)
{
#ifdef __CUDA_ARCH__
#define SVB_BF_EMIT(B, R, F, C, M)                                                        \
    asm("{\n\t.reg ." R " x, y;\n\t"                                                      \
        "fma.rn." F " x, %4, %2, %0;\n\tfma.rn." F " y, %4, %3, %1;\n\t"                  \
        "fma.rn." F " x, %7, %3, x;\n\tfma.rn." F " y, %6, %2, y;\n\t"                    \
        "fma.rn." F " %2, %5, %0, %2;\n\tfma.rn." F " %3, %5, %1, %3;\n\t"                \
        "fma.rn." F " %2, %7, %1, %2;\n\tfma.rn." F " %3, %6, %0, %3;\n\t"                \
        "mov." R " %0, x;\n\tmov." R " %1, y;\n\t}"                                       \
        : "+" C(a.re M), "+" C(a.im M), "+" C(b.re M), "+" C(b.im M)                      \
        : C(r M), C(nr M), C(s M), C(ns M));
    SVB_BF_ASM()
#undef SVB_BF_EMIT
#else
    using B = BfScalar<T>;
    const BfUnit<T> x = a, y = b;
    a.re = B::fma_(ns, y.im, B::fma_(r, y.re, x.re));
    a.im = B::fma_(s, y.re, B::fma_(r, y.im, x.im));
    b.re = B::fma_(ns, x.im, B::fma_(nr, x.re, y.re));
    b.im = B::fma_(s, x.re, B::fma_(nr, x.im, y.im));
#endif
}

// a, b <- p a + w b, p b - conj(w) a
template <typename T>
SVB_HD void bf_srot_pair(BfUnit<T>& a, BfUnit<T>& b, typename BfScalar<T>::S p, typename BfScalar<T>::S r,
                         typename BfScalar<T>::S nr, typename BfScalar<T>::S s, typename BfScalar<T>::S ns)
{
#ifdef __CUDA_ARCH__
#define SVB_BF_EMIT(B, R, F, C, M)                                                        \
    asm("{\n\t.reg ." R " x, y;\n\t"                                                      \
        "mul.rn." F " x, %8, %0;\n\tmul.rn." F " y, %8, %1;\n\t"                          \
        "fma.rn." F " x, %4, %2, x;\n\tfma.rn." F " y, %4, %3, y;\n\t"                    \
        "fma.rn." F " x, %7, %3, x;\n\tfma.rn." F " y, %6, %2, y;\n\t"                    \
        "mul.rn." F " %2, %8, %2;\n\tmul.rn." F " %3, %8, %3;\n\t"                        \
        "fma.rn." F " %2, %5, %0, %2;\n\tfma.rn." F " %3, %5, %1, %3;\n\t"                \
        "fma.rn." F " %2, %7, %1, %2;\n\tfma.rn." F " %3, %6, %0, %3;\n\t"                \
        "mov." R " %0, x;\n\tmov." R " %1, y;\n\t}"                                       \
        : "+" C(a.re M), "+" C(a.im M), "+" C(b.re M), "+" C(b.im M)                      \
        : C(r M), C(nr M), C(s M), C(ns M), C(p M));
    SVB_BF_ASM()
#undef SVB_BF_EMIT
#else
    using B = BfScalar<T>;
    const BfUnit<T> x = a, y = b;
    a.re = B::fma_(ns, y.im, B::fma_(r, y.re, B::mul(p, x.re)));
    a.im = B::fma_(s, y.re, B::fma_(r, y.im, B::mul(p, x.im)));
    b.re = B::fma_(ns, x.im, B::fma_(nr, x.re, B::mul(p, y.re)));
    b.im = B::fma_(s, x.re, B::fma_(nr, x.im, B::mul(p, y.im)));
#endif
}

// between the halves of a packed unit: v <- p v + e swap(v), e complex per half
SVB_HD void bf_half_srot(BfUnit<float>& u, F2 p, F2 er, F2 ei, F2 nei)
{
#ifdef __CUDA_ARCH__
    asm("{\n\t.reg .b64 w, z;\n\t.reg .b32 l, h;\n\t"
        "mov.b64 {l, h}, %0;\n\tmov.b64 w, {h, l};\n\tmov.b64 {l, h}, %1;\n\tmov.b64 z, {h, l};\n\t"
        "mul.rn.f32x2 %0, %2, %0;\n\tmul.rn.f32x2 %1, %2, %1;\n\t"
        "fma.rn.f32x2 %0, %3, w, %0;\n\tfma.rn.f32x2 %1, %3, z, %1;\n\t"
        "fma.rn.f32x2 %0, %5, z, %0;\n\tfma.rn.f32x2 %1, %4, w, %1;\n\t}"
        : "+l"(u.re.b), "+l"(u.im.b) : "l"(p.b), "l"(er.b), "l"(ei.b), "l"(nei.b));
#else
    using B = BfScalar<float>;
    const F2 w = B::swap(u.re), z = B::swap(u.im);
    u.re = B::fma_(nei, z, B::fma_(er, w, B::mul(p, u.re)));
    u.im = B::fma_(ei, w, B::fma_(er, z, B::mul(p, u.im)));
#endif
}
// the same with p = 1
SVB_HD void bf_half_rot(BfUnit<float>& u, F2 er, F2 ei, F2 nei)
{
#ifdef __CUDA_ARCH__
    asm("{\n\t.reg .b64 w, z;\n\t.reg .b32 l, h;\n\t"
        "mov.b64 {l, h}, %0;\n\tmov.b64 w, {h, l};\n\tmov.b64 {l, h}, %1;\n\tmov.b64 z, {h, l};\n\t"
        "fma.rn.f32x2 %0, %2, w, %0;\n\tfma.rn.f32x2 %1, %2, z, %1;\n\t"
        "fma.rn.f32x2 %0, %4, z, %0;\n\tfma.rn.f32x2 %1, %3, w, %1;\n\t}"
        : "+l"(u.re.b), "+l"(u.im.b) : "l"(er.b), "l"(ei.b), "l"(nei.b));
#else
    using B = BfScalar<float>;
    const F2 w = B::swap(u.re), z = B::swap(u.im);
    u.re = B::fma_(nei, z, B::fma_(er, w, u.re));
    u.im = B::fma_(ei, w, B::fma_(er, z, u.im));
#endif
}

// [[1, u], [-conj u, 1]], u = r + i s, on register bit TGT.  4 FMAs per unit: bound by the
// FP64 (FFMA2) pipe, 256 cycles a tile and SM at its full rate.
template <typename T, int TGT>
SVB_HD void bf_rot(BfUnit<T>* v, typename BfScalar<T>::S r, typename BfScalar<T>::S s)
{
    using B = BfScalar<T>;
    const typename B::S nr = B::neg(r), ns = B::neg(s);
#pragma unroll
    for (int k = 0; k < BF_NR; k++)
        if (!(k & (1 << TGT))) bf_rot_pair<T>(v[k], v[k | (1 << TGT)], r, nr, s, ns);
}

// [[p, w], [-conj w, p]], w = r + i s, on register bit TGT: for p too small to divide by
template <typename T, int TGT>
SVB_HD void bf_srot(BfUnit<T>* v, typename BfScalar<T>::S p, typename BfScalar<T>::S r, typename BfScalar<T>::S s)
{
    using B = BfScalar<T>;
    const typename B::S nr = B::neg(r), ns = B::neg(s);
#pragma unroll
    for (int k = 0; k < BF_NR; k++)
        if (!(k & (1 << TGT))) bf_srot_pair<T>(v[k], v[k | (1 << TGT)], p, r, nr, s, ns);
}

// CX from register bit (or packed half) CTL on register bit TGT, or on the packed half
template <typename T, int TGT, int CTL>
SVB_HD void bf_cx_regs(BfUnit<T>* v)
{
#pragma unroll
    for (int k = 0; k < BF_NR; k++) {
        if constexpr (TGT == BF_PACK) {
            if ((k >> CTL) & 1) bf_swap_halves(v[k]);
        } else {
            if (k & (1 << TGT)) continue;
            if constexpr (CTL == BF_PACK) bf_swap_high(v[k], v[k | (1 << TGT)]);
            else if ((k >> CTL) & 1) bf_exchange<T>(v[k], v[k | (1 << TGT)]);
        }
    }
}

// a complex factor c + i s on every unit whose slot has odd parity of RM; with the packed bit
// (half) on the amplitudes whose slot and half have odd parity together
template <typename T, int RM>
SVB_HD void bf_phase(BfUnit<T>* v, T c, T s, bool half)
{
    using B = BfScalar<T>;
    if (B::packed && half) {
        const typename B::S ce = B::lohi(T(1), c), se = B::lohi(T(0), s);   // even slots: high half
        const typename B::S co = B::lohi(c, T(1)), so = B::lohi(s, T(0));   // odd slots: low half
        const typename B::S nse = B::neg(se), nso = B::neg(so);
#pragma unroll
        for (int k = 0; k < BF_NR; k++) {
            const bool odd = (((k & RM) >> 3) ^ ((k & RM) >> 2) ^ ((k & RM) >> 1) ^ (k & RM)) & 1;
            bf_scale_unit<T>(v[k], odd ? co : ce, odd ? so : se, odd ? nso : nse);
        }
    } else {
        const typename B::S cc = B::dup(c), ss = B::dup(s), ns = B::neg(ss);
#pragma unroll
        for (int k = 0; k < BF_NR; k++) {
            const bool odd = (((k & RM) >> 3) ^ ((k & RM) >> 2) ^ ((k & RM) >> 1) ^ (k & RM)) & 1;
            if (odd) bf_scale_unit<T>(v[k], cc, ss, ns);
        }
    }
}

// register slots' XOR combination of four bit images
template <typename I>
SVB_HD I bf_comb(const I* reg, int k)
{
    I r = 0;
#pragma unroll
    for (int i = 0; i < BF_RB; i++)
        if ((k >> i) & 1) r ^= reg[i];
    return r;
}
template <typename I>
SVB_HD I bf_thr(const I* thr, int tid)
{
    I r = 0;
#pragma unroll
    for (int b = 0; b < BF_TB; b++)
        if ((tid >> b) & 1) r ^= thr[b];
    return r;
}

SVB_HD int bf_parity(uint32_t x)
{
#ifdef __CUDA_ARCH__
    return __popc(x) & 1;
#else
    return __builtin_popcount(x) & 1;
#endif
}
SVB_HD int bf_parity64(uint64_t x) { return bf_parity((uint32_t)x ^ (uint32_t)(x >> 32)); }

// A thread's pending factors, in FP64 for either precision and in shared memory, so that the
// gates have the registers: `own` collects the phases that are the same for all of the
// thread's units and is multiplied in before they leave it (BF_FLUSH); `run` the factor on
// the odd slots of a run of phases over one register mask, multiplied in at the run's end.
struct BfPhase {
    double2 own, run;
};

SVB_HD double2 bf_cmul(double2 a, double c, double s) { return make_double2(a.x * c - a.y * s, a.x * s + a.y * c); }

#define SVB_BF_CX(t, c) \
    case (t) * 8 + (c): bf_cx_regs<T, t, c>(v); break;

template <typename T>
SVB_HD void bf_cx_op(int tgt, int ctl, BfUnit<T>* v)
{
    if constexpr (BfScalar<T>::packed) {
        switch (tgt * 8 + ctl) {
        SVB_BF_CX(0, 4) SVB_BF_CX(1, 4) SVB_BF_CX(2, 4) SVB_BF_CX(3, 4)
        SVB_BF_CX(4, 0) SVB_BF_CX(4, 1) SVB_BF_CX(4, 2) SVB_BF_CX(4, 3)
        default: break;
        }
    }
    switch (tgt * 8 + ctl) {
    SVB_BF_CX(0, 1) SVB_BF_CX(0, 2) SVB_BF_CX(0, 3)
    SVB_BF_CX(1, 0) SVB_BF_CX(1, 2) SVB_BF_CX(1, 3)
    SVB_BF_CX(2, 0) SVB_BF_CX(2, 1) SVB_BF_CX(2, 3)
    SVB_BF_CX(3, 0) SVB_BF_CX(3, 1) SVB_BF_CX(3, 2)
    default: break;
    }
}

SVB_HD void bf_coef(const BfOp& op, int flip, double& r, double& s)
{
    r = flip ? -op.d[0] : op.d[0];
    s = op.d[1];
}
SVB_HD void bf_coef(const BfOp& op, int flip, float& r, float& s)
{
    r = flip ? -op.f[0] : op.f[0];
    s = op.f[1];
}

// A gate on a register bit (BF_ROT).
template <typename T>
SVB_HD void bf_apply_rot(const BfOp& op, BfUnit<T>* v, int tid, uint64_t tiles)
{
    using B = BfScalar<T>;
    const int flip = (bf_parity(op.thr_mask & (uint32_t)tid) ^ (int)(tiles >> op.tile_bit)) & 1;
    T r1, s1;
    bf_coef(op, flip, r1, s1);
    const typename B::S r = B::dup(r1), s = B::dup(s1);
    switch (op.tgt) {
    case 0: bf_rot<T, 0>(v, r, s); break;
    case 1: bf_rot<T, 1>(v, r, s); break;
    case 2: bf_rot<T, 2>(v, r, s); break;
    default: bf_rot<T, 3>(v, r, s); break;
    }
}

// Any other op that needs no other thread (everything but BF_RELAYOUT).  tiles: bit i is the
// parity of the pass's tile mask i on this tile.
template <typename T>
SVB_HD void bf_apply(const BfOp& op, const T* coefs, BfUnit<T>* v, BfPhase* ph, int tid, uint64_t tiles)
{
    using B = BfScalar<T>;
    const int flip = (bf_parity(op.thr_mask & (uint32_t)tid) ^ (int)(tiles >> op.tile_bit)) & 1;
    const int tgt = op.tgt;
    const T* m = coefs + op.coef;
    switch (op.kind) {
    case BF_PROT:
        if constexpr (B::packed) {
            T r1, s1;
            bf_coef(op, flip, r1, s1);
            const F2 er = f2_make(r1, -r1), ei = B::dup(s1), nei = B::neg(ei);
#pragma unroll
            for (int k = 0; k < BF_NR; k++) bf_half_rot(v[k], er, ei, nei);
        }
        break;
    case BF_SROT: {
        T r1, s1;
        bf_coef(op, flip, r1, s1);
        const typename B::S p = B::dup(m[0]), r = B::dup(r1), s = B::dup(s1);
        switch (tgt) {
        case 0: bf_srot<T, 0>(v, p, r, s); break;
        case 1: bf_srot<T, 1>(v, p, r, s); break;
        case 2: bf_srot<T, 2>(v, p, r, s); break;
        case 3: bf_srot<T, 3>(v, p, r, s); break;
        default:
            if constexpr (B::packed) {
                const F2 er = f2_make(r1, -r1);
#pragma unroll
                for (int k = 0; k < BF_NR; k++) bf_half_srot(v[k], p, er, s, B::neg(s));
            }
            break;
        }
        break;
    }
    case BF_CX:
        bf_cx_op<T>(tgt, op.ctl, v);
        break;
    case BF_DIAG: {
        // d_{parity} = d_flip on the even slots and d_{1-flip} on the odd ones: d_flip on the
        // whole thread, and the ratio (both have modulus 1) on the odd slots
        const double* d = reinterpret_cast<const double*>(m);
        const double fc = flip ? d[2] : d[0], fs = flip ? d[3] : d[1];
        ph->own = bf_cmul(ph->own, fc, fs);
        if (op.rmask == 0) break;
        const double oc = flip ? d[0] : d[2], os = flip ? d[1] : d[3];
        double2 h = make_double2(oc * fc + os * fs, os * fc - oc * fs);
        if (!(op.run & 1)) h = bf_cmul(h, ph->run.x, ph->run.y);
        if (!(op.run & 2)) {
            ph->run = h;
            break;
        }
        const T c = (T)h.x, s = (T)h.y;
        const bool half = (op.rmask >> BF_PACK) & 1;
        switch (op.rmask & (BF_NR - 1)) {
        case 0: bf_phase<T, 0>(v, c, s, half); break;
        case 1: bf_phase<T, 1>(v, c, s, half); break;
        case 2: bf_phase<T, 2>(v, c, s, half); break;
        case 3: bf_phase<T, 3>(v, c, s, half); break;
        case 4: bf_phase<T, 4>(v, c, s, half); break;
        case 5: bf_phase<T, 5>(v, c, s, half); break;
        case 6: bf_phase<T, 6>(v, c, s, half); break;
        case 8: bf_phase<T, 8>(v, c, s, half); break;
        case 9: bf_phase<T, 9>(v, c, s, half); break;
        case 10: bf_phase<T, 10>(v, c, s, half); break;
        case 12: bf_phase<T, 12>(v, c, s, half); break;
        default: break;                  // the planner makes no phase over more register bits
        }
        break;
    }
    case BF_FLUSH: {
        const typename B::S c = B::dup((T)ph->own.x), s = B::dup((T)ph->own.y), ns = B::neg(s);
#pragma unroll
        for (int k = 0; k < BF_NR; k++) bf_scale_unit<T>(v[k], c, s, ns);
        ph->own = make_double2(1.0, 0.0);
        break;
    }
    case BF_PFIX:
        if (B::packed && flip) {
#pragma unroll
            for (int k = 0; k < BF_NR; k++) bf_swap_halves(v[k]);
        }
        break;
    default:
        break;
    }
}

#undef SVB_BF_CX
#ifdef __CUDA_ARCH__
#undef SVB_BF_ASM
#endif

}  // namespace svb
