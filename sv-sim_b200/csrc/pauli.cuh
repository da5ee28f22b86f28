// Pauli-sum observables over a state in global memory: a thread's share of
// Re <psi| sum_t c_t P_t |psi>, and of (sum_t c_t P_t) |psi>.
//
// A term reads the amplitude at i ^ x_mask.  What bounds a plain loop (one amplitude, all
// terms, one after the other) is the latency of those reads: 7.8 ms for 64 states of 20
// qubits and 40 terms, where reading the states takes 0.2.  Here a thread takes PAULI_U
// amplitudes through the terms together, so that as many reads are in flight; terms without
// X or Y read nothing (their signs add up to one factor on |a|^2); and of the two equal
// contributions of a pair (i, i ^ x_mask) to the energy one is computed.
//
// That takes enough amplitudes to fill the chip with a quarter of the threads, and enough terms
// to pay for the amplitudes of its four: pauli_by_four.  Below, one amplitude with the terms
// in a loop without a branch, whose loads the compiler moves ahead, is the faster form.
// Kernel times of one state, 1 / four amplitudes in us: 300 random strings on 10, 16, 18, 19, 20,
// 26 qubits 38 / 77, 77 / 129, 167 / 222, 314 / 269, 579 / 483, 70,900 / 38,700; one X on 19,
// 22, 24 qubits 4.7 / 6.6, 14.6 / 17.1, 70 / 75, five strings on 19, 20, 22 qubits 9.1 / 10.5,
// 14.8 / 14.8, 48 / 39.  Batches, where a warp takes a chunk, the whole call: 64 states of 4, 8,
// 12 qubits and 300 strings 109 / 167, 661 / 343, 14,900 / 5,100.
#pragma once

#include "gate_math.cuh"

namespace svb {

constexpr int PAULI_U = 4;

__device__ __forceinline__ double pauli_signed(double c, uint64_t bits)
{
    return (__popcll(bits) & 1) ? -c : c;
}

constexpr int PAULI_FEW = 4;             // terms
constexpr int PAULI_STATE_BITS = 19, PAULI_APPLY_BITS = 17, PAULI_CHUNK_BITS = 8;
// bits: the state's size from which on a whole state, resp. a warp's chunk, has amplitudes enough
__host__ __device__ constexpr bool pauli_by_four(uint64_t dim, int n_terms, int bits)
{
    return n_terms >= PAULI_FEW && dim >= 1ull << bits;
}

// (P psi)[i] from the amplitude b at j = i ^ x_mask
__device__ __forceinline__ double2 pauli_image(double br, double bi, uint64_t j, uint64_t xm, uint64_t zm)
{
    if (__popcll(j & zm) & 1) { br = -br; bi = -bi; }
    switch (__popcll(xm & zm) & 3) {         // i^(number of Y factors)
    case 0: return make_double2(br, bi);
    case 1: return make_double2(-bi, br);
    case 2: return make_double2(-br, -bi);
    default: return make_double2(bi, -br);
    }
}

// amplitude i's part of the energy
template <typename T>
__device__ __forceinline__ double pauli_energy_one(const typename VecOf<T>::type* sv, uint64_t i,
                                                   const svb_pauli_term* terms, int n_terms)
{
    const auto a = sv[i];
    const double ar = (double)a.x, ai = (double)a.y;
    double acc = 0.0;
    for (int t = 0; t < n_terms; t++) {
        const svb_pauli_term P = terms[t];
        const uint64_t j = i ^ P.x_mask;
        const auto b = sv[j];
        const double2 p = pauli_image((double)b.x, (double)b.y, j, P.x_mask, P.z_mask);
        acc += P.coef * (ar * p.x + ai * p.y);
    }
    return acc;
}

// (sum_t c_t P_t psi)[i]
__device__ __forceinline__ double2 pauli_apply_one(const double2* __restrict__ psi, uint64_t i,
                                                   const svb_pauli_term* terms, int n_terms)
{
    double2 acc = make_double2(0.0, 0.0);
    for (int t = 0; t < n_terms; t++) {
        const uint64_t xm = terms[t].x_mask, j = i ^ xm;
        const double2 b = psi[j], p = pauli_image(b.x, b.y, j, xm, terms[t].z_mask);
        acc.x += terms[t].coef * p.x;
        acc.y += terms[t].coef * p.y;
    }
    return acc;
}

// amplitudes first, first + step, ... (PAULI_U of them, those below end); terms in shared or
// global memory
template <typename T>
__device__ __forceinline__ double pauli_energy(const typename VecOf<T>::type* __restrict__ sv, uint64_t first,
                                               uint64_t step, uint64_t end, const svb_pauli_term* terms, int n_terms)
{
    double ar[PAULI_U], ai[PAULI_U], diag[PAULI_U], acc = 0.0;
#pragma unroll
    for (int u = 0; u < PAULI_U; u++) {
        const uint64_t i = first + u * step;
        const auto a = sv[i < end ? i : 0];
        ar[u] = i < end ? (double)a.x : 0.0;
        ai[u] = i < end ? (double)a.y : 0.0;
        diag[u] = 0.0;
    }
    for (int t = 0; t < n_terms; t++) {
        const double c = terms[t].coef;
        const uint64_t xm = terms[t].x_mask, zm = terms[t].z_mask;
        if (xm == 0) {
#pragma unroll
            for (int u = 0; u < PAULI_U; u++) diag[u] += pauli_signed(c, (first + u * step) & zm);
            continue;
        }
        const uint64_t top = 1ull << (63 - __clzll((long long)xm));
        const int ny = __popcll(xm & zm) & 3;
        double br[PAULI_U], bi[PAULI_U];
        bool on[PAULI_U];
#pragma unroll
        for (int u = 0; u < PAULI_U; u++) {
            const uint64_t i = first + u * step;
            on[u] = i < end && !(i & top);
            if (on[u]) {
                const auto b = sv[i ^ xm];
                br[u] = (double)b.x;
                bi[u] = (double)b.y;
            }
        }
#pragma unroll
        for (int u = 0; u < PAULI_U; u++) {
            if (!on[u]) continue;
            // i^ny times b, then its product with conj(a): real part
            double v = (ny & 1) ? ai[u] * br[u] - ar[u] * bi[u] : ar[u] * br[u] + ai[u] * bi[u];
            if (ny & 2) v = -v;
            acc += pauli_signed(2.0 * c, ((first + u * step) ^ xm) & zm) * v;
        }
    }
#pragma unroll
    for (int u = 0; u < PAULI_U; u++)       // 0 without Z strings, also where |a|^2 is no double
        acc += diag[u] * ar[u] * ar[u] + diag[u] * ai[u] * ai[u];
    return acc;
}

// out[i] = (sum_t c_t P_t psi)[i] at the same amplitudes
__device__ __forceinline__ void pauli_apply(const double2* __restrict__ psi, double2* __restrict__ out, uint64_t first,
                                            uint64_t step, uint64_t end, const svb_pauli_term* terms, int n_terms)
{
    double re[PAULI_U], im[PAULI_U], diag[PAULI_U];
#pragma unroll
    for (int u = 0; u < PAULI_U; u++) re[u] = im[u] = diag[u] = 0.0;
    for (int t = 0; t < n_terms; t++) {
        const double c = terms[t].coef;
        const uint64_t xm = terms[t].x_mask, zm = terms[t].z_mask;
        if (xm == 0) {
#pragma unroll
            for (int u = 0; u < PAULI_U; u++) diag[u] += pauli_signed(c, (first + u * step) & zm);
            continue;
        }
        const int ny = __popcll(xm & zm) & 3;
        double2 b[PAULI_U];
#pragma unroll
        for (int u = 0; u < PAULI_U; u++) {
            const uint64_t i = first + u * step;
            b[u] = psi[i < end ? i ^ xm : 0];
        }
#pragma unroll
        for (int u = 0; u < PAULI_U; u++) {
            double s = pauli_signed(c, ((first + u * step) ^ xm) & zm);
            if (ny & 2) s = -s;
            re[u] += s * ((ny & 1) ? -b[u].y : b[u].x);
            im[u] += s * ((ny & 1) ? b[u].x : b[u].y);
        }
    }
#pragma unroll
    for (int u = 0; u < PAULI_U; u++) {
        const uint64_t i = first + u * step;
        if (i >= end) continue;
        const double2 a = psi[i];
        out[i] = make_double2(re[u] + diag[u] * a.x, im[u] + diag[u] * a.y);
    }
}

}  // namespace svb
