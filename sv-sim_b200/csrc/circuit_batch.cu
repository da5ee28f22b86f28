// Batched circuits (no counterpart in the reference): many independent circuits, each on
// its own state of n_i qubits (any mix of sizes up to 24), run from |0..0> by one
// persistent cooperative launch that a CUDA graph replays, with an optional Pauli-sum
// energy per circuit.  The reference runs one circuit per Simulation and one launch per
// sim() (svsim_nvgpu_sin.cuh:306-339) with a fixed launch shape (:309-316, config.hpp:48);
// here the tile size and block size are chosen per batch by timing candidates (the
// autotuner below).
//
// Plan.  Each circuit is lowered to the reference's elementary ops (lower.cpp).  A circuit
// of n <= MB qubits is one tile holding its whole state: all its ops in one pass.  Larger
// circuits are cut into passes of MB local qubits by the shared pass cut (select_passes):
// dense and CX targets are local; a diagonal op or a CX control on a non-local qubit is
// resolved per tile (the qubit's value is fixed across the tile).
//
// Launch.  Phase p processes pass p of every circuit that has one: the work items are
// (circuit, pass, tile), spread over the resident CTAs; phases are separated by a grid
// barrier whose wait is bounded (an error flag, then the host reports the failure).  A CTA
// loads its tile into shared memory (gather through two offset tables per pass), applies
// the pass's ops in order with one sweep over the tile each, and writes the tile back.
// After the last phase, each circuit's energy sum_t c_t Re <psi| P_t |psi> is summed per
// chunk of 4,096 amplitudes by one warp each and per circuit in a fixed order (FP64,
// repeatable).
//
// FP64 circuits of 12 or more qubits can instead run on the pair engine's machinery
// (pairs_core.cuh): each is planned by plan_pairs (two-qubit blocks on the FP64 tensor
// cores, 4,096-amplitude tiles), the plans are concatenated, and a second persistent
// cooperative launch k_cb_pairs runs phase p = pass p of every such circuit, a CTA taking a
// contiguous run of (circuit, pass, tile) items so that it stages a pass's ops, layouts and
// gate fragments in shared memory once for many tiles.  That launch goes first; the sweep
// launch then runs the other circuits and the energies of all.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <tuple>
#include <vector>

#include "pairs_core.cuh"
#include "pauli.cuh"

namespace svb {
namespace {

constexpr unsigned kCbSpinLimit = 1u << 24;    // x >= 64 ns sleeps: > 1 s per barrier
constexpr int CB_CHUNK = 4096;                 // amplitudes per energy chunk
constexpr int CB_MAX_QUBITS = 24;

struct CbOp {                    // 80 bytes
    uint8_t form;
    uint8_t p;                   // local position of the target (dense, CX) or of a local diagonal qubit
    uint8_t c;                   // CX: local position of a local control
    uint8_t flags;               // 1: the diagonal qubit is non-local; 2: the CX control is non-local
    uint8_t tb;                  // the tile-index bit of that non-local qubit
    uint8_t pad[3];
    double m[8];
    uint64_t pad2;
};
static_assert(sizeof(CbOp) == 80, "CbOp layout");

struct CbPass {
    uint64_t g_lo[64];           // local index bits 0..5 -> offset in the circuit's state
    uint64_t g_hi[128];          // local index bits 6..12 -> offset
    uint8_t nonlocal_q[64];      // tile-index bit j -> qubit
    int32_t n_nonlocal, M, op_begin, op_end;
};
static_assert(sizeof(CbPass) % 16 == 0, "CbPass layout");

struct CbCircuit {
    uint64_t state_off;          // first amplitude of the circuit in the pool
    uint32_t n;
    uint32_t term_begin, term_end;
    uint32_t chunk_begin;        // its first energy chunk
};

struct CbItem {
    uint32_t circuit;
    uint32_t pass;
    uint64_t tile;
};

struct CbArgs {
    void* pool;
    const CbCircuit* circ;
    const CbPass* passes;
    const CbOp* ops;
    const CbItem* items;
    const uint32_t* phase_off;   // [n_phases + 1]
    const svb_pauli_term* terms;
    const uint32_t* chunk_circ;  // energy chunk -> circuit
    double* partial;             // [n_chunks]
    double* energy;              // [n_circ]
    unsigned* barrier;           // [0] arrivals (zeroed before each launch), [1] error flag
    int n_phases;
    int n_circ;
    uint32_t n_chunks;
    int pad;
};

svb_status cb_invalid(const std::string& msg)
{
    set_error(msg);
    return SVB_ERR_INVALID;
}

svb_status cb_cuda_fail(cudaError_t e, const char* what)
{
    set_error(std::string(what) + ": " + cudaGetErrorString(e));
    (void)cudaGetLastError();
    return e == cudaErrorMemoryAllocation ? SVB_ERR_OOM : SVB_ERR_CUDA;
}

__device__ __forceinline__ unsigned cb_ld_acquire(const unsigned* p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Grid-wide barrier with a bounded wait (the launch is cooperative, so every block is
// resident and the wait ends; past the limit the error flag is raised and the block goes on).
__device__ __forceinline__ void cb_grid_barrier(unsigned* bar, unsigned target)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(bar, 1u);
        unsigned spins = 0;
        while (cb_ld_acquire(bar) < target) {
            if (++spins > kCbSpinLimit || cb_ld_acquire(bar + 1) != 0u) {
                atomicOr(bar + 1, 1u);
                break;
            }
            __nanosleep(64);
        }
        __threadfence();
    }
    __syncthreads();
}

__device__ __forceinline__ uint32_t insert_zero32(uint32_t x, int b)
{
    return ((x >> b) << (b + 1)) | (x & ((1u << b) - 1u));
}

template <typename T>
__device__ void cb_apply(typename VecOf<T>::type* tile, int M, const CbOp& op, uint64_t tile_index)
{
    const Coef<T> c = load_coef<T>(op.m);
    const uint32_t half = 1u << (M - 1);
    const uint32_t pd = 1u << op.p;
    if (op.form == F_CX) {
        if ((op.flags & 2) && !((tile_index >> op.tb) & 1ull)) return;
        for (uint32_t t = threadIdx.x; t < half; t += blockDim.x) {
            const uint32_t l0 = insert_zero32(t, op.p);
            if (!(op.flags & 2) && !((l0 >> op.c) & 1u)) continue;
            const auto a = tile[l0];
            tile[l0] = tile[l0 | pd];
            tile[l0 | pd] = a;
        }
    } else if (form_is_diag(op.form)) {
        if (op.flags & 1) {              // the qubit is fixed across the tile
            const bool one = (tile_index >> op.tb) & 1ull;
            if (!one && op.form != F_DIAG) return;
            for (uint32_t l = threadIdx.x; l < 2 * half; l += blockDim.x) {
                if (one) diag_one<T>(op.form, c, tile[l]);
                else diag_zero<T>(op.form, c, tile[l]);
            }
        } else {
            for (uint32_t t = threadIdx.x; t < half; t += blockDim.x) {
                const uint32_t l0 = insert_zero32(t, op.p);
                diag_one<T>(op.form, c, tile[l0 | pd]);
                if (op.form == F_DIAG) diag_zero<T>(op.form, c, tile[l0]);
            }
        }
    } else {
        for (uint32_t t = threadIdx.x; t < half; t += blockDim.x) {
            const uint32_t l0 = insert_zero32(t, op.p);
            dense_pair<T>(op.form, c, tile[l0], tile[l0 | pd]);
        }
    }
}

__device__ __forceinline__ double cb_warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// partial energies, one warp per chunk
template <typename T, bool FOUR>
__device__ __forceinline__ void cb_chunk_energies(const CbArgs& A)
{
    using V = typename VecOf<T>::type;
    const int lane = threadIdx.x & 31;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < A.n_chunks; k += warps) {
        const CbCircuit C = A.circ[A.chunk_circ[k]];
        const uint64_t dim = 1ull << C.n;
        const uint64_t start = (uint64_t)(k - C.chunk_begin) * CB_CHUNK;
        const uint64_t end = start + CB_CHUNK < dim ? start + CB_CHUNK : dim;
        const V* sv = static_cast<const V*>(A.pool) + C.state_off;
        const svb_pauli_term* terms = A.terms + C.term_begin;
        const int n_terms = (int)(C.term_end - C.term_begin);
        double acc = 0.0;
        if (FOUR && pauli_by_four(dim, n_terms, PAULI_CHUNK_BITS))
            for (uint64_t i = start + lane; i < end; i += 32 * PAULI_U)
                acc += pauli_energy<T>(sv, i, 32, end, terms, n_terms);
        else
            for (uint64_t i = start + lane; i < end; i += 32) acc += pauli_energy_one<T>(sv, i, terms, n_terms);
        acc = cb_warp_sum(acc);
        if (lane == 0) A.partial[k] = acc;
    }
}

// one warp per circuit over its chunks in order
__device__ __forceinline__ void cb_sum_energies(const CbArgs& A)
{
    const int lane = threadIdx.x & 31;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < (uint32_t)A.n_circ; c += warps) {
        const CbCircuit C = A.circ[c];
        if (C.term_end == C.term_begin) {
            if (lane == 0) A.energy[c] = 0.0;
            continue;
        }
        const uint64_t nch = ((1ull << C.n) + CB_CHUNK - 1) / CB_CHUNK;
        double s = 0.0;
        for (uint64_t k = lane; k < nch; k += 32) s += A.partial[C.chunk_begin + k];
        s = cb_warp_sum(s);
        if (lane == 0) A.energy[c] = s;
    }
}

template <typename T>
__global__ void __launch_bounds__(512) k_cbatch(CbArgs A)
{
    using V = typename VecOf<T>::type;
    extern __shared__ __align__(16) unsigned char cb_smem[];
    CbPass* sp = reinterpret_cast<CbPass*>(cb_smem);
    V* tile = reinterpret_cast<V*>(cb_smem + sizeof(CbPass));
    __shared__ int cur_pass;
    V* pool = static_cast<V*>(A.pool);
    if (threadIdx.x == 0) cur_pass = -1;
    __syncthreads();
    unsigned target = 0;
    for (int ph = 0; ph < A.n_phases; ph++) {
        for (uint32_t it = A.phase_off[ph] + blockIdx.x; it < A.phase_off[ph + 1]; it += gridDim.x) {
            const CbItem item = A.items[it];
            if ((int)item.pass != cur_pass) {
                const uint4* src = reinterpret_cast<const uint4*>(A.passes + item.pass);
                uint4* dst = reinterpret_cast<uint4*>(sp);
                for (int w = threadIdx.x; w < (int)(sizeof(CbPass) / 16); w += blockDim.x) dst[w] = src[w];
                __syncthreads();
                if (threadIdx.x == 0) cur_pass = (int)item.pass;
            }
            const CbCircuit C = A.circ[item.circuit];
            const int M = sp->M;
            const uint32_t TL = 1u << M;
            // the tile's offset within the circuit's state (state_off is not aligned to 2^n)
            uint64_t off = 0;
            for (int j = 0; j < sp->n_nonlocal; j++) off |= ((item.tile >> j) & 1ull) << sp->nonlocal_q[j];
            const uint64_t base = C.state_off + off;
            for (uint32_t l = threadIdx.x; l < TL; l += blockDim.x) tile[l] = pool[base + sp->g_lo[l & 63u] + sp->g_hi[l >> 6]];
            __syncthreads();
            for (int o = sp->op_begin; o < sp->op_end; o++) {
                const CbOp op = A.ops[o];
                cb_apply<T>(tile, M, op, item.tile);
                __syncthreads();
            }
            for (uint32_t l = threadIdx.x; l < TL; l += blockDim.x) pool[base + sp->g_lo[l & 63u] + sp->g_hi[l >> 6]] = tile[l];
            __syncthreads();
        }
        target += gridDim.x;
        cb_grid_barrier(A.barrier, target);
    }
    if (A.n_chunks == 0) return;
    cb_chunk_energies<T, false>(A);
    target += gridDim.x;
    cb_grid_barrier(A.barrier, target);
    cb_sum_energies(A);
}

// The energies of a batch in which some circuit's go four amplitudes at a time, after k_cbatch
// (which then has no chunks): in one kernel with the passes that form's registers (84 instead of
// 50) halved the CTAs an SM held during the passes (512 circuits of 14 qubits, a layer and one
// string each: 0.80 -> 1.15 ms).
template <typename T>
__global__ void __launch_bounds__(256) k_cb_energies(CbArgs A)
{
    cb_chunk_energies<T, true>(A);
}
__global__ void __launch_bounds__(256) k_cb_energy_sums(CbArgs A)
{
    cb_sum_energies(A);
}

template <typename T>
__global__ void k_cb_ones(void* pool, const CbCircuit* circ, int n_circ)
{
    using V = typename VecOf<T>::type;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n_circ; c += gridDim.x * blockDim.x) {
        V one;
        one.x = 1;
        one.y = 0;
        static_cast<V*>(pool)[circ[c].state_off] = one;
    }
}

struct CbPairArgs {
    double2* pool;
    const CbCircuit* circ;
    const PairPass* passes;
    const PairOp* ops;
    const DevStage* layouts;
    const double2* gates;
    const CbItem* items;
    const uint32_t* phase_off;   // [n_phases + 1]
    unsigned* barrier;           // [0] arrivals (zeroed before each launch), [1] error flag
    int n_phases;
    int pad;
};

// Phase p runs pass p of every pair-planned circuit.  The items of a phase are ordered by
// circuit and tile, and each CTA takes a contiguous share of them, so it changes pass (and
// stages the new pass's data) at most a few times per phase.
__global__ void __launch_bounds__(PR_THREADS, 2) k_cb_pairs(CbPairArgs A)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* sm = reinterpret_cast<double2*>(smem_raw);
    __shared__ PairPass sP;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    int cur = -1;
    PairStaged S{};
    PairGOffs gin{}, gout{};
    unsigned target = 0;
    for (int ph = 0; ph < A.n_phases; ph++) {
        const uint32_t lo = A.phase_off[ph];
        const uint64_t cnt = A.phase_off[ph + 1] - lo;
        const uint32_t b0 = lo + (uint32_t)(cnt * blockIdx.x / gridDim.x);
        const uint32_t b1 = lo + (uint32_t)(cnt * (blockIdx.x + 1) / gridDim.x);
        for (uint32_t it = b0; it < b1; it++) {
            const CbItem item = A.items[it];
            if ((int)item.pass != cur) {
                __syncthreads();       // every thread is done with the previous pass's data
                const uint32_t* src = reinterpret_cast<const uint32_t*>(A.passes + item.pass);
                uint32_t* dst = reinterpret_cast<uint32_t*>(&sP);
                for (int w = tid; w < (int)(sizeof(PairPass) / 4); w += PR_THREADS) dst[w] = src[w];
                __syncthreads();
                S = pair_stage(smem_raw, sP, A.ops, A.layouts, A.gates, tid);
                pair_goffs(S.lay[0], sP.local_q, tid, gin);
                pair_goffs(S.lay[S.n_lay - 1], sP.local_q, tid, gout);
                cur = (int)item.pass;
            }
            pair_tile(A.pool + A.circ[item.circuit].state_off, sm, sP, S, gin, gout, item.tile, tid, lane);
        }
        target += gridDim.x;
        cb_grid_barrier(A.barrier, target);
    }
}

// ---- host side ----------------------------------------------------------------------

// The pair-engine part of a batch plan: the circuits' pair plans concatenated (indices
// rebased), and the (circuit, pass, tile) items of each phase.
struct CbPairPlan {
    std::vector<PairPass> passes;
    std::vector<PairOp> ops;
    std::vector<DevStage> layouts;
    std::vector<double> gates;
    std::vector<CbItem> items;
    std::vector<uint32_t> phase_off;
    size_t stage_bytes = 0;
    uint32_t circuits = 0;
    std::vector<PairPlan> each;          // the circuits' own plans, without their gates
    std::vector<size_t> gate_at;         // where each one's gates begin
};

struct CbPlan {
    std::vector<CbCircuit> circ;
    std::vector<CbPass> passes;
    std::vector<CbOp> ops;
    std::vector<CbItem> items;
    std::vector<uint32_t> phase_off;
    std::vector<uint32_t> chunk_circ;
    bool by_four = false;                // energies by k_cb_energies
    uint64_t pool_amps = 0;
    double moved_bytes = 0;
    CbPairPlan pairs;
};

CbPass make_pass(uint64_t L, int n)
{
    CbPass P;
    std::memset(&P, 0, sizeof(P));
    int local_q[64], nl = 0, nn = 0;
    for (int q = 0; q < n; q++) {
        if ((L >> q) & 1ull) local_q[nl++] = q;
        else P.nonlocal_q[nn++] = (uint8_t)q;
    }
    P.n_nonlocal = nn;
    P.M = nl;
    for (int j = 0; j < 64; j++)
        for (int b = 0; b < 6 && b < nl; b++)
            if ((j >> b) & 1) P.g_lo[j] |= 1ull << local_q[b];
    for (int j = 0; j < 128; j++)
        for (int b = 0; b < 7 && 6 + b < nl; b++)
            if ((j >> b) & 1) P.g_hi[j] |= 1ull << local_q[6 + b];
    return P;
}

// Appends circuit ops `taken` (indices into eops) as one pass over local mask L.
void emit_pass(CbPlan& plan, const std::vector<EOp>& eops, const std::vector<int>& taken, uint64_t L, int n)
{
    CbPass P = make_pass(L, n);
    int pos[64], tbit[64];
    for (int q = 0; q < 64; q++) pos[q] = tbit[q] = -1;
    int nl = 0;
    for (int q = 0; q < n; q++)
        if ((L >> q) & 1ull) pos[q] = nl++;
    for (int j = 0; j < P.n_nonlocal; j++) tbit[P.nonlocal_q[j]] = j;
    P.op_begin = (int32_t)plan.ops.size();
    for (int i : taken) {
        const EOp& e = eops[i];
        CbOp o;
        std::memset(&o, 0, sizeof(o));
        o.form = e.form;
        std::memcpy(o.m, e.m, sizeof(o.m));
        if (e.form == F_CX) {
            o.p = (uint8_t)pos[e.q];
            if (pos[e.c] >= 0) o.c = (uint8_t)pos[e.c];
            else { o.flags |= 2; o.tb = (uint8_t)tbit[e.c]; }
        } else if (form_is_diag(e.form)) {
            if (pos[e.q] >= 0) o.p = (uint8_t)pos[e.q];
            else { o.flags |= 1; o.tb = (uint8_t)tbit[e.q]; }
        } else {
            o.p = (uint8_t)pos[e.q];
        }
        plan.ops.push_back(o);
    }
    P.op_end = (int32_t)plan.ops.size();
    plan.passes.push_back(P);
}

}  // namespace
}  // namespace svb

struct svb_circuit_batch {
    int device = 0;
    int precision = SVB_FP64;
    uint32_t n_circ = 0;
    int tile_bits = 12;
    int threads = 512;
    bool use_pairs = false;      // pair engine for the FP64 circuits of >= 12 qubits
    bool tuned = false;
    std::vector<uint32_t> n;
    std::vector<uint64_t> gate_off;
    std::vector<svb_gate> gates;
    std::vector<uint64_t> term_off;
    std::vector<svb_pauli_term> terms;
    svb::CbPlan plan;
    // device
    void* pool = nullptr;
    svb::CbCircuit* d_circ = nullptr;
    svb::CbPass* d_passes = nullptr;
    svb::CbOp* d_ops = nullptr;
    svb::CbItem* d_items = nullptr;
    uint32_t* d_phase_off = nullptr;
    svb_pauli_term* d_terms = nullptr;
    uint32_t* d_chunk_circ = nullptr;
    double* d_partial = nullptr;
    double* d_energy = nullptr;
    unsigned* d_bar = nullptr;   // [0, 1] the sweep launch's barrier, [2, 3] the pair launch's
    svb::PairPass* d_ppasses = nullptr;
    svb::PairOp* d_pops = nullptr;
    svb::DevStage* d_playouts = nullptr;
    double* d_pgates = nullptr;
    svb::CbItem* d_pitems = nullptr;
    uint32_t* d_pphase_off = nullptr;
    // pinned host
    svb::CbOp* h_ops = nullptr;
    double* h_pgates = nullptr;
    double* h_energy = nullptr;
    unsigned* h_err = nullptr;   // the 4 barrier words after a run
    cudaStream_t stream = nullptr;
    cudaGraphExec_t graph = nullptr;
    bool graphed = false;
    unsigned grid = 0;
    size_t smem = 0;
    unsigned pgrid = 0;
    size_t psmem = 0;
};

namespace svb {
namespace {

void cb_free(svb_circuit_batch* b)
{
    if (!b) return;
    if (b->graph) cudaGraphExecDestroy(b->graph);
    if (b->stream) cudaStreamDestroy(b->stream);
    cudaFree(b->pool);
    cudaFree(b->d_circ);
    cudaFree(b->d_passes);
    cudaFree(b->d_ops);
    cudaFree(b->d_items);
    cudaFree(b->d_phase_off);
    cudaFree(b->d_terms);
    cudaFree(b->d_chunk_circ);
    cudaFree(b->d_partial);
    cudaFree(b->d_energy);
    cudaFree(b->d_bar);
    cudaFree(b->d_ppasses);
    cudaFree(b->d_pops);
    cudaFree(b->d_playouts);
    cudaFree(b->d_pgates);
    cudaFree(b->d_pitems);
    cudaFree(b->d_pphase_off);
    cudaFreeHost(b->h_ops);
    cudaFreeHost(b->h_pgates);
    cudaFreeHost(b->h_energy);
    cudaFreeHost(b->h_err);
    delete b;
}

// Runs f(i) for i in [0, count) on up to 16 host threads.
template <typename F>
void cb_parallel_for(size_t count, F&& f)
{
    const size_t hw = std::max<size_t>(1, std::thread::hardware_concurrency());
    const size_t nt = std::min<size_t>({hw, (size_t)16, count});
    if (nt <= 1) {
        for (size_t i = 0; i < count; i++) f(i);
        return;
    }
    std::vector<std::thread> pool;
    for (size_t t = 0; t < nt; t++)
        pool.emplace_back([&, t] {
            for (size_t i = t; i < count; i += nt) f(i);
        });
    for (auto& th : pool) th.join();
}

// Appends circuit c's pair plan to the batch's (indices rebased) and its items per phase;
// false (nothing appended) when the concatenated layouts would outgrow the 16-bit indices.
bool cb_append_pairs(CbPairPlan& P, const PairPlan& pp, uint32_t c, int n,
                     std::vector<std::vector<CbItem>>& phase_items)
{
    const size_t op0 = P.ops.size(), lay0 = P.layouts.size(), g0 = P.gates.size() / 64, pass0 = P.passes.size();
    if (lay0 + pp.layouts.size() > 65535) return false;
    for (PairPass Q : pp.passes) {
        Q.op_begin += (int32_t)op0;
        Q.op_end += (int32_t)op0;
        Q.load_layout += (int32_t)lay0;
        Q.store_layout += (int32_t)lay0;
        Q.gate_begin += (int32_t)g0;
        P.passes.push_back(Q);
    }
    for (PairOp o : pp.ops) {
        if (o.kind == PO_BLOCK) o.gate += (uint32_t)g0;
        if (o.kind == PO_RELAYOUT) {
            o.src = (uint16_t)(o.src + lay0);
            o.layout = (uint16_t)(o.layout + lay0);
        }
        P.ops.push_back(o);
    }
    P.layouts.insert(P.layouts.end(), pp.layouts.begin(), pp.layouts.end());
    P.gates.insert(P.gates.end(), pp.gates.begin(), pp.gates.end());
    P.stage_bytes = std::max(P.stage_bytes, pp.stage_bytes);
    P.circuits++;
    const uint64_t tiles = 1ull << (n - PR_TILE_BITS);
    for (size_t k = 0; k < pp.passes.size(); k++) {
        if (phase_items.size() <= k) phase_items.resize(k + 1);
        for (uint64_t t = 0; t < tiles; t++) phase_items[k].push_back(CbItem{c, (uint32_t)(pass0 + k), t});
    }
    return true;
}

// The plan for tile size MB (and, with use_pairs, the pair engine for every FP64 circuit
// of at least 12 qubits that it can run); false (with a message) on an invalid gate.
bool cb_build_plan(const svb_circuit_batch* b, const svb_gate* gates, int MB, bool use_pairs, CbPlan& plan,
                   std::string& err)
{
    plan = CbPlan{};
    const size_t amp = b->precision == SVB_FP64 ? 16 : 8;
    std::vector<std::vector<EOp>> eops(b->n_circ);
    for (uint32_t c = 0; c < b->n_circ; c++) {
        const int n = (int)b->n[c];
        for (uint64_t g = b->gate_off[c]; g < b->gate_off[c + 1]; g++) {
            const svb_gate& gg = gates[g];
            const int slots = gate_qubit_slots(gg.op);
            if (slots == 0) { err = "gate " + std::to_string(g) + ": unknown op"; return false; }
            for (int k = 0; k < slots; k++) {
                if (gg.qb[k] >= (uint32_t)n) {
                    err = "circuit " + std::to_string(c) + ", gate " + std::to_string(g) + ": qubit >= n";
                    return false;
                }
                for (int j = 0; j < k; j++)
                    if (gg.qb[j] == gg.qb[k]) { err = "gate " + std::to_string(g) + " repeats a qubit"; return false; }
            }
            lower_gate(gg, (int32_t)g, eops[c]);
        }
    }
    // pair plans of the eligible circuits (independent: planned on several host threads)
    std::vector<PairPlan> pp(b->n_circ);
    std::vector<char> is_pair(b->n_circ, 0);
    if (use_pairs && b->precision == SVB_FP64) {
        std::vector<uint32_t> cand;
        for (uint32_t c = 0; c < b->n_circ; c++)
            if ((int)b->n[c] >= PR_TILE_BITS) cand.push_back(c);
        cb_parallel_for(cand.size(), [&](size_t i) {
            const uint32_t c = cand[i];
            is_pair[c] = plan_pairs(eops[c], (int)b->n[c], pp[c]) ? 1 : 0;
        });
    }
    std::vector<std::vector<CbItem>> phase_items, pair_items;
    uint32_t chunks = 0;
    for (uint32_t c = 0; c < b->n_circ; c++) {
        const int n = (int)b->n[c];
        CbCircuit C;
        C.state_off = plan.pool_amps;
        C.n = (uint32_t)n;
        C.term_begin = (uint32_t)b->term_off[c];
        C.term_end = (uint32_t)b->term_off[c + 1];
        C.chunk_begin = chunks;
        if (C.term_end > C.term_begin) {
            const uint64_t nch = ((1ull << n) + CB_CHUNK - 1) / CB_CHUNK;
            for (uint64_t k = 0; k < nch; k++) plan.chunk_circ.push_back(c);
            chunks += (uint32_t)nch;
            plan.by_four |= pauli_by_four(1ull << n, (int)(C.term_end - C.term_begin), PAULI_CHUNK_BITS);
        }
        plan.pool_amps += 1ull << n;
        plan.circ.push_back(C);
        const size_t gate_at = plan.pairs.gates.size();
        if (is_pair[c] && cb_append_pairs(plan.pairs, pp[c], c, n, pair_items)) {
            plan.pairs.gate_at.push_back(gate_at);
            pp[c].gates.clear();
            pp[c].gates.shrink_to_fit();
            plan.pairs.each.push_back(std::move(pp[c]));
            plan.moved_bytes += 2.0 * amp * (double)(1ull << n) * (double)plan.pairs.each.back().passes.size();
            continue;
        }
        const int M = std::min(n, MB);
        std::vector<uint32_t> my_passes;
        if (n <= MB) {
            std::vector<int> all(eops[c].size());
            for (size_t i = 0; i < eops[c].size(); i++) all[i] = (int)i;
            my_passes.push_back((uint32_t)plan.passes.size());
            emit_pass(plan, eops[c], all, n >= 64 ? ~0ull : ((1ull << n) - 1), n);
        } else {
            select_passes(eops[c], n, M, std::min(3, M), [&](uint64_t L, const std::vector<int>& taken) {
                my_passes.push_back((uint32_t)plan.passes.size());
                emit_pass(plan, eops[c], taken, L, n);
                return std::vector<int>{};
            });
        }
        const uint64_t tiles = 1ull << (n - M);
        for (size_t p = 0; p < my_passes.size(); p++) {
            if (phase_items.size() <= p) phase_items.resize(p + 1);
            for (uint64_t t = 0; t < tiles; t++) phase_items[p].push_back(CbItem{c, my_passes[p], t});
            plan.moved_bytes += 2.0 * amp * (double)(1ull << n);
        }
    }
    plan.phase_off.push_back(0);
    for (auto& v : phase_items) {
        plan.items.insert(plan.items.end(), v.begin(), v.end());
        plan.phase_off.push_back((uint32_t)plan.items.size());
    }
    plan.pairs.phase_off.push_back(0);
    for (auto& v : pair_items) {
        plan.pairs.items.insert(plan.pairs.items.end(), v.begin(), v.end());
        plan.pairs.phase_off.push_back((uint32_t)plan.pairs.items.size());
    }
    return true;
}

// New angles for a batch whose circuits all run on the pair engine: every circuit lowered and
// planned with the cut its plan was made with, on the host threads, its structure compared
// and its gate fragments copied to the upload buffer.  (Building the whole batch plan again,
// one circuit's lowering after the other, with both cuts of each circuit, its work items and
// three copies of the fragments, took 13 ms of the 44 of 64 circuits of 20 qubits.)  False,
// with nothing changed, if a plan came out different.
bool cb_replan_pairs(svb_circuit_batch* b, const svb_gate* gates)
{
    const CbPairPlan& old = b->plan.pairs;
    std::vector<PairPlan> fresh(b->n_circ);
    std::vector<char> ok(b->n_circ, 0);
    auto same = [](const auto& x, const auto& y) {
        return x.size() == y.size() && (x.empty() || std::memcmp(x.data(), y.data(), x.size() * sizeof(x[0])) == 0);
    };
    cb_parallel_for(b->n_circ, [&](size_t c) {
        std::vector<EOp> eops;
        eops.reserve(2 * (b->gate_off[c + 1] - b->gate_off[c]));
        for (uint64_t g = b->gate_off[c]; g < b->gate_off[c + 1]; g++) lower_gate(gates[g], (int32_t)g, eops);
        const PairPlan& was = old.each[c];
        PairPlan& now = fresh[c];
        const size_t end = c + 1 < b->n_circ ? old.gate_at[c + 1] : old.gates.size();
        ok[c] = plan_pairs_cut(eops, (int)b->n[c], now, nullptr, was.seeds) && same(now.passes, was.passes) &&
                same(now.ops, was.ops) && same(now.layouts, was.layouts) && now.gates.size() == end - old.gate_at[c];
    });
    if (std::find(ok.begin(), ok.end(), 0) != ok.end()) return false;
    cb_parallel_for(b->n_circ, [&](size_t c) {
        if (!fresh[c].gates.empty())
            std::memcpy(b->h_pgates + old.gate_at[c], fresh[c].gates.data(), fresh[c].gates.size() * sizeof(double));
    });
    return true;
}

template <typename T>
cudaError_t cb_launch(svb_circuit_batch* b, cudaStream_t s)
{
    CbArgs a;
    a.pool = b->pool;
    a.circ = b->d_circ;
    a.passes = b->d_passes;
    a.ops = b->d_ops;
    a.items = b->d_items;
    a.phase_off = b->d_phase_off;
    a.terms = b->d_terms;
    a.chunk_circ = b->d_chunk_circ;
    a.partial = b->d_partial;
    a.energy = b->d_energy;
    a.barrier = b->d_bar;
    a.n_phases = (int)b->plan.phase_off.size() - 1;
    a.n_circ = (int)b->n_circ;
    const uint32_t chunks = (uint32_t)b->plan.chunk_circ.size();
    a.n_chunks = b->plan.by_four ? 0 : chunks;
    a.pad = 0;
    void* args[] = {&a};
    cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_cbatch<T>, dim3(b->grid), dim3(b->threads), args, b->smem, s);
    if (e == cudaSuccess && b->plan.by_four) {
        a.n_chunks = chunks;
        k_cb_energies<T><<<std::min<unsigned>((chunks + 7) / 8, 148 * 16), 256, 0, s>>>(a);
        k_cb_energy_sums<<<std::min<unsigned>((b->n_circ + 7) / 8, 148 * 4), 256, 0, s>>>(a);
        e = cudaGetLastError();
    }
    return e;
}

cudaError_t cb_launch_pairs(svb_circuit_batch* b, cudaStream_t s)
{
    CbPairArgs a;
    a.pool = static_cast<double2*>(b->pool);
    a.circ = b->d_circ;
    a.passes = b->d_ppasses;
    a.ops = b->d_pops;
    a.layouts = b->d_playouts;
    a.gates = reinterpret_cast<const double2*>(b->d_pgates);
    a.items = b->d_pitems;
    a.phase_off = b->d_pphase_off;
    a.barrier = b->d_bar + 2;
    a.n_phases = (int)b->plan.pairs.phase_off.size() - 1;
    a.pad = 0;
    void* args[] = {&a};
    return cudaLaunchCooperativeKernel((const void*)k_cb_pairs, dim3(b->pgrid), dim3(PR_THREADS), args, b->psmem, s);
}

// one evaluation: angles in, reset, launches, energies and the error flags out
cudaError_t cb_enqueue(svb_circuit_batch* b, cudaStream_t s)
{
    const size_t amp = b->precision == SVB_FP64 ? 16 : 8;
    const bool pairs = b->plan.pairs.circuits > 0;
    cudaError_t e = cudaSuccess;
    if (!b->plan.ops.empty())
        e = cudaMemcpyAsync(b->d_ops, b->h_ops, b->plan.ops.size() * sizeof(CbOp), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess && pairs && !b->plan.pairs.gates.empty())
        e = cudaMemcpyAsync(b->d_pgates, b->h_pgates, b->plan.pairs.gates.size() * sizeof(double),
                            cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(b->d_bar, 0, 4 * sizeof(unsigned), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(b->pool, 0, b->plan.pool_amps * amp, s);
    if (e == cudaSuccess) {
        const unsigned g = (unsigned)std::min<uint64_t>((b->n_circ + 255) / 256, 1024);
        if (b->precision == SVB_FP64) k_cb_ones<double><<<g, 256, 0, s>>>(b->pool, b->d_circ, (int)b->n_circ);
        else k_cb_ones<float><<<g, 256, 0, s>>>(b->pool, b->d_circ, (int)b->n_circ);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && pairs) e = cb_launch_pairs(b, s);
    if (e == cudaSuccess) e = b->precision == SVB_FP64 ? cb_launch<double>(b, s) : cb_launch<float>(b, s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(b->h_energy, b->d_energy, b->n_circ * sizeof(double), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(b->h_err, b->d_bar, 4 * sizeof(unsigned), cudaMemcpyDeviceToHost, s);
    return e;
}

template <typename Tp>
cudaError_t upload(Tp** dst, const std::vector<Tp>& v, cudaStream_t s)
{
    cudaError_t e = cudaMalloc(dst, std::max<size_t>(1, v.size()) * sizeof(Tp));
    if (e == cudaSuccess && !v.empty())
        e = cudaMemcpyAsync(*dst, v.data(), v.size() * sizeof(Tp), cudaMemcpyHostToDevice, s);
    return e;
}

// Builds a batch with tile size MB, block size `threads` and (use_pairs) the pair engine for
// the circuits it can run: device buffers, graph.
svb_status cb_create_with(svb_circuit_batch* proto, int MB, int threads, bool use_pairs, svb_circuit_batch** out)
{
    svb_circuit_batch* b = new svb_circuit_batch(*proto);
    b->tile_bits = MB;
    b->threads = threads;
    b->use_pairs = use_pairs;
    auto fail = [&](const std::string& what, cudaError_t e) {
        set_error("svb_cbatch_create: " + what + (e != cudaSuccess ? std::string(": ") + cudaGetErrorString(e) : ""));
        (void)cudaGetLastError();
        cb_free(b);
        return e == cudaErrorMemoryAllocation ? SVB_ERR_OOM : (e == cudaSuccess ? SVB_ERR_INVALID : SVB_ERR_CUDA);
    };
    std::string err;
    if (!cb_build_plan(b, b->gates.data(), MB, use_pairs, b->plan, err)) return fail(err, cudaSuccess);
    const size_t amp = b->precision == SVB_FP64 ? 16 : 8;
    // the uploads on the stream that the batch runs on: in order with its first evaluation
    cudaError_t e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMalloc(&b->pool, std::max<uint64_t>(1, b->plan.pool_amps) * amp);
    if (e == cudaSuccess) e = upload(&b->d_circ, b->plan.circ, b->stream);
    if (e == cudaSuccess) e = upload(&b->d_passes, b->plan.passes, b->stream);
    if (e == cudaSuccess) e = upload(&b->d_ops, b->plan.ops, b->stream);
    if (e == cudaSuccess) e = upload(&b->d_items, b->plan.items, b->stream);
    if (e == cudaSuccess) e = upload(&b->d_phase_off, b->plan.phase_off, b->stream);
    if (e == cudaSuccess) e = upload(&b->d_terms, b->terms, b->stream);
    if (e == cudaSuccess) e = upload(&b->d_chunk_circ, b->plan.chunk_circ, b->stream);
    if (e == cudaSuccess) e = cudaMalloc(&b->d_partial, std::max<size_t>(1, b->plan.chunk_circ.size()) * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc(&b->d_energy, std::max<size_t>(1, b->n_circ) * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc(&b->d_bar, 4 * sizeof(unsigned));
    const CbPairPlan& PP = b->plan.pairs;
    if (e == cudaSuccess) e = upload(&b->d_ppasses, PP.passes, b->stream);
    if (e == cudaSuccess) e = upload(&b->d_pops, PP.ops, b->stream);
    if (e == cudaSuccess) e = upload(&b->d_playouts, PP.layouts, b->stream);
    if (e == cudaSuccess) e = upload(&b->d_pgates, PP.gates, b->stream);
    if (e == cudaSuccess) e = upload(&b->d_pitems, PP.items, b->stream);
    if (e == cudaSuccess) e = upload(&b->d_pphase_off, PP.phase_off, b->stream);
    if (e == cudaSuccess) e = cudaMallocHost(&b->h_ops, std::max<size_t>(1, b->plan.ops.size()) * sizeof(CbOp));
    if (e == cudaSuccess) e = cudaMallocHost(&b->h_pgates, std::max<size_t>(1, PP.gates.size()) * sizeof(double));
    if (e == cudaSuccess) e = cudaMallocHost(&b->h_energy, std::max<size_t>(1, b->n_circ) * sizeof(double));
    if (e == cudaSuccess) e = cudaMallocHost(&b->h_err, 4 * sizeof(unsigned));
    if (e != cudaSuccess) return fail("allocation", e);
    if (!b->plan.ops.empty()) std::memcpy(b->h_ops, b->plan.ops.data(), b->plan.ops.size() * sizeof(CbOp));
    if (!PP.gates.empty()) std::memcpy(b->h_pgates, PP.gates.data(), PP.gates.size() * sizeof(double));
    b->smem = sizeof(CbPass) + (amp << MB);
    const void* fn = b->precision == SVB_FP64 ? (const void*)k_cbatch<double> : (const void*)k_cbatch<float>;
    int per_sm = 0, sms = 0;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b->smem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, b->smem);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->device);
    if (e != cudaSuccess || per_sm < 1) return fail("kernel setup", e);
    const uint64_t most = b->plan.items.empty() ? 1 : [&] {
        uint64_t m = 1;
        for (size_t p = 0; p + 1 < b->plan.phase_off.size(); p++)
            m = std::max<uint64_t>(m, b->plan.phase_off[p + 1] - b->plan.phase_off[p]);
        return m;
    }();
    b->grid = (unsigned)std::min<uint64_t>((uint64_t)per_sm * sms, std::max<uint64_t>(most, (uint64_t)sms));
    if (PP.circuits > 0) {
        // the pair launch: two CTAs of 256 threads per SM, the tile and the largest pass's data
        b->psmem = (sizeof(double2) << PR_TILE_BITS) + PP.stage_bytes;
        int pper = 0;
        e = b->psmem <= PR_SMEM_CAP ? cudaFuncSetAttribute((const void*)k_cb_pairs,
                                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PR_SMEM_CAP)
                                    : cudaErrorInvalidValue;
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&pper, (const void*)k_cb_pairs, PR_THREADS, b->psmem);
        if (e != cudaSuccess || pper < 1) return fail("pair kernel setup", e);
        uint64_t pmost = 1;
        for (size_t p = 0; p + 1 < PP.phase_off.size(); p++)
            pmost = std::max<uint64_t>(pmost, PP.phase_off[p + 1] - PP.phase_off[p]);
        b->pgrid = (unsigned)std::min<uint64_t>((uint64_t)pper * sms, pmost);
    }
    cudaGraph_t g = nullptr;
    if (cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
        const cudaError_t le = cb_enqueue(b, b->stream);
        const cudaError_t ce = cudaStreamEndCapture(b->stream, &g);
        if (le == cudaSuccess && ce == cudaSuccess && g && cudaGraphInstantiate(&b->graph, g, 0) == cudaSuccess)
            b->graphed = true;
        else
            b->graph = nullptr;
        if (g) cudaGraphDestroy(g);
        (void)cudaGetLastError();
    }
    *out = b;
    return SVB_OK;
}

svb_status cb_run(svb_circuit_batch* b)
{
    std::memset(b->h_err, 0, 4 * sizeof(unsigned));
    cudaError_t e = b->graphed ? cudaGraphLaunch(b->graph, b->stream) : cb_enqueue(b, b->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(b->stream);
    if (e != cudaSuccess) return cb_cuda_fail(e, "svb_cbatch_run");
    if (b->h_err[1] | b->h_err[3]) {
        set_error("svb_cbatch_run: a grid barrier timed out; results are invalid");
        return SVB_ERR_STATE;
    }
    return SVB_OK;
}

// Autotuner cache: batch signature -> (tile bits, threads, pair engine).
std::mutex g_tune_mutex;
std::map<std::vector<uint64_t>, std::tuple<int, int, bool>> g_tune_cache;

std::vector<uint64_t> signature(const svb_circuit_batch* b)
{
    std::vector<uint64_t> sig = {(uint64_t)b->precision, (uint64_t)b->device};
    for (uint32_t c = 0; c < b->n_circ; c++)
        sig.push_back(((uint64_t)b->n[c] << 40) | (b->gate_off[c + 1] - b->gate_off[c]));
    return sig;
}

}  // namespace
}  // namespace svb

using namespace svb;

extern "C" {

svb_status svb_cbatch_create(int device, int precision, uint32_t n_circuits, const uint32_t* n_qubits,
                             const uint64_t* gate_offsets, const svb_gate* gates, const uint64_t* term_offsets,
                             const svb_pauli_term* terms, int tile_bits, svb_circuit_batch** out)
{
    if (!out || !n_qubits || !gate_offsets || (gate_offsets[n_circuits] && !gates)) {
        set_error("svb_cbatch_create: NULL argument");
        return SVB_ERR_INVALID;
    }
    *out = nullptr;
    if (precision != SVB_FP64 && precision != SVB_FP32) return cb_invalid("svb_cbatch_create: bad precision");
    if (n_circuits == 0) return cb_invalid("svb_cbatch_create: no circuits");
    const int max_tb = precision == SVB_FP64 ? 12 : 13;
    if (tile_bits != 0 && tile_bits != SVB_CBATCH_PAIRS && (tile_bits < 6 || tile_bits > max_tb))
        return cb_invalid("svb_cbatch_create: tile_bits must be 0 (tune), SVB_CBATCH_PAIRS or in [6, " +
                          std::to_string(max_tb) + "]");
    svb_circuit_batch proto;
    proto.device = device;
    proto.precision = precision;
    proto.n_circ = n_circuits;
    uint32_t max_n = 0;
    for (uint32_t c = 0; c < n_circuits; c++) {
        if (n_qubits[c] < 1 || n_qubits[c] > CB_MAX_QUBITS)
            return cb_invalid("svb_cbatch_create: circuit " + std::to_string(c) + " needs 1..24 qubits");
        if (gate_offsets[c + 1] < gate_offsets[c]) return cb_invalid("svb_cbatch_create: gate_offsets decrease");
        max_n = std::max(max_n, n_qubits[c]);
        proto.n.push_back(n_qubits[c]);
    }
    if (gate_offsets[0] != 0) return cb_invalid("svb_cbatch_create: gate_offsets[0] must be 0");
    proto.gate_off.assign(gate_offsets, gate_offsets + n_circuits + 1);
    proto.gates.assign(gates, gates + gate_offsets[n_circuits]);
    if (term_offsets) {
        if (term_offsets[0] != 0) return cb_invalid("svb_cbatch_create: term_offsets[0] must be 0");
        if (term_offsets[n_circuits] && !terms) return cb_invalid("svb_cbatch_create: NULL terms");
        proto.term_off.assign(term_offsets, term_offsets + n_circuits + 1);
        proto.terms.assign(terms, terms + term_offsets[n_circuits]);
        for (uint32_t c = 0; c < n_circuits; c++) {
            if (term_offsets[c + 1] < term_offsets[c]) return cb_invalid("svb_cbatch_create: term_offsets decrease");
            for (uint64_t t = term_offsets[c]; t < term_offsets[c + 1]; t++)
                if ((terms[t].x_mask | terms[t].z_mask) >> n_qubits[c])
                    return cb_invalid("svb_cbatch_create: a term of circuit " + std::to_string(c) + " acts on a qubit >= n");
        }
    } else {
        proto.term_off.assign(n_circuits + 1, 0);
    }
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return cb_cuda_fail(e, "svb_cbatch_create");
    if (tile_bits == SVB_CBATCH_PAIRS) return cb_create_with(&proto, max_tb, 512, true, out);
    if (tile_bits != 0) return cb_create_with(&proto, tile_bits, 512, false, out);

    // autotune: the cached choice for this signature, else time the candidates
    const std::vector<uint64_t> sig = signature(&proto);
    {
        std::lock_guard<std::mutex> lock(g_tune_mutex);
        auto it = g_tune_cache.find(sig);
        if (it != g_tune_cache.end()) {
            svb_status st = cb_create_with(&proto, std::get<0>(it->second), std::get<1>(it->second),
                                           std::get<2>(it->second), out);
            if (st == SVB_OK) (*out)->tuned = true;
            return st;
        }
    }
    // candidates: the sweep at three tile sizes and two block sizes, and (FP64, when a
    // circuit has 12 or more qubits) the pair engine with the sweep's largest tile for the rest
    std::vector<std::tuple<int, int, bool>> cands;
    for (int tb = max_tb - 2; tb <= max_tb; tb++)
        for (int threads : {256, 512}) cands.emplace_back(tb, threads, false);
    if (precision == SVB_FP64 && max_n >= (uint32_t)PR_TILE_BITS) cands.emplace_back(max_tb, 512, true);
    svb_circuit_batch* best = nullptr;
    double best_ms = 0;
    for (const auto& cfg : cands) {
        const int tb = std::get<0>(cfg), threads = std::get<1>(cfg);
        svb_circuit_batch* cand = nullptr;
        if (cb_create_with(&proto, tb, threads, std::get<2>(cfg), &cand) != SVB_OK) continue;
        if (std::get<2>(cfg) && cand->plan.pairs.circuits == 0) {      // nothing for the pair engine
            cb_free(cand);
            continue;
        }
        double ms = 1e300;
        bool ok = cb_run(cand) == SVB_OK;           // warm-up
        for (int r = 0; ok && r < 3; r++) {
            const auto t0 = std::chrono::steady_clock::now();
            ok = cb_run(cand) == SVB_OK;
            const auto t1 = std::chrono::steady_clock::now();
            ms = std::min(ms, std::chrono::duration<double, std::milli>(t1 - t0).count());
        }
        if (ok && (!best || ms < best_ms)) {
            if (best) cb_free(best);
            best = cand;
            best_ms = ms;
        } else {
            cb_free(cand);
        }
    }
    if (!best) {
        set_error("svb_cbatch_create: no candidate configuration ran");
        return SVB_ERR_CUDA;
    }
    best->tuned = true;
    {
        std::lock_guard<std::mutex> lock(g_tune_mutex);
        g_tune_cache[sig] = std::make_tuple(best->tile_bits, best->threads, best->use_pairs);
    }
    *out = best;
    return SVB_OK;
}

svb_status svb_cbatch_run(svb_circuit_batch* b, const svb_gate* gates, double* energies)
{
    if (!b) return cb_invalid("svb_cbatch_run: NULL batch");
    cudaError_t e = cudaSetDevice(b->device);
    if (e != cudaSuccess) return cb_cuda_fail(e, "svb_cbatch_run");
    if (gates) {
        // new angles for the same gate structure: re-plan and check that nothing moved
        for (uint64_t g = 0; g < b->gate_off[b->n_circ]; g++)
            if (gates[g].op != b->gates[g].op || std::memcmp(gates[g].qb, b->gates[g].qb, sizeof(gates[g].qb)) != 0)
                return cb_invalid("svb_cbatch_run: gate " + std::to_string(g) + " differs from the batch's structure");
        if (b->plan.pairs.each.size() == b->n_circ) {
            if (!cb_replan_pairs(b, gates)) return cb_invalid("svb_cbatch_run: the plan's structure changed");
            std::copy(gates, gates + b->gate_off[b->n_circ], b->gates.begin());
            svb_status st = cb_run(b);
            if (st != SVB_OK) return st;
            if (energies) std::memcpy(energies, b->h_energy, b->n_circ * sizeof(double));
            return SVB_OK;
        }
        CbPlan plan;
        std::string err;
        if (!cb_build_plan(b, gates, b->tile_bits, b->use_pairs, plan, err)) return cb_invalid("svb_cbatch_run: " + err);
        if (plan.ops.size() != b->plan.ops.size()) return cb_invalid("svb_cbatch_run: the plan's structure changed");
        for (size_t i = 0; i < plan.ops.size(); i++)
            if (plan.ops[i].form != b->plan.ops[i].form || plan.ops[i].p != b->plan.ops[i].p ||
                plan.ops[i].flags != b->plan.ops[i].flags)
                return cb_invalid("svb_cbatch_run: the plan's structure changed");
        // the pair part: the same passes, ops and layouts, new gate fragments
        const CbPairPlan &np = plan.pairs, &op = b->plan.pairs;
        if (np.circuits != op.circuits || np.passes.size() != op.passes.size() || np.ops.size() != op.ops.size() ||
            np.layouts.size() != op.layouts.size() || np.gates.size() != op.gates.size() ||
            (!np.passes.empty() && std::memcmp(np.passes.data(), op.passes.data(), np.passes.size() * sizeof(PairPass))) ||
            (!np.ops.empty() && std::memcmp(np.ops.data(), op.ops.data(), np.ops.size() * sizeof(PairOp))) ||
            (!np.layouts.empty() && std::memcmp(np.layouts.data(), op.layouts.data(), np.layouts.size() * sizeof(DevStage))))
            return cb_invalid("svb_cbatch_run: the plan's structure changed");
        std::memcpy(b->h_ops, plan.ops.data(), plan.ops.size() * sizeof(CbOp));
        if (!np.gates.empty()) std::memcpy(b->h_pgates, np.gates.data(), np.gates.size() * sizeof(double));
        b->plan.pairs.gates = np.gates;
        std::copy(gates, gates + b->gate_off[b->n_circ], b->gates.begin());
    }
    svb_status st = cb_run(b);
    if (st != SVB_OK) return st;
    if (energies) std::memcpy(energies, b->h_energy, b->n_circ * sizeof(double));
    return SVB_OK;
}

svb_status svb_cbatch_get_state(svb_circuit_batch* b, uint32_t circuit, double* re, double* im)
{
    if (!b || circuit >= b->n_circ) return cb_invalid("svb_cbatch_get_state: bad batch or circuit");
    cudaError_t e = cudaSetDevice(b->device);
    if (e != cudaSuccess) return cb_cuda_fail(e, "svb_cbatch_get_state");
    const uint64_t dim = 1ull << b->n[circuit];
    const size_t amp = b->precision == SVB_FP64 ? 16 : 8;
    std::vector<char> host(dim * amp);
    e = cudaMemcpy(host.data(), static_cast<char*>(b->pool) + b->plan.circ[circuit].state_off * amp, dim * amp,
                   cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cb_cuda_fail(e, "svb_cbatch_get_state");
    for (uint64_t i = 0; i < dim; i++) {
        double r, m;
        if (b->precision == SVB_FP64) {
            r = reinterpret_cast<const double*>(host.data())[2 * i];
            m = reinterpret_cast<const double*>(host.data())[2 * i + 1];
        } else {
            r = reinterpret_cast<const float*>(host.data())[2 * i];
            m = reinterpret_cast<const float*>(host.data())[2 * i + 1];
        }
        if (re) re[i] = r;
        if (im) im[i] = m;
    }
    return SVB_OK;
}

svb_status svb_cbatch_info(const svb_circuit_batch* b, svb_cbatch_stats* out)
{
    if (!b || !out) return cb_invalid("svb_cbatch_info: NULL argument");
    out->n_circuits = b->n_circ;
    out->n_phases = (uint32_t)b->plan.phase_off.size() - 1;
    out->tile_bits = (uint32_t)b->tile_bits;
    out->threads = (uint32_t)b->threads;
    out->pool_amplitudes = b->plan.pool_amps;
    out->items = b->plan.items.size();
    out->grid = b->grid;
    out->graphed = b->graphed ? 1u : 0u;
    out->moved_bytes = b->plan.moved_bytes;
    out->tuned = b->tuned ? 1u : 0u;
    out->n_passes = (uint32_t)b->plan.passes.size();
    out->pair_circuits = b->plan.pairs.circuits;
    out->pair_passes = (uint32_t)b->plan.pairs.passes.size();
    out->pair_phases = (uint32_t)b->plan.pairs.phase_off.size() - 1;
    out->pair_grid = b->pgrid;
    out->n_phases = std::max(out->n_phases, out->pair_phases);
    out->items += b->plan.pairs.items.size();
    return SVB_OK;
}

svb_status svb_cbatch_destroy(svb_circuit_batch* b)
{
    if (!b) return SVB_OK;
    cudaSetDevice(b->device);
    cb_free(b);
    return SVB_OK;
}

}  // extern "C"
