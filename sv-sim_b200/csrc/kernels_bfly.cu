// Kernel of the butterfly engine (bfly.h): one launch per pass, two persistent CTAs of 256
// threads per SM, a tile of 4,096 16-byte units (64 KiB) at a time in registers, redistributed
// through shared memory where a stage ends.
//
// What bounds it (n = 28, FP64, depth-40 random circuit, 44 passes, 1,134 gates, 145
// redistributions: 196 ms): the gates 73-90 ms (390 cycles each per tile and SM where their
// 64 FMAs a warp take 256: the register file feeds a 64-bit FMA's operands in its two issue
// slots, so every other instruction adds to them), a redistribution 1,500 cycles, tile loads
// and stores 58 ms.  The two CTAs of an SM overlap these little; handing the right to compute
// from one to the other made it 242 ms, prefetching the next tile into L2 and starting half
// of the CTAs later changed nothing, loading tiles without cp.async made it 259 ms.  So neither
// memory nor the FP64 pipe is full: 25% of the DRAM rate and 35% of the pipe's in a pass at 26
// qubits.  Registers: 128, the most that two CTAs leave; <float> spills 128 bytes a thread.
#include <cstring>
#include <vector>

#include "bfly_core.cuh"

namespace svb {
namespace {

constexpr size_t BF_TILE_BYTES = size_t(16) << BF_UNIT_BITS;

// global index bits of a tile
__device__ __forceinline__ uint64_t tile_base(const BfPass& P, uint64_t tile)
{
    uint64_t base = 0;
    for (int j = 0; j < P.n_nonlocal; j++) base |= ((tile >> j) & 1ull) << P.nonlocal_q[j];
    return base;
}

// bit i: parity of the tile mask i on the tile (the same in every lane)
__device__ __forceinline__ uint64_t tile_bits(const BfPass& P, uint64_t base, int lane)
{
    if (P.n_tile_masks == 0) return 0;
    const int a = lane < P.n_tile_masks && bf_parity64(P.tile_mask[lane] & base);
    const uint32_t lo = __ballot_sync(0xffffffffu, a);
    if (P.n_tile_masks <= 32) return lo;
    const int b = lane + 32 < P.n_tile_masks && bf_parity64(P.tile_mask[min(lane + 32, BF_NO_TILE - 1)] & base);
    return (uint64_t)__ballot_sync(0xffffffffu, b) << 32 | lo;
}

// starts the copies of a tile's units into this thread's own 16 slots of the tile buffer
template <typename T>
__device__ __forceinline__ void prefetch(const typename BfWord<T>::type* __restrict__ src, const BfPass& P,
                                         BfUnit<T>* sm, int tid)
{
    constexpr int SH = BfScalar<T>::packed ? 1 : 0;
#pragma unroll
    for (int k = 0; k < BF_NR; k++) {
        const uint32_t to = (uint32_t)__cvta_generic_to_shared(sm + k * BF_THREADS + tid);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(src + (bf_comb(P.in_reg, k) >> SH)));
    }
}

template <typename T>
__global__ void __launch_bounds__(BF_THREADS, 2)
k_bfly(typename BfWord<T>::type* __restrict__ sv, const BfPass* __restrict__ passes, const BfOp* __restrict__ ops,
       const BfRelayout* __restrict__ rels, const T* __restrict__ coefs, int pass_index, uint64_t tiles)
{
    using W = typename BfWord<T>::type;
    constexpr int SH = BfScalar<T>::packed ? 1 : 0;      // amplitudes per unit, log2
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ BfPass P;
    BfUnit<T>* sm = reinterpret_cast<BfUnit<T>*>(smem);
    const int tid = threadIdx.x;
    {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(passes + pass_index);
        uint32_t* dst = reinterpret_cast<uint32_t*>(&P);
        for (int w = tid; w < (int)(sizeof(BfPass) / 4); w += BF_THREADS) dst[w] = src[w];
        __syncthreads();
    }
    // the pass's ops, relayouts, slot tables and coefficients in shared memory, once per CTA,
    // and what each thread would otherwise keep in registers beside its 16 units
    BfPhase* sph = reinterpret_cast<BfPhase*>(smem + BF_TILE_BYTES);
    ulonglong2* sgo = reinterpret_cast<ulonglong2*>(sph + BF_THREADS);
    BfOp* so = reinterpret_cast<BfOp*>(sgo + BF_THREADS);
    BfRelayout* sr = reinterpret_cast<BfRelayout*>(so + P.n_ops);
    uint16_t* tab = reinterpret_cast<uint16_t*>(sr + P.n_rel);
    T* sc = reinterpret_cast<T*>(tab + (size_t)P.n_rel * 2 * BF_THREADS);
    {
        const uint4* o4 = reinterpret_cast<const uint4*>(ops + P.op_begin);
        for (int w = tid; w < P.n_ops * 2; w += BF_THREADS) reinterpret_cast<uint4*>(so)[w] = o4[w];
        const uint32_t* src = reinterpret_cast<const uint32_t*>(rels + P.rel_begin);
        for (int w = tid; w < P.n_rel * (int)(sizeof(BfRelayout) / 4); w += BF_THREADS)
            reinterpret_cast<uint32_t*>(sr)[w] = src[w];
        for (int w = tid; w < P.n_coef; w += BF_THREADS) sc[w] = coefs[P.coef_begin + w];
        __syncthreads();
        // from here on a thread reads only the entries it wrote itself
        for (int r = 0; r < P.n_rel; r++) {
            tab[(2 * r) * BF_THREADS + tid] = bf_thr(sr[r].wthr, tid);
            tab[(2 * r + 1) * BF_THREADS + tid] = bf_thr(sr[r].rthr, tid);
        }
        sph[tid].own = make_double2(1.0, 0.0);
        sgo[tid] = make_ulonglong2(bf_thr(P.in_thr, tid), bf_thr(P.out_thr, tid));
    }

    // Tiles arrive by cp.async in the tile buffer, each thread's units in slots of its own (it
    // waits for no one else's): the next tile's copies start as soon as the last relayout has
    // left the buffer, and run beside the pass's last gates and its stores.
    uint64_t base = tile_base(P, blockIdx.x), next = base;
    prefetch<T>(sv + ((base | sgo[tid].x) >> SH), P, sm, tid);
    for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, base = next) {
        const bool more = tile + gridDim.x < tiles;
        BfUnit<T> v[BF_NR];
        asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
        for (int k = 0; k < BF_NR; k++) {
            const W w = *reinterpret_cast<const W*>(sm + k * BF_THREADS + tid);
            bf_load(w, v[k]);
        }
        const uint64_t flips = tile_bits(P, base, tid & 31);
        for (int o = 0;; o++) {
            // runs of gates in a loop of their own: with every kind of op in one loop the
            // compiler moved the 16 units between registers at every op (n = 28: 201 ms
            // instead of 196)
            BfOp op = so[o];
            while (op.kind == BF_ROT) {
                const BfOp cur = op;
                op = so[++o];                // read while the gate runs; the list ends with BF_END
                bf_apply_rot<T>(cur, v, tid, flips);
            }
            if (op.kind == BF_END) break;
            if (op.kind != BF_RELAYOUT) {
                bf_apply<T>(op, sc, v, sph + tid, tid, flips);
                continue;
            }
            const BfRelayout& R = sr[op.lay];
            const uint32_t w = tab[(2 * op.lay) * BF_THREADS + tid];
            uint32_t reg[BF_RB];
#pragma unroll
            for (int i = 0; i < BF_RB; i++) reg[i] = R.wreg[i];
            __syncthreads();                 // the last relayout's (or the tile's) readers are done
#pragma unroll
            for (int k = 0; k < BF_NR; k++) sm[w ^ bf_comb(reg, k)] = v[k];
            const uint32_t r = tab[(2 * op.lay + 1) * BF_THREADS + tid];
#pragma unroll
            for (int i = 0; i < BF_RB; i++) reg[i] = R.rreg[i];
            __syncthreads();
#pragma unroll
            for (int k = 0; k < BF_NR; k++) v[k] = sm[r ^ bf_comb(reg, k)];
            if (op.lay + 1 == P.n_rel && more) {
                __syncthreads();
                next = tile_base(P, tile + gridDim.x);
                prefetch<T>(sv + ((next | sgo[tid].x) >> SH), P, sm, tid);
            }
        }
        if (P.n_rel == 0) {
            // the buffer's slots are this thread's own; but a store may land where another
            // thread of the tile still has to load: the barriers of a relayout part the two, a
            // pass without one needs its own
            if (more) {
                next = tile_base(P, tile + gridDim.x);
                prefetch<T>(sv + ((next | sgo[tid].x) >> SH), P, sm, tid);
            }
            __syncthreads();
        }
        uint64_t off = sgo[tid].y;
        for (int f = 0; f < P.n_flips; f++)
            if (bf_parity64(P.flips[f].tile & base)) off ^= P.flips[f].off;
        const typename BfScalar<T>::S scale = BfScalar<T>::dup(sc[P.n_coef - 1]);
        W* dst = sv + (base >> SH);
#pragma unroll
        for (int k = 0; k < BF_NR; k++) {
            BfUnit<T> u;
            u.re = BfScalar<T>::mul(v[k].re, scale);
            u.im = BfScalar<T>::mul(v[k].im, scale);
            W w;
            bf_store(u, w);
            dst[(off ^ bf_comb(P.out_reg, k)) >> SH] = w;
        }
    }
}

}  // namespace

cudaError_t upload_bfly(const BfPlan& plan, int precision, GrowBuf& buf, DevBfBuffers& dev)
{
    const bool fp32 = precision == SVB_FP32;
    // BfOp is read in 16-byte words: the passes' part is rounded up
    const size_t sp = (plan.passes.size() * sizeof(BfPass) + 15) / 16 * 16, so = plan.ops.size() * sizeof(BfOp);
    const size_t sr = plan.rels.size() * sizeof(BfRelayout), sc = plan.coefs.size() * (fp32 ? 4 : 8);
    std::vector<unsigned char> host(sp + so + sr + sc);     // every part a multiple of 8 bytes
    unsigned char* h = host.data();
    if (sp) std::memcpy(h, plan.passes.data(), plan.passes.size() * sizeof(BfPass));
    if (so) std::memcpy(h + sp, plan.ops.data(), so);
    if (sr) std::memcpy(h + sp + so, plan.rels.data(), sr);
    if (fp32) {
        const std::vector<float> f = bfly_coefs32(plan);
        if (sc) std::memcpy(h + sp + so + sr, f.data(), sc);
    } else if (sc) {
        std::memcpy(h + sp + so + sr, plan.coefs.data(), sc);
    }
    cudaError_t e = grow(buf, host.size());
    if (e == cudaSuccess && !host.empty()) e = cudaMemcpyAsync(buf.p, h, host.size(), cudaMemcpyHostToDevice, nullptr);
    unsigned char* d = static_cast<unsigned char*>(buf.p);
    dev.passes = reinterpret_cast<BfPass*>(d);
    dev.ops = reinterpret_cast<BfOp*>(d + sp);
    dev.rels = reinterpret_cast<BfRelayout*>(d + sp + so);
    dev.coefs = d + sp + so + sr;
    dev.smem_bytes = plan.smem_bytes;
    return e;
}

template <typename T>
cudaError_t launch_bfly_pass(void* state, int n, int pass_index, const DevBfBuffers& b, cudaStream_t s)
{
    using W = typename BfWord<T>::type;
    constexpr int M = BF_UNIT_BITS + (BfScalar<T>::packed ? 1 : 0);
    static int max_ctas[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (n < M || b.smem_bytes > BF_SMEM_CAP) return cudaErrorInvalidValue;
    if (dev < 64 && max_ctas[dev] == 0) {
        cudaError_t e = cudaFuncSetAttribute(k_bfly<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BF_SMEM_CAP);
        if (e != cudaSuccess) return e;
        int per_sm = 0, sms = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bfly<T>, BF_THREADS, BF_SMEM_CAP);
        if (e != cudaSuccess) return e;
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        max_ctas[dev] = (per_sm > 0 ? per_sm : 1) * sms;
    }
    const uint64_t tiles = 1ull << (n - M);
    uint64_t grid = tiles;
    if (dev < 64 && grid > (uint64_t)max_ctas[dev]) grid = (uint64_t)max_ctas[dev];
    k_bfly<T><<<(unsigned)grid, BF_THREADS, b.smem_bytes, s>>>(static_cast<W*>(state), b.passes, b.ops, b.rels,
                                                              static_cast<const T*>(b.coefs), pass_index, tiles);
    return cudaGetLastError();
}
template cudaError_t launch_bfly_pass<double>(void*, int, int, const DevBfBuffers&, cudaStream_t);
template cudaError_t launch_bfly_pass<float>(void*, int, int, const DevBfBuffers&, cudaStream_t);

}  // namespace svb
