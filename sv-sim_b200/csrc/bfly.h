// Plan of the butterfly engine (bfly.cpp plans, bfly_core.cuh executes, kernels_bfly.cu
// launches): circuits of unitary 2x2 matrices, CX and phases applied in registers, many
// gates per pass over the state.
//
// What it rests on.  A gate U on a qubit before a CX splits into a left factor that
// commutes with the CX and so waits for the qubit's next gate, and a rest that is a scale
// times [[1, u], [-conj(u), 1]]:
//   * control: U = D W with D diagonal;
//   * target:  U = (a I + b X) W.
// So a gate costs one complex multiply-add per amplitude (4 real FMAs; a general 2x2 matrix
// is 8, the 4x4 block of two gates and their CX on the tensor cores 16), the scales of a
// pass are multiplied into its stores, and a CX itself only renames amplitudes.
//
// A tile is 2^12 units of 16 bytes: one complex<double>, or two complex<float> whose index
// differs in qubit 0 (a packed pair of real parts and one of imaginary parts, the operands
// of fma.rn.f32x2).  256 threads hold 16 units each; a unit's index bits sit on 4 register
// bits, 5 lane bits and 3 warp bits.  The value of local position p in register slot k
// (k's bit 4: the half of a packed unit) of thread t in tile b is
//     x_p = parity(k & rm_p) ^ parity(t & tm_p) ^ parity(b & xm_p),
// and a CX adds its control's masks to its target's: nothing moves.  Only where the target
// sits in a register are the registers permuted, which keeps
// rm_p of a register-held position a single bit, the form a gate needs.
#pragma once

#include "svb_internal.h"

namespace svb {

constexpr int BF_RB = 4;                 // register bits: 16 units per thread
constexpr int BF_TB = 8;                 // thread bits: 256 threads
constexpr int BF_UNIT_BITS = BF_RB + BF_TB;
constexpr int BF_THREADS = 1 << BF_TB;
constexpr int BF_NR = 1 << BF_RB;
constexpr int BF_PACK = BF_RB;           // "register bit" 4: the half of a packed FP32 unit
constexpr int BF_MAX_POS = BF_UNIT_BITS + 1;
// Gates leave amplitudes unscaled within a pass: they grow by up to 1 / least, and the gate that
// would exceed it takes the scale into its matrix (BF_SROT).  So runs stay finite for
// amplitudes up to the type's largest value times least, 3e35 (FP32) and 1.5e290 (FP64).  Of
// the 1,215 gates of the depth-40 random circuit of 30 qubits one is a BF_SROT (37 with 2^-30),
// of the 50 of a Fourier transform of 25 qubits in FP32 one.
constexpr double BF_LEAST32 = 0x1p-10, BF_LEAST64 = 0x1p-60;
// positions 0..1 (FP64), resp. 1..2 beside the packed 0 (FP32), sit on lanes 0 and 1 when a
// tile is loaded and stored: whole 64-byte runs
constexpr int BF_COAL = 2;

enum BfKind : uint8_t {
    BF_ROT = 0,      // v0 += u v1, v1 -= conj(u) v0 on register bit tgt
    BF_PROT,         // the same between the halves of packed units
    BF_SROT,         // p v0 + b v1, p v1 - conj(b) v0 (p = coef[0]), with the scale so far in p and b
    BF_CX,           // register permutation: swap along tgt where register bit ctl is 1
    BF_DIAG,         // phase d0 (coef[0..1]) on even, d1 (coef[2..3]) on odd parity; doubles in
                     // both precisions (two float coefficients each)
    BF_FLUSH,        // multiplies in what the phases left to the whole thread
    BF_PFIX,         // swap the halves of packed units where the thread/tile parity is odd
    BF_RELAYOUT,     // redistribute the tile through shared memory
    BF_END           // end of the pass's list
};

// One op, 32 bytes: two 16-byte shared-memory reads, made while the op before it runs.
struct alignas(16) BfOp {
    uint8_t kind;
    uint8_t tgt;                         // register bit, or BF_PACK
    uint8_t ctl;                         // CX: register bit of the control, or BF_PACK
    uint8_t rmask;                       // DIAG: register mask (bit 4: packed half)
    uint8_t thr_mask;                    // parity of thread bits and
    uint8_t tile_bit;                    // of tile mask number tile_bit (BF_NO_TILE: none): exchanges v0, v1
    uint8_t run;                         // DIAG: bit 0 begins, bit 1 ends a run over one rmask
    uint8_t lay;                         // RELAYOUT: index among the pass's relayouts
    uint32_t coef;                       // SROT, DIAG: first coefficient, relative to the pass's
    uint32_t pad;
    union {
        double d[2];                     // ROT, SROT: real and imaginary part of u (b)
        float f[4];
    };
};
static_assert(sizeof(BfOp) == 32, "BfOp layout");
constexpr int BF_NO_TILE = 63;           // distinct tile masks of a pass: 0..62

struct BfRelayout {                      // shared-memory unit slots, combined by XOR
    uint16_t wthr[BF_TB], wreg[BF_RB];   // written: slot of each thread and register bit
    uint16_t rthr[BF_TB], rreg[BF_RB];   // read
};
static_assert(sizeof(BfRelayout) == 48, "BfRelayout layout");

struct BfFlip {                          // stores of tiles with odd parity(base & tile) move by off
    uint64_t tile;
    uint64_t off;
};

struct BfPass {
    uint64_t in_thr[BF_TB], in_reg[BF_RB];    // global amplitude offsets, combined by XOR
    uint64_t out_thr[BF_TB], out_reg[BF_RB];
    BfFlip flips[BF_MAX_POS];
    uint64_t tile_mask[BF_NO_TILE];
    uint8_t nonlocal_q[64 - BF_UNIT_BITS];
    int32_t n_nonlocal, n_flips, n_tile_masks, pad;
    int32_t op_begin, n_ops;
    int32_t rel_begin, n_rel;
    int32_t coef_begin, n_coef;          // the last one is the scale of the pass
};
static_assert(sizeof(BfPass) % 8 == 0, "BfPass layout");

// Most relayouts and ops of a pass: slot tables (1 KiB a relayout), ops and coefficients sit
// in shared memory beside the 64 KiB tile and 48 bytes a thread (its global offsets and
// pending phases), all within what two CTAs per SM can hold.  A pass that would need more is
// continued in another one.
constexpr int BF_MAX_REL = 16;
constexpr int BF_MAX_OPS = 256;
constexpr int BF_MAX_COEF = 768;
constexpr size_t BF_SMEM_CAP = 110 * 1024;
// dynamic shared memory of a pass: tile, phases, offsets, ops, relayouts, slot tables,
// coefficients
constexpr size_t bfly_smem(int n_ops, int n_rel, int n_coef, bool fp32)
{
    return (size_t(16) << BF_UNIT_BITS) + 48 * BF_THREADS + sizeof(BfOp) * (size_t)n_ops +
           (sizeof(BfRelayout) + 4 * BF_THREADS) * (size_t)n_rel + (fp32 ? 4 : 8) * (size_t)n_coef;
}
static_assert(bfly_smem(BF_MAX_OPS, BF_MAX_REL, BF_MAX_COEF, false) <= BF_SMEM_CAP, "pass limits");

struct BfPlan {
    int tile_bits = 0;                   // local qubits of a pass: 12 (FP64) or 13 (FP32)
    std::vector<BfPass> passes;
    std::vector<BfOp> ops;
    std::vector<BfRelayout> rels;
    std::vector<double> coefs;
    std::vector<size_t> raw;             // FP32: first of four doubles' slots (each takes two floats)
    size_t n_gates2 = 0, n_diags = 0, n_moves = 0;   // ROT and SROT, DIAG, register CX
    size_t smem_bytes = 0;               // largest pass
};

// whether every op is a unitary 2x2 matrix, a phase or a CX, and the state is big enough
bool bfly_supported(const std::vector<EOp>& ops, int n, int precision);
// The faster form by a circuit's counts, where those tell (butterflies only if bfly_supported).
enum class BfChoice { BLOCKS, BUTTERFLIES, COMPARE };
BfChoice bfly_choice(const std::vector<EOp>& ops, int n, int precision);
// the comparison of the FP64 plans of one circuit
bool bfly_cheaper(const BfPlan& b, const PairPlan& p);
// False if a layout came out that the kernel cannot address, or a pass that does nothing of
// what is left (neither has been seen; the caller then takes another engine).
bool plan_bfly(const std::vector<EOp>& ops, int n, int precision, BfPlan& plan);

// The coefficients as the kernel of FP32 states reads them.
std::vector<float> bfly_coefs32(const BfPlan& plan);
// The plan in one device buffer, copied from the host on the default stream (it may return before
// the copy has arrived); `buf` grows as needed and no kernel may still be reading it.
cudaError_t upload_bfly(const BfPlan& plan, int precision, GrowBuf& buf, DevBfBuffers& dev);
// one pass over the state
template <typename T>
cudaError_t launch_bfly_pass(void* state, int n, int pass_index, const DevBfBuffers& b, cudaStream_t s);

}  // namespace svb
