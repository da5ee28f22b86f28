// FP64 probability reductions and measurement sampling on the GPU.
//
// The reference samples on the host (svsim/src/svsim_nvgpu_sin.cuh:359-383): it copies
// the whole state back, builds the sequential inclusive scan S_0 = 0,
// S_{i+1} = fl(S_i + p_i) with p_i = fl(fl(re_i*re_i) + fl(im_i*im_i)) (2^n+1 doubles),
// and for each shot keeps the j with S_j <= r < S_{j+1} (0 if none).  The samples here
// are those of that exact S, bit for bit, without a sequential pass and without a 2^n
// scan array.
//
// Why a parallel pass can give the sequential sums exactly: while S stays inside one
// binade [2^e, 2^(e+1)), every value S takes is an integer multiple m of the grid unit
// u = 2^(e-52) (m in [2^52, 2^53)), and fl(S + p) = (m + round(p/u)) u, where round is
// to the nearest integer — unless p/u has a fractional part of exactly one half (a
// tie: round-half-even then depends on the last bit of m) or m + p/u reaches 2^53 (the
// sum leaves the binade and the grid doubles).  So a run of elements without ties
// that stays in the binade advances m by an exact integer sum of per-element
// roundings, which adds up in any order.  After a tie m is even whatever it was, so a
// run with ties depends on m's first parity alone: it is a pair (d for even m, d + t for
// odd m, t = -1, 0 or 1) and runs join associatively (struct Run).  Binade crossings (at
// most a few dozen, S being non-decreasing) are added one element at a time with IEEE
// adds in index order.
//
// Passes (B = 4096 amplitudes per block, 64 blocks per superblock):
//   1. k_block_sums   approximate FP64 block sums (any order) -> k_scan_single gives
//                     an approximate prefix, used only to guess each block's binade;
//   2. k_cdf_blocks   per block: the exact run D_b of its round(p_i/u) on the guessed
//                     binade's grid, or "zero block" / "no delta" (a guessed crossing,
//                     or no normal start);
//   3. k_cdf_super    per superblock: its blocks' D_b joined when they share one
//                     binade, else "no delta";
//   4. k_cdf_chain    one CTA walks the superblocks in order from S = 0: a delta
//                     applies when S is in its binade and stays there (checked on the
//                     exact S), otherwise the CTA descends to blocks and, where a
//                     block's delta does not apply either, through the block's chunks
//                     of 32 elements (walk_block);
//   5. k_cdf_fill     the exact S at every block start of the superblocks the chain
//                     did not descend into;
//   6. k_sample_exact one warp per shot: binary search over the exact block starts,
//                     then groups of 512 elements, their chunks and one chunk's exact sums
//                     to the first index whose inclusive S exceeds r.
// States of at most WALK_BLOCKS blocks skip passes 1-3 and 5: the chain walks every block.
// Every step computes the reference's sequential values themselves, so equal inputs
// give the reference's samples whatever the summation order of pass 1.
#include "pauli.cuh"

namespace svb {
namespace {

constexpr int BLOCK_AMPS = 1 << MEAS_BLOCK_BITS;   // 4096
constexpr int CHUNKS = BLOCK_AMPS / 32;            // 128
constexpr int SUPER_BLOCKS = 1 << MEAS_SUPER_BITS; // 64
// Up to here walking every block (a few us each) is shorter than the five launches that
// would spare the chain some of them; a state this small has a binade crossing in most.
constexpr uint64_t WALK_BLOCKS = 4;
constexpr uint64_t FRAC_MASK = (1ull << 52) - 1;
constexpr uint64_t HIDDEN = 1ull << 52;
constexpr uint64_t M_MAX = (1ull << 53) - 1;       // largest grid count inside one binade
// A block or superblock entry: bits 0..52 hold its run (d below DELTA_END), bits 53..63
// the biased exponent code of its binade (e + 1023, in [1, 2046]); code 0 = no delta
// (the field is then 1 if no probability of the range is NaN), code 2047 = every
// probability of the range is zero.
constexpr uint32_t CODE_NONE = 0, CODE_ZERO = 2047;

__device__ __forceinline__ uint64_t pack_entry(uint64_t d, uint32_t code) { return (uint64_t)code << 53 | d; }
__device__ __forceinline__ uint32_t entry_code(uint64_t w) { return (uint32_t)(w >> 53); }
__device__ __forceinline__ uint64_t entry_delta(uint64_t w) { return w & M_MAX; }
constexpr uint64_t DELTA_END = ((1ull << 53) - 1) / 3;   // 3 d + t + 1 fits the field

// Elements added in one binade: m advances by d if it is even, by d + t if it is odd.
struct Run {
    uint64_t d;
    int t;
};
// A run in 64 bits (d up to 2^57: 32 elements below 2^52).
__device__ __forceinline__ uint64_t pack_run(Run a) { return a.d << 2 | (uint64_t)(a.t + 1); }
__device__ __forceinline__ Run unpack_run(uint64_t w) { return {w >> 2, (int)(w & 3) - 1}; }
__device__ __forceinline__ uint64_t entry_field(Run a) { return a.d * 3 + (uint64_t)(a.t + 1); }
__device__ __forceinline__ Run entry_run(uint64_t w)
{
    const uint64_t f = entry_delta(w), d = f / 3;
    return {d, (int)(f - d * 3) - 1};
}
__device__ __forceinline__ Run join(Run a, Run b)  // a, then b
{
    const bool odd = a.d & 1;
    return {a.d + b.d + (uint64_t)(int64_t)(odd ? b.t : 0), a.t ? a.t : (odd ? -b.t : b.t)};
}
__device__ __forceinline__ uint64_t units_from(uint64_t m, Run a) { return a.d + (uint64_t)(int64_t)((m & 1) ? a.t : 0); }

// One element per lane joined in lane order.  m is even after a tie, so what a tie adds
// depends on the odd elements between it and the tie before, which two ballots show: a lane
// receives its own element's units for even m at lane 0 (their sum is the run's d), and *t
// and *odd (the sum's parity) are the run's.
__device__ __forceinline__ uint64_t warp_run(Run a, int lane, int* t, int* odd)
{
    const uint32_t ones = __ballot_sync(0xffffffffu, a.t == 0 && (a.d & 1));
    const uint32_t ties = __ballot_sync(0xffffffffu, a.t != 0);
    *t = 0;
    *odd = __popc(ones) & 1;
    if (ties == 0) return a.d;
    const uint32_t lt = (1u << lane) - 1, before = ties & lt;
    const uint32_t since = before ? lt & ~((2u << (31 - __clz(before))) - 1) : lt;
    const bool from_odd = __popc(ones & since) & 1;
    *t = __shfl_sync(0xffffffffu, from_odd ? -a.t : a.t, __ffs(ties) - 1);
    *odd = __popc(ones & ~((2u << (31 - __clz(ties))) - 1)) & 1;
    return a.d + (uint64_t)(int64_t)(from_odd ? a.t : 0);
}

// The runs of a warp's lanes joined in lane order; lane 0 has the result.
__device__ __forceinline__ Run warp_join(Run a)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
        a = join(a, unpack_run(__shfl_down_sync(0xffffffffu, pack_run(a), o)));
    return a;
}

// Lane l: the runs of lanes 0..l joined.
__device__ __forceinline__ Run warp_scan(Run a, int lane)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const Run b = unpack_run(__shfl_up_sync(0xffffffffu, pack_run(a), o));
        if (lane >= o) a = join(b, a);
    }
    return a;
}

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ uint64_t warp_sum_u64(uint64_t v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// |a_i|^2 as the reference forms it (svsim_nvgpu_sin.cuh:362-365): both products
// rounded, then added; never contracted into an FMA.
template <typename T>
__device__ __forceinline__ double prob_at(const typename VecOf<T>::type* sv, uint64_t dim, uint64_t i)
{
    if (i >= dim) return 0.0;
    const auto a = sv[i];
    const double r = (double)a.x, m = (double)a.y;
    return __dadd_rn(__dmul_rn(r, r), __dmul_rn(m, m));
}

// Binade code of a positive normal double (e + 1023), or 0 for 0, subnormals, inf,
// NaN and negatives; *m receives its significand as an integer in [2^52, 2^53).
__device__ __forceinline__ uint32_t binade_of(double s, uint64_t* m)
{
    const uint64_t b = (uint64_t)__double_as_longlong(s);
    const uint32_t code = (uint32_t)(b >> 52);      // sign bit included: negatives give >= 2048
    if (code == 0 || code >= 2047) return 0;
    *m = (b & FRAC_MASK) | HIDDEN;
    return code;
}

__device__ __forceinline__ double from_grid(uint32_t code, uint64_t m)   // m in [2^52, 2^53)
{
    return __longlong_as_double((long long)(((uint64_t)code << 52) | (m - HIDDEN)));
}

// A binade's grid unit as two factors, p / 2^(e-52) = p * a * b with e = code - 1023 in
// [-1022, 1023]: 2^(52-e) alone can lie outside the doubles.
struct Grid { double a, b; };
__device__ __forceinline__ Grid grid_of(uint32_t code)
{
    const int k = 52 + 1023 - (int)code, h = k >> 1;
    return {__longlong_as_double((long long)(1023 + h) << 52), __longlong_as_double((long long)(1023 + k - h) << 52)};
}

// p / 2^(e-52) rounded to the nearest integer, for p >= 0, as a run (a tie goes to the even
// integer, so an odd m takes one unit more where that was down and one less where it was
// up).  *ok is cleared where p alone leaves the binade (p / u >= 2^52) and for NaN or inf;
// the result is then not used.  Both products are exact (or below 2^-900, rounded
// to 0 units either way), x + 2^52 rounds to an integer, and x - round(x) is exact.  In
// doubles without a branch: shifts of the significand took some fifty instructions in
// five branches, which also kept a lane's loads from being in flight together.
__device__ __forceinline__ Run grid_run(double p, Grid g, bool* ok)
{
    constexpr double TWO52 = 4503599627370496.0;
    const double x = __dmul_rn(__dmul_rn(p, g.a), g.b);
    const double y = __dadd_rn(x, TWO52);
    const double frac = __dadd_rn(x, -__dadd_rn(y, -TWO52));
    if (!(x < TWO52)) *ok = false;
    return {(uint64_t)(__double_as_longlong(y) - __double_as_longlong(TWO52)),
            frac == 0.5 ? 1 : frac == -0.5 ? -1 : 0};
}

// The same where a tie is not wanted: it clears *ok too.
__device__ __forceinline__ uint64_t grid_units(double p, Grid g, bool* ok)
{
    const Run a = grid_run(p, g, ok);
    if (a.t) *ok = false;
    return a.d;
}

// S advanced by a run of binade `code`, if S lies in that binade and stays there; returns
// false (S unchanged) otherwise.
__device__ __forceinline__ bool advance(double* s, uint32_t code, Run a)
{
    uint64_t m;
    if (binade_of(*s, &m) != code || code == 0) return false;
    const uint64_t d = units_from(m, a);
    if (d > M_MAX - m) return false;
    *s = from_grid(code, m + d);
    return true;
}

// The reference's inclusive sums over one chunk of 32 consecutive elements, exactly:
// lane l receives S_{j0+l+1} given s_in = S_{j0} (warp-uniform) and its own p.
// Integer grid deltas when no lane ties and the chunk stays in s_in's binade; else
// 32 IEEE adds in index order, evaluated by every lane.
__device__ __forceinline__ double chunk_scan_exact(double s_in, double p, int lane)
{
    uint64_t m;
    const uint32_t code = binade_of(s_in, &m);
    if (code != 0) {
        bool ok = true;
        const uint64_t d = grid_units(p, grid_of(code), &ok);
        uint64_t incl = d;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        const uint64_t total = __shfl_sync(0xffffffffu, incl, 31);
        if (__all_sync(0xffffffffu, ok) && total <= M_MAX - m) return from_grid(code, m + incl);
    } else if (s_in == 0.0 && __all_sync(0xffffffffu, p == 0.0)) {
        return 0.0;
    }
    double s = s_in, mine = 0.0;
#pragma unroll 8
    for (int k = 0; k < 32; k++) {
        s = __dadd_rn(s, __shfl_sync(0xffffffffu, p, k));
        if (k == lane) mine = s;
    }
    return mine;
}

// The chain's CTA.  Its 16 warps share one block's probabilities in shared memory; one warp
// alone walked a block in 48-190 us (128 dependent chunk loads and scans), and a state has
// a walked block per binade that S crosses, 12 to 25 of them.  Bound by that chain of
// crossings, each a chunk's dependent adds and the deltas after it formed again.  The chain
// of 2^16 / 2^23 amplitudes: 749 / 2,227 us with one warp, 91 / 299 with the CTA, 61 / 252
// with the branch-free rounding, 54 / 137 since blocks with ties (one in b at block b, in a
// state of even weight) have deltas and are not walked.
constexpr int CHAIN_THREADS = 512;
struct WalkSmem {
    double p[BLOCK_AMPS];
    uint64_t run[CHUNKS];            // a chunk's run in the current binade
    uint32_t ok[CHUNKS];             // no NaN or inf in it, and none that leaves the binade alone
    double s;                        // warp 0's sum and the chunks it has added
    int cur;
};

// S after block b, exactly, from s at its start; every thread of the CTA calls it with the
// same s and receives the same result.  The chunks' runs are formed for the current binade
// by all warps at once; a warp-wide scan over the 128 chunks (four a lane, the same in every
// warp) finds the first chunk that leaves the binade, that chunk is added element by
// element, and the runs of the chunks after it are formed again for the new binade.
template <typename T>
__device__ double walk_block(const typename VecOf<T>::type* __restrict__ sv, uint64_t dim, uint64_t b,
                             double s, WalkSmem& sm)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t base = b * BLOCK_AMPS;
    const int chunks = dim - base < BLOCK_AMPS ? (int)((dim - base + 31) / 32) : CHUNKS;
#pragma unroll
    for (int k = 0; k < BLOCK_AMPS / CHAIN_THREADS; k++)
        sm.p[tid + k * CHAIN_THREADS] = prob_at<T>(sv, dim, base + tid + k * CHAIN_THREADS);
    __syncthreads();
    for (int cur = 0; cur < chunks;) {
        uint64_t m = 0;
        const uint32_t code = binade_of(s, &m);
        if (code != 0) {
#pragma unroll
            for (int k = 0; k < CHUNKS * 32 / CHAIN_THREADS; k++) {
                const int c = warp + k * (CHAIN_THREADS / 32);
                if (c < cur) continue;
                bool ok = true;
                Run a = grid_run(sm.p[c * 32 + lane], grid_of(code), &ok);
                ok = __all_sync(0xffffffffu, ok);
                int odd;
                a.d = warp_sum_u64(warp_run(a, lane, &a.t, &odd));
                if (lane == 0) {
                    sm.run[c] = pack_run(a);
                    sm.ok[c] = ok;
                }
            }
        }
        __syncthreads();                 // sm.run is written; sm.s has been read by all
        // one warp goes on until the binade changes: in all sixteen the scan took four times
        // as many issue slots
        if (warp == 0) {
            do {
                int f = cur;                 // chunk to add element by element
                if (code != 0) {
                    // inclusive runs of the chunks from cur on.  They are capped just above M_MAX, as
                    // is a chunk that is not ok, so that 128 of them cannot wrap.
                    constexpr uint64_t OVER = 1ull << 54;
                    Run v[4], run = {0, 0};
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const int c = lane * 4 + k;
                        Run a = {0, 0};
                        if (c >= cur && c < chunks) a = sm.ok[c] ? unpack_run(sm.run[c]) : Run{OVER, 0};
                        run = join(run, a);
                        if (run.d > OVER) run.d = OVER;
                        v[k] = run;
                    }
                    const Run incl = warp_scan(run, lane);   // up to 32 times OVER
                    Run excl = unpack_run(__shfl_up_sync(0xffffffffu, pack_run(incl), 1));
                    if (lane == 0) excl = {0, 0};
                    int bad = 4;                     // first of this lane's chunks that does not fit
                    uint64_t mine = units_from(m, excl);     // grid units before it
#pragma unroll
                    for (int k = 3; k >= 0; k--)
                        if (units_from(m, join(excl, v[k])) > M_MAX - m) bad = k;
#pragma unroll
                    for (int k = 0; k < 3; k++)
                        if (bad == k + 1) mine = units_from(m, join(excl, v[k]));
                    const unsigned who = __ballot_sync(0xffffffffu, bad < 4);
                    uint64_t pre = 0;                // grid units before chunk f
                    if (who) {
                        const int l = __ffs(who) - 1;
                        pre = __shfl_sync(0xffffffffu, mine, l);
                        f = l * 4 + __shfl_sync(0xffffffffu, bad, l);
                    } else {
                        pre = __shfl_sync(0xffffffffu, units_from(m, incl), 31);
                        f = chunks;
                    }
                    s = from_grid(code, m + pre);
                    if (f >= chunks) {
                        cur = chunks;
                        break;
                    }
                } else if (s != s) {         // NaN stays NaN
                    cur = chunks;
                    break;
                }
                if (code != 0 || !(s == 0.0 && __all_sync(0xffffffffu, sm.p[f * 32 + lane] == 0.0))) {
#pragma unroll
                    for (int k = 0; k < 32; k++) s = __dadd_rn(s, sm.p[f * 32 + k]);
                }
                cur = f + 1;
            } while (cur < chunks && binade_of(s, &m) == code);
            if (lane == 0) {
                sm.s = s;
                sm.cur = cur;
            }
        }
        __syncthreads();
        s = sm.s;
        cur = sm.cur;
    }
    return s;
}

// One CTA per block of 4,096 amplitudes, 16 loads in flight a thread: HBM-bound for large
// states; with one warp per block a 2^16-amplitude state took 75 us on 16 warps.
template <typename T>
__global__ void __launch_bounds__(256)
k_block_sums(const typename VecOf<T>::type* __restrict__ sv, uint64_t dim, uint64_t nblocks,
             double* __restrict__ out)
{
    __shared__ double red[8];
    const int tid = threadIdx.x, lane = tid & 31;
    for (uint64_t b = blockIdx.x; b < nblocks; b += gridDim.x) {
        const uint64_t base = b * BLOCK_AMPS + tid;
        double q[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int k = 0; k < 16; k++) q[k & 3] += prob_at<T>(sv, dim, base + k * 256);
        const double acc = warp_sum((q[0] + q[1]) + (q[2] + q[3]));
        if (lane == 0) red[tid >> 5] = acc;
        __syncthreads();
        if (tid == 0) {
            double t = 0.0;
#pragma unroll
            for (int w = 0; w < 8; w++) t += red[w];
            out[b] = t;
        }
        __syncthreads();
    }
}

// Exclusive scan of `in[0..count)` into out[0..count], out[count] = total.  One block
// of 1024 threads: each owns a contiguous segment (sequential sums), the segment
// totals are scanned across the block, then each segment is rewritten.
__global__ void __launch_bounds__(1024)
k_scan_single(const double* __restrict__ in, uint64_t count, double* __restrict__ out)
{
    __shared__ double wsum[32];
    const int t = threadIdx.x;
    const uint64_t seg = (count + 1023) / 1024;
    const uint64_t b = (uint64_t)t * seg;
    const uint64_t e = b + seg < count ? b + seg : count;
    double local = 0.0;
    for (uint64_t i = b; i < e; i++) local += in[i];
    // block exclusive scan of `local`
    const int lane = t & 31, w = t >> 5;
    double incl = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    if (w == 0) {
        double x = wsum[lane];
        double xi = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, xi, o);
            if (lane >= o) xi += y;
        }
        wsum[lane] = xi - x;   // exclusive over warps
    }
    __syncthreads();
    double run = wsum[w] + (incl - local);
    for (uint64_t i = b; i < e; i++) {
        out[i] = run;
        run += in[i];
    }
    if (t == 1023) out[count] = wsum[31] + incl;
}

// Pass 2: one CTA per block.  The binade guess is that of the approximate prefix at
// the block's start; a block whose approximate end lies in another binade is left
// without a delta (the chain adds it element by element).
template <typename T>
__global__ void __launch_bounds__(256)
k_cdf_blocks(const typename VecOf<T>::type* __restrict__ sv, uint64_t dim, uint64_t nblocks,
             const double* __restrict__ approx, uint64_t* __restrict__ entry)
{
    __shared__ uint64_t red[8];
    __shared__ uint32_t redf[8];
    __shared__ uint64_t runs[CHUNKS], redt[8];
    constexpr uint32_t NONZERO = 1, NAN_SEEN = 2, NOT_OK = 4, TIE = 8;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (uint64_t b = blockIdx.x; b < nblocks; b += gridDim.x) {
        uint64_t m0, m1;
        const uint32_t c0 = binade_of(approx[b], &m0);
        const uint32_t c1 = binade_of(approx[b + 1], &m1);
        const uint32_t code = (c0 != 0 && c0 == c1) ? c0 : 0;
        const Grid grid = grid_of(code);
        const uint64_t base = b * BLOCK_AMPS + tid;
        double p[16];
#pragma unroll
        for (int k = 0; k < 16; k++) p[k] = prob_at<T>(sv, dim, base + k * 256);
        uint64_t acc = 0;
        uint32_t flags = 0;
#pragma unroll
        for (int k = 0; k < 16; k++) {
            bool ok = true;
            const Run a = grid_run(p[k], grid, &ok);
            acc += a.d;
            flags |= (p[k] != 0.0 ? NONZERO : 0) | (p[k] != p[k] ? NAN_SEEN : 0) | (ok ? 0 : NOT_OK) | (a.t ? TIE : 0);
        }
        acc = warp_sum_u64(acc);               // 4096 terms of at most 2^52: no wrap
        flags = __reduce_or_sync(0xffffffffu, flags);
        if (lane == 0) {
            red[warp] = acc;
            redf[warp] = flags;
        }
        __syncthreads();
        flags = 0;
#pragma unroll
        for (int w = 0; w < 8; w++) flags |= redf[w];
        const bool use = code != 0 && !(flags & NOT_OK);
        if (use && (flags & TIE)) {
            // in index order: each chunk with its first m even, then the chunks' parities and
            // what their first ties add for odd m, by one warp
            uint64_t more = 0;                 // modulo 2^64: -1 or 1 a tie
#pragma unroll
            for (int k = 0; k < 16; k++) {
                bool ok = true;
                int t, odd;
                const Run a = grid_run(p[k], grid, &ok);
                more += warp_run(a, lane, &t, &odd) - a.d;
                if (lane == 0) runs[k * 8 + warp] = pack_run({(uint64_t)odd, t});
            }
            more = warp_sum_u64(more);
            if (lane == 0) redt[warp] = red[warp] + more;
            __syncthreads();
            if (warp == 0) {
                Run a = {0, 0};
                uint64_t odds = 0;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const Run c = unpack_run(runs[lane * 4 + k]);
                    a = k ? join(a, c) : c;
                    odds += c.d;
                }
                // a joined run of parities can be negative by its ties: an offset per lane
                // that is even keeps it packable and no parity changes
                a.d += 8;
                a = warp_join(a);
                odds = warp_sum_u64(odds) + 8 * 32;
                if (lane == 0) {
                    uint64_t sum = a.d - odds;
#pragma unroll
                    for (int w = 0; w < 8; w++) sum += redt[w];
                    entry[b] = sum < DELTA_END ? pack_entry(entry_field({sum, a.t}), code) : pack_entry(1, CODE_NONE);
                }
            }
        } else if (tid == 0) {
            acc = 0;
#pragma unroll
            for (int w = 0; w < 8; w++) acc += red[w];
            uint64_t w = pack_entry(flags & NAN_SEEN ? 0 : 1, CODE_NONE);
            if (!(flags & NONZERO)) w = pack_entry(0, CODE_ZERO);
            else if (use && acc < DELTA_END) w = pack_entry(entry_field({acc, 0}), code);
            entry[b] = w;
        }
        __syncthreads();
    }
}

// Pass 3: one thread per superblock.
__global__ void __launch_bounds__(256)
k_cdf_super(const uint64_t* __restrict__ entry, uint64_t nblocks, uint64_t nsuper,
            uint64_t* __restrict__ sentry)
{
    const uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nsuper) return;
    const uint64_t b0 = s * SUPER_BLOCKS;
    const uint64_t b1 = b0 + SUPER_BLOCKS < nblocks ? b0 + SUPER_BLOCKS : nblocks;
    uint32_t code = CODE_ZERO;
    Run d = {0, 0};
    bool ok = true, nan_free = true;
    for (uint64_t b = b0; b < b1; b++) {
        const uint64_t w = entry[b];
        const uint32_t c = entry_code(w);
        if (c == CODE_ZERO) continue;
        if (c == CODE_NONE) {
            ok = false;
            nan_free = nan_free && entry_delta(w) == 1;
            continue;
        }
        if (code != CODE_ZERO && c != code) ok = false;
        code = c;
        d = join(d, entry_run(w));   // each below 2^52, at most 64 of them
        if (d.d >= DELTA_END) ok = false;
    }
    sentry[s] = ok ? pack_entry(code == CODE_ZERO ? 0 : entry_field(d), code) : pack_entry(nan_free ? 1 : 0, CODE_NONE);
}

// S can no longer change over a range: S is NaN, or S is +inf and no probability of
// the range is NaN.
__device__ __forceinline__ bool stuck(double s, uint64_t w)
{
    if (s != s) return true;
    return isinf(s) && (entry_code(w) != CODE_NONE || entry_delta(w) == 1);
}

// S over consecutive superblocks (or blocks), up to 32 at once: lane l holds entry w of the
// l-th of them, and lanes from..cnt-1 are to be added.  Returns the first that S cannot be
// advanced past (a delta of another binade or none, or S leaves the binade), or cnt; *s is
// then S at its start, and *excl S at this lane's start for lanes from..that one.
__device__ __forceinline__ int advance_32(double* s, uint64_t w, int from, int cnt, int lane, double* excl)
{
    uint64_t m = 0;
    const uint32_t code = binade_of(*s, &m), c = entry_code(w);
    const bool in = lane >= from && lane < cnt;
    if (code == 0) {                         // zeros change no S
        const unsigned stop = __ballot_sync(0xffffffffu, in && c != CODE_ZERO);
        *excl = *s;
        return stop ? __ffs(stop) - 1 : cnt;
    }
    const Run a = in && c == code ? entry_run(w) : Run{0, 0};
    const uint64_t d = units_from(m, warp_scan(a, lane));    // up to 32 below 2^52
    const uint64_t up = __shfl_up_sync(0xffffffffu, d, 1);
    const uint64_t before = lane ? up : 0;
    const unsigned stop = __ballot_sync(0xffffffffu, in && ((c != CODE_ZERO && c != code) || d > M_MAX - m));
    const int f = stop ? __ffs(stop) - 1 : cnt;
    *excl = from_grid(code, m + before);
    *s = from_grid(code, m + __shfl_sync(0xffffffffu, stop ? before : d, stop ? f : 31));
    return f;
}

// Pass 4: one CTA; every warp follows the same chain (S and the entries are the same in
// all), warp 0 writes it down, and all of them share the work of a walked block.  Entries
// are read 32 at a time (one per lane) and added by one scan up to the first that does not
// apply, which is descended into.  desc[s] = 1 marks a superblock whose block starts the
// chain wrote itself.  entry == nullptr: no deltas, every block is walked.
template <typename T>
__global__ void __launch_bounds__(CHAIN_THREADS)
k_cdf_chain(const typename VecOf<T>::type* __restrict__ sv, uint64_t dim, uint64_t nblocks,
            uint64_t nsuper, const uint64_t* __restrict__ entry, const uint64_t* __restrict__ sentry,
            double* __restrict__ start, double* __restrict__ sstart, uint32_t* __restrict__ desc)
{
    __shared__ WalkSmem sm;
    const int lane = threadIdx.x & 31;
    const bool writer = threadIdx.x == 0, wwarp = threadIdx.x < 32;
    double s_val = 0.0, at;
    if (!entry) {
        for (uint64_t b = 0; b < nblocks; b++) {
            if (writer) start[b] = s_val;
            s_val = walk_block<T>(sv, dim, b, s_val, sm);
        }
        if (writer) start[nblocks] = s_val;
        return;
    }
    for (uint64_t g = 0; g < nsuper; g += 32) {
        const uint64_t mine = g + lane < nsuper ? sentry[g + lane] : 0;
        const int cnt = nsuper - g < 32 ? (int)(nsuper - g) : 32;
        for (int k = 0; k < cnt; k++) {
            const int from = k;
            k = advance_32(&s_val, mine, from, cnt, lane, &at);
            if (wwarp && lane >= from && lane < k) {
                sstart[g + lane] = at;
                desc[g + lane] = 0;
            }
            if (k == cnt) break;
            const uint64_t sidx = g + k;
            const uint64_t w = __shfl_sync(0xffffffffu, mine, k);
            const bool skip = stuck(s_val, w);
            if (writer) {
                sstart[sidx] = s_val;
                desc[sidx] = !skip;
            }
            if (skip) continue;
            const uint64_t b0 = sidx * SUPER_BLOCKS;
            const uint64_t b1 = b0 + SUPER_BLOCKS < nblocks ? b0 + SUPER_BLOCKS : nblocks;
            for (uint64_t h = b0; h < b1; h += 32) {
                const uint64_t bm = h + lane < b1 ? entry[h + lane] : 0;
                const int bc = b1 - h < 32 ? (int)(b1 - h) : 32;
                for (int j = 0; j < bc; j++) {
                    const int first = j;
                    j = advance_32(&s_val, bm, first, bc, lane, &at);
                    if (wwarp && lane >= first && lane < j) start[h + lane] = at;
                    if (j == bc) break;
                    if (writer) start[h + j] = s_val;
                    if (!stuck(s_val, __shfl_sync(0xffffffffu, bm, j)))
                        s_val = walk_block<T>(sv, dim, h + j, s_val, sm);
                }
            }
        }
    }
    if (writer) {
        start[nblocks] = s_val;
        sstart[nsuper] = s_val;
    }
}

// Pass 5: one thread per superblock the chain did not descend into; its blocks'
// deltas all apply (they share the superblock's binade and their sum stays in it).
__global__ void __launch_bounds__(256)
k_cdf_fill(const uint64_t* __restrict__ entry, uint64_t nblocks, uint64_t nsuper,
           const double* __restrict__ sstart, const uint32_t* __restrict__ desc,
           double* __restrict__ start)
{
    const uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nsuper || desc[s]) return;
    const uint64_t b0 = s * SUPER_BLOCKS;
    const uint64_t b1 = b0 + SUPER_BLOCKS < nblocks ? b0 + SUPER_BLOCKS : nblocks;
    double v = sstart[s];
    for (uint64_t b = b0; b < b1; b++) {
        start[b] = v;
        const uint64_t w = entry[b];
        const uint32_t c = entry_code(w);
        if (c != CODE_ZERO && c != CODE_NONE && v == v) advance(&v, c, entry_run(w));
    }
}

// Grid units of 16 consecutive chunks on binade `code`'s grid: lanes 2c and 2c + 1 receive
// chunk c's sum and whether it has no tie, NaN or inf.  The 16 loads a lane are in flight
// together and the 16 sums share one exchange (31 shuffles a lane instead of 160).
constexpr int SHOT_GROUP = 16;
// A state of few chunks is walked chunk by chunk: its shots lie a few chunks in, where a group's
// 16 loads and the kernel's 63 registers (34 without) only cost when there are many shots.
// svb_measure, chunks / groups in us, FP32 random state: 50,000 shots on 8, 10, 11, 12 qubits
// 332 / 451, 579 / 788, 865 / 1,125, 1,429 (chunks before groups) / 1,415; 1,000 shots on 10 and
// 11 qubits (FP64, uniform state) 81 / 73, 96 / 82.
constexpr bool shot_groups(int n, uint32_t shots) { return n >= 12 || (n >= 10 && shots <= 2048); }
template <typename T>
__device__ __forceinline__ uint64_t group_units(const typename VecOf<T>::type* __restrict__ sv, uint64_t dim,
                                                uint64_t first, uint32_t code, int lane, bool* fits)
{
    const Grid grid = grid_of(code);
    double p[SHOT_GROUP];
    uint64_t d[SHOT_GROUP];
    uint32_t bad = 0;
#pragma unroll
    for (int c = 0; c < SHOT_GROUP; c++) p[c] = prob_at<T>(sv, dim, first + (uint64_t)c * 32 + lane);
#pragma unroll
    for (int c = 0; c < SHOT_GROUP; c++) {
        bool ok = true;
        d[c] = grid_units(p[c], grid, &ok);
        if (!ok) bad |= 1u << c;
    }
    *fits = !(__reduce_or_sync(0xffffffffu, bad) >> (lane >> 1) & 1);
#pragma unroll
    for (int h = SHOT_GROUP / 2; h >= 1; h >>= 1) {
        const bool up = lane & (2 * h);          // this lane keeps the upper half of its sums
#pragma unroll
        for (int k = 0; k < h; k++) {
            const uint64_t mine = up ? d[k + h] : d[k], theirs = up ? d[k] : d[k + h];
            d[k] = mine + __shfl_xor_sync(0xffffffffu, theirs, 2 * h);
        }
    }
    return d[0] + __shfl_xor_sync(0xffffffffu, d[0], 1);
}

// Pass 6: one warp per shot.  start[] holds the reference's S at every block start
// (start[nblocks] = S_{2^n}); the block with start[b] <= r < start[b+1] is walked with
// the exact chunk sums until the first index j whose S_{j+1} exceeds r, which is the
// reference's j with S_j <= r < S_{j+1}.  A group of 16 chunks is summed at once; its first
// chunk that ties, leaves the binade or ends above r is added element by element, and only a
// new binade forms the sums again.  Bound by the slowest shot's chain of groups and chunks,
// which lies in block 0, where S crosses a binade or ties every few chunks: 1,024 shots took
// 94 us while such a group was added element by element throughout, 34 us now (n = 16; 30 at
// n = 23).  Shots with no such j (r >= S_{2^n}, r < 0 or
// NaN) give 0 as in the reference.
template <typename T, bool GROUPS>
__global__ void __launch_bounds__(256)
k_sample_exact(const typename VecOf<T>::type* __restrict__ sv, uint64_t dim, uint64_t nblocks,
               const double* __restrict__ start, const double* __restrict__ uniforms, uint32_t shots,
               uint64_t* __restrict__ out)
{
    const int lane = threadIdx.x & 31;
    const uint64_t shot = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (shot >= shots) return;
    const double r = uniforms[shot];
    uint64_t result = 0;
    if (r >= 0.0 && r < start[nblocks]) {
        uint64_t lo = 0, hi = nblocks;   // start[lo] <= r < start[hi]
        while (hi - lo > 1) {
            const uint64_t mid = lo + (hi - lo) / 2;
            if (start[mid] <= r) lo = mid;
            else hi = mid;
        }
        const uint64_t base = lo * BLOCK_AMPS;
        double s = start[lo];
        result = ~0ull;                  // replaced below: start[lo+1] > r is met inside the block
        uint32_t have = 0;               // binade code and group that the sums are formed for
        int group = -1;
        uint64_t units = 0;              // grid units of chunk group + lane / 2, and its ties
        bool fits = false;
        for (int cur = 0; cur < CHUNKS && base + (uint64_t)cur * 32 < dim;) {
            uint64_t m = 0;
            const uint32_t code = binade_of(s, &m);
            int f = cur;                 // chunk to add element by element
            if (GROUPS && code != 0) {
                const int g = cur & ~(SHOT_GROUP - 1);
                if (code != have || g != group) {
                    units = group_units<T>(sv, dim, base + (uint64_t)g * 32, code, lane, &fits);
                    have = code;
                    group = g;
                }
                const int c = g + (lane >> 1);
                const bool in = !(lane & 1) && c >= cur;
                const uint64_t v = in ? units : 0;
                uint64_t incl = v;       // 16 sums of at most 2^58: no wrap
#pragma unroll
                for (int o = 2; o < 32; o <<= 1) {
                    const uint64_t y = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += y;
                }
                const unsigned stop = __ballot_sync(
                    0xffffffffu, in && (!fits || incl > M_MAX - m || from_grid(code, m + incl) > r));
                const int l = stop ? __ffs(stop) - 1 : 30;
                s = from_grid(code, m + __shfl_sync(0xffffffffu, stop ? incl - v : incl, l));
                if (!stop) {
                    cur = g + SHOT_GROUP;
                    continue;
                }
                f = g + (l >> 1);
            }
            const uint64_t i0 = base + (uint64_t)f * 32;
            const double incl = chunk_scan_exact(s, prob_at<T>(sv, dim, i0 + lane), lane);
            const unsigned hit = __ballot_sync(0xffffffffu, incl > r);
            if (hit) {
                result = i0 + (uint64_t)(__ffs(hit) - 1);
                break;
            }
            s = __shfl_sync(0xffffffffu, incl, 31);
            cur = f + 1;
        }
    }
    if (lane == 0) out[shot] = result;
}

template <typename T, bool FOUR>
__global__ void __launch_bounds__(256)
k_pauli_expect(const typename VecOf<T>::type* __restrict__ sv, uint64_t dim,
               const svb_pauli_term* __restrict__ terms, int n_terms, double* __restrict__ partial)
{
    extern __shared__ svb_pauli_term sterms[];
    __shared__ double red[8];
    for (int t = threadIdx.x; t < n_terms; t += blockDim.x) sterms[t] = terms[t];
    __syncthreads();
    double acc = 0.0;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < dim; i += (FOUR ? PAULI_U : 1) * stride)
        acc += FOUR ? pauli_energy<T>(sv, i, stride, dim, sterms, n_terms)
                    : pauli_energy_one<T>(sv, i, sterms, n_terms);
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += red[w];
        partial[blockIdx.x] = s;
    }
}

__global__ void k_sum_partials(const double* __restrict__ partial, int count, double* __restrict__ out)
{
    // one warp, fixed order: deterministic
    double s = 0.0;
    for (int i = threadIdx.x; i < count; i += 32) s += partial[i];
    s = warp_sum(s);
    if (threadIdx.x == 0) *out = s;
}

template <typename TA, typename TB>
__global__ void __launch_bounds__(256)
k_compare(const typename VecOf<TA>::type* __restrict__ a, const typename VecOf<TB>::type* __restrict__ b,
          uint64_t dim, double* __restrict__ partial)
{
    __shared__ double red[5][8];
    double re = 0, im = 0, na = 0, nb = 0, mx = 0;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < dim; i += stride) {
        const double ar = (double)a[i].x, ai = (double)a[i].y;
        const double br = (double)b[i].x, bi = (double)b[i].y;
        re += ar * br + ai * bi;            // conj(a) b
        im += ar * bi - ai * br;
        na += ar * ar + ai * ai;
        nb += br * br + bi * bi;
        const double dr = ar - br, di = ai - bi;
        mx = fmax(mx, sqrt(dr * dr + di * di));
    }
    double v[5] = {re, im, na, nb, mx};
#pragma unroll
    for (int q = 0; q < 5; q++) {
        double x = v[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double y = __shfl_xor_sync(0xffffffffu, x, o);
            x = (q == 4) ? fmax(x, y) : x + y;
        }
        if ((threadIdx.x & 31) == 0) red[q][threadIdx.x >> 5] = x;
    }
    __syncthreads();
    if (threadIdx.x < 5) {
        const int q = threadIdx.x;
        double x = red[q][0];
        for (int w = 1; w < (int)(blockDim.x >> 5); w++) x = (q == 4) ? fmax(x, red[q][w]) : x + red[q][w];
        partial[(size_t)q * gridDim.x + blockIdx.x] = x;
    }
}

__global__ void k_compare_final(const double* __restrict__ partial, int blocks, double* __restrict__ out)
{
    if (threadIdx.x != 0) return;
    double v[5] = {0, 0, 0, 0, 0};
    for (int q = 0; q < 5; q++)
        for (int i = 0; i < blocks; i++) {
            const double x = partial[(size_t)q * blocks + i];
            v[q] = (q == 4) ? fmax(v[q], x) : v[q] + x;
        }
    for (int q = 0; q < 5; q++) out[q] = v[q];
}

}  // namespace

template <typename TA, typename TB>
cudaError_t compare_device(const void* a, const void* b, int n, double* d_out5, double* d_partial5,
                           cudaStream_t s)
{
    const uint64_t dim = 1ull << n;
    k_compare<TA, TB><<<REDUCE_BLOCKS, 256, 0, s>>>(static_cast<const typename VecOf<TA>::type*>(a),
                                                   static_cast<const typename VecOf<TB>::type*>(b), dim,
                                                   d_partial5);
    k_compare_final<<<1, 32, 0, s>>>(d_partial5, REDUCE_BLOCKS, d_out5);
    return cudaGetLastError();
}
template cudaError_t compare_device<double, double>(const void*, const void*, int, double*, double*, cudaStream_t);
template cudaError_t compare_device<double, float>(const void*, const void*, int, double*, double*, cudaStream_t);
template cudaError_t compare_device<float, double>(const void*, const void*, int, double*, double*, cudaStream_t);
template cudaError_t compare_device<float, float>(const void*, const void*, int, double*, double*, cudaStream_t);

size_t measure_scratch_doubles(int n) { return (size_t)measure_layout(n).doubles; }

template <typename T>
cudaError_t measure_device(const void* state, int n, const double* d_uniforms, uint32_t shots,
                           uint64_t* d_samples, double* d_total, MeasureScratch& scr, cudaStream_t s)
{
    using V = typename VecOf<T>::type;
    const MeasureLayout L = measure_layout(n);
    if (!scr.cdf || scr.cap_doubles < L.doubles) return cudaErrorInvalidValue;
    const V* sv = static_cast<const V*>(state);
    const uint64_t dim = 1ull << n;
    double* base = scr.cdf;
    uint64_t* entry = reinterpret_cast<uint64_t*>(base + L.off_entry);
    double* start = base + L.off_start;
    uint64_t* sentry = reinterpret_cast<uint64_t*>(base + L.off_sentry);
    double* sstart = base + L.off_sstart;
    uint32_t* desc = reinterpret_cast<uint32_t*>(base + L.off_desc);
    const unsigned blocks = (unsigned)(L.nblocks < 148u * 16 ? L.nblocks : 148u * 16);
    if (L.nblocks <= WALK_BLOCKS) {
        k_cdf_chain<T><<<1, CHAIN_THREADS, 0, s>>>(sv, dim, L.nblocks, L.nsuper, nullptr, nullptr, start, sstart, desc);
    } else {
        // 1. approximate block sums (into the entry array) and their prefix (into start)
        k_block_sums<T><<<blocks, 256, 0, s>>>(sv, dim, L.nblocks, base + L.off_entry);
        k_scan_single<<<1, 1024, 0, s>>>(base + L.off_entry, L.nblocks, start);
        // 2-5. exact block starts
        k_cdf_blocks<T><<<blocks, 256, 0, s>>>(sv, dim, L.nblocks, start, entry);
        const unsigned sb = (unsigned)((L.nsuper + 255) / 256);
        k_cdf_super<<<sb, 256, 0, s>>>(entry, L.nblocks, L.nsuper, sentry);
        k_cdf_chain<T><<<1, CHAIN_THREADS, 0, s>>>(sv, dim, L.nblocks, L.nsuper, entry, sentry, start, sstart, desc);
        k_cdf_fill<<<sb, 256, 0, s>>>(entry, L.nblocks, L.nsuper, sstart, desc, start);
    }
    // 6. samples
    if (shots > 0) {
        const unsigned sblocks = (unsigned)(((uint64_t)shots * 32 + 255) / 256);
        if (shot_groups(n, shots))
            k_sample_exact<T, true><<<sblocks, 256, 0, s>>>(sv, dim, L.nblocks, start, d_uniforms, shots, d_samples);
        else
            k_sample_exact<T, false><<<sblocks, 256, 0, s>>>(sv, dim, L.nblocks, start, d_uniforms, shots, d_samples);
    }
    cudaError_t e = cudaSuccess;
    if (d_total)
        e = cudaMemcpyAsync(d_total, start + L.nblocks, sizeof(double), cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

template <typename T>
cudaError_t norm2_device(const void* state, int n, double* d_total, MeasureScratch& scr, cudaStream_t s)
{
    using V = typename VecOf<T>::type;
    const MeasureLayout L = measure_layout(n);
    if (!scr.cdf || scr.cap_doubles < L.doubles) return cudaErrorInvalidValue;
    double* base = scr.cdf;
    const unsigned blocks = (unsigned)(L.nblocks < 148u * 16 ? L.nblocks : 148u * 16);
    k_block_sums<T><<<blocks, 256, 0, s>>>(static_cast<const V*>(state), 1ull << n, L.nblocks, base + L.off_entry);
    k_scan_single<<<1, 1024, 0, s>>>(base + L.off_entry, L.nblocks, base + L.off_start);
    cudaError_t e = cudaMemcpyAsync(d_total, base + L.off_start + L.nblocks, sizeof(double),
                                    cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

template <typename T>
cudaError_t expectation_device(const void* state, int n, const svb_pauli_term* d_terms, int n_terms,
                               double* d_out, double* d_partial, cudaStream_t s)
{
    using V = typename VecOf<T>::type;
    const uint64_t dim = 1ull << n;
    const size_t smem = sizeof(svb_pauli_term) * (size_t)n_terms;
    if (pauli_by_four(dim, n_terms, PAULI_STATE_BITS))
        k_pauli_expect<T, true><<<REDUCE_BLOCKS, 256, smem, s>>>(static_cast<const V*>(state), dim, d_terms,
                                                                  n_terms, d_partial);
    else
        k_pauli_expect<T, false><<<REDUCE_BLOCKS, 256, smem, s>>>(static_cast<const V*>(state), dim, d_terms,
                                                                   n_terms, d_partial);
    k_sum_partials<<<1, 32, 0, s>>>(d_partial, REDUCE_BLOCKS, d_out);
    return cudaGetLastError();
}

#define SVB_MEAS_INST(T)                                                                    \
    template cudaError_t measure_device<T>(const void*, int, const double*, uint32_t,       \
                                           uint64_t*, double*, MeasureScratch&, cudaStream_t); \
    template cudaError_t norm2_device<T>(const void*, int, double*, MeasureScratch&, cudaStream_t); \
    template cudaError_t expectation_device<T>(const void*, int, const svb_pauli_term*, int, \
                                               double*, double*, cudaStream_t);
SVB_MEAS_INST(double)
SVB_MEAS_INST(float)

}  // namespace svb
