// Shared device utilities for the subsetix B200 kernels.
//
// * Device flag codes raised by kernels and reported through the C ABI.
// * Single-pass chained scan with decoupled look-back for block tiles.  Tile
//   ids are handed out dynamically.  Every launch clears its own state first
//   (a memset on its stream), so the workspace may hold any earlier scratch.
// * A block-wide exclusive scan.
#pragma once

#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>

#define SX_MAX_LEAVES 9
#define SX_TABLE_MAX_LEAVES 8
#define SX_BLOCK 256

// Bits of the device flag word that kernels raise.
#define SXF_CONTRACT 1u   // input outside the fast path's contract: rerun the exact path
#define SXF_LONG_TILE 2u  // a row too long, or a tile too wide, for the staged sweep that was asked for
#define SXF_CAPACITY 4u   // an output would have exceeded the caller's capacity
#define SXF_TIMEOUT 8u    // a bounded wait gave up (look-back predecessor never published)

// Scan state kept in caller workspace.  status[t] holds the published value
// of tile t: bits 0-31 the value, bits 32-33 the kind (1 = tile aggregate,
// 2 = inclusive prefix), bits 34-63 the launch epoch.  counters[0] hands out
// tile tickets, counters[1] counts finished tiles, counters[2] is the epoch
// and counters[3] accumulates the SXF_* flags.
struct SxScanState {
    unsigned long long* status;
    unsigned int* counters;
    int max_tiles;
};

#define SX_EPOCH_MASK 0x3FFFFFFFu
#define SX_KIND_AGG 1ull
#define SX_KIND_PREFIX 2ull
#define SX_LOOKBACK_SPIN_LIMIT (1u << 22)

__device__ __forceinline__ unsigned long long sx_pack(unsigned epoch, unsigned long long kind, int value)
{
    return ((unsigned long long)(epoch & SX_EPOCH_MASK) << 34) | (kind << 32) | (unsigned long long)(unsigned)value;
}

__device__ __forceinline__ void sx_publish(unsigned long long* slot, unsigned long long word)
{
    atomicExch(slot, word);
}

// Thread 0 takes a tile ticket and reads the epoch.  Every thread of the
// block gets both back through shared memory.
__device__ __forceinline__ void sx_ticket(const SxScanState& st, int* s_tile, unsigned* s_epoch)
{
    if (threadIdx.x == 0) {
        *s_tile = (int)atomicAdd(&st.counters[0], 1u);
        *s_epoch = *((volatile unsigned*)&st.counters[2]) & SX_EPOCH_MASK;
    }
    __syncthreads();
}

// Decoupled look-back, run by one full warp.  Returns the exclusive prefix
// of tile `tile` and publishes its inclusive prefix.  Every wait is bounded.
// If a predecessor never publishes, SXF_TIMEOUT is raised in `flags` and its
// value counts as zero, so the kernel always finishes.
__device__ __forceinline__ int sx_lookback_warp(const SxScanState& st, int tile, unsigned epoch, int aggregate,
                                                unsigned& flags)
{
    const int lane = threadIdx.x & 31;
    if (tile == 0) {
        if (lane == 0) sx_publish(&st.status[0], sx_pack(epoch, SX_KIND_PREFIX, aggregate));
        return 0;
    }
    if (lane == 0) sx_publish(&st.status[tile], sx_pack(epoch, SX_KIND_AGG, aggregate));
    int exclusive = 0;
    int pos = tile - 1;
    bool timed_out = false;
    while (true) {
        int t = pos - lane;
        unsigned long long word = 0ull;
        unsigned kind = SX_KIND_PREFIX;  // lanes past tile 0 act as a zero prefix
        int value = 0;
        if (t >= 0) {
            unsigned spins = 0;
            while (true) {
                word = *((volatile unsigned long long*)&st.status[t]);
                unsigned e = (unsigned)(word >> 34) & SX_EPOCH_MASK;
                kind = (unsigned)((word >> 32) & 3ull);
                if (e == epoch && kind != 0) break;
                if (++spins > SX_LOOKBACK_SPIN_LIMIT) {
                    timed_out = true;
                    kind = SX_KIND_PREFIX;
                    word = 0ull;
                    break;
                }
                if (spins > 8) __nanosleep(64);
            }
            value = (int)(unsigned)(word & 0xFFFFFFFFull);
        }
        unsigned prefix_mask = __ballot_sync(0xFFFFFFFFu, kind == SX_KIND_PREFIX);
        int stop_lane = prefix_mask ? (__ffs(prefix_mask) - 1) : 32;
        int contrib = (lane <= stop_lane) ? value : 0;
        for (int o = 16; o > 0; o >>= 1) contrib += __shfl_xor_sync(0xFFFFFFFFu, contrib, o);
        exclusive += contrib;
        if (prefix_mask) break;
        pos -= 32;
    }
    if (__any_sync(0xFFFFFFFFu, timed_out)) flags |= SXF_TIMEOUT;
    if (lane == 0) sx_publish(&st.status[tile], sx_pack(epoch, SX_KIND_PREFIX, exclusive + aggregate));
    return exclusive;
}

// End of kernel.  Every block ORs its flags into counters[3].  The last
// block to finish then writes result[0] (the inclusive prefix of the last
// tile, i.e. the grand total) and result[1] (the flags).
__device__ __forceinline__ void sx_retire(const SxScanState& st, unsigned epoch, unsigned block_flags, int* result)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        if (block_flags) atomicOr(&st.counters[3], block_flags);
        __threadfence();
        unsigned prev = atomicAdd(&st.counters[1], 1u);
        if (prev == gridDim.x - 1) {
            __threadfence();
            unsigned long long last = *((volatile unsigned long long*)&st.status[gridDim.x - 1]);
            unsigned flags = atomicExch(&st.counters[3], 0u);
            if (result) {
                result[0] = (int)(unsigned)(last & 0xFFFFFFFFull);
                result[1] = (int)flags;
            }
            atomicExch(&st.counters[2], (epoch + 1u) & SX_EPOCH_MASK);
        }
    }
}

// Block-wide exclusive scan of one int per thread (blockDim.x == SX_BLOCK).
// Returns the exclusive prefix; *total receives the block total.
__device__ __forceinline__ int sx_block_exclusive_scan(int v, int* s_warp, int* total)
{
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = (lane < (SX_BLOCK / 32)) ? s_warp[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xFFFFFFFFu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < (SX_BLOCK / 32)) s_warp[lane] = w;
    }
    __syncthreads();
    int warp_prefix = warp > 0 ? s_warp[warp - 1] : 0;
    int result = warp_prefix + x - v;
    if (total) *total = s_warp[SX_BLOCK / 32 - 1];
    __syncthreads();
    return result;
}

// ---------------------------------------------------------------------------
// The reference's float32 formulas with the contraction its NVRTC build
// applies.  The reference compiles its kernels with NVRTC's default
// --fmad=true, which fuses each multiply into the add that consumes it:
//   upwind  c - dt * (a * du_dx + b * du_dy)  ->  fma(-dt, fma(a, du_dx, b * du_dy), c)
//   |grad|  sqrtf(gx * gx + gy * gy)           ->  sqrt(fma(gx, gx, gy * gy))
// (interval_stencil.py:105-111, regrid.py:196-217; established on a B200 by
// running the reference's own kernels, compiled with its NVRTC options,
// against every candidate grouping: only this one agrees on every cell).
// Float64 has no reference counterpart and rounds every operation once.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float sx_upwind_update(float c, float du_dx, float du_dy, float a, float b, float dt)
{
    return __fmaf_rn(-dt, __fmaf_rn(a, du_dx, __fmul_rn(b, du_dy)), c);
}

__device__ __forceinline__ double sx_upwind_update(double c, double du_dx, double du_dy, double a, double b, double dt)
{
    return __dsub_rn(c, __dmul_rn(dt, __dadd_rn(__dmul_rn(a, du_dx), __dmul_rn(b, du_dy))));
}

__device__ __forceinline__ float sx_grad_norm(float gx, float gy)
{
    return __fsqrt_rn(__fmaf_rn(gx, gx, __fmul_rn(gy, gy)));
}

// ---------------------------------------------------------------------------
// Division by a divisor known beforehand: with z = RN(1 / d), q = RN(x z) and the
// remainder r = q d - x, which one fma gives exactly, RN(q - r z) is the correctly
// rounded x / d (P. Markstein, IBM J. Res. Dev. 34, 1990; N. Brisebarre, J.-M. Muller
// and S. K. Raina, IEEE Trans. Computers 53, 2004) as long as nothing under- or
// overflows: three operations instead of a general division.  For d within
// 2^-60 .. 2^24 (SX_BY_CONST is only chosen then) that holds for x = 0 (either sign: r
// is +0 then, so -r z is -0 and leaves q as it is; x - q d would turn -0 into +0)
// and for |x| >= 2^-100 (float32) or 2^-900 (float64); a quotient that
// overflows comes out as NaN.  So callers test for smaller x and for results that
// are not finite, and divide there.  (Float32: 2^64 x is large enough for every x, and
// 2^-64 times the quotient is exact unless the result is subnormal: SX_BY_SCALED, for
// fields with tails below 2^-76.  For those the three operations in float64 and one
// rounding to float32 are exact: a quotient of 24-bit numbers is either a tie of two
// neighbours, and a float64 number, or at least 2^-49 of itself away from it.)
// ---------------------------------------------------------------------------
#define SX_BY_DIVISION 0  // divide
#define SX_BY_POW2 1      // multiply by the exact reciprocal of a power of two
#define SX_BY_CONST 2     // the three operations above
#define SX_BY_SCALED 3    // the same on 2^64 x (float32), for small x
#define SX_BY_DOUBLE 4    // the same in float64 (float32), for subnormal quotients

// Magnitudes below which a nonzero value counts as small, as high words shifted left
// by one: differences of values that are zero or above it are zero or above
// 2^-100 (float32) and 2^-900 (float64), where the remainder is exact.
#define SX_SMALL_F32 ((unsigned)(127 - 76) << 24)
#define SX_SMALL_F64 ((unsigned)(1023 - 840) << 21)

// Order key of |x| in which zero comes last: min over several values < SX_SMALL says
// that one of them is small and not zero.
__device__ __forceinline__ unsigned sx_small_key(float x) { return 2u * __float_as_uint(x) - 1u; }
__device__ __forceinline__ unsigned sx_small_key(double x)
{
    return (2u * (unsigned)__double2hiint(x) | (__double2loint(x) != 0 ? 1u : 0u)) - 1u;
}
// The same for the differences themselves (x above): 2^-100 and 2^-900, and the
// magnitudes from which a quotient may overflow (d >= 2^-60): 2^60 and 2^900.
#define SX_SMALL_DIFF_F32 ((unsigned)(127 - 100) << 24)
#define SX_SMALL_DIFF_F64 ((unsigned)(1023 - 900) << 21)
#define SX_LARGE_DIFF_F32 ((unsigned)(127 + 60) << 24)
#define SX_LARGE_DIFF_F64 ((unsigned)(1023 + 900) << 21)
__device__ __forceinline__ unsigned sx_large_key(float x) { return 2u * __float_as_uint(x); }
__device__ __forceinline__ unsigned sx_large_key(double x) { return 2u * (unsigned)__double2hiint(x); }

// x / d by the three operations, z = RN(1 / d).
__device__ __forceinline__ float sx_by_const(float x, float d, float z)
{
    const float q = __fmul_rn(x, z);
    return __fmaf_rn(-__fmaf_rn(q, d, -x), z, q);
}
__device__ __forceinline__ double sx_by_const(double x, double d, double z)
{
    const double q = __dmul_rn(x, z);
    return __fma_rn(-__fma_rn(q, d, -x), z, q);
}

template <typename T>
__host__ __device__ inline bool sx_known_divisor(T d)
{
    return d >= (T)0x1p-60 && d <= (T)0x1p24;
}
// The key of a subnormal value, nonzero.
template <typename T>
__device__ __forceinline__ bool sx_is_subnormal(unsigned key)
{
    return key < (sizeof(T) == 4 ? 1u << 24 : 1u << 21) - 1u;
}
template <typename T>
__device__ __forceinline__ bool sx_is_small(unsigned key)
{
    return key < (sizeof(T) == 4 ? SX_SMALL_F32 : SX_SMALL_F64);
}

// ---------------------------------------------------------------------------
// Arithmetic helpers without contraction (float and double)
// ---------------------------------------------------------------------------
__device__ __forceinline__ float sx_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sx_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float sx_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float sx_div(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ float sx_sqrt(float a) { return __fsqrt_rn(a); }
__device__ __forceinline__ double sx_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sx_sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double sx_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double sx_div(double a, double b) { return __ddiv_rn(a, b); }

// x / d, or x * d when the launcher passed the reciprocal of a power-of-two
// spacing instead (pow2 != 0): dividing by 2^k and multiplying by 2^-k have
// the same exact real result, so the rounded results are identical.
template <typename T>
__device__ __forceinline__ T sx_over(T x, T d, int pow2)
{
    return pow2 ? sx_mul(x, d) : sx_div(x, d);
}

// Spacings that are powers of two (in the kernel's precision) become their
// exact reciprocals.
template <typename T>
inline int sx_pow2_pair(T& dx, T& dy)
{
    int ex, ey;
    if (!(frexp((double)dx, &ex) == 0.5 && frexp((double)dy, &ey) == 0.5)) return 0;
    const T ix = (T)1 / dx, iy = (T)1 / dy;
    if (!std::isfinite((double)ix) || !std::isfinite((double)iy)) return 0;  // reciprocal out of range
    dx = ix;
    dy = iy;
    return 1;
}

// Row ordinal of interval i: the last p with off[p] <= i and off[p+1] > i.
__device__ __forceinline__ int sx_row_of(const int* __restrict__ off, int rows, int i)
{
    int lo = 0, hi = rows - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= i) lo = mid; else hi = mid - 1;
    }
    return lo;
}
