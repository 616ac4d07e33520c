// Threshold run-length encoding and gradient magnitude of a full width x height
// grid (subsetix_amr2/regrid.py:20-124,172-333).
//
//   sx_threshold_mask  one bit per cell: value >= threshold, the value being the
//                      grid itself or its gradient magnitude (formulas of
//                      sx_threshold_rle), then the exclusive scan of the rows'
//                      run counts (a look-back over blocks of rows);
//   sx_mask_runs       the runs of the bit mask, written at the rows' offsets.
//
// The number of runs has to be known before they can be stored, and counting
// with one warp per row and then doing it all again (sx_threshold_rle) reads the
// field twice with 28 warps per SM whose loads wait for a ballot each: 161 us for
// both passes on 4096^2, where one read of the field takes 10 us at the copy
// rate.  The mask is 1/32 of the field and stays in L2.  A warp takes 128 columns
// of RLE_ROWS rows, four cells per lane by 16-byte loads, all loaded before the
// first is used.  Measured (B200, gradient tags on 4096^2): mask 27 us, count
// 7.9 us, runs 3 us; one kernel with the counts and the look-back inside the mask
// pass took 36 us (blocks wait at its barriers and in its tail), 49 us with the
// square root that sx_least_radicand removes.

#include <cmath>
#include <cstring>

#include "sx_internal.cuh"

namespace {

constexpr int RLE_THREADS = 256;
// Rows per warp: 2, 4 and 8 took 29, 26.6 and 30 us on 4096^2 (gradient tags).
constexpr int RLE_ROWS = 4;
constexpr int NARROW = 48;  // columns below which the gradient takes a cell per thread

// Cells of one row in a warp's 128-column strip: lane's cells are x0 + 4 lane ..
// + 3 with VEC (rows 16-byte aligned, width a multiple of 4), else x0 + lane +
// 32 k.  `before` and `after` are the cells next to the strip (lanes 0 and 31).
struct Strip {
    float v[4];
    float before, after;
};

template <bool GRAD, bool VEC>
__device__ __forceinline__ Strip load_strip(const float* __restrict__ d, int x0, int y, int W, int H, int lane)
{
    Strip s;
#pragma unroll
    for (int k = 0; k < 4; ++k) s.v[k] = 0.0f;
    s.before = s.after = 0.0f;
    if (y < 0 || y >= H) return s;
    const float* row = d + (long long)y * W;
    if (VEC) {
        const int x = x0 + 4 * lane;
        if (x < W) {  // the width is a multiple of 4
            const float4 q = *(const float4*)(row + x);
            s.v[0] = q.x; s.v[1] = q.y; s.v[2] = q.z; s.v[3] = q.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int x = x0 + lane + 32 * k;
            if (x < W) s.v[k] = row[x];
        }
    }
    if (GRAD) {
        if (lane == 0 && x0 > 0 && x0 <= W) s.before = row[x0 - 1];
        if (lane == 31 && x0 + 128 < W) s.after = row[x0 + 128];
    }
    return s;
}

// The radicand of sx_grad_norm.  A correctly rounded square root never falls, so
// sqrt(s) >= threshold is s >= the smallest radicand whose root reaches the
// threshold (sx_least_radicand, found on the host): same bits, no square root.
__device__ __forceinline__ float grad_square(float gx, float gy) { return __fmaf_rn(gx, gx, __fmul_rn(gy, gy)); }

// Left and right neighbours of a strip's cells.
template <bool VEC>
__device__ __forceinline__ void strip_sides(const Strip& cur, int lane, float (&left)[4], float (&right)[4])
{
    if (VEC) {
        float l = __shfl_up_sync(0xFFFFFFFFu, cur.v[3], 1);
        float r = __shfl_down_sync(0xFFFFFFFFu, cur.v[0], 1);
        if (lane == 0) l = cur.before;
        if (lane == 31) r = cur.after;
        left[0] = l; left[1] = cur.v[0]; left[2] = cur.v[1]; left[3] = cur.v[2];
        right[0] = cur.v[1]; right[1] = cur.v[2]; right[2] = cur.v[3]; right[3] = r;
    } else {
        const float first = __shfl_sync(0xFFFFFFFFu, cur.before, 0), last = __shfl_sync(0xFFFFFFFFu, cur.after, 31);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            left[k] = __shfl_up_sync(0xFFFFFFFFu, cur.v[k], 1);
            right[k] = __shfl_down_sync(0xFFFFFFFFu, cur.v[k], 1);
            const float l = k > 0 ? __shfl_sync(0xFFFFFFFFu, cur.v[k > 0 ? k - 1 : 0], 31) : first;
            const float r = k < 3 ? __shfl_sync(0xFFFFFFFFu, cur.v[k < 3 ? k + 1 : 3], 0) : last;
            if (lane == 0) left[k] = l;
            if (lane == 31) right[k] = r;
        }
    }
}

// Gradient components of a cell: half central differences inside, one-sided at
// the grid's edges.  INNER: the strip holds no edge cell.
template <bool INNER>
__device__ __forceinline__ void cell_gradient(float c, float left, float right, float up, float down, int x, int y,
                                              int W, int H, float& gx, float& gy)
{
    if (INNER) {
        gx = __fmul_rn(__fsub_rn(right, left), 0.5f);
        gy = __fmul_rn(__fsub_rn(down, up), 0.5f);
        return;
    }
    gx = gy = 0.0f;
    if (W > 1) {
        if (x == 0) gx = __fsub_rn(right, c);
        else if (x == W - 1) gx = __fsub_rn(c, left);
        else gx = __fmul_rn(__fsub_rn(right, left), 0.5f);
    }
    if (H > 1) {
        if (y == 0) gy = __fsub_rn(down, c);
        else if (y == H - 1) gy = __fsub_rn(c, up);
        else gy = __fmul_rn(__fsub_rn(down, up), 0.5f);
    }
}

// The strip's predicate bits of one row as four words, the same on every lane.
template <bool GRAD, bool VEC>
__device__ __forceinline__ void strip_words(const Strip& up, const Strip& cur, const Strip& down, int x0, int y, int W,
                                            int H, float thr, int lane, unsigned (&words)[4])
{
    float left[4], right[4];
    if (GRAD) strip_sides<VEC>(cur, lane, left, right);
    // a strip without the grid's first and last columns and rows takes the plain central differences
    const bool inner = GRAD && x0 > 0 && x0 + 128 < W && y > 0 && y + 1 < H;
    unsigned mine = 0u;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int x = VEC ? x0 + 4 * lane + k : x0 + lane + 32 * k;
        bool on;
        if (!GRAD) {
            on = cur.v[k] >= thr && x < W && y < H;
        } else {
            float gx, gy;
            if (inner) cell_gradient<true>(cur.v[k], left[k], right[k], up.v[k], down.v[k], x, y, W, H, gx, gy);
            else cell_gradient<false>(cur.v[k], left[k], right[k], up.v[k], down.v[k], x, y, W, H, gx, gy);
            on = grad_square(gx, gy) >= thr && (inner || (x < W && y < H));
        }
        if (VEC) mine |= (on ? 1u : 0u) << k;
        else words[k] = __ballot_sync(0xFFFFFFFFu, on);
    }
    if (VEC) {  // lanes 8 k .. 8 k + 7 hold word k, four bits each
        unsigned w = mine << (4 * (lane & 7));
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) w |= __shfl_xor_sync(0xFFFFFFFFu, w, o);
#pragma unroll
        for (int k = 0; k < 4; ++k) words[k] = __shfl_sync(0xFFFFFFFFu, w, 8 * k);
    }
}

// One warp per 128 columns and RLE_ROWS rows; neighbouring warps take neighbouring strips.
template <bool GRAD, bool VEC>
__global__ void __launch_bounds__(RLE_THREADS)
    mask_kernel(const float* __restrict__ d, int W, int H, float thr, unsigned* __restrict__ mask, int words_per_row,
                int strips, long long tasks)
{
    const long long task = ((long long)blockIdx.x * RLE_THREADS + threadIdx.x) >> 5;
    if (task >= tasks) return;
    const int lane = threadIdx.x & 31;
    const int x0 = (int)(task % strips) * 128, y0 = (int)(task / strips) * RLE_ROWS;
    // every row is loaded before the first is used: one round trip per task
    Strip rows[RLE_ROWS + 2];
    if (GRAD) rows[0] = load_strip<false, VEC>(d, x0, y0 - 1, W, H, lane);
#pragma unroll
    for (int r = 0; r < RLE_ROWS; ++r) rows[r + 1] = load_strip<GRAD, VEC>(d, x0, y0 + r, W, H, lane);
    if (GRAD) rows[RLE_ROWS + 1] = load_strip<false, VEC>(d, x0, y0 + RLE_ROWS, W, H, lane);
#pragma unroll
    for (int r = 0; r < RLE_ROWS; ++r) {
        unsigned words[4];
        strip_words<GRAD, VEC>(rows[r], rows[r + 1], rows[r + 2], x0, y0 + r, W, H, thr, lane, words);
        const unsigned lo = lane & 1 ? words[1] : words[0], hi = lane & 1 ? words[3] : words[2];
        const int w = (x0 >> 5) + lane;
        if (lane < 4 && w < words_per_row && y0 + r < H)
            mask[(long long)(y0 + r) * words_per_row + w] = lane & 2 ? hi : lo;
    }
}

// Gradient magnitude of every cell, the same strips (90 us with one thread and
// five loads per cell on 4096^2, 32 us here; 20 us at the copy rate).
template <bool VEC>
__global__ void __launch_bounds__(RLE_THREADS)
    gradient_kernel(const float* __restrict__ d, int W, int H, float* __restrict__ out, int strips, long long tasks)
{
    const long long task = ((long long)blockIdx.x * RLE_THREADS + threadIdx.x) >> 5;
    if (task >= tasks) return;
    const int lane = threadIdx.x & 31;
    const int x0 = (int)(task % strips) * 128, y0 = (int)(task / strips) * RLE_ROWS;
    Strip rows[RLE_ROWS + 2];
    rows[0] = load_strip<false, VEC>(d, x0, y0 - 1, W, H, lane);
#pragma unroll
    for (int r = 0; r < RLE_ROWS; ++r) rows[r + 1] = load_strip<true, VEC>(d, x0, y0 + r, W, H, lane);
    rows[RLE_ROWS + 1] = load_strip<false, VEC>(d, x0, y0 + RLE_ROWS, W, H, lane);
#pragma unroll
    for (int r = 0; r < RLE_ROWS; ++r) {
        const int y = y0 + r;
        const bool inner = x0 > 0 && x0 + 128 < W && y > 0 && y + 1 < H;
        float left[4], right[4], g[4];
        strip_sides<VEC>(rows[r + 1], lane, left, right);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int x = VEC ? x0 + 4 * lane + k : x0 + lane + 32 * k;
            float gx, gy;
            if (inner)
                cell_gradient<true>(rows[r + 1].v[k], left[k], right[k], rows[r].v[k], rows[r + 2].v[k], x, y, W, H, gx,
                                    gy);
            else
                cell_gradient<false>(rows[r + 1].v[k], left[k], right[k], rows[r].v[k], rows[r + 2].v[k], x, y, W, H,
                                     gx, gy);
            g[k] = sx_grad_norm(gx, gy);
        }
        if (y >= H) continue;
        float* o = out + (long long)y * W;
        if (VEC) {
            if (x0 + 4 * lane < W) *(float4*)(o + x0 + 4 * lane) = make_float4(g[0], g[1], g[2], g[3]);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (x0 + lane + 32 * k < W) o[x0 + lane + 32 * k] = g[k];
        }
    }
}

// The same for narrow grids, a cell per thread: strips leave most lanes of a warp
// without a cell (200,000 rows, strips and this kernel: 3 columns 62 and 6.3 us, 16
// columns 55 and 17, 32 columns 55 and 25; strips take 55 us for 64 columns too).
__global__ void __launch_bounds__(RLE_THREADS)
    narrow_gradient_kernel(const float* __restrict__ d, int W, int H, float* __restrict__ out)
{
    const long long cells = (long long)W * H, step = (long long)gridDim.x * RLE_THREADS;
    for (long long i = (long long)blockIdx.x * RLE_THREADS + threadIdx.x; i < cells; i += step) {
        const int y = (int)(i / W), x = (int)(i - (long long)y * W);
        const float left = x > 0 ? d[i - 1] : 0.0f, right = x + 1 < W ? d[i + 1] : 0.0f;
        const float up = y > 0 ? d[i - W] : 0.0f, down = y + 1 < H ? d[i + W] : 0.0f;
        float gx, gy;
        cell_gradient<false>(d[i], left, right, up, down, x, y, W, H, gx, gy);
        out[i] = sx_grad_norm(gx, gy);
    }
}

// Exclusive scan of the rows' run counts: a warp counts the run starts of a row,
// a block of eight rows takes its place by a look-back.
__global__ void __launch_bounds__(RLE_THREADS) mask_count_kernel(const unsigned* __restrict__ mask, int H,
                                                                 int words_per_row, int* __restrict__ offsets,
                                                                 int* result, SxScanState st)
{
    __shared__ int s_count[8];
    __shared__ int s_tile;
    __shared__ unsigned s_epoch, s_flags;
    sx_ticket(st, &s_tile, &s_epoch);
    const int tile = s_tile;
    const unsigned epoch = s_epoch;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int y0 = tile * 8, y = y0 + warp;
    int runs = 0;
    if (y < H) {
        const unsigned* row = mask + (long long)y * words_per_row;
#pragma unroll 4
        for (int w = lane; w < words_per_row; w += 32) {
            const unsigned m = row[w], prev = w > 0 ? row[w - 1] >> 31 : 0u;
            runs += __popc(m & ~((m << 1) | prev));
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) runs += __shfl_xor_sync(0xFFFFFFFFu, runs, o);
    if (lane == 0) s_count[warp] = runs;
    __syncthreads();
    if (warp == 0) {
        const int mine = lane < 8 ? s_count[lane] : 0;
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += v;
        }
        unsigned f = 0u;
        const int base = sx_lookback_warp(st, tile, epoch, __shfl_sync(0xFFFFFFFFu, incl, 31), f);
        if (lane < 8 && y0 + lane < H) offsets[y0 + lane] = base + incl - mine;
        if (lane < 8 && y0 + lane == H - 1) offsets[H] = base + incl;
        if (lane == 0) s_flags = f;
    }
    __syncthreads();
    sx_retire(st, epoch, s_flags, result);
}

// One warp per row; a lane writes the run starts and ends of its word.
__global__ void __launch_bounds__(256) mask_runs_kernel(const unsigned* __restrict__ mask, int W, int H,
                                                        int words_per_row, const int* __restrict__ offsets,
                                                        int* __restrict__ ob, int* __restrict__ oe)
{
    const unsigned y = blockIdx.x * 8u + (threadIdx.x >> 5);  // not from the thread number: 2^27 rows take 2^32 threads
    const int lane = threadIdx.x & 31;
    if (y >= (unsigned)H) return;
    const int first = offsets[y], count = offsets[y + 1] - first;
    if (count == 0) return;
    const unsigned* row = mask + (long long)y * words_per_row;
    unsigned carry = 0u;
    int done = 0;  // starts in the words before this round
    for (int w0 = 0; w0 < words_per_row; w0 += 32) {
        const unsigned m = w0 + lane < words_per_row ? row[w0 + lane] : 0u;
        unsigned prev = __shfl_up_sync(0xFFFFFFFFu, m, 1) >> 31;
        if (lane == 0) prev = carry;
        carry = __shfl_sync(0xFFFFFFFFu, m, 31) >> 31;
        const unsigned shifted = (m << 1) | prev;
        unsigned starts = m & ~shifted, stops = shifted & ~m;
        const int n = __popc(starts);
        int incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += v;
        }
        const int x = 32 * (w0 + lane);
        int s = first + done + incl - n, t = s - (int)prev;  // a run open at the word's start ends at t
        for (; starts; starts &= starts - 1u) ob[s++] = x + __ffs(starts) - 1;
        for (; stops; stops &= stops - 1u, ++t)
            if (x + __ffs(stops) - 1 < W) oe[t] = x + __ffs(stops) - 1;
        done += __shfl_sync(0xFFFFFFFFu, incl, 31);
    }
    // a run that reaches the last column ends with the row
    const bool open = (row[words_per_row - 1] >> ((W - 1) & 31)) & 1u;
    if (lane == 0 && open) oe[first + count - 1] = W;
}

template <bool GRAD, bool VEC>
void mask_go(const float* d, int W, int H, float thr, unsigned* mask, cudaStream_t stream)
{
    const int strips = (W + 127) / 128;
    const long long tasks = (long long)strips * (((long long)H + RLE_ROWS - 1) / RLE_ROWS);
    mask_kernel<GRAD, VEC><<<(int)((tasks + RLE_THREADS / 32 - 1) / (RLE_THREADS / 32)), RLE_THREADS, 0, stream>>>(
        d, W, H, thr, mask, (W + 31) / 32, strips, tasks);
}

}  // namespace

// Smallest non-negative float whose correctly rounded square root is >= thr
// (NaN for a NaN threshold: no cell passes, as in the comparison itself).
float sx_least_radicand(float thr)
{
    if (!(thr > 0.0f)) return thr != thr ? thr : 0.0f;
    unsigned lo = 0u, hi = 0x7F800000u;  // sqrt(+inf) passes for every threshold
    while (lo < hi) {
        const unsigned mid = lo + (hi - lo) / 2;
        float s;
        memcpy(&s, &mid, 4);
        if (sqrtf(s) >= thr) hi = mid; else lo = mid + 1;
    }
    float s;
    memcpy(&s, &lo, 4);
    return s;
}

int sx_mask_tiles(int H) { return (int)(((long long)H + 7) / 8); }

cudaError_t sx_mask_launch(const float* d, int W, int H, float thr, int grad, unsigned* mask, int* offsets, int* result,
                           const SxScanState& st, cudaStream_t stream)
{
    const int tiles = sx_mask_tiles(H);
    cudaError_t err = cudaMemsetAsync(st.counters, 0, 16 + (size_t)tiles * 8, stream);
    if (err != cudaSuccess) return err;
    const bool vec = (W & 3) == 0 && ((uintptr_t)d & 15u) == 0;
    if (grad) {
        thr = sx_least_radicand(thr);
        if (vec) mask_go<true, true>(d, W, H, thr, mask, stream);
        else mask_go<true, false>(d, W, H, thr, mask, stream);
    } else {
        if (vec) mask_go<false, true>(d, W, H, thr, mask, stream);
        else mask_go<false, false>(d, W, H, thr, mask, stream);
    }
    mask_count_kernel<<<tiles, RLE_THREADS, 0, stream>>>(mask, H, (W + 31) / 32, offsets, result, st);
    return cudaGetLastError();
}

cudaError_t sx_gradient_launch(const float* d, int W, int H, float* out, cudaStream_t stream)
{
    if (W <= 0 || H <= 0) return cudaSuccess;
    if (W < NARROW) {
        const long long need = ((long long)W * H + RLE_THREADS - 1) / RLE_THREADS;
        narrow_gradient_kernel<<<(int)(need < 148 * 32 ? need : 148 * 32), RLE_THREADS, 0, stream>>>(d, W, H, out);
        return cudaGetLastError();
    }
    const int strips = (W + 127) / 128;
    const long long tasks = (long long)strips * (((long long)H + RLE_ROWS - 1) / RLE_ROWS);
    const int blocks = (int)((tasks + RLE_THREADS / 32 - 1) / (RLE_THREADS / 32));
    if ((W & 3) == 0 && ((uintptr_t)d & 15u) == 0 && ((uintptr_t)out & 15u) == 0)
        gradient_kernel<true><<<blocks, RLE_THREADS, 0, stream>>>(d, W, H, out, strips, tasks);
    else
        gradient_kernel<false><<<blocks, RLE_THREADS, 0, stream>>>(d, W, H, out, strips, tasks);
    return cudaGetLastError();
}

cudaError_t sx_mask_runs_launch(const unsigned* mask, int W, int H, const int* offsets, int* ob, int* oe,
                                cudaStream_t stream)
{
    mask_runs_kernel<<<sx_mask_tiles(H), 256, 0, stream>>>(mask, W, H, (W + 31) / 32, offsets, ob, oe);
    return cudaGetLastError();
}
