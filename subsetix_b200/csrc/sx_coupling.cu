// Level coupling of a nested multi-level field by index tables: ghost
// filling from the coarser level, restriction onto it, and the transposes of
// both.  The tables are built once per fixed geometry on the host side
// (subsetix_b200/adjoint.py), so every kernel here is a gather or a
// scatter over precomputed indices, bound by HBM bandwidth:
//
//   sx_index_copy            dst[dst_idx[i]] = src[src_idx[i]]
//                            (ghost fill: a fine ghost cell takes its coarse
//                            parent's value, as injection does in
//                            subsetix_cupy/multilevel.py:365-407);
//   sx_index_block_mean      out[out_idx[j]] = (sum_m in[in_idx[j*g+m]]) * norm
//                            summed in table order (sub-row outer, column
//                            inner), then scaled: the order of
//                            restrict_field's mean (multilevel.py:410-479);
//   sx_index_block_mean_adj  its transpose: in_bar[in_idx[j*g+m]] +=
//                            out_bar[out_idx[j]] * norm, out_bar[out_idx[j]] = 0
//                            (the in_idx entries are distinct, so no two
//                            threads write one cell);
//   sx_run_block_mean{,_adj} the same two on runs: consecutive coarse cells have
//                            consecutive children in each sub-row, so a run of
//                            up to 64 coarse cells needs only where its cells
//                            and its sub-rows' children start;
//   sx_index_segment_add     transpose of a gather with repeats: dst[dst_idx[s]]
//                            += sum of src[src_idx[t]] over segment s, in
//                            segment order, then src[src_idx[t]] = 0 when asked
//                            (deterministic: one thread per segment).
//
// Float arithmetic uses explicit round-to-nearest operations, so float32
// and float64 results do not depend on the compiler's contraction choices.

#include "sx_internal.cuh"

namespace {

__device__ __forceinline__ float cp_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double cp_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float cp_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double cp_mul(double a, double b) { return __dmul_rn(a, b); }

template <typename T>
__global__ void index_copy_kernel(long long n, const int* dst_idx, const int* src_idx,
                                  const T* src, T* __restrict__ dst)
{
    sx_after_previous();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const long long s = src_idx ? src_idx[i] : i;
        const long long d = dst_idx ? dst_idx[i] : i;
        dst[d] = src[s];
    }
}

template <typename T>
__global__ void block_mean_kernel(long long n, int group, T norm, const int* __restrict__ out_idx,
                                  const int* __restrict__ in_idx, const T* __restrict__ in, T* __restrict__ out)
{
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (long long)gridDim.x * blockDim.x) {
        const int* idx = in_idx + j * group;
        T acc = T(0);
        for (int m = 0; m < group; ++m) acc = cp_add(acc, in[idx[m]]);
        out[out_idx[j]] = cp_mul(acc, norm);
    }
}

template <typename T>
__global__ void block_mean_adj_kernel(long long n, int group, T norm, const int* __restrict__ out_idx,
                                      const int* __restrict__ in_idx, T* __restrict__ out_bar, T* __restrict__ in_bar)
{
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (long long)gridDim.x * blockDim.x) {
        const int* idx = in_idx + j * group;
        const T w = cp_mul(out_bar[out_idx[j]], norm);
        for (int m = 0; m < group; ++m) in_bar[idx[m]] = cp_add(in_bar[idx[m]], w);
        out_bar[out_idx[j]] = T(0);
    }
}

// A segment holds a few sources (the ghost children of one parent).  Their
// indices are loaded together, then their values, so a thread waits for three
// memory round trips instead of two per source (ghost rings of about 10,000
// cells: 11.6 -> 5.4 us per launch); the sum keeps the segment order.
template <typename T>
__global__ void segment_add_kernel(long long nseg, const int* seg_off, const int* src_idx,
                                   const int* dst_idx, T* __restrict__ src, T* __restrict__ dst,
                                   int zero_src)
{
    sx_after_previous();
    constexpr int BATCH = 4;
    for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < nseg;
         s += (long long)gridDim.x * blockDim.x) {
        const int d = dst_idx[s], t0 = seg_off[s], t1 = seg_off[s + 1];
        T acc = dst[d];
        for (int t = t0; t < t1; t += BATCH) {
            int idx[BATCH];
            T val[BATCH];
#pragma unroll
            for (int k = 0; k < BATCH; ++k) idx[k] = t + k < t1 ? src_idx[t + k] : -1;
#pragma unroll
            for (int k = 0; k < BATCH; ++k) val[k] = idx[k] >= 0 ? src[idx[k]] : T(0);
#pragma unroll
            for (int k = 1; k < BATCH; ++k)
#pragma unroll
                for (int j = 0; j < k; ++j)
                    if (zero_src && idx[k] == idx[j]) val[k] = T(0);  // a source listed twice is cleared by then
#pragma unroll
            for (int k = 0; k < BATCH; ++k) {
                if (idx[k] >= 0) acc = cp_add(acc, val[k]);
                if (zero_src && idx[k] >= 0) src[idx[k]] = T(0);
            }
        }
        dst[d] = acc;
    }
}

// Runs of coarse cells, two per warp, two cells of each per lane.  Plan entry of a run:
// first coarse value, cells (at most 64), then the first child of each of
// the r sub-rows; `stride` ints per entry (a multiple of 4).  Bound by the fine
// values' bytes.  Per coarse cell the index tables took 4 (1 + r^2) bytes and a
// dependent gather per child, here 16 bytes per run and loads of consecutive
// values, in pairs where a sub-row of a run starts at an even value (PAIR: r = 2
// and arrays aligned to a pair).  Measured (B200, 1.18 M coarse cells, float32):
// mean 11.4 -> 7.0 us, transpose 30.8 -> 11.9 us (27.6 us while its stores stood
// between its loads).  With every load of a run, then of two, before the first use, and
// plan entries as one load each, a pass of the composite (190 means, 100 transposes)
// went from 9.45 to 9.11 and 8.79 ms; four runs per warp 8.85.
template <typename T>
struct Pair;
template <>
struct Pair<float> {
    typedef float2 type;
};
template <>
struct Pair<double> {
    typedef double2 type;
};

constexpr int RUNS_PER_WARP = 2;

template <typename T, bool PAIR>
__global__ void __launch_bounds__(256) run_block_mean_kernel(int runs, int rr, int stride, T norm,
                                                             const int* plan, const T* in,
                                                             T* __restrict__ out)
{
    sx_after_previous();
    typedef typename Pair<T>::type P2;
    const int first = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * RUNS_PER_WARP, lane = threadIdx.x & 31;
    if constexpr (PAIR) {
        int count[RUNS_PER_WARP];
        long long c0[RUNS_PER_WARP], f[RUNS_PER_WARP][2];
#pragma unroll
        for (int q = 0; q < RUNS_PER_WARP; ++q) {
            const int4 p = first + q < runs ? *(const int4*)(plan + (long long)(first + q) * stride) : make_int4(0, 0, 0, 0);
            c0[q] = p.x;
            count[q] = p.y;
            f[q][0] = p.z;
            f[q][1] = p.w;
        }
        P2 v[RUNS_PER_WARP][2][2];
#pragma unroll
        for (int q = 0; q < RUNS_PER_WARP; ++q)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int dy = 0; dy < 2; ++dy) {
                    const int k = lane + 32 * h;
                    if (k >= count[q]) continue;
                    const T* src = in + f[q][dy] + 2ll * k;
                    if ((f[q][dy] & 1) == 0) {
                        v[q][h][dy] = *(const P2*)src;
                    } else {
                        v[q][h][dy].x = src[0];
                        v[q][h][dy].y = src[1];
                    }
                }
#pragma unroll
        for (int q = 0; q < RUNS_PER_WARP; ++q)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int k = lane + 32 * h;
                if (k >= count[q]) continue;
                const T a = cp_add(cp_add(T(0), v[q][h][0].x), v[q][h][0].y);
                out[c0[q] + k] = cp_mul(cp_add(cp_add(a, v[q][h][1].x), v[q][h][1].y), norm);
            }
    } else {
        for (int run = first; run < min(runs, first + RUNS_PER_WARP); ++run) {
            const int* p = plan + (long long)run * stride;
            const int count = p[1];
            const long long c0 = p[0];
            T acc[2] = {T(0), T(0)};
            for (int dy = 0; dy < rr; ++dy) {
                const long long f0 = p[2 + dy];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int k = lane + 32 * h;
                    if (k >= count) continue;
                    const T* src = in + f0 + (long long)k * rr;
                    for (int dx = 0; dx < rr; ++dx) acc[h] = cp_add(acc[h], src[dx]);
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (lane + 32 * h < count) out[c0 + lane + 32 * h] = cp_mul(acc[h], norm);
        }
    }
}

template <typename T, bool PAIR>
__global__ void __launch_bounds__(256) run_block_mean_adj_kernel(int runs, int rr, int stride, T norm,
                                                                 const int* plan, T* __restrict__ out_bar,
                                                                 T* __restrict__ in_bar)
{
    sx_after_previous();
    typedef typename Pair<T>::type P2;
    const int first = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * RUNS_PER_WARP, lane = threadIdx.x & 31;
    if constexpr (PAIR) {
        // every load before the first store, so a warp waits for one round trip
        int count[RUNS_PER_WARP];
        long long c0[RUNS_PER_WARP], f[RUNS_PER_WARP][2];
#pragma unroll
        for (int q = 0; q < RUNS_PER_WARP; ++q) {
            const int4 p = first + q < runs ? *(const int4*)(plan + (long long)(first + q) * stride) : make_int4(0, 0, 0, 0);
            c0[q] = p.x;
            count[q] = p.y;
            f[q][0] = p.z;
            f[q][1] = p.w;
        }
        T w[RUNS_PER_WARP][2];
        P2 v[RUNS_PER_WARP][2][2];
#pragma unroll
        for (int q = 0; q < RUNS_PER_WARP; ++q)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int k = lane + 32 * h;
                if (k >= count[q]) continue;
                w[q][h] = out_bar[c0[q] + k];
#pragma unroll
                for (int dy = 0; dy < 2; ++dy) {
                    const T* src = in_bar + f[q][dy] + 2ll * k;
                    if ((f[q][dy] & 1) == 0) {
                        v[q][h][dy] = *(const P2*)src;
                    } else {
                        v[q][h][dy].x = src[0];
                        v[q][h][dy].y = src[1];
                    }
                }
            }
#pragma unroll
        for (int q = 0; q < RUNS_PER_WARP; ++q)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int k = lane + 32 * h;
                if (k >= count[q]) continue;
                const T a = cp_mul(w[q][h], norm);
                out_bar[c0[q] + k] = T(0);
#pragma unroll
                for (int dy = 0; dy < 2; ++dy) {
                    T* dst = in_bar + f[q][dy] + 2ll * k;
                    v[q][h][dy].x = cp_add(v[q][h][dy].x, a);
                    v[q][h][dy].y = cp_add(v[q][h][dy].y, a);
                    if ((f[q][dy] & 1) == 0) {
                        *(P2*)dst = v[q][h][dy];
                    } else {
                        dst[0] = v[q][h][dy].x;
                        dst[1] = v[q][h][dy].y;
                    }
                }
            }
    } else {
        for (int run = first; run < min(runs, first + RUNS_PER_WARP); ++run) {
            const int* p = plan + (long long)run * stride;
            const int count = p[1];
            const long long c0 = p[0];
            T w[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int k = lane + 32 * h;
                w[h] = k < count ? cp_mul(out_bar[c0 + k], norm) : T(0);
                if (k < count) out_bar[c0 + k] = T(0);
            }
            for (int dy = 0; dy < rr; ++dy) {
                const long long f0 = p[2 + dy];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int k = lane + 32 * h;
                    if (k >= count) continue;
                    T* dst = in_bar + f0 + (long long)k * rr;
                    for (int dx = 0; dx < rr; ++dx) dst[dx] = cp_add(dst[dx], w[h]);
                }
            }
        }
    }
}

int grid_for(long long n)
{
    long long g = (n + 255) / 256;
    if (g > 148 * 32) g = 148 * 32;
    return (int)(g < 1 ? 1 : g);
}

}  // namespace

cudaError_t sx_index_copy_launch(int dtype, long long n, const int* dst_idx, const int* src_idx, const void* src,
                                 void* dst, cudaStream_t stream)
{
    if (n <= 0) return cudaSuccess;
    if (dtype == 1)
        sx_launch_early(index_copy_kernel<double>, dim3(grid_for(n)), dim3(256), 0, stream, n, dst_idx, src_idx, (const double*)src,
                                                                    (double*)dst);
    else
        sx_launch_early(index_copy_kernel<float>, dim3(grid_for(n)), dim3(256), 0, stream, n, dst_idx, src_idx, (const float*)src, (float*)dst);
    return cudaGetLastError();
}

cudaError_t sx_index_block_mean_launch(int dtype, long long n, int group, double norm, const int* out_idx,
                                       const int* in_idx, const void* in, void* out, cudaStream_t stream)
{
    if (n <= 0) return cudaSuccess;
    if (dtype == 1)
        block_mean_kernel<double><<<grid_for(n), 256, 0, stream>>>(n, group, norm, out_idx, in_idx, (const double*)in,
                                                                    (double*)out);
    else
        block_mean_kernel<float><<<grid_for(n), 256, 0, stream>>>(n, group, (float)norm, out_idx, in_idx,
                                                                   (const float*)in, (float*)out);
    return cudaGetLastError();
}

cudaError_t sx_index_block_mean_adj_launch(int dtype, long long n, int group, double norm, const int* out_idx,
                                           const int* in_idx, void* out_bar, void* in_bar, cudaStream_t stream)
{
    if (n <= 0) return cudaSuccess;
    if (dtype == 1)
        block_mean_adj_kernel<double><<<grid_for(n), 256, 0, stream>>>(n, group, norm, out_idx, in_idx,
                                                                        (double*)out_bar, (double*)in_bar);
    else
        block_mean_adj_kernel<float><<<grid_for(n), 256, 0, stream>>>(n, group, (float)norm, out_idx, in_idx,
                                                                       (float*)out_bar, (float*)in_bar);
    return cudaGetLastError();
}

cudaError_t sx_index_segment_add_launch(int dtype, long long nseg, const int* seg_off, const int* src_idx,
                                        const int* dst_idx, void* src, void* dst, int zero_src, cudaStream_t stream)
{
    if (nseg <= 0) return cudaSuccess;
    if (dtype == 1)
        sx_launch_early(segment_add_kernel<double>, dim3(grid_for(nseg)), dim3(256), 0, stream, nseg, seg_off, src_idx, dst_idx, (double*)src,
                                                                        (double*)dst, zero_src);
    else
        sx_launch_early(segment_add_kernel<float>, dim3(grid_for(nseg)), dim3(256), 0, stream, nseg, seg_off, src_idx, dst_idx, (float*)src,
                                                                       (float*)dst, zero_src);
    return cudaGetLastError();
}

namespace {

template <typename T, bool ADJ>
void run_go(long long runs, int ratio, int stride, double norm, const int* plan, T* coarse, T* fine,
            cudaStream_t stream)
{
    const int blocks = (int)((runs + 8 * RUNS_PER_WARP - 1) / (8 * RUNS_PER_WARP));
    const bool pair = ratio == 2 && stride % 4 == 0 && ((uintptr_t)plan & 15u) == 0 &&
                      ((uintptr_t)fine & (2 * sizeof(T) - 1)) == 0;
    if (ADJ) {
        if (pair)
            sx_launch_early(run_block_mean_adj_kernel<T, true>, dim3(blocks), dim3(256), 0, stream, (int)runs, ratio, stride, (T)norm, plan,
                                                                           coarse, fine);
        else
            sx_launch_early(run_block_mean_adj_kernel<T, false>, dim3(blocks), dim3(256), 0, stream, (int)runs, ratio, stride, (T)norm, plan,
                                                                            coarse, fine);
    } else {
        if (pair)
            sx_launch_early(run_block_mean_kernel<T, true>, dim3(blocks), dim3(256), 0, stream, (int)runs, ratio, stride, (T)norm, plan, fine,
                                                                       coarse);
        else
            sx_launch_early(run_block_mean_kernel<T, false>, dim3(blocks), dim3(256), 0, stream, (int)runs, ratio, stride, (T)norm, plan, fine,
                                                                        coarse);
    }
}

}  // namespace

cudaError_t sx_run_block_mean_launch(int dtype, int adjoint, long long runs, int ratio, int stride, double norm,
                                     const int* plan, void* coarse, void* fine, cudaStream_t stream)
{
    if (runs <= 0) return cudaSuccess;
    if (dtype == 1) {
        if (adjoint) run_go<double, true>(runs, ratio, stride, norm, plan, (double*)coarse, (double*)fine, stream);
        else run_go<double, false>(runs, ratio, stride, norm, plan, (double*)coarse, (double*)fine, stream);
    } else {
        if (adjoint) run_go<float, true>(runs, ratio, stride, norm, plan, (float*)coarse, (float*)fine, stream);
        else run_go<float, false>(runs, ratio, stride, norm, plan, (float*)coarse, (float*)fine, stream);
    }
    return cudaGetLastError();
}
