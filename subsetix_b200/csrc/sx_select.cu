// The value that a fraction of a field's larger values reaches: the selection behind
// gradient_tag_set (subsetix_amr2/regrid.py:353-380), which sorts the values above
// epsilon and takes the one that ceil(fraction * their number) of them reach.
//
// Three passes over the values, each a histogram of the next 11 (11, 10) bits of their
// order keys among the values that agree with the bits chosen so far; the last block of
// a pass finds the bin that holds the wanted rank.  Bound by reading the values three
// times, from the second time on from L2 where they fit.  Neighbouring values of a
// smooth field share their leading bits, which would put a warp's shared-memory atomics
// on one address: a thread takes 16 consecutive values and adds a run of equal bins at
// once.  Measured (B200, gradients of a 4096^2 grid, 67 MB): 68 us for the three passes;
// compacting the values and torch.kthvalue took 33 ms (700^2:
// 22 us against 1.0 ms).

#include "sx_internal.cuh"

namespace {

constexpr int SEL_THREADS = 256;
constexpr int SEL_BINS = 2048;
constexpr int SEL_RUN = 16;

struct SelState {
    unsigned hist[SEL_BINS];
    unsigned prefix;  // key bits chosen so far
    unsigned want;    // rank from above among the values that have them
    unsigned total;   // values above epsilon
    unsigned done;    // blocks of the pass that have finished
};

// Larger floats have larger keys.
__device__ __forceinline__ unsigned order_key(float v)
{
    const unsigned b = __float_as_uint(v);
    return b ^ ((b >> 31) ? 0xFFFFFFFFu : 0x80000000u);
}

template <bool VEC>
__global__ void __launch_bounds__(SEL_THREADS) select_kernel(const float* __restrict__ values, long long n, float eps,
                                                             double fraction, int pass, SelState* __restrict__ state,
                                                             int* __restrict__ result)
{
    __shared__ unsigned s_hist[SEL_BINS];
    __shared__ unsigned s_sum[SEL_THREADS / 32], s_pick[2];
    __shared__ bool s_last;
    const int shift = pass == 0 ? 21 : pass == 1 ? 10 : 0, bits = pass == 2 ? 10 : 11;
    const unsigned bins = 1u << bits, prefix = pass == 0 ? 0u : state->prefix;
    for (int i = threadIdx.x; i < SEL_BINS; i += SEL_THREADS) s_hist[i] = 0u;
    __syncthreads();
    const long long runs = (n + SEL_RUN - 1) / SEL_RUN;
    for (long long r = (long long)blockIdx.x * SEL_THREADS + threadIdx.x; r < runs; r += (long long)gridDim.x * SEL_THREADS) {
        float v[SEL_RUN];
        const long long at = r * SEL_RUN;
        if (VEC && at + SEL_RUN <= n) {
#pragma unroll
            for (int q = 0; q < SEL_RUN / 4; ++q) {
                const float4 f = __ldg((const float4*)(values + at) + q);
                v[4 * q] = f.x; v[4 * q + 1] = f.y; v[4 * q + 2] = f.z; v[4 * q + 3] = f.w;
            }
        } else {
#pragma unroll
            for (int q = 0; q < SEL_RUN; ++q) v[q] = at + q < n ? __ldg(values + at + q) : eps;
        }
        unsigned bin = 0u, count = 0u;
#pragma unroll
        for (int q = 0; q < SEL_RUN; ++q) {
            const unsigned key = order_key(v[q]);
            const bool in = v[q] > eps && (pass == 0 || (key >> (shift + bits)) == prefix);
            const unsigned b = (key >> shift) & (bins - 1u);
            if (in && b != bin) {
                if (count) atomicAdd(&s_hist[bin], count);
                bin = b;
                count = 0u;
            }
            count += in ? 1u : 0u;
        }
        if (count) atomicAdd(&s_hist[bin], count);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < (int)bins; i += SEL_THREADS)
        if (s_hist[i]) atomicAdd(&state->hist[i], s_hist[i]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&state->done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // the last block: thread t has the bins from bins - 1 - t per downwards
    const int per = (int)bins / SEL_THREADS, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned mine = 0u;
    for (int i = 0; i < per; ++i) mine += __ldcg(&state->hist[bins - 1 - (threadIdx.x * per + i)]);
    unsigned incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_sum[wid] = incl;
    __syncthreads();
    unsigned before = incl - mine, total = 0u;
    for (int w = 0; w < SEL_THREADS / 32; ++w) {
        if (w < wid) before += s_sum[w];
        total += s_sum[w];
    }
    unsigned want = state->want;
    if (pass == 0) {
        const double share = ceil((double)total * fraction);
        want = share < 1.0 ? 1u : share > (double)total ? total : (unsigned)share;
    }
    if (threadIdx.x == 0) s_pick[0] = s_pick[1] = 0u;
    __syncthreads();
    if (before < want && before + mine >= want) {
        unsigned seen = before;
        for (int i = 0; i < per; ++i) {
            const unsigned b = bins - 1 - (threadIdx.x * per + i), c = __ldcg(&state->hist[b]);
            if (seen + c >= want) {
                s_pick[0] = b;
                s_pick[1] = want - seen;
                break;
            }
            seen += c;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < (int)bins; i += SEL_THREADS) state->hist[i] = 0u;
    if (threadIdx.x == 0) {
        const unsigned chosen = (prefix << bits) | s_pick[0];
        state->prefix = chosen;
        state->want = s_pick[1];
        state->done = 0u;
        if (pass == 0) state->total = total;
        if (pass == 2) {
            result[0] = __float_as_int(__uint_as_float(chosen ^ ((chosen >> 31) ? 0x80000000u : 0xFFFFFFFFu)));
            result[1] = (int)state->total;
        }
    }
}

}  // namespace

size_t sx_select_bytes() { return sizeof(SelState); }

cudaError_t sx_select_launch(const float* values, long long n, float eps, double fraction, void* workspace, int* result,
                             cudaStream_t stream)
{
    cudaError_t err = cudaMemsetAsync(workspace, 0, sizeof(SelState), stream);
    if (err != cudaSuccess) return err;
    long long blocks = (n + SEL_THREADS * SEL_RUN - 1) / (SEL_THREADS * SEL_RUN);
    if (blocks > 148 * 4) blocks = 148 * 4;
    if (blocks < 1) blocks = 1;
    const bool vec = ((uintptr_t)values & 15u) == 0;
    for (int pass = 0; pass < 3; ++pass) {
        if (vec)
            select_kernel<true><<<(int)blocks, SEL_THREADS, 0, stream>>>(values, n, eps, fraction, pass,
                                                                         (SelState*)workspace, result);
        else
            select_kernel<false><<<(int)blocks, SEL_THREADS, 0, stream>>>(values, n, eps, fraction, pass,
                                                                          (SelState*)workspace, result);
    }
    return cudaGetLastError();
}
