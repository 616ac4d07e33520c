// Staging and look-back helpers shared by the tile sweeps (sx_sweep.cu,
// sx_box.cu): bulk copies into shared memory counted on an mbarrier with a
// bounded wait, and the single-level decoupled look-back over tiles.
#pragma once

#include "sx_internal.cuh"

#define SX_GROUP 32
#define SXS_WAIT_LIMIT (1u << 16)
#define SXS_WAIT_HINT_NS 20000

// Look-back state in the workspace: counters[4] | tile status[tiles] |
// group status[groups] | group sum[groups] | group count[groups].
struct SxSweepState {
    unsigned* counters;
    unsigned long long* tile_status;
    unsigned long long* group_status;
    int* group_sum;
    unsigned* group_count;
};

__device__ __forceinline__ unsigned long long sx_ld_status(const unsigned long long* p)
{
    return *((volatile const unsigned long long*)p);
}

__device__ __forceinline__ unsigned sxs_saddr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void sxs_bar_init(unsigned long long* bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sxs_saddr(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// The single arrival of a phase of the barrier, announcing `bytes` of copies.
__device__ __forceinline__ void sxs_bar_expect(unsigned long long* bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sxs_saddr(bar)), "r"(bytes)
                 : "memory");
}

// Bulk copy of `bytes` (a multiple of 16) between 16-byte aligned addresses,
// global to this block's shared memory, counted on `bar`.
__device__ __forceinline__ void sxs_bulk_copy(void* dst, const void* src, unsigned bytes, unsigned long long* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     sxs_saddr(dst)),
                 "l"(src), "r"(bytes), "r"(sxs_saddr(bar))
                 : "memory");
}

// Bounded wait for the phase of `bar` with the given parity (0, then 1, ...);
// false if it did not complete.  Each
// try_wait may suspend the thread for up to SXS_WAIT_HINT_NS (it resumes as
// soon as the phase completes), so waiting warps take no issue slots; the
// whole wait is bounded by SXS_WAIT_LIMIT tries.
__device__ __forceinline__ bool sxs_bar_wait(unsigned long long* bar, unsigned parity = 0u)
{
    const unsigned a = sxs_saddr(bar);
    for (unsigned i = 0; i < SXS_WAIT_LIMIT; ++i) {
        unsigned done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %3, %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(a), "n"(SXS_WAIT_HINT_NS), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// Wait until a tile status word is published, backing off from 32 ns to
// 512 ns between polls so that waiting warps leave the issue slots to the
// warps that sweep; bounded by SX_LOOKBACK_SPIN_LIMIT polls.
__device__ __forceinline__ unsigned long long sxs_wait_status(const unsigned long long* p, bool& timed_out,
                                                             unsigned limit)
{
    unsigned sleep = 32;
    for (unsigned spins = 0;; ++spins) {
        const unsigned long long w = sx_ld_status(p);
        if ((w >> 32) & 3ull) return w;
        if (spins > limit) {
            timed_out = true;
            return (SX_KIND_PREFIX << 32);  // treat as a zero prefix so the kernel finishes
        }
        __nanosleep(sleep);
        if (sleep < 512) sleep <<= 1;
    }
}

// Single-level decoupled look-back for the segmented sweeps (whole warp).
// Status word of a tile: bits 0-31 the value, bits 32-33 the kind (1 tile
// aggregate, 2 inclusive prefix), bits 34-37 the OR of the SXF_* flags of
// the tiles the value covers.  The tile publishes its aggregate, then reads
// its 32 nearest predecessors at once (each wait bounded) and adds values up
// to the nearest inclusive prefix, 32 tiles per step.  Returns the exclusive
// prefix; `flags` comes back as the OR over this tile and all before it.
// A.wait_limit (when set) bounds every wait instead of SX_LOOKBACK_SPIN_LIMIT,
// and the tile A.withhold_tile - 1 publishes nothing: both exist only so that
// tests can make the waits give up.
__device__ __forceinline__ int sxs_lookback(const SxBoolArgs& A, const SxSweepState& st, int tile, int aggregate,
                                            unsigned& flags)
{
    const int lane = threadIdx.x & 31;
    const unsigned limit = A.wait_limit ? A.wait_limit : SX_LOOKBACK_SPIN_LIMIT;
    const bool publish = A.withhold_tile != tile + 1;
    const unsigned long long own = ((unsigned long long)(flags & 15u) << 34) | (unsigned long long)(unsigned)aggregate;
    if (tile == 0) {
        if (lane == 0 && publish) atomicExch(&st.tile_status[0], own | (SX_KIND_PREFIX << 32));
        return 0;
    }
    if (lane == 0 && publish) atomicExch(&st.tile_status[tile], own | (SX_KIND_AGG << 32));
    int exclusive = 0;
    unsigned fl = flags;
    bool timed_out = false;
    for (int pos = tile - 1;; pos -= 32) {
        const int t = pos - lane;
        unsigned long long w = SX_KIND_PREFIX << 32;  // before tile 0: an empty prefix
        if (t >= 0) w = sxs_wait_status(&st.tile_status[t], timed_out, limit);
        const unsigned pm = __ballot_sync(0xFFFFFFFFu, ((w >> 32) & 3ull) == SX_KIND_PREFIX);
        const int stop = pm ? __ffs(pm) - 1 : 32;
        int v = lane <= stop ? (int)(unsigned)(w & 0xFFFFFFFFull) : 0;
        unsigned f = lane <= stop ? (unsigned)(w >> 34) & 15u : 0u;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
            f |= __shfl_xor_sync(0xFFFFFFFFu, f, o);
        }
        exclusive += v;
        fl |= f;
        if (pm) break;
    }
    if (__any_sync(0xFFFFFFFFu, timed_out)) fl |= SXF_TIMEOUT;
    if (lane == 0 && publish)
        atomicExch(&st.tile_status[tile], ((unsigned long long)(fl & 15u) << 34) | (SX_KIND_PREFIX << 32) |
                                              (unsigned long long)(unsigned)(exclusive + aggregate));
    flags = fl;
    return exclusive;
}

// The last tile in ticket order reports the grand total and the flags of
// every tile; an output beyond the capacity shows as a total above it.
__device__ __forceinline__ void sxs_report(const SxBoolArgs& A, int tile, int tiles, int base, int aggregate,
                                           unsigned flags)
{
    if (tile == tiles - 1 && (threadIdx.x & 31) == 0) {
        const long long total = (long long)base + aggregate;
        A.result[0] = (int)total;
        A.result[1] = (int)(flags | (total > A.capacity ? SXF_CAPACITY : 0u));
    }
}

static inline size_t a256(size_t x) { return (x + 255) & ~(size_t)255; }

static inline SxSweepState sx_sweep_state(void* ws, long long tiles)
{
    const long long groups = (tiles + SX_GROUP - 1) / SX_GROUP;
    char* p = (char*)ws;
    SxSweepState st;
    st.counters = (unsigned*)p;
    p += a256(16);
    st.tile_status = (unsigned long long*)p;
    p += a256((size_t)tiles * 8);
    st.group_status = (unsigned long long*)p;
    p += a256((size_t)groups * 8);
    st.group_sum = (int*)p;
    p += a256((size_t)groups * 4);
    st.group_count = (unsigned*)p;
    return st;
}
