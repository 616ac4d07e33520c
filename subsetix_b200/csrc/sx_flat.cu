// First-order upwind and its adjoint on a flat plan: fixed geometry whose rows
// are sorted and disjoint and whose cells all lie in the domain.
//
// Values are packed in interval order, so the cell to the left of cell c is
// cell c - 1 whenever it is in the set, and the cells under a stretch of
// consecutive cells are consecutive too.  The plan splits the value array into
// groups of four consecutive cells, whatever intervals they belong to, and
// holds per group
//   bits     16 flags: 0-3 which cells have a neighbour below, 4-7 above,
//            8-11 on the left, 14 whether the last cell has one on the right
//            (the right neighbour of the others is the left flag of the next
//            cell), 12 and 13 that the group is irregular below and above;
//   dn, up   value index of the group's first neighbour in that row.  The
//            others follow it one by one unless the group is irregular (an
//            interval starts inside it, so the neighbours may jump): then the
//            entry is a slot of side_dn / side_up, which holds all four
//            indices.  The slot is the interval of the group's last cell,
//            which is unique, because that interval starts inside the group.
// A thread updates one group: one 16-byte load of its values (two in float64),
// 6 bytes of plan, four neighbour values (consecutive lanes read consecutive
// addresses), one 16-byte store; the horizontal neighbour comes from a shuffle.
//
// Bound and why this form: the kernel on 128-cell chunks of single intervals
// (sx_upwind_chunk_kernel) was limited by instructions: a chunk's plan entry
// is 64 bytes, intervals end inside chunks (110 cells on average in the uneven
// batch), and every cell carries its own index arithmetic and domain tests.
// Groups are always full, so nothing is done for padding, and with all cells in
// the domain (span_kernel checks it when the plan is built) no test is left:
// a neighbour in the set is a neighbour in the domain.  Geometry with cells
// outside the domain keeps the chunk kernel.  Measured (B200): one float64 step
// on 2500^2 26.1 -> 15.1 us (12.3 with over_group), the uneven batch 1337 -> 644 us (327 M cells; its
// 9.5 bytes a cell take 475 us at the copy rate), the three-level composite's
// 300 level steps 5.1 -> 2.8 ms and its 150 transposed ones, sums over blocks
// included, 5.2 -> 3.2 ms.  Same values as sx_upwind, bit for bit; the adjoint's
// velocity gradient adds the same products in another fixed order.

#include <climits>

#include "sx_internal.cuh"

namespace {

constexpr int FLAT_THREADS = 256;
// Runs of groups per block of the banded step: a block pays one search for its
// band, so a large batch takes 16 runs (256 uneven sets, 327 M cells, float32:
// 1106 us with 1, 651 with 8, 626 with 16, 630 with 32, 659 with 64; the chunk
// kernel 1337 us).  Below BAND_BLOCKS such blocks per SM one run per block keeps
// the chip busy: at 4, 30 sets take 76 us against 91, 8 sets 13.5 against 18.4.
constexpr int BAND_ROUNDS = 16;
constexpr int BAND_BLOCKS = 4;
// Resident blocks per SM asked of the compiler.  One run: six (float64 on
// 2500^2 15.1 against 17.0 us without, 8192^2 120 against 138 us; float32 the
// same).  Several runs hold two runs' values: five in float32 (six 767 us, four
// 691 against 626 us), four in float64.
constexpr int STEP_BLOCKS = 6;
constexpr int BAND_STEP_BLOCKS_F32 = 5;
constexpr int BAND_STEP_BLOCKS_F64 = 4;
// Blocks per SM of the adjoint, all resident at once: every block ends with a reduction
// and its share of the last block's sum, so more blocks cost more than they hide (the
// three-level composite, 50 steps with gradients: 9.67 ms with 4 per SM, 9.94 with 8,
// 10.5 with 16; 9.45 with the next group's plan loaded early).  Float64 takes 80
// registers, three blocks.
constexpr int ADJOINT_BLOCKS = 4;
constexpr int ADJOINT_BLOCKS_F64 = 3;

// Smallest begin and largest end over all intervals into span[0], span[1]
// (which start at INT_MAX, INT_MIN).
__global__ void __launch_bounds__(256) span_kernel(const int* __restrict__ b, const int* __restrict__ e, int n,
                                                   int* __restrict__ span)
{
    int lo = INT_MAX, hi = INT_MIN;
    for (long long i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        lo = min(lo, b[i]);
        hi = max(hi, e[i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&span[0], lo);
        atomicMax(&span[1], hi);
    }
}

__global__ void span_init_kernel(int* span)
{
    span[0] = INT_MAX;
    span[1] = INT_MIN;
}

// Last index in [lo, hi] whose entry is not above v (a[lo] <= v holds).
__device__ __forceinline__ int last_not_above(const int* a, int lo, int hi, int v)
{
    while (lo < hi) {
        const int mid = lo + ((hi - lo + 1) >> 1);
        if (a[mid] <= v) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Value index of column x in the row of ordinal ord (-1: no such row), -1 when
// it is not in the set.  [j, je) is the part of the row not yet passed; x must
// not decrease between calls on one row.
__device__ __forceinline__ int neighbour(int& j, int je, int x, const int* __restrict__ b, const int* __restrict__ e,
                                         const int* __restrict__ coff)
{
    int lo = j, hi = je;  // first interval ending after x; usually the current one
    if (lo < hi && e[lo] <= x) {
        ++lo;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (e[mid] <= x) lo = mid + 1; else hi = mid;
        }
    }
    j = lo;
    return lo < je && b[lo] <= x ? coff[lo] + (x - b[lo]) : -1;
}

// One thread per group.  The block's first and last interval and row are found
// once, so a thread searches only among those.
__global__ void __launch_bounds__(FLAT_THREADS)
    flat_plan_kernel(const int* __restrict__ rows, const int* __restrict__ off, int row_count,
                     const int* __restrict__ b, const int* __restrict__ e, const int* __restrict__ coff, int n,
                     int cells, const int* __restrict__ lookup, int height, int* __restrict__ dn, int* __restrict__ up,
                     unsigned short* __restrict__ bits, int4* __restrict__ side_dn, int4* __restrict__ side_up)
{
    __shared__ int s_i[2], s_p[2];
    const int groups = (int)(((long long)cells + 3) >> 2);  // cells may be 2^31 - 1
    const int g0 = blockIdx.x * FLAT_THREADS;
    if (threadIdx.x == 0 || threadIdx.x == 32) {
        const int side = threadIdx.x >> 5;
        const long long c = side == 0 ? 4ll * g0 : 4ll * (g0 + FLAT_THREADS) - 1;
        const int i = last_not_above(coff, 0, n - 1, (int)min(c, (long long)cells - 1));
        s_i[side] = i;
        s_p[side] = last_not_above(off, 0, row_count - 1, i);
    }
    __syncthreads();
    const int g = g0 + threadIdx.x;
    if (g >= groups) return;
    const int c0 = 4 * g;
    int i = last_not_above(coff, s_i[0], s_i[1], c0);
    int p = last_not_above(off, s_p[0], s_p[1], i);
    int idn[4], iup[4];
    unsigned m = 0u;
    int jd = 0, jde = 0, ju = 0, jue = 0;
    bool fresh = true;  // the neighbour rows of p are still to be looked up
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        idn[k] = iup[k] = -1;
        const int c = c0 + k;
        if (c < cells) {
            while (i + 1 < n && coff[i + 1] <= c) ++i;
            while (off[p + 1] <= i) {
                ++p;
                fresh = true;
            }
            const int x = b[i] + (c - coff[i]);
            if (fresh) {
                const int row = rows[p];
                const int od = row >= 1 && row - 1 < height ? lookup[row - 1] : -1;
                const int ou = row < height - 1 && row >= -1 ? lookup[row + 1] : -1;
                jd = od >= 0 ? off[od] : 0;
                jde = od >= 0 ? off[od + 1] : 0;
                ju = ou >= 0 ? off[ou] : 0;
                jue = ou >= 0 ? off[ou + 1] : 0;
                fresh = false;
            }
            idn[k] = neighbour(jd, jde, x, b, e, coff);
            iup[k] = neighbour(ju, jue, x, b, e, coff);
            if (idn[k] >= 0) m |= 1u << k;
            if (iup[k] >= 0) m |= 16u << k;
            if (x > b[i] || (i > off[p] && e[i - 1] == b[i])) m |= 256u << k;
            if (k == 3 && (x + 1 < e[i] || (i + 1 < off[p + 1] && b[i + 1] == e[i]))) m |= 1u << 14;
        }
    }
    int fd = -1, fu = -1, nd = 0, nu = 0;
    bool rd = true, ru = true;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (idn[k] >= 0) {
            if (fd < 0) fd = idn[k];
            rd = rd && idn[k] == fd + nd;
            ++nd;
        }
        if (iup[k] >= 0) {
            if (fu < 0) fu = iup[k];
            ru = ru && iup[k] == fu + nu;
            ++nu;
        }
    }
    if (!rd) {
        m |= 1u << 12;
        side_dn[i] = make_int4(idn[0], idn[1], idn[2], idn[3]);
        fd = i;
    }
    if (!ru) {
        m |= 1u << 13;
        side_up[i] = make_int4(iup[0], iup[1], iup[2], iup[3]);
        fu = i;
    }
    dn[g] = max(fd, 0);
    up[g] = max(fu, 0);
    bits[g] = (unsigned short)m;
}

// Four consecutive values from c0: one vector load (two for float64) with VEC,
// which needs a 16-byte aligned array and a whole group.
template <typename T, bool VEC>
__device__ __forceinline__ void load_group(const T* v, long long c0, long long cells, T (&r)[4])
{
    if (VEC && c0 + 4 <= cells) {
        if (sizeof(T) == 4) {
            const float4 q = *(const float4*)(v + c0);
            r[0] = q.x; r[1] = q.y; r[2] = q.z; r[3] = q.w;
        } else {
            const double2 q = *(const double2*)(v + c0), w = *(const double2*)(v + c0 + 2);
            r[0] = (T)q.x; r[1] = (T)q.y; r[2] = (T)w.x; r[3] = (T)w.y;
        }
        return;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) r[k] = c0 + k < cells ? v[c0 + k] : (T)0;
}

template <typename T, bool VEC>
__device__ __forceinline__ void store_group(T* __restrict__ v, long long c0, long long cells, const T (&r)[4])
{
    if (VEC && c0 + 4 <= cells) {
        if (sizeof(T) == 4) {
            *(float4*)(v + c0) = make_float4((float)r[0], (float)r[1], (float)r[2], (float)r[3]);
        } else {
            *(double2*)(v + c0) = make_double2((double)r[0], (double)r[1]);
            *(double2*)(v + c0 + 2) = make_double2((double)r[2], (double)r[3]);
        }
        return;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (c0 + k < cells) v[c0 + k] = r[k];
}

// The neighbours of a group in one row: presence flags nm, the group's plan
// entry base, and the side array when the group is irregular.
template <typename T>
__device__ __forceinline__ void row_group(const T* v, int base, unsigned nm, bool irregular,
                                          const int4* side, T (&r)[4])
{
    int idx[4];
    idx[0] = base;
    idx[1] = base + (int)(nm & 1u);
    idx[2] = idx[1] + (int)((nm >> 1) & 1u);
    idx[3] = idx[2] + (int)((nm >> 2) & 1u);
    if (irregular) {
        const int4 s = side[base];
        idx[0] = s.x; idx[1] = s.y; idx[2] = s.z; idx[3] = s.w;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) r[k] = (nm >> k) & 1u ? v[idx[k]] : (T)0;
}

// The neighbours on one side within the value array: LEFT those at c - 1, else
// those at c + 1; 0 where the cell has none.  Lanes hold consecutive groups.
template <typename T, bool LEFT>
__device__ __forceinline__ void side_group(const T* v, const T (&cen)[4], unsigned m, long long c0,
                                           int lane, T (&r)[4])
{
    const unsigned hm = (m >> 8) & 15u;
    if (LEFT) {
        T prev = __shfl_up_sync(0xFFFFFFFFu, cen[3], 1);
        if (lane == 0 && (hm & 1u)) prev = v[c0 - 1];
        r[0] = hm & 1u ? prev : (T)0;
#pragma unroll
        for (int k = 1; k < 4; ++k) r[k] = (hm >> k) & 1u ? cen[k - 1] : (T)0;
    } else {
        T next = __shfl_down_sync(0xFFFFFFFFu, cen[0], 1);
        const bool has = (m >> 14) & 1u;
        if (lane == 31 && has) next = v[c0 + 4];
        r[3] = has ? next : (T)0;
#pragma unroll
        for (int k = 0; k < 3; ++k) r[k] = (hm >> (k + 1)) & 1u ? cen[k + 1] : (T)0;
    }
}

// Divides eight differences by the spacings: by their exact reciprocals
// (SX_BY_POW2: dx and dy hold those), or by the three operations for a known divisor
// (zx and zy: RN of the reciprocals) unless a difference is too small or too large
// for those, or by division.  One branch for the group.  Spacings that are no powers of
// two, before (division) and after: one float64 step on 2500^2 15.1 -> 12.3 us, float32
// on 3000^2 12.6 -> 10.4, the 120 level steps and 60 transposed ones of a composite of
// base 600 in float32 389 -> 257 and 470 -> 370 us.  Not in the banded step (CONST):
// with a reciprocal to keep per axis and band its 626 us became 654.
template <typename T, bool CONST>
__device__ __forceinline__ void over_group(T (&x)[4], T (&y)[4], T dx, T dy, T zx, T zy, int way)
{
    if (way == SX_BY_POW2) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            x[k] = sx_mul(x[k], dx);
            y[k] = sx_mul(y[k], dy);
        }
        return;
    }
    if (CONST && way == SX_BY_CONST) {
        unsigned small = 0xFFFFFFFFu, large = 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            small = min(small, min(sx_small_key(x[k]), sx_small_key(y[k])));
            large = max(large, max(sx_large_key(x[k]), sx_large_key(y[k])));
        }
        if (small >= (sizeof(T) == 4 ? SX_SMALL_DIFF_F32 : SX_SMALL_DIFF_F64) &&
            large < (sizeof(T) == 4 ? SX_LARGE_DIFF_F32 : SX_LARGE_DIFF_F64)) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                x[k] = sx_by_const(x[k], dx, zx);
                y[k] = sx_by_const(y[k], dy, zy);
            }
            return;
        }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        x[k] = sx_div(x[k], dx);
        y[k] = sx_div(y[k], dy);
    }
}

// How to divide by the spacings (dx and dy become their reciprocals for SX_BY_POW2).
template <typename T>
int spacing_way(T& dx, T& dy)
{
    if (sx_pow2_pair(dx, dy)) return SX_BY_POW2;
    return sx_known_divisor(dx) && sx_known_divisor(dy) ? SX_BY_CONST : SX_BY_DIVISION;
}

// One step.  SGN holds the upwind sides the velocity selects (bit 0: a >= 0,
// the left neighbour; bit 1: b >= 0, the row below), as in the reference's
// formula, which reads one side per axis.  With BANDS, cells band_cell[q] ..
// band_cell[q + 1] - 1 belong to band q with its own spacing and time step
// (band_table[4 q ..]: dx, dy or their exact reciprocals, dt, 1 when the
// reciprocals are given); a block searches its first band once and walks on.
// A block takes ROUNDS runs of groups and, with several, loads a run's plan and values before
// it works on the run before, so a warp waits for one memory round trip per
// run, that of the neighbour row.
template <typename T, bool BANDS, bool VEC, int SGN, int ROUNDS>
__global__ void __launch_bounds__(FLAT_THREADS,
                                  ROUNDS == 1      ? STEP_BLOCKS
                                  : sizeof(T) == 4 ? BAND_STEP_BLOCKS_F32
                                                   : BAND_STEP_BLOCKS_F64)
    flat_step_kernel(const T* v, T* __restrict__ out, long long cells, const int* nbr,
                     const unsigned short* bits, const int4* side, T a, T bb, T dt, T dx,
                     T dy, T zx, T zy, int way, const int* band_cell, const T* band_table,
                     int nbands)
{
    sx_after_previous();
    constexpr bool LEFT = (SGN & 1) != 0, DOWN = (SGN & 2) != 0;
    const int lane = threadIdx.x & 31;
    const long long groups = (cells + 3) >> 2;
    long long g = (long long)blockIdx.x * (FLAT_THREADS * ROUNDS) + threadIdx.x;
    int q = 0;
    long long band_end = cells;
    if (BANDS) {
        q = last_not_above(band_cell, 0, nbands - 1, (int)min(4 * (g - lane), cells - 1));
        band_end = -1;  // the band's values are still to be loaded
    }
    T cen[4];
    unsigned m = 0u;
    int base = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) cen[k] = (T)0;
    if (g < groups) {
        m = bits[g];
        base = nbr[g];
        load_group<T, VEC>(v, 4 * g, cells, cen);
    }
#pragma unroll 1
    for (int round = 0; round < ROUNDS; ++round) {
        const bool act = g < groups;
        const long long c0 = 4 * g;
        g += FLAT_THREADS;
        T nxt[4];
        unsigned mn = 0u;
        int bn = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) nxt[k] = (T)0;
        if (ROUNDS > 1 && round + 1 < ROUNDS && g < groups) {
            mn = bits[g];
            bn = nbr[g];
            load_group<T, VEC>(v, 4 * g, cells, nxt);
        }
        if (BANDS && c0 >= band_end) {
            while (q + 1 < nbands && c0 >= band_cell[q + 1]) ++q;
            band_end = q + 1 < nbands ? band_cell[q + 1] : cells;
            dx = band_table[4 * q];
            dy = band_table[4 * q + 1];
            dt = band_table[4 * q + 2];
            way = band_table[4 * q + 3] != (T)0 ? SX_BY_POW2 : SX_BY_DIVISION;
        }
        T vn[4], vs[4], x[4], y[4], res[4];
        row_group<T>(v, base, DOWN ? m & 15u : (m >> 4) & 15u, (m >> (DOWN ? 12 : 13)) & 1u, side, vn);
        side_group<T, LEFT>(v, cen, m, c0, lane, vs);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            x[k] = LEFT ? sx_sub(cen[k], vs[k]) : sx_sub(vs[k], cen[k]);
            y[k] = DOWN ? sx_sub(cen[k], vn[k]) : sx_sub(vn[k], cen[k]);
        }
        if (BANDS && c0 + 3 >= band_end && act) {  // a band starts inside the group: cell by cell
            int qk = q;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                while (qk + 1 < nbands && c0 + k >= band_cell[qk + 1]) ++qk;
                const T* t = band_table + 4 * qk;
                const int p = t[3] != (T)0;
                res[k] = sx_upwind_update(cen[k], sx_over(x[k], t[0], p), sx_over(y[k], t[1], p), a, bb,
                                          t[2]);
            }
        } else {
            over_group<T, !BANDS>(x, y, dx, dy, zx, zy, way);
#pragma unroll
            for (int k = 0; k < 4; ++k) res[k] = sx_upwind_update(cen[k], x[k], y[k], a, bb, dt);
        }
        if (act) store_group<T, VEC>(out, c0, cells, res);
        m = mn;
        base = bn;
#pragma unroll
        for (int k = 0; k < 4; ++k) cen[k] = nxt[k];
    }
}

// Transpose of one step and the velocity gradient (formulas of
// sx_upwind_adjoint): u is read on the upwind side, w on the other one.  The
// gradient is the sum of exact float64 products w * du (float32 fields),
// reduced per block; the last block to finish adds the blocks' sums in a fixed
// order and scales by -dt, so no second launch is needed.  scratch: a counter
// (zero before the first call, left zero), then two doubles per block.
template <typename T, bool VEC, int SGN>
__global__ void __launch_bounds__(FLAT_THREADS, sizeof(T) == 4 ? ADJOINT_BLOCKS : ADJOINT_BLOCKS_F64)
    flat_adjoint_kernel(const T* w, const T* u, T* __restrict__ ubar, long long cells,
                        const int* dn, const int* up,
                        const unsigned short* bits, const int4* side_dn,
                        const int4* side_up, T a, T bb, T dt, T dx, T dy, T zx, T zy, int way,
                        unsigned* __restrict__ counter, double* __restrict__ partial, double* __restrict__ grads,
                        int accumulate)
{
    sx_after_previous();
    constexpr bool LEFT = (SGN & 1) != 0, DOWN = (SGN & 2) != 0;
    __shared__ double s_a[FLAT_THREADS], s_b[FLAT_THREADS];
    __shared__ bool s_last;
    const int lane = threadIdx.x & 31;
    const long long groups = (cells + 3) >> 2;
    double ga = 0.0, gb = 0.0;
    unsigned mn = 0u;  // the next group's plan: with it at hand, a round waits for memory once
    int bdn = 0, bun = 0;
    const long long first = (long long)blockIdx.x * FLAT_THREADS + threadIdx.x;
    if (first < groups) {
        mn = bits[first];
        bdn = dn[first];
        bun = up[first];
    }
    // whole warps stay in the loop together (the shuffles need every lane)
    for (long long gw = first - lane; gw < groups; gw += (long long)gridDim.x * FLAT_THREADS) {
        const long long g = gw + lane;
        const bool act = g < groups;
        const long long c0 = 4 * g;
        T wc[4], uc[4], wr[4], ur[4], ws[4], us[4], res[4];
        const unsigned m = mn;
        const int bd = bdn, bu = bun;
#pragma unroll
        for (int k = 0; k < 4; ++k) wc[k] = uc[k] = (T)0;
        if (act) {
            load_group<T, VEC>(w, c0, cells, wc);
            load_group<T, VEC>(u, c0, cells, uc);
        }
        mn = 0u;
        const long long gn = g + (long long)gridDim.x * FLAT_THREADS;
        if (gn < groups) {
            mn = bits[gn];
            bdn = dn[gn];
            bun = up[gn];
        }
        const unsigned md = m & 15u, mu = (m >> 4) & 15u;
        const bool id = (m >> 12) & 1u, iu = (m >> 13) & 1u;
        row_group<T>(u, DOWN ? bd : bu, DOWN ? md : mu, DOWN ? id : iu, DOWN ? side_dn : side_up, ur);
        row_group<T>(w, DOWN ? bu : bd, DOWN ? mu : md, DOWN ? iu : id, DOWN ? side_up : side_dn, wr);
        side_group<T, LEFT>(u, uc, m, c0, lane, us);
        side_group<T, !LEFT>(w, wc, m, c0, lane, ws);
        T tx[4], ty[4], dux[4], duy[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            tx[k] = LEFT ? sx_sub(wc[k], ws[k]) : sx_sub(ws[k], wc[k]);
            ty[k] = DOWN ? sx_sub(wc[k], wr[k]) : sx_sub(wr[k], wc[k]);
            dux[k] = LEFT ? sx_sub(uc[k], us[k]) : sx_sub(us[k], uc[k]);
            duy[k] = DOWN ? sx_sub(uc[k], ur[k]) : sx_sub(ur[k], uc[k]);
        }
        over_group<T, true>(tx, ty, dx, dy, zx, zy, way);
        over_group<T, true>(dux, duy, dx, dy, zx, zy, way);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            res[k] = sx_sub(wc[k], sx_mul(dt, sx_add(sx_mul(a, tx[k]), sx_mul(bb, ty[k]))));
            ga = fma((double)wc[k], (double)dux[k], ga);  // cells past the end hold zeros
            gb = fma((double)wc[k], (double)duy[k], gb);
        }
        if (act) store_group<T, VEC>(ubar, c0, cells, res);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ga += __shfl_down_sync(0xFFFFFFFFu, ga, o);
        gb += __shfl_down_sync(0xFFFFFFFFu, gb, o);
    }
    if (lane == 0) {
        s_a[threadIdx.x >> 5] = ga;
        s_b[threadIdx.x >> 5] = gb;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double ta = 0.0, tb = 0.0;
        for (int k = 0; k < FLAT_THREADS / 32; ++k) {
            ta += s_a[k];
            tb += s_b[k];
        }
        partial[2 * blockIdx.x] = ta;
        partial[2 * blockIdx.x + 1] = tb;
        __threadfence();
        s_last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    double ta = 0.0, tb = 0.0;
    for (int k = threadIdx.x; k < (int)gridDim.x; k += FLAT_THREADS) {
        ta += __ldcg(partial + 2 * k);
        tb += __ldcg(partial + 2 * k + 1);
    }
    s_a[threadIdx.x] = ta;
    s_b[threadIdx.x] = tb;
    __syncthreads();
    for (int h = FLAT_THREADS / 2; h > 0; h >>= 1) {
        if (threadIdx.x < h) {
            s_a[threadIdx.x] += s_a[threadIdx.x + h];
            s_b[threadIdx.x] += s_b[threadIdx.x + h];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double sa = -(double)dt * s_a[0], sb = -(double)dt * s_b[0];
        grads[0] = accumulate ? grads[0] + sa : sa;
        grads[1] = accumulate ? grads[1] + sb : sb;
        *counter = 0u;
    }
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

template <typename T, bool BANDS, bool VEC, int ROUNDS>
void step_go(int sgn, int blocks, const T* v, T* out, const SxFlatPlan& P, T a, T bb, T dt, T dx, T dy, int way,
             const int* band_cell, const T* band_table, int nbands, cudaStream_t stream)
{
    const T zx = (T)1 / dx, zy = (T)1 / dy;
    switch (sgn) {
        case 0:
            sx_launch_early(flat_step_kernel<T, BANDS, VEC, 0, ROUNDS>, dim3(blocks), dim3(FLAT_THREADS), 0, stream,
                v, out, P.cells, P.up, P.bits, P.side_up, a, bb, dt, dx, dy, zx, zy, way, band_cell, band_table, nbands);
            break;
        case 1:
            sx_launch_early(flat_step_kernel<T, BANDS, VEC, 1, ROUNDS>, dim3(blocks), dim3(FLAT_THREADS), 0, stream,
                v, out, P.cells, P.up, P.bits, P.side_up, a, bb, dt, dx, dy, zx, zy, way, band_cell, band_table, nbands);
            break;
        case 2:
            sx_launch_early(flat_step_kernel<T, BANDS, VEC, 2, ROUNDS>, dim3(blocks), dim3(FLAT_THREADS), 0, stream,
                v, out, P.cells, P.dn, P.bits, P.side_dn, a, bb, dt, dx, dy, zx, zy, way, band_cell, band_table, nbands);
            break;
        default:
            sx_launch_early(flat_step_kernel<T, BANDS, VEC, 3, ROUNDS>, dim3(blocks), dim3(FLAT_THREADS), 0, stream,
                v, out, P.cells, P.dn, P.bits, P.side_dn, a, bb, dt, dx, dy, zx, zy, way, band_cell, band_table, nbands);
            break;
    }
}

template <typename T, bool BANDS, int ROUNDS>
void step_rounds(const SxFlatPlan& P, const T* v, T* out, T a, T bb, T dt, T dx, T dy, int way, const int* band_cell,
                 const T* band_table, int nbands, cudaStream_t stream)
{
    const long long per = (long long)FLAT_THREADS * 4 * ROUNDS;
    const int blocks = (int)((P.cells + per - 1) / per);
    const int sgn = (a >= (T)0 ? 1 : 0) | (bb >= (T)0 ? 2 : 0);
    if (aligned16(v) && aligned16(out))
        step_go<T, BANDS, true, ROUNDS>(sgn, blocks, v, out, P, a, bb, dt, dx, dy, way, band_cell, band_table, nbands,
                                        stream);
    else
        step_go<T, BANDS, false, ROUNDS>(sgn, blocks, v, out, P, a, bb, dt, dx, dy, way, band_cell, band_table, nbands,
                                         stream);
}

template <typename T, bool BANDS>
void step_run(const SxFlatPlan& P, const T* v, T* out, T a, T bb, T dt, T dx, T dy, int way, const int* band_cell,
              const T* band_table, int nbands, cudaStream_t stream)
{
    // Without bands one run per block is faster at every size (33 M cells, float32: 86 us against 98 to 108).
    if (BANDS && P.cells >= (long long)FLAT_THREADS * 4 * BAND_ROUNDS * 148 * BAND_BLOCKS)
        step_rounds<T, BANDS, BANDS ? BAND_ROUNDS : 1>(P, v, out, a, bb, dt, dx, dy, way, band_cell, band_table,
                                                       nbands, stream);
    else
        step_rounds<T, BANDS, 1>(P, v, out, a, bb, dt, dx, dy, way, band_cell, band_table, nbands, stream);
}

template <typename T, bool VEC>
void adjoint_go(int blocks, const SxFlatPlan& P, const T* w, const T* u, T* ubar, T a, T bb, T dt, T dx, T dy, int way,
                unsigned* counter, double* partial, double* grads, int accumulate, cudaStream_t stream)
{
    const T zx = (T)1 / dx, zy = (T)1 / dy;
    switch ((a >= (T)0 ? 1 : 0) | (bb >= (T)0 ? 2 : 0)) {
        case 0:
            sx_launch_early(flat_adjoint_kernel<T, VEC, 0>, dim3(blocks), dim3(FLAT_THREADS), 0, stream,
                w, u, ubar, P.cells, P.dn, P.up, P.bits, P.side_dn, P.side_up, a, bb, dt, dx, dy, zx, zy, way,
                counter,
                partial, grads, accumulate);
            break;
        case 1:
            sx_launch_early(flat_adjoint_kernel<T, VEC, 1>, dim3(blocks), dim3(FLAT_THREADS), 0, stream,
                w, u, ubar, P.cells, P.dn, P.up, P.bits, P.side_dn, P.side_up, a, bb, dt, dx, dy, zx, zy, way,
                counter,
                partial, grads, accumulate);
            break;
        case 2:
            sx_launch_early(flat_adjoint_kernel<T, VEC, 2>, dim3(blocks), dim3(FLAT_THREADS), 0, stream,
                w, u, ubar, P.cells, P.dn, P.up, P.bits, P.side_dn, P.side_up, a, bb, dt, dx, dy, zx, zy, way,
                counter,
                partial, grads, accumulate);
            break;
        default:
            sx_launch_early(flat_adjoint_kernel<T, VEC, 3>, dim3(blocks), dim3(FLAT_THREADS), 0, stream,
                w, u, ubar, P.cells, P.dn, P.up, P.bits, P.side_dn, P.side_up, a, bb, dt, dx, dy, zx, zy, way,
                counter,
                partial, grads, accumulate);
            break;
    }
}

template <typename T>
void adjoint_run(const SxFlatPlan& P, const T* w, const T* u, T* ubar, T a, T bb, T dt, T dx, T dy, void* scratch,
                 double* grads, int accumulate, cudaStream_t stream)
{
    const int way = spacing_way(dx, dy);
    int blocks = sx_flat_adjoint_parts(P.cells);
    if (sizeof(T) == 8 && blocks > 148 * ADJOINT_BLOCKS_F64) blocks = 148 * ADJOINT_BLOCKS_F64;
    unsigned* counter = (unsigned*)scratch;
    double* partial = (double*)scratch + 2;
    if (aligned16(w) && aligned16(u) && aligned16(ubar))
        adjoint_go<T, true>(blocks, P, w, u, ubar, a, bb, dt, dx, dy, way, counter, partial, grads, accumulate,
                            stream);
    else
        adjoint_go<T, false>(blocks, P, w, u, ubar, a, bb, dt, dx, dy, way, counter, partial, grads, accumulate,
                             stream);
}

}  // namespace

// Blocks of the adjoint kernel: enough to fill the chip once, few enough that
// the last block adds their sums quickly.
int sx_flat_adjoint_parts(long long cells)
{
    long long g = (cells + 4 * FLAT_THREADS - 1) / (4 * FLAT_THREADS);
    if (g < 1) g = 1;
    if (g > 148 * ADJOINT_BLOCKS) g = 148 * ADJOINT_BLOCKS;
    return (int)g;
}

cudaError_t sx_flat_plan_launch(const int* rows, const int* off, int row_count, const int* b, const int* e,
                                const int* coff, int n, long long cells, const int* lookup, int height, int* dn,
                                int* up, unsigned short* bits, void* side, int* span, cudaStream_t stream)
{
    span_init_kernel<<<1, 1, 0, stream>>>(span);
    if (n > 0) span_kernel<<<n < 148 * 4 * 256 ? (n + 255) / 256 : 148 * 4, 256, 0, stream>>>(b, e, n, span);
    if (n > 0 && cells > 0) {
        const long long groups = (cells + 3) / 4;
        const int blocks = (int)((groups + FLAT_THREADS - 1) / FLAT_THREADS);
        flat_plan_kernel<<<blocks, FLAT_THREADS, 0, stream>>>(rows, off, row_count, b, e, coff, n, (int)cells, lookup,
                                                              height, dn, up, bits, (int4*)side, (int4*)side + n);
    }
    return cudaGetLastError();
}

cudaError_t sx_flat_step_launch(const SxFlatPlan& P, int dbl, const void* v, void* out, double a, double bb, double dt,
                                double dx, double dy, cudaStream_t stream)
{
    if (P.cells <= 0) return cudaSuccess;
    if (dbl) {
        const int p = spacing_way(dx, dy);
        step_run<double, false>(P, (const double*)v, (double*)out, a, bb, dt, dx, dy, p, nullptr, nullptr, 0, stream);
    } else {
        float fx = (float)dx, fy = (float)dy;
        const int p = spacing_way(fx, fy);
        step_run<float, false>(P, (const float*)v, (float*)out, (float)a, (float)bb, (float)dt, fx, fy, p, nullptr,
                               nullptr, 0, stream);
    }
    return cudaGetLastError();
}

cudaError_t sx_flat_step_bands_launch(const SxFlatPlan& P, int dbl, const void* v, void* out, double a, double bb,
                                      const int* band_cell, const void* band_table, int nbands, cudaStream_t stream)
{
    if (P.cells <= 0 || nbands <= 0) return cudaSuccess;
    if (dbl)
        step_run<double, true>(P, (const double*)v, (double*)out, a, bb, 0.0, 1.0, 1.0, 0, band_cell,
                               (const double*)band_table, nbands, stream);
    else
        step_run<float, true>(P, (const float*)v, (float*)out, (float)a, (float)bb, 0.0f, 1.0f, 1.0f, 0, band_cell,
                              (const float*)band_table, nbands, stream);
    return cudaGetLastError();
}

cudaError_t sx_flat_adjoint_launch(const SxFlatPlan& P, int dbl, const void* w, const void* u, void* ubar, double a,
                                   double bb, double dt, double dx, double dy, void* scratch, double* grads,
                                   int accumulate, cudaStream_t stream)
{
    if (dbl)
        adjoint_run<double>(P, (const double*)w, (const double*)u, (double*)ubar, a, bb, dt, dx, dy, scratch, grads,
                            accumulate, stream);
    else
        adjoint_run<float>(P, (const float*)w, (const float*)u, (float*)ubar, (float)a, (float)bb, (float)dt,
                           (float)dx, (float)dy, scratch, grads, accumulate, stream);
    return cudaGetLastError();
}
