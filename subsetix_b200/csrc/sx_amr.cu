// Two-level AMR step on full grids, batched over independent simulations.
//
// In the reference's AMR2Simulation both levels are full rectangles: the
// coarse field covers [0, W) x [0, H) and the fine field [0, rW) x [0, rH),
// one interval per row (subsetix_amr2/simulation.py:159-213).  On such sets
// the interval kernels reduce to dense ones, and this file runs them
// directly on [batch][rows][cols] arrays:
//
//   sx_upwind_full     the upwind update of interval_stencil.py:59-113 with
//                      zero exterior (cells outside the grid read 0);
//   sx_amr_sync_full   synchronize_interval_fields with the mean reducer and
//                      copy=False (fields.py:570-612): a coarse cell marked
//                      REFINE takes the mean of its r x r fine block, summed
//                      sub-row outer, column inner, times 1/r^2
//                      (kernels.py:458-527); any other coarse cell is copied
//                      into its fine block (kernels.py:384-418).  Refine and
//                      coarse-only cells partition the grid, so one pass per
//                      coarse cell does both halves;
//   sx_amr_step_full   upwind on both levels and the synchronisation in one kernel
//                      (ratio 2), sx_amr_steps_full up to five such steps;
//   sx_amr_tag_full    the gradient tag of regrid.py:172-223,336-350: the
//                      field is read as float32, the gradient has central
//                      differences inside and one-sided ones at the edges,
//                      and a cell is tagged when sqrt(gx^2 + gy^2) >=
//                      threshold;
//   sx_amr_grade_full  enforce_two_level_grading_set (regrid.py:404-442) as
//                      a cell set: a coarse cell is refined when a tagged
//                      cell lies within `padding` along a row or a column
//                      (von Neumann) or within the (2p+1)^2 box (Moore),
//                      clipped to the grid.  The action byte is REFINE (1)
//                      or KEEP (0), as ActionField.set_from_interval_set
//                      writes it (fields.py:520-546).
//
// Float formulas use explicit rounding intrinsics, including the float32
// fusions the reference's NVRTC build makes (sx_upwind_update and
// sx_grad_norm), so results are bit-identical to the interval kernels (and
// to the reference) on the same inputs, in float32 and in float64.

#include <cmath>

#include "sx_internal.cuh"

__device__ __forceinline__ float sxa_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sxa_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float sxa_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float sxa_div(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ double sxa_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sxa_sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double sxa_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double sxa_div(double a, double b) { return __ddiv_rn(a, b); }

// x / d, or x * d when the launcher passed the reciprocal of a power-of-two
// spacing instead (pow2 != 0).  Dividing by 2^k and multiplying by 2^-k
// have the same exact real result, so the rounded results are identical.
template <typename T>
__device__ __forceinline__ T sxa_over(T x, T d, int pow2)
{
    return pow2 ? sxa_mul(x, d) : sxa_div(x, d);
}

// One thread per cell; x fastest.  blockIdx.z is the batch entry.
// The upwind update of one cell from the neighbours the velocity selects:
// SGN bit 0 (a >= 0) the left one in h, else the right one; bit 1 (b >= 0)
// the one below in v, else the one above.  The reference's formula uses one
// side per axis, so the other side is never read.
template <typename T, int SGN>
__device__ __forceinline__ T sxa_upwind_side(T c, T h, T v, T a, T b, T dt, T dx, T dy, int pow2)
{
    const T du_dx = (SGN & 1) ? sxa_over(sxa_sub(c, h), dx, pow2) : sxa_over(sxa_sub(h, c), dx, pow2);
    const T du_dy = (SGN & 2) ? sxa_over(sxa_sub(c, v), dy, pow2) : sxa_over(sxa_sub(v, c), dy, pow2);
    return sx_upwind_update(c, du_dx, du_dy, a, b, dt);
}

template <typename T, int SGN>
__global__ void __launch_bounds__(256) sx_upwind_full_kernel(const T* __restrict__ in, T* __restrict__ out, int W,
                                                             int H, T a, T b, T dt, T dx, T dy, int pow2)
{
    const long long plane = (long long)W * H;
    const T* v = in + plane * blockIdx.z;
    T* o = out + plane * blockIdx.z;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= W) return;
    const long long idx = (long long)y * W + x;
    const T c = v[idx];
    const T h = (SGN & 1) ? (x > 0 ? v[idx - 1] : (T)0) : (x + 1 < W ? v[idx + 1] : (T)0);
    const T w = (SGN & 2) ? (y > 0 ? v[idx - W] : (T)0) : (y + 1 < H ? v[idx + W] : (T)0);
    o[idx] = sxa_upwind_side<T, SGN>(c, h, w, a, b, dt, dx, dy, pow2);
}

// One thread per coarse cell.  R is the refinement ratio (template for the
// common 2, runtime otherwise).
template <typename T, int RT>
__global__ void __launch_bounds__(256) sx_amr_sync_full_kernel(T* __restrict__ coarse, T* __restrict__ fine,
                                                               const signed char* __restrict__ actions, int W, int H,
                                                               int rr, T norm)
{
    const int R = RT > 0 ? RT : rr;
    const int b = blockIdx.z;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= W) return;
    const long long plane = (long long)W * H;
    const long long ci = plane * b + (long long)y * W + x;
    const int FW = W * R;
    T* f = fine + plane * R * R * b + ((long long)y * R) * FW + (long long)x * R;
    if (actions[ci] == 1) {
        T acc = (T)0;
        for (int dy = 0; dy < R; ++dy)
            for (int dx = 0; dx < R; ++dx) acc = sxa_add(acc, f[(long long)dy * FW + dx]);
        coarse[ci] = sxa_mul(acc, norm);
    } else {
        const T c = coarse[ci];
        for (int dy = 0; dy < R; ++dy)
            for (int dx = 0; dx < R; ++dx) f[(long long)dy * FW + dx] = c;
    }
}

// The synchronisation into new arrays, both read and written once: bound by
// their bytes (1001^2 float64: 80 MB, 12 us at the copy rate, 8.4 us measured as part of it stays in L2).
// Without it a copying synchronisation of whole-grid fields was two clones, a
// restriction, two gathers, two scatters and a prolongation over interval sets,
// 60 launches and 13 read-backs.  `actions` may be null: nothing refined.  For
// ratio 2 a thread moves the two values of a sub-row at once (PAIR: fine rows
// have an even length, so pairs are aligned when the arrays are).
template <typename T>
struct SxaPair;
template <>
struct SxaPair<float> {
    typedef float2 type;
};
template <>
struct SxaPair<double> {
    typedef double2 type;
};

template <typename T, bool PAIR>
__global__ void __launch_bounds__(256) sx_amr_sync_copy_kernel(const T* __restrict__ coarse, const T* __restrict__ fine,
                                                               const signed char* __restrict__ actions,
                                                               T* __restrict__ coarse_out, T* __restrict__ fine_out,
                                                               int W, int H, int rr, T norm)
{
    typedef typename SxaPair<T>::type P2;
    const int R = PAIR ? 2 : rr;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= W) return;
    const long long plane = (long long)W * H, ci = plane * blockIdx.z + (long long)y * W + x;
    const long long FW = (long long)W * R;
    const long long fi = plane * R * R * blockIdx.z + (long long)y * R * FW + (long long)x * R;
    if (actions && actions[ci] == 1) {
        T acc = (T)0;
        if (PAIR) {
            const P2 a = *(const P2*)(fine + fi), b = *(const P2*)(fine + fi + FW);
            acc = sxa_add(sxa_add(sxa_add(sxa_add(acc, a.x), a.y), b.x), b.y);
            *(P2*)(fine_out + fi) = a;
            *(P2*)(fine_out + fi + FW) = b;
        } else {
            for (int dy = 0; dy < R; ++dy)
                for (int dx = 0; dx < R; ++dx) {
                    const T v = fine[fi + dy * FW + dx];
                    acc = sxa_add(acc, v);
                    fine_out[fi + dy * FW + dx] = v;
                }
        }
        coarse_out[ci] = sxa_mul(acc, norm);
    } else {
        const T c = coarse[ci];
        coarse_out[ci] = c;
        if (PAIR) {
            P2 q;
            q.x = c;
            q.y = c;
            *(P2*)(fine_out + fi) = q;
            *(P2*)(fine_out + fi + FW) = q;
        } else {
            for (int dy = 0; dy < R; ++dy)
                for (int dx = 0; dx < R; ++dx) fine_out[fi + dy * FW + dx] = c;
        }
    }
}

// Whole fixed-geometry step for ratio 2: upwind of the coarse cell and of
// its 2 x 2 fine block (from the previous values, zero exterior), then the
// synchronisation of that coarse cell with its block.  A step's
// synchronisation of a coarse cell reads only that cell's and that block's
// new values, so this equals upwind(coarse); upwind(fine); sync, value for
// value.  in/out are distinct buffers.  SGN: the velocity's upwind sides, as
// in sxa_upwind_side.
template <typename T, int SGN>
__global__ void __launch_bounds__(256) sx_amr_step_full_kernel(const T* __restrict__ cin, const T* __restrict__ fin,
                                                               T* __restrict__ cout, T* __restrict__ fout,
                                                               const signed char* __restrict__ actions, int W, int H,
                                                               T a, T b, T dt, T dxc, T dyc, T dxf, T dyf, T norm,
                                                               int pow2c, int pow2f)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= W) return;
    const long long plane = (long long)W * H;
    const int FW = 2 * W, FH = 2 * H;
    const T* C = cin + plane * blockIdx.z;
    const T* F = fin + 4 * plane * blockIdx.z;
    const long long ci = (long long)y * W + x;
    // coarse cell, with the neighbours the velocity selects
    const T c = C[ci];
    const T ch = (SGN & 1) ? (x > 0 ? C[ci - 1] : (T)0) : (x + 1 < W ? C[ci + 1] : (T)0);
    const T cv = (SGN & 2) ? (y > 0 ? C[ci - W] : (T)0) : (y + 1 < H ? C[ci + W] : (T)0);
    const T cn = sxa_upwind_side<T, SGN>(c, ch, cv, a, b, dt, dxc, dyc, pow2c);
    const int fx = 2 * x, fy = 2 * y;
    T* CO = cout + plane * blockIdx.z;
    T* FO = fout + 4 * plane * blockIdx.z;
    if (actions[plane * blockIdx.z + ci] != 1) {
        // not refined: the synchronisation overwrites the fine block with the
        // new coarse value, so its own upwind update is never needed
        CO[ci] = cn;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            T* row = FO + (long long)(fy + j) * FW + fx;
            row[0] = cn;
            row[1] = cn;
        }
        return;
    }
    // refined: fine block, rows 2y-1 .. 2y+2, columns 2x-1 .. 2x+2; only the
    // 2 x 2 block and the column and row on its upwind sides are read
    T v[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int yy = fy - 1 + j;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int xx = fx - 1 + i;
            const bool inner_row = j == 1 || j == 2, inner_col = i == 1 || i == 2;
            const bool needed = (inner_row && inner_col) ||
                                (inner_row && (((SGN & 1) && i == 0) || (!(SGN & 1) && i == 3))) ||
                                (inner_col && (((SGN & 2) && j == 0) || (!(SGN & 2) && j == 3)));
            v[j][i] = (needed && yy >= 0 && yy < FH && xx >= 0 && xx < FW) ? F[(long long)yy * FW + xx] : (T)0;
        }
    }
    T fn[2][2];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i)
            fn[j][i] = sxa_upwind_side<T, SGN>(v[j + 1][i + 1], (SGN & 1) ? v[j + 1][i] : v[j + 1][i + 2],
                                               (SGN & 2) ? v[j][i + 1] : v[j + 2][i + 1], a, b, dt, dxf, dyf, pow2f);
    T acc = sxa_add(sxa_add(sxa_add(sxa_add((T)0, fn[0][0]), fn[0][1]), fn[1][0]), fn[1][1]);
    CO[ci] = sxa_mul(acc, norm);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        T* row = FO + (long long)(fy + j) * FW + fx;
        row[0] = fn[j][0];
        row[1] = fn[j][1];
    }
}

// Several fixed-geometry steps in one pass over the arrays (ratio 2), value for
// value those of sx_amr_step_full_kernel.
//
// A block owns a tile: its warps' lanes hold 32 lanes' coarse columns (two per lane in
// float32, one in float64) of SXA_ROWS rows each, with their fine blocks, in registers.
// Columns and rows count from the velocity's upwind side, so every cell depends on its
// own and the lower indices only: a step goes through a warp's rows from the last to
// the first, takes the left column by a shuffle and the row below the warp's first from
// shared memory, one barrier per step.  The arrays are read once and written once for
// all the steps.  The first `steps` columns and rows of a tile only serve the others
// (they depend on cells the tile does not have); at the grid's edges those cells are
// the zero exterior instead.
//
// Bound: one step per pass moves 42 MB at 1024^2 (float32) and takes 6.4 us, close to
// what L2 gives; five in one pass take 14.9 us and are bound by instructions (the
// repeated columns and rows are a third of the work).  Walking up single strips with
// the steps following one another in registers or shared memory took 22 to 26 us (a
// chain of dependent operations, and each band repeats the rows before it); 2, 3, 4, 8
// rows per warp 15.6, 14.9, 17.2, 27 us.  Float32 cells go two by two through the
// packed instructions, which round each half as the scalar ones do.  Twenty steps,
// before and after, without the regrids: 1024^2 float32 129 -> 60 us, float64 206 -> 96,
// 2048^2 568 -> 208; spacings that are no powers of two: 777^2 float32 122 -> 91,
// 1200^2 float64 327 -> 244, 300^2 float64 75 -> 39, and with a general division per
// difference 207, 309 and 141: those divide by a known divisor (sx_common.cuh) unless
// a value is too small or not finite.
// An unrefined coarse cell's fine block is its coarse value after every step, and a
// refined one's coarse value is its block's mean: a row without refined (or
// unrefined) cells skips the fine (or coarse) updates.

// SxaP<T>: the coarse columns of one lane, in one register pair.
template <typename T>
struct SxaP;
template <>
struct SxaP<double> {
    static constexpr int CPL = 1;
    double v;
};
template <>
struct SxaP<float> {
    static constexpr int CPL = 2;
    unsigned long long v;  // column 0 in the low half
};
typedef SxaP<float> SxaPf;
typedef SxaP<double> SxaPd;

__device__ __forceinline__ SxaPd sxp_set(double x) { return SxaPd{x}; }
__device__ __forceinline__ SxaPf sxp_set(float x, float y)
{
    SxaPf p;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p.v) : "f"(x), "f"(y));
    return p;
}
__device__ __forceinline__ void sxp_get(const SxaPf& p, float (&x)[2])
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x[0]), "=f"(x[1]) : "l"(p.v));
}
__device__ __forceinline__ void sxp_get(const SxaPd& p, double (&x)[1]) { x[0] = p.v; }
__device__ __forceinline__ SxaPf sxp_make(const float (&x)[2]) { return sxp_set(x[0], x[1]); }
__device__ __forceinline__ SxaPd sxp_make(const double (&x)[1]) { return sxp_set(x[0]); }
__device__ __forceinline__ SxaPf sxp_all(float x) { return sxp_set(x, x); }
__device__ __forceinline__ SxaPd sxp_all(double x) { return sxp_set(x); }
__device__ __forceinline__ SxaPf sxp_add(SxaPf a, SxaPf b)
{
    SxaPf r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ SxaPf sxp_sub(SxaPf a, SxaPf b)
{
    SxaPf r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ SxaPf sxp_mul(SxaPf a, SxaPf b)
{
    SxaPf r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ SxaPf sxp_fma(SxaPf a, SxaPf b, SxaPf c)
{
    SxaPf r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ SxaPd sxp_add(SxaPd a, SxaPd b) { return SxaPd{sxa_add(a.v, b.v)}; }
__device__ __forceinline__ SxaPd sxp_sub(SxaPd a, SxaPd b) { return SxaPd{sxa_sub(a.v, b.v)}; }
__device__ __forceinline__ SxaPd sxp_mul(SxaPd a, SxaPd b) { return SxaPd{sxa_mul(a.v, b.v)}; }
__device__ __forceinline__ SxaPd sxp_fma(SxaPd a, SxaPd b, SxaPd c) { return SxaPd{__fma_rn(a.v, b.v, c.v)}; }
__device__ __forceinline__ SxaPd sxp_div(SxaPd a, double d) { return SxaPd{sxa_div(a.v, d)}; }
__device__ __forceinline__ SxaPf sxp_div(SxaPf a, float d)
{
    float x[2];
    sxp_get(a, x);
    return sxp_set(sxa_div(x[0], d), sxa_div(x[1], d));
}
// sx_upwind_update, term for term; ndt is -dt in float32, dt in float64
__device__ __forceinline__ SxaPf sxp_update(SxaPf c, SxaPf dux, SxaPf duy, SxaPf a, SxaPf b, SxaPf ndt)
{
    return sxp_fma(ndt, sxp_fma(a, dux, sxp_mul(b, duy)), c);
}
__device__ __forceinline__ SxaPd sxp_update(SxaPd c, SxaPd dux, SxaPd duy, SxaPd a, SxaPd b, SxaPd dt)
{
    return sxp_sub(c, sxp_mul(dt, sxp_add(sxp_mul(a, dux), sxp_mul(b, duy))));
}
// the values one column to the left; the first lane's left column is zero
__device__ __forceinline__ SxaPf sxp_left(SxaPf p, int lane)
{
    float x[2];
    sxp_get(p, x);
    const float l = __shfl_up_sync(0xFFFFFFFFu, x[1], 1);
    return sxp_set(lane == 0 ? 0.0f : l, x[0]);
}
__device__ __forceinline__ SxaPd sxp_left(SxaPd p, int lane)
{
    const double l = __shfl_up_sync(0xFFFFFFFFu, p.v, 1);
    return sxp_set(lane == 0 ? 0.0 : l);
}
// column k from a where bit k of m is set, else from b
__device__ __forceinline__ SxaPf sxp_pick(unsigned m, SxaPf a, SxaPf b)
{
    float x[2], y[2];
    sxp_get(a, x);
    sxp_get(b, y);
    return sxp_set(m & 1u ? x[0] : y[0], m & 2u ? x[1] : y[1]);
}
__device__ __forceinline__ SxaPd sxp_pick(unsigned m, SxaPd a, SxaPd b) { return m & 1u ? a : b; }

// by the three operations in float64 (float32 only; z = RN(1 / d) there)
__device__ __forceinline__ SxaPf sxp_div_double(SxaPf a, float d, double z)
{
    float x[2];
    sxp_get(a, x);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const double t = (double)x[k], q = __dmul_rn(t, z);
        x[k] = (float)__fma_rn(-__fma_rn(q, (double)d, -t), z, q);
    }
    return sxp_make(x);
}
__device__ __forceinline__ SxaPd sxp_div_double(SxaPd a, double d, double) { return sxp_div(a, d); }
__device__ __forceinline__ unsigned sxp_small_key(SxaPf p)
{
    float x[2];
    sxp_get(p, x);
    return min(sx_small_key(x[0]), sx_small_key(x[1]));
}
__device__ __forceinline__ unsigned sxp_small_key(SxaPd p) { return sx_small_key(p.v); }
__device__ __forceinline__ bool sxp_is_zero(SxaPf p)
{
    float x[2];
    sxp_get(p, x);
    return x[0] == 0.0f && x[1] == 0.0f;
}
__device__ __forceinline__ bool sxp_is_zero(SxaPd p) { return p.v == 0.0; }

// One row of a lane: coarse values c, and f[r][i] the fine values of sub-row r and
// sub-column i, upwind ones first; bit k of act: column k is refined.
template <typename T>
struct SxaRow {
    SxaP<T> c, f[2][2];
    unsigned act;
};

template <typename T, int SGN>
__device__ __forceinline__ void sxa_load_row(SxaRow<T>& R, const T* __restrict__ C, const T* __restrict__ F,
                                             const signed char* __restrict__ A, int W, int y, int xm, int vec)
{
    constexpr bool LEFT = (SGN & 1) != 0, DOWN = (SGN & 2) != 0;
    constexpr int CPL = SxaP<T>::CPL;
    const T* cr = C + (long long)y * W;
    const signed char* ar = A + (long long)y * W;
    R.act = 0u;
    T c[CPL], f[2][2][CPL];
    if (vec && xm + CPL <= W) {
        const int x = LEFT ? xm : W - CPL - xm;
        if constexpr (CPL == 2) {
            const float2 q = *(const float2*)(cr + x);
            const char2 p = *(const char2*)(ar + x);
            c[LEFT ? 0 : 1] = q.x;
            c[LEFT ? 1 : 0] = q.y;
            R.act = (p.x == 1 ? (LEFT ? 1u : 2u) : 0u) | (p.y == 1 ? (LEFT ? 2u : 1u) : 0u);
        } else {
            c[0] = cr[x];
            R.act = ar[x] == 1 ? 1u : 0u;
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const T* fr = F + (2ll * y + (DOWN ? r : 1 - r)) * (2ll * W) + 2ll * x;
            if constexpr (CPL == 2) {
                const float4 q = *(const float4*)fr;
                f[r][0][0] = LEFT ? q.x : q.w;
                f[r][1][0] = LEFT ? q.y : q.z;
                f[r][0][1] = LEFT ? q.z : q.y;
                f[r][1][1] = LEFT ? q.w : q.x;
            } else {
                const double2 q = *(const double2*)fr;
                f[r][0][0] = LEFT ? q.x : q.y;
                f[r][1][0] = LEFT ? q.y : q.x;
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < CPL; ++k) {
            const bool in = xm + k < W;
            const int x = LEFT ? xm + k : W - 1 - xm - k;
            c[k] = in ? cr[x] : (T)0;
            if (in && ar[x] == 1) R.act |= 1u << k;
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    f[r][i][k] = in ? F[(2ll * y + (DOWN ? r : 1 - r)) * (2ll * W) + 2ll * x + (LEFT ? i : 1 - i)] : (T)0;
        }
    }
    R.c = sxp_make(c);
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int i = 0; i < 2; ++i) R.f[r][i] = sxp_make(f[r][i]);
}

template <typename T, int SGN>
__device__ __forceinline__ void sxa_store_row(const SxaRow<T>& R, T* __restrict__ C, T* __restrict__ F, int W, int y,
                                              int xm, int vec)
{
    constexpr bool LEFT = (SGN & 1) != 0, DOWN = (SGN & 2) != 0;
    constexpr int CPL = SxaP<T>::CPL;
    T c[CPL], f[2][2][CPL];
    sxp_get(R.c, c);
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int i = 0; i < 2; ++i) sxp_get(R.f[r][i], f[r][i]);
    if (vec && xm + CPL <= W) {
        const int x = LEFT ? xm : W - CPL - xm;
        T* cr = C + (long long)y * W + x;
        if constexpr (CPL == 2)
            *(float2*)cr = make_float2(c[LEFT ? 0 : 1], c[LEFT ? 1 : 0]);
        else
            *cr = c[0];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            T* fr = F + (2ll * y + (DOWN ? r : 1 - r)) * (2ll * W) + 2ll * x;
            if constexpr (CPL == 2)
                *(float4*)fr = LEFT ? make_float4(f[r][0][0], f[r][1][0], f[r][0][1], f[r][1][1])
                                    : make_float4(f[r][1][1], f[r][0][1], f[r][1][0], f[r][0][0]);
            else
                *(double2*)fr = make_double2(f[r][LEFT ? 0 : 1][0], f[r][LEFT ? 1 : 0][0]);
        }
        return;
    }
#pragma unroll
    for (int k = 0; k < CPL; ++k) {
        if (xm + k >= W) continue;
        const int x = LEFT ? xm + k : W - 1 - xm - k;
        C[(long long)y * W + x] = c[k];
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int i = 0; i < 2; ++i)
                F[(2ll * y + (DOWN ? r : 1 - r)) * (2ll * W) + 2ll * x + (LEFT ? i : 1 - i)] = f[r][i][k];
    }
}

constexpr int SXA_WARPS = 8;  // warps of a block
constexpr int SXA_ROWS = 3;   // coarse rows of a warp

// Spacing of one axis: d, or its reciprocal z = RN(1 / d) as well.
template <typename T>
struct SxaSpan {
    T d, z;
    double zz;  // RN(1 / d) in float64
};
template <typename T>
struct SxaStep {
    T a, b, dt, norm;
    SxaSpan<T> xc, yc, xf, yf;
};

// Whether sxa_over gives the negated quotient: for the three operations on pairs, which
// have no negated operands, that is what keeps the sign of a zero (see sx_by_const)
// without a fourth one.
template <int DIV>
constexpr bool sxa_negated = DIV == SX_BY_CONST || DIV == SX_BY_SCALED;

// t over the spacing; key takes the smallest key of the scaled quotients.
template <typename T, int DIV>
__device__ __forceinline__ SxaP<T> sxa_over(SxaP<T> t, const SxaSpan<T>& w, unsigned& key)
{
    if constexpr (DIV == SX_BY_POW2) return sxp_mul(t, sxp_all(w.z));
    if constexpr (DIV == SX_BY_CONST) {
        const SxaP<T> nz = sxp_all(-w.z), nq = sxp_mul(t, nz);
        return sxp_fma(sxp_fma(nq, sxp_all(w.d), t), nz, nq);
    }
    if constexpr (DIV == SX_BY_SCALED) {
        const SxaP<T> u = sxp_mul(t, sxp_all((T)0x1p64)), nz = sxp_all(-w.z), nq = sxp_mul(u, nz);
        const SxaP<T> v = sxp_mul(sxp_fma(sxp_fma(nq, sxp_all(w.d), u), nz, nq), sxp_all((T)0x1p-64));
        key = min(key, sxp_small_key(v));
        return v;
    }
    if constexpr (DIV == SX_BY_DOUBLE) return sxp_div_double(t, w.d, w.zz);
    return sxp_div(t, w.d);
}

// One step of a row whose lower neighbour row had coarse values vc and, in its nearer
// fine row, v0 and v1: the new coarse values cn and fine values fn before the
// synchronisation (the ones the row's refinement asks for).
template <typename T, int SGN, int DIV>
__device__ __forceinline__ void sxa_step_row(const SxaRow<T>& Q, SxaP<T> vc, SxaP<T> v0, SxaP<T> v1, int lane,
                                             bool some, bool all, const SxaStep<T>& S, SxaP<T>& cn, SxaP<T> (&fn)[2][2],
                                             unsigned& key)
{
    typedef SxaP<T> P;
    constexpr bool LEFT = (SGN & 1) != 0, DOWN = (SGN & 2) != 0;
    const P a = sxp_all(sxa_negated<DIV> ? -S.a : S.a), b = sxp_all(sxa_negated<DIV> ? -S.b : S.b);
    const P ndt = sxp_all(sizeof(T) == 4 ? -S.dt : S.dt);
    auto update = [&](P c, P h, P v, const SxaSpan<T>& wx, const SxaSpan<T>& wy) {
        const P tx = LEFT ? sxp_sub(c, h) : sxp_sub(h, c), ty = DOWN ? sxp_sub(c, v) : sxp_sub(v, c);
        return sxp_update(c, sxa_over<T, DIV>(tx, wx, key), sxa_over<T, DIV>(ty, wy, key), a, b, ndt);
    };
    if (!all) cn = update(Q.c, sxp_left(Q.c, lane), vc, S.xc, S.yc);
    if (some) {
        fn[0][0] = update(Q.f[0][0], sxp_left(Q.f[0][1], lane), v0, S.xf, S.yf);
        fn[0][1] = update(Q.f[0][1], Q.f[0][0], v1, S.xf, S.yf);
        fn[1][0] = update(Q.f[1][0], sxp_left(Q.f[1][1], lane), Q.f[0][0], S.xf, S.yf);
        fn[1][1] = update(Q.f[1][1], Q.f[1][0], Q.f[0][1], S.xf, S.yf);
    }
}

// Not zero once a new value is not finite.
template <typename T>
__device__ __forceinline__ bool sxa_not_finite(const SxaP<T>& cn, const SxaP<T> (&fn)[2][2])
{
    const SxaP<T> zero = sxp_all((T)0);
    SxaP<T> x = sxp_mul(cn, zero);
#pragma unroll
    for (int q = 0; q < 4; ++q) x = sxp_fma(fn[q >> 1][q & 1], zero, x);
    return !sxp_is_zero(x);
}

// sxa_step_row for rows with small or overflowing values, out of line: by the scaled
// quotients (float32), and by divisions where that does not hold.
template <typename T>
struct SxaNew {
    SxaP<T> c, f[2][2];
};
template <typename T, int SGN>
__device__ __noinline__ SxaNew<T> sxa_divide_row(SxaRow<T> Q, SxaP<T> vc, SxaP<T> v0, SxaP<T> v1, int lane, bool some,
                                                 bool all, const SxaStep<T>& S)
{
    SxaNew<T> n;
    n.c = n.f[0][0] = n.f[0][1] = n.f[1][0] = n.f[1][1] = sxp_all((T)0);
    unsigned key = 0xFFFFFFFFu;
    if (sizeof(T) == 4) {
        sxa_step_row<T, SGN, SX_BY_SCALED>(Q, vc, v0, v1, lane, some, all, S, n.c, n.f, key);
        if (!__any_sync(0xFFFFFFFFu, sx_is_subnormal<T>(key) || sxa_not_finite<T>(n.c, n.f))) return n;
        sxa_step_row<T, SGN, SX_BY_DOUBLE>(Q, vc, v0, v1, lane, some, all, S, n.c, n.f, key);
        if (!__any_sync(0xFFFFFFFFu, sxa_not_finite<T>(n.c, n.f))) return n;
    }
    sxa_step_row<T, SGN, SX_BY_DIVISION>(Q, vc, v0, v1, lane, some, all, S, n.c, n.f, key);
    return n;
}

template <typename T, int SGN, int DIV>
__global__ void __launch_bounds__(32 * SXA_WARPS, DIV == SX_BY_POW2 ? 4 : 3)
    sx_amr_steps_full_kernel(const T* __restrict__ cin, const T* __restrict__ fin, T* __restrict__ cout,
                             T* __restrict__ fout, const signed char* __restrict__ actions, int W, int H, int steps,
                             int strips, int vec, const __grid_constant__ SxaStep<T> S)
{
    typedef SxaP<T> P;
    constexpr bool LEFT = (SGN & 1) != 0, DOWN = (SGN & 2) != 0;
    constexpr int CPL = P::CPL, NR = SXA_ROWS;
    // every warp's last row before a step: coarse values and those of the nearer fine row
    __shared__ P s_c[2][SXA_WARPS][32], s_f[2][SXA_WARPS][2][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int strip = blockIdx.x % strips, band = blockIdx.x / strips;
    const int halo = (steps + CPL - 1) / CPL * CPL;
    const int xm = strip * (32 * CPL - halo) + lane * CPL;      // first column of this lane, upwind side first
    const int jm = band * (SXA_WARPS * NR - steps) + wid * NR;  // first row of this warp
    const long long plane = (long long)W * H;
    const T* C = cin + plane * blockIdx.z;
    const T* F = fin + 4 * plane * blockIdx.z;
    const signed char* A = actions + plane * blockIdx.z;
    const P zero = sxp_all((T)0);
    SxaRow<T> R[NR];
    bool some[NR], all[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        if (jm + r < H) {
            sxa_load_row<T, SGN>(R[r], C, F, A, W, DOWN ? jm + r : H - 1 - jm - r, xm, vec);
        } else {
            R[r].act = 0u;
            R[r].c = R[r].f[0][0] = R[r].f[0][1] = R[r].f[1][0] = R[r].f[1][1] = zero;
        }
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        some[r] = __any_sync(0xFFFFFFFFu, R[r].act != 0u);
        all[r] = __all_sync(0xFFFFFFFFu, R[r].act == (1u << CPL) - 1u);
    }
#pragma unroll 1
    for (int s = 0; s < steps; ++s) {
        const int par = s & 1;
        s_c[par][wid][lane] = R[NR - 1].c;
        s_f[par][wid][0][lane] = R[NR - 1].f[1][0];
        s_f[par][wid][1][lane] = R[NR - 1].f[1][1];
        __syncthreads();  // the other half holds the step before, which a late warp may still read
        const P bc = wid > 0 ? s_c[par][wid - 1][lane] : zero;
        const P b0 = wid > 0 ? s_f[par][wid - 1][0][lane] : zero, b1 = wid > 0 ? s_f[par][wid - 1][1][lane] : zero;
        bool small = false;
        if constexpr (DIV == SX_BY_CONST) {
            unsigned key = min(sxp_small_key(bc), min(sxp_small_key(b0), sxp_small_key(b1)));
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                key = min(key, sxp_small_key(R[r].c));
#pragma unroll
                for (int q = 0; q < 4; ++q) key = min(key, sxp_small_key(R[r].f[q >> 1][q & 1]));
            }
            small = __any_sync(0xFFFFFFFFu, sx_is_small<T>(key));
        }
        // rows from the last to the first: each reads its lower neighbour before that changes
#pragma unroll
        for (int r = NR - 1; r >= 0; --r) {
            SxaRow<T>& Q = R[r];
            const P vc = r > 0 ? R[r > 0 ? r - 1 : 0].c : bc;
            const P v0 = r > 0 ? R[r > 0 ? r - 1 : 0].f[1][0] : b0, v1 = r > 0 ? R[r > 0 ? r - 1 : 0].f[1][1] : b1;
            P cn = zero, fn[2][2];
            fn[0][0] = fn[0][1] = fn[1][0] = fn[1][1] = zero;
            unsigned key = 0u;
            if (!small) sxa_step_row<T, SGN, DIV>(Q, vc, v0, v1, lane, some[r], all[r], S, cn, fn, key);
            if constexpr (DIV == SX_BY_CONST) {
                if (small || __any_sync(0xFFFFFFFFu, sxa_not_finite<T>(cn, fn))) {
                    const SxaNew<T> n = sxa_divide_row<T, SGN>(Q, vc, v0, v1, lane, some[r], all[r], S);
                    cn = n.c;
#pragma unroll
                    for (int q = 0; q < 4; ++q) fn[q >> 1][q & 1] = n.f[q >> 1][q & 1];
                }
            }
            if (!some[r]) {
                Q.c = Q.f[0][0] = Q.f[0][1] = Q.f[1][0] = Q.f[1][1] = cn;
                continue;
            }
            // the synchronisation, the block's values in the grid's order
            constexpr int R0 = DOWN ? 0 : 1, C0 = LEFT ? 0 : 1;
            P acc = sxp_add(zero, fn[R0][C0]);
            acc = sxp_add(acc, fn[R0][1 - C0]);
            acc = sxp_add(acc, fn[1 - R0][C0]);
            acc = sxp_mul(sxp_add(acc, fn[1 - R0][1 - C0]), sxp_all(S.norm));
            if (all[r]) {
                Q.c = acc;
#pragma unroll
                for (int q = 0; q < 4; ++q) Q.f[q >> 1][q & 1] = fn[q >> 1][q & 1];
            } else {
                Q.c = sxp_pick(Q.act, acc, cn);
#pragma unroll
                for (int q = 0; q < 4; ++q) Q.f[q >> 1][q & 1] = sxp_pick(Q.act, fn[q >> 1][q & 1], cn);
            }
        }
    }
    if (strip > 0 && lane * CPL < halo) return;
#pragma unroll
    for (int r = 0; r < NR; ++r)
        if (jm + r < H && (band == 0 || wid * NR + r >= steps))
            sxa_store_row<T, SGN>(R[r], cout + plane * blockIdx.z, fout + 4 * plane * blockIdx.z, W,
                                  DOWN ? jm + r : H - 1 - jm - r, xm, vec);
}

template <typename T>
__global__ void __launch_bounds__(256) sx_amr_tag_full_kernel(const T* __restrict__ in, unsigned char* __restrict__ tags,
                                                              int W, int H, float thr)
{
    const long long plane = (long long)W * H;
    const T* v = in + plane * blockIdx.z;
    unsigned char* t = tags + plane * blockIdx.z;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= W) return;
    const long long idx = (long long)y * W + x;
    const float c = (float)v[idx];
    float gx = 0.0f, gy = 0.0f;
    if (W > 1) {
        if (x == 0) gx = __fsub_rn((float)v[idx + 1], c);
        else if (x == W - 1) gx = __fsub_rn(c, (float)v[idx - 1]);
        else gx = __fmul_rn(__fsub_rn((float)v[idx + 1], (float)v[idx - 1]), 0.5f);
    }
    if (H > 1) {
        if (y == 0) gy = __fsub_rn((float)v[idx + W], c);
        else if (y == H - 1) gy = __fsub_rn(c, (float)v[idx - W]);
        else gy = __fmul_rn(__fsub_rn((float)v[idx + W], (float)v[idx - W]), 0.5f);
    }
    t[idx] = sx_grad_norm(gx, gy) >= thr ? 1 : 0;
}

// Tag and grade in one pass for paddings up to SXA_GRADE_MAX.  A warp walks up a strip of 32 columns: the gradient's neighbours are the
// lanes beside and the rows before and after, a ballot has the row's tags, and shift
// registers the 2 p + 1 last rows', so each value is read once.  The p + 1 columns on
// either side of a strip and the p rows before and after a band serve their
// neighbours' results.  mode as in sx_amr_grade_full_kernel; p = 0 grades nothing.
// The two kernels, one thread per cell, spend their time on the square root and on a
// byte load per neighbour: 13.1 us at 1024^2, 41 at 2048^2; here 7.9 and 23 us with 16
// rows per band (12 us with the square root, see sx_least_radicand).  Small grids have
// few warps and wait for the rows one after another: bands of 8 rows there (300^2:
// 5.2 us, 7.8 with 16; 777^2 6.0 and 7.1; 1024^2 8.4 and 7.9).
#define SXA_GRADE_MAX 8

template <typename T>
__global__ void __launch_bounds__(128) sx_amr_tag_grade_kernel(const T* __restrict__ in, unsigned char* __restrict__ tags,
                                                               signed char* __restrict__ actions, int W, int H,
                                                               float least, int p, int mode, int strips, int rows)
{
    constexpr int CHUNK = 4;  // rows loaded together
    const int lane = threadIdx.x & 31;
    const int gw = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int strip = gw % strips, j0 = gw / strips * rows;
    if (j0 >= H) return;  // whole warps
    const int j1 = min(H, j0 + rows);
    const int x = strip * (30 - 2 * p) - p - 1 + lane;
    const bool inside = x >= 0 && x < W, store = inside && lane > p && lane < 31 - p;
    const long long plane = (long long)W * H;
    const T* v = in + plane * blockIdx.z;
    auto value = [&](int j) { return inside && j >= 0 && j < H ? (float)v[(long long)j * W + x] : 0.0f; };
    const unsigned window = (2u << (2 * p)) - 1u;
    unsigned tag_rows = 0u, hit_rows = 0u;  // bit k: k rows ago
    float below = value(j0 - p - 1), c = value(j0 - p), next[CHUNK];
#pragma unroll
    for (int k = 0; k < CHUNK; ++k) next[k] = value(j0 - p + 1 + k);
    for (int jb = j0 - p; jb < j1 + p; jb += CHUNK) {
        float above[CHUNK];
#pragma unroll
        for (int k = 0; k < CHUNK; ++k) above[k] = next[k];
#pragma unroll
        for (int k = 0; k < CHUNK; ++k) next[k] = value(jb + CHUNK + 1 + k);
#pragma unroll
        for (int k = 0; k < CHUNK; ++k) {
            const int j = jb + k;
            const float l = __shfl_up_sync(0xFFFFFFFFu, c, 1), r = __shfl_down_sync(0xFFFFFFFFu, c, 1);
            float gx = 0.0f, gy = 0.0f;
            if (W > 1)
                gx = x == 0 ? __fsub_rn(r, c) : x == W - 1 ? __fsub_rn(c, l) : __fmul_rn(__fsub_rn(r, l), 0.5f);
            if (H > 1)
                gy = j == 0 ? __fsub_rn(above[k], c)
                            : j == H - 1 ? __fsub_rn(c, below) : __fmul_rn(__fsub_rn(above[k], below), 0.5f);
            const bool tag = inside && j >= 0 && j < H && __fmaf_rn(gx, gx, __fmul_rn(gy, gy)) >= least;
            const unsigned row = __ballot_sync(0xFFFFFFFFu, tag);
            const bool hit = lane >= p && ((row >> (lane - p)) & window) != 0u;
            tag_rows = tag_rows << 1 | (tag ? 1u : 0u);
            hit_rows = hit_rows << 1 | (hit ? 1u : 0u);
            if (store && j >= j0 && j < j1) tags[plane * blockIdx.z + (long long)j * W + x] = tag ? 1 : 0;
            const int jo = j - p;  // its window is complete
            if (store && jo >= j0 && jo < j1) {
                const bool on = mode == 1 ? (hit_rows & window) != 0u
                                          : ((hit_rows >> p) & 1u) != 0u || (tag_rows & window) != 0u;
                actions[plane * blockIdx.z + (long long)jo * W + x] = on ? 1 : 0;
            }
            below = c;
            c = above[k];
        }
    }
}

// mode 0: von Neumann (row or column within p), 1: Moore (box), 2: no grading
__global__ void __launch_bounds__(256) sx_amr_grade_full_kernel(const unsigned char* __restrict__ tags,
                                                               signed char* __restrict__ actions, int W, int H, int p,
                                                               int mode)
{
    const long long plane = (long long)W * H;
    const unsigned char* t = tags + plane * blockIdx.z;
    signed char* a = actions + plane * blockIdx.z;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= W) return;
    bool on = t[(long long)y * W + x] != 0;
    if (!on && mode != 2) {
        const int x0 = max(0, x - p), x1 = min(W - 1, x + p);
        const int y0 = max(0, y - p), y1 = min(H - 1, y + p);
        if (mode == 1) {
            for (int yy = y0; yy <= y1 && !on; ++yy)
                for (int xx = x0; xx <= x1; ++xx)
                    if (t[(long long)yy * W + xx]) {
                        on = true;
                        break;
                    }
        } else {
            for (int xx = x0; xx <= x1 && !on; ++xx) on = t[(long long)y * W + xx] != 0;
            for (int yy = y0; yy <= y1 && !on; ++yy) on = t[(long long)yy * W + x] != 0;
        }
    }
    a[(long long)y * W + x] = on ? 1 : 0;
}

static dim3 sxa_grid(int W, int H, int batch) { return dim3((unsigned)((W + 255) / 256), (unsigned)H, (unsigned)batch); }

// Spacings that are powers of two (in the kernel's precision) are passed
// as their exact reciprocals, turning divisions into multiplications.
template <typename T>
static int sxa_pow2_pair(T& dx, T& dy)
{
    int ex, ey;
    const bool p = frexp((double)dx, &ex) == 0.5 && frexp((double)dy, &ey) == 0.5;
    if (!p) return 0;
    const T ix = (T)1 / dx, iy = (T)1 / dy;
    if (!std::isfinite((double)ix) || !std::isfinite((double)iy)) return 0;  // reciprocal out of range
    dx = ix;
    dy = iy;
    return 1;
}

// Kernel instances by the velocity's upwind sides, tested in the kernel's precision.
template <typename T>
static void sxa_upwind_full_go(dim3 g, const T* in, T* out, int W, int H, T a, T b, T dt, T dx, T dy, int p,
                               cudaStream_t stream)
{
    switch ((a >= (T)0 ? 1 : 0) | (b >= (T)0 ? 2 : 0)) {
        case 0: sx_upwind_full_kernel<T, 0><<<g, 256, 0, stream>>>(in, out, W, H, a, b, dt, dx, dy, p); break;
        case 1: sx_upwind_full_kernel<T, 1><<<g, 256, 0, stream>>>(in, out, W, H, a, b, dt, dx, dy, p); break;
        case 2: sx_upwind_full_kernel<T, 2><<<g, 256, 0, stream>>>(in, out, W, H, a, b, dt, dx, dy, p); break;
        default: sx_upwind_full_kernel<T, 3><<<g, 256, 0, stream>>>(in, out, W, H, a, b, dt, dx, dy, p); break;
    }
}

template <typename T>
static void sxa_step_full_go(dim3 g, const T* cin, const T* fin, T* cout, T* fout, const signed char* actions, int W,
                             int H, T a, T b, T dt, T cx, T cy, T fx, T fy, T norm, int pc, int pf,
                             cudaStream_t stream)
{
    switch ((a >= (T)0 ? 1 : 0) | (b >= (T)0 ? 2 : 0)) {
        case 0:
            sx_amr_step_full_kernel<T, 0><<<g, 256, 0, stream>>>(cin, fin, cout, fout, actions, W, H, a, b, dt, cx, cy,
                                                                 fx, fy, norm, pc, pf);
            break;
        case 1:
            sx_amr_step_full_kernel<T, 1><<<g, 256, 0, stream>>>(cin, fin, cout, fout, actions, W, H, a, b, dt, cx, cy,
                                                                 fx, fy, norm, pc, pf);
            break;
        case 2:
            sx_amr_step_full_kernel<T, 2><<<g, 256, 0, stream>>>(cin, fin, cout, fout, actions, W, H, a, b, dt, cx, cy,
                                                                 fx, fy, norm, pc, pf);
            break;
        default:
            sx_amr_step_full_kernel<T, 3><<<g, 256, 0, stream>>>(cin, fin, cout, fout, actions, W, H, a, b, dt, cx, cy,
                                                                 fx, fy, norm, pc, pf);
            break;
    }
}

cudaError_t sx_upwind_full_launch(int dbl, const void* in, void* out, int W, int H, int batch, double a, double b,
                                  double dt, double dx, double dy, cudaStream_t stream)
{
    const dim3 g = sxa_grid(W, H, batch);
    if (dbl) {
        double ddx = dx, ddy = dy;
        const int p = sxa_pow2_pair(ddx, ddy);
        sxa_upwind_full_go<double>(g, (const double*)in, (double*)out, W, H, a, b, dt, ddx, ddy, p, stream);
    } else {
        float fdx = (float)dx, fdy = (float)dy;
        const int p = sxa_pow2_pair(fdx, fdy);
        sxa_upwind_full_go<float>(g, (const float*)in, (float*)out, W, H, (float)a, (float)b, (float)dt, fdx, fdy, p,
                                  stream);
    }
    return cudaGetLastError();
}

cudaError_t sx_amr_sync_full_launch(int dbl, void* coarse, void* fine, const signed char* actions, int W, int H,
                                    int batch, int ratio, cudaStream_t stream)
{
    const dim3 g = sxa_grid(W, H, batch);
    const double norm = 1.0 / ((double)ratio * ratio);
    if (dbl) {
        if (ratio == 2)
            sx_amr_sync_full_kernel<double, 2><<<g, 256, 0, stream>>>((double*)coarse, (double*)fine, actions, W, H, 2,
                                                                      norm);
        else
            sx_amr_sync_full_kernel<double, 0><<<g, 256, 0, stream>>>((double*)coarse, (double*)fine, actions, W, H,
                                                                      ratio, norm);
    } else {
        if (ratio == 2)
            sx_amr_sync_full_kernel<float, 2><<<g, 256, 0, stream>>>((float*)coarse, (float*)fine, actions, W, H, 2,
                                                                     (float)norm);
        else
            sx_amr_sync_full_kernel<float, 0><<<g, 256, 0, stream>>>((float*)coarse, (float*)fine, actions, W, H, ratio,
                                                                     (float)norm);
    }
    return cudaGetLastError();
}

template <typename T>
static void sxa_sync_copy_go(dim3 g, const T* coarse, const T* fine, const signed char* actions, T* coarse_out,
                             T* fine_out, int W, int H, int ratio, T norm, cudaStream_t stream)
{
    const bool pair = ratio == 2 && (((uintptr_t)fine | (uintptr_t)fine_out) & (2 * sizeof(T) - 1)) == 0;
    if (pair)
        sx_amr_sync_copy_kernel<T, true><<<g, 256, 0, stream>>>(coarse, fine, actions, coarse_out, fine_out, W, H, 2,
                                                                norm);
    else
        sx_amr_sync_copy_kernel<T, false><<<g, 256, 0, stream>>>(coarse, fine, actions, coarse_out, fine_out, W, H,
                                                                 ratio, norm);
}

cudaError_t sx_amr_sync_copy_launch(int dbl, const void* coarse, const void* fine, const signed char* actions,
                                    void* coarse_out, void* fine_out, int W, int H, int batch, int ratio,
                                    cudaStream_t stream)
{
    const dim3 g = sxa_grid(W, H, batch);
    const double norm = 1.0 / ((double)ratio * ratio);
    if (dbl)
        sxa_sync_copy_go<double>(g, (const double*)coarse, (const double*)fine, actions, (double*)coarse_out,
                                 (double*)fine_out, W, H, ratio, norm, stream);
    else
        sxa_sync_copy_go<float>(g, (const float*)coarse, (const float*)fine, actions, (float*)coarse_out,
                                (float*)fine_out, W, H, ratio, (float)norm, stream);
    return cudaGetLastError();
}

cudaError_t sx_amr_regrid_full_launch(int dbl, const void* coarse, unsigned char* tags, signed char* actions, int W,
                                      int H, int batch, float threshold, int padding, int mode, cudaStream_t stream)
{
    const int p = padding <= 0 ? 0 : padding;
    const float least = sx_least_radicand(threshold);
    if (p <= SXA_GRADE_MAX) {
        const int strips = (W + 29 - 2 * p) / (30 - 2 * p);
        const int rows = (long long)strips * ((H + 15) / 16) * batch >= 148 * 16 ? 16 : 8;
        const long long warps = (long long)strips * ((H + rows - 1) / rows);
        const dim3 gs((unsigned)((warps + 3) / 4), 1, (unsigned)batch);
        if (dbl)
            sx_amr_tag_grade_kernel<double><<<gs, 128, 0, stream>>>((const double*)coarse, tags, actions, W, H, least,
                                                                    p, mode, strips, rows);
        else
            sx_amr_tag_grade_kernel<float><<<gs, 128, 0, stream>>>((const float*)coarse, tags, actions, W, H, least,
                                                                   p, mode, strips, rows);
        return cudaGetLastError();
    }
    const dim3 g = sxa_grid(W, H, batch);
    if (dbl)
        sx_amr_tag_full_kernel<double><<<g, 256, 0, stream>>>((const double*)coarse, tags, W, H, threshold);
    else
        sx_amr_tag_full_kernel<float><<<g, 256, 0, stream>>>((const float*)coarse, tags, W, H, threshold);
    sx_amr_grade_full_kernel<<<g, 256, 0, stream>>>(tags, actions, W, H, padding, padding <= 0 ? 2 : mode);
    return cudaGetLastError();
}

cudaError_t sx_amr_step_full_launch(int dbl, const void* cin, const void* fin, void* cout, void* fout,
                                    const signed char* actions, int W, int H, int batch, double a, double b, double dt,
                                    double dxc, double dyc, double dxf, double dyf, cudaStream_t stream)
{
    const dim3 g = sxa_grid(W, H, batch);
    if (dbl) {
        double cx = dxc, cy = dyc, fx = dxf, fy = dyf;
        const int pc = sxa_pow2_pair(cx, cy), pf = sxa_pow2_pair(fx, fy);
        sxa_step_full_go<double>(g, (const double*)cin, (const double*)fin, (double*)cout, (double*)fout, actions, W,
                                 H, a, b, dt, cx, cy, fx, fy, 0.25, pc, pf, stream);
    } else {
        float cx = (float)dxc, cy = (float)dyc, fx = (float)dxf, fy = (float)dyf;
        const int pc = sxa_pow2_pair(cx, cy), pf = sxa_pow2_pair(fx, fy);
        sxa_step_full_go<float>(g, (const float*)cin, (const float*)fin, (float*)cout, (float*)fout, actions, W, H,
                                (float)a, (float)b, (float)dt, cx, cy, fx, fy, 0.25f, pc, pf, stream);
    }
    return cudaGetLastError();
}

template <typename T, int DIV>
static void sxa_steps_full_go(int batch, const T* cin, const T* fin, T* cout, T* fout, const signed char* actions,
                              int W, int H, int steps, const SxaStep<T>& S, cudaStream_t stream)
{
    constexpr int CPL = SxaP<T>::CPL, TALL = SXA_WARPS * SXA_ROWS;
    const int halo = (steps + CPL - 1) / CPL * CPL, wide = 32 * CPL - halo, high = TALL - steps;
    const int strips = W <= 32 * CPL ? 1 : (W - halo + wide - 1) / wide;
    const int bands = H <= TALL ? 1 : (H - steps + high - 1) / high;
    const int vec = (W % CPL == 0 && (((uintptr_t)cin | (uintptr_t)fin | (uintptr_t)cout | (uintptr_t)fout) & 15u) == 0 &&
                     ((uintptr_t)actions & 1u) == 0) ? 1 : 0;
    const dim3 g((unsigned)((long long)strips * bands), 1, (unsigned)batch);
    const int sgn = (S.a >= (T)0 ? 1 : 0) | (S.b >= (T)0 ? 2 : 0);
    auto* kernel = sgn == 0   ? sx_amr_steps_full_kernel<T, 0, DIV>
                   : sgn == 1 ? sx_amr_steps_full_kernel<T, 1, DIV>
                   : sgn == 2 ? sx_amr_steps_full_kernel<T, 2, DIV>
                              : sx_amr_steps_full_kernel<T, 3, DIV>;
    kernel<<<g, 32 * SXA_WARPS, 0, stream>>>(cin, fin, cout, fout, actions, W, H, steps, strips, vec, S);
}

template <typename T>
static void sxa_steps_full(int batch, const T* cin, const T* fin, T* cout, T* fout, const signed char* actions, int W,
                           int H, int steps, double a, double b, double dt, double dxc, double dyc, double dxf,
                           double dyf, cudaStream_t stream)
{
    const T d[4] = {(T)dxc, (T)dyc, (T)dxf, (T)dyf};
    SxaSpan<T> w[4];
    bool pow2 = true, known = true;
    for (int q = 0; q < 4; ++q) {
        int e;
        w[q].d = d[q];
        w[q].z = (T)1 / d[q];
        w[q].zz = 1.0 / (double)d[q];
        pow2 = pow2 && frexp((double)d[q], &e) == 0.5 && std::isfinite((double)w[q].z);
        known = known && sx_known_divisor(d[q]);
    }
    const SxaStep<T> S = {(T)a, (T)b, (T)dt, (T)0.25, w[0], w[1], w[2], w[3]};
    if (pow2)
        sxa_steps_full_go<T, SX_BY_POW2>(batch, cin, fin, cout, fout, actions, W, H, steps, S, stream);
    else if (known)
        sxa_steps_full_go<T, SX_BY_CONST>(batch, cin, fin, cout, fout, actions, W, H, steps, S, stream);
    else
        sxa_steps_full_go<T, SX_BY_DIVISION>(batch, cin, fin, cout, fout, actions, W, H, steps, S, stream);
}

cudaError_t sx_amr_steps_full_launch(int dbl, const void* cin, const void* fin, void* cout, void* fout,
                                     const signed char* actions, int W, int H, int batch, int steps, double a, double b,
                                     double dt, double dxc, double dyc, double dxf, double dyf, cudaStream_t stream)
{
    if (dbl)
        sxa_steps_full<double>(batch, (const double*)cin, (const double*)fin, (double*)cout, (double*)fout, actions, W,
                               H, steps, a, b, dt, dxc, dyc, dxf, dyf, stream);
    else
        sxa_steps_full<float>(batch, (const float*)cin, (const float*)fin, (float*)cout, (float*)fout, actions, W, H,
                              steps, a, b, dt, dxc, dyc, dxf, dyf, stream);
    return cudaGetLastError();
}
