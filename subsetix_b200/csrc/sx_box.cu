// Box morphology of one set in one launch: dilation, clipping to a domain,
// grading and erosion over consecutive output rows.
//
// Output row y looks at the source rows y - hy .. y + hy of the set itself, so
// nothing is aligned first: with dense rows the source row's ordinal is
// arithmetic, otherwise one binary search per output row finds the first and the
// others follow.
//   dilate   the merged union of the rows' intervals, widened by w_center (source
//            row y) or w_other (the others) and clipped to [xlo, xhi)
//            (morphology.py:211-319, regrid.py:404-442);
//   erode    the columns of [0, xhi) that no widened gap of those rows covers, a
//            gap being a stretch of [0, xhi) outside the set; rows that the set
//            lacks are one gap, rows outside the domain none
//            (morphology.py:361-386).
//   restrict the merged union of [floor(b / K), ceil(e / K)) over the K sub-rows
//            K y .. K y + K - 1 (multilevel.py:272-362), K = 2, 3 or 4.
// With out_rows only rows with runs are kept (their ids, compacted offsets), which
// is the row list of an unbounded dilation.
//
// The sweep is that of sx_union_kernel (sx_sweep.cu): a warp owns a tile of rows,
// the source intervals under the tile are staged once, several lanes cut a row
// into pieces at begins of its longest view and walk elements instead of
// boundaries.  Chained over separate launches, an erosion was a clip, a
// difference, an alignment, a dilation, a clip and a difference with 75 launches
// and 13 read-backs (1114 us on 3001^2, of which 20 us were the dilation's sweep),
// a dilation an alignment of six launches before its sweep.  Measured (B200): kernel
// 34 us for hy = 3 on 3001 rows of 34 intervals and for hy = 1 on 32,768 such rows,
// 11 us for the grading of 4096 short rows; public calls: erosion 1114 -> 112 us,
// dilation of eight 4096^2 copies 247 -> 120 us, tags and grading on 4096^2
// 1499 -> 206 us.
//
// Contract as for the union sweep (non-decreasing begins and ends in a row, no
// empty interval), and no begin - w or end + w may leave int32; anything else
// raises SXF_CONTRACT and the caller runs the general path.

#include <climits>

#include "sx_tile.cuh"

#define SXB_WARPS 4
#define SXB_HDR_WORDS 4

namespace {

__host__ __device__ inline int slice_words(int cap) { return SXB_HDR_WORDS + 2 * ((cap + 11) & ~3); }

enum { SXB_UNION = 0, SXB_ERODE = 1, SXB_RESTRICT = 2 };

template <int K>
__device__ __forceinline__ int floor_div(int a)
{
    const int q = a / K;
    return a - q * K < 0 ? q - 1 : q;
}

// Source row of view l under output row y.
template <int K, int MODE>
__device__ __forceinline__ int source_row(int y, int l) { return MODE == SXB_RESTRICT ? K * y + l : y + l - K / 2; }

// One view's elements: interval j of the row for dilate, gap j (before interval
// j; the last one after the row's end) for erode.  B, E point at the row.
struct Element {
    int b, e;    // transformed; empty when e <= b
    bool empty, bad;
};

template <int MODE>
__device__ __forceinline__ int elements(int n, bool valid) { return MODE == SXB_ERODE ? (valid ? n + 1 : 0) : n; }

// Transformed begin of element j: the sweep's key, never falling along a row.
// Elements beyond the right edge share the key of the edge, so the element
// before a piece is never one of them.
template <int K, int MODE>
__device__ __forceinline__ int key(const SxBoxArgs& A, const int* B, const int* E, int n, int j, int w)
{
    if (MODE == SXB_ERODE) return (j == 0 ? 0 : min(max(E[j - 1], 0), A.xhi)) - w;
    if (MODE == SXB_RESTRICT) return floor_div<K>(B[j]);
    const int b = B[j];
    return b < A.xlo + w ? A.xlo : min(b - w, A.xhi);  // the launcher keeps xlo + w inside int32
}

template <int K, int MODE>
__device__ __forceinline__ Element element(const SxBoxArgs& A, const int* B, const int* E, int n, int j, int w)
{
    Element r;
    if (MODE == SXB_RESTRICT) {
        r.bad = E[j] <= B[j];
        r.empty = false;
        r.b = floor_div<K>(B[j]);
        r.e = -floor_div<K>(-E[j]);
    } else if (MODE == SXB_ERODE) {
        const int g0 = j == 0 ? 0 : min(max(E[j - 1], 0), A.xhi), g1 = j == n ? A.xhi : min(B[j], A.xhi);
        r.bad = j < n && E[j] <= B[j];
        r.empty = g1 <= g0;
        r.b = g0 - w;
        r.e = g1 + w;
    } else {
        const int b = B[j], e = E[j];
        r.bad = e <= b || b < INT_MIN + w || e > INT_MAX - w;
        r.b = b < A.xlo + w ? A.xlo : min(b - w, A.xhi);
        r.e = e > A.xhi - w ? A.xhi : e + w;
        r.empty = r.e <= r.b;
    }
    return r;
}

// One piece of an output row; see sxu_sweep.  Returns the intervals it emits.
template <int K, int MODE, bool WRITE>
__device__ __forceinline__ int sweep(const SxBoxArgs& A, const int* SB, const int* SE, const int (&lo)[K],
                                     const int (&n)[K], const int (&m)[K], const int (&p0)[K], int khi, long long rank,
                                     int (&pos)[K], int& ce, bool& open, bool& bad)
{
    int h[K], el[K];
    open = false;
    ce = INT_MIN;
#pragma unroll
    for (int l = 0; l < K; ++l) {
        const int w = l == K / 2 ? A.w_center : A.w_other;
        const int *B = SB + lo[l], *E = SE + lo[l];
        pos[l] = p0[l];
        h[l] = pos[l] < m[l] ? key<K, MODE>(A, B, E, n[l], pos[l], w) : INT_MAX;
        el[l] = INT_MIN;
        // the running end: of the last element before the piece that is not empty
        for (int q = pos[l] - 1; q >= 0; --q) {
            const Element x = element<K, MODE>(A, B, E, n[l], q, w);
            if (q == pos[l] - 1) el[l] = x.e;
            if (!x.empty) {
                ce = max(ce, x.e);
                open = true;
                break;
            }
            if (MODE != SXB_ERODE || (q < n[l] && B[q] <= 0)) break;  // clipped away on the left, as is everything before it
        }
    }
    int out = 0;
    while (true) {
        int c = h[0];
#pragma unroll
        for (int l = 1; l < K; ++l) c = min(c, h[l]);
        if (c >= khi) break;
        int reach = INT_MIN;
        bool some = false;
#pragma unroll
        for (int l = 0; l < K; ++l) {
            if (h[l] == c && pos[l] < m[l]) {
                const int w = l == K / 2 ? A.w_center : A.w_other;
                const int *B = SB + lo[l], *E = SE + lo[l];
                const Element x = element<K, MODE>(A, B, E, n[l], pos[l], w);
                if (x.bad || x.e < el[l]) bad = true;
                el[l] = x.e;
                if (!x.empty) {
                    reach = max(reach, x.e);
                    some = true;
                }
                const int q = ++pos[l];
                h[l] = q < m[l] ? key<K, MODE>(A, B, E, n[l], q, w) : INT_MAX;
                if (h[l] < c) bad = true;
            }
        }
        if (!some) continue;
        if (!open || c > ce) {
            const long long o = rank + out;
            if (MODE == SXB_ERODE) {  // the stretch before this gap
                const int from = open ? ce : 0;
                if (c > from) {
                    if (WRITE && o < A.capacity) {
                        A.out_begin[o] = from;
                        A.out_end[o] = c;
                    }
                    ++out;
                }
            } else {
                if (WRITE && o < A.capacity) {
                    A.out_begin[o] = c;
                    if (open) A.out_end[o - 1] = ce;
                }
                ++out;
            }
            open = true;
        }
        ce = max(ce, reach);
    }
    return out;
}

// Look-back over tiles carrying two sums, intervals (32 bits) and kept rows (26
// bits); otherwise sxs_lookback.  Status word: intervals, kind (2 bits), flags (4
// bits), rows.
__device__ __forceinline__ int lookback(const SxSweepState& st, int tile, int intervals, int rows, unsigned& flags,
                                        int& row_base)
{
    const int lane = threadIdx.x & 31;
    const unsigned long long own = ((unsigned long long)(unsigned)rows << 38) |
                                   ((unsigned long long)(flags & 15u) << 34) | (unsigned)intervals;
    row_base = 0;
    if (tile == 0) {
        if (lane == 0) atomicExch(&st.tile_status[0], own | (SX_KIND_PREFIX << 32));
        return 0;
    }
    if (lane == 0) atomicExch(&st.tile_status[tile], own | (SX_KIND_AGG << 32));
    int exclusive = 0, rex = 0;
    unsigned fl = flags;
    bool timed_out = false;
    for (int pos = tile - 1;; pos -= 32) {
        const int t = pos - lane;
        unsigned long long w = SX_KIND_PREFIX << 32;  // before tile 0: an empty prefix
        if (t >= 0) w = sxs_wait_status(&st.tile_status[t], timed_out, SX_LOOKBACK_SPIN_LIMIT);
        const unsigned pm = __ballot_sync(0xFFFFFFFFu, ((w >> 32) & 3ull) == SX_KIND_PREFIX);
        const int stop = pm ? __ffs(pm) - 1 : 32;
        int v = lane <= stop ? (int)(unsigned)(w & 0xFFFFFFFFull) : 0;
        int r = lane <= stop ? (int)(w >> 38) : 0;
        unsigned f = lane <= stop ? (unsigned)(w >> 34) & 15u : 0u;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
            r += __shfl_xor_sync(0xFFFFFFFFu, r, o);
            f |= __shfl_xor_sync(0xFFFFFFFFu, f, o);
        }
        exclusive += v;
        rex += r;
        fl |= f;
        if (pm) break;
    }
    if (__any_sync(0xFFFFFFFFu, timed_out)) fl |= SXF_TIMEOUT;
    if (lane == 0)
        atomicExch(&st.tile_status[tile], ((unsigned long long)(unsigned)(rex + rows) << 38) |
                                              ((unsigned long long)(fl & 15u) << 34) | (SX_KIND_PREFIX << 32) |
                                              (unsigned long long)(unsigned)(exclusive + intervals));
    flags = fl;
    row_base = rex;
    return exclusive;
}

template <int K, int MODE>
__global__ void __launch_bounds__(32 * SXB_WARPS) box_kernel(SxBoxArgs A, SxSweepState st, int tiles, int lg, int cap)
{
    extern __shared__ __align__(16) int sxb_smem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (blockIdx.x * SXB_WARPS + wid >= tiles) return;  // exactly `tiles` warps take tickets
    int* const slice = sxb_smem + wid * slice_words(cap);
    unsigned long long* bar = (unsigned long long*)slice;
    int* const raw = slice + SXB_HDR_WORDS;
    int tile = 0;
    if (lane == 0) {
        tile = (int)atomicAdd(&st.counters[0], 1u);
        sxs_bar_init(bar);
    }
    tile = __shfl_sync(0xFFFFFFFFu, tile, 0);
    const int TR = 32 >> lg;
    const int row = lane >> lg, piece = lane & ((1 << lg) - 1);
    const int i = tile * TR + row;  // output row number
    const int y = A.ybase + i;
    const bool act = i < A.nrows, last = piece == (1 << lg) - 1;
    // source rows y - K/2 .. y + K/2: first interval and count; valid: a row of the domain (erode)
    int lo[K], n[K], m[K];
    int gs = INT_MAX, ge = INT_MIN;
    bool bad = false;
    int at = 0;  // ordinal of the first source row at or after the current one
    if (!A.dense && act) {
        int a = 0, b = A.row_count;
        const int v = source_row<K, MODE>(y, 0);
        while (a < b) {
            const int mid = (a + b) >> 1;
            if (A.rows[mid] < v) a = mid + 1; else b = mid;
        }
        at = a;
    }
#pragma unroll
    for (int l = 0; l < K; ++l) {
        const int v = source_row<K, MODE>(y, l);
        int ord = -1;
        if (act) {
            if (A.dense) {
                const long long o = (long long)v - A.row0;
                if (o >= 0 && o < A.row_count) ord = (int)o;
            } else if (at < A.row_count && A.rows[at] == v) {
                ord = at++;
            }
        }
        const bool valid = act && (MODE != SXB_ERODE || (v >= 0 && v < A.nrows));
        const int a = ord >= 0 && valid ? A.off[ord] : 0, b = ord >= 0 && valid ? A.off[ord + 1] : 0;
        if (b < a) bad = true;  // row offsets must not run backwards
        lo[l] = a;
        n[l] = b > a ? b - a : 0;
        m[l] = elements<MODE>(n[l], valid);
        if (n[l] > 0) {
            gs = min(gs, a);
            ge = max(ge, b);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        gs = min(gs, __shfl_xor_sync(0xFFFFFFFFu, gs, o));
        ge = max(ge, __shfl_xor_sync(0xFFFFFFFFu, ge, o));
    }
    const int ns = gs < ge ? ge - gs : 0;
    unsigned flags = 0u;
    const int *SB = A.begin, *SE = A.end;
    if (ns > 0 && ns <= cap) {
        const int *gb = A.begin + gs, *gq = A.end + gs;
        const uintptr_t b0 = (uintptr_t)gb & ~(uintptr_t)15, e0 = (uintptr_t)gq & ~(uintptr_t)15;
        const unsigned nb = (unsigned)((((uintptr_t)(gb + ns) + 15) & ~(uintptr_t)15) - b0);
        const unsigned ne = (unsigned)((((uintptr_t)(gq + ns) + 15) & ~(uintptr_t)15) - e0);
        int* const second = raw + ((ns + 11) & ~3);  // at most ns + 6 copied words
        if (lane == 0) {
            sxs_bar_expect(bar, nb + ne);
            sxs_bulk_copy(raw, (const void*)b0, nb, bar);
            sxs_bulk_copy(second, (const void*)e0, ne, bar);
        }
        __syncwarp();
        if (__all_sync(0xFFFFFFFFu, sxs_bar_wait(bar))) {
            SB = raw + (((uintptr_t)gb & 15) >> 2);
            SE = second + (((uintptr_t)gq & 15) >> 2);
#pragma unroll
            for (int l = 0; l < K; ++l) lo[l] = n[l] > 0 ? lo[l] - gs : 0;
        } else {
            flags |= SXF_TIMEOUT;
        }
    }
    // this lane's piece: between two begins of the row's longest view
    int p0[K], pos[K], khi = INT_MAX, ce;
    bool open;
#pragma unroll
    for (int l = 0; l < K; ++l) p0[l] = 0;
    if (lg > 0) {
        int big_m = 0, big_lo = 0, big_n = 0, big_w = 0;
#pragma unroll
        for (int l = 0; l < K; ++l)
            if (m[l] > big_m) {
                big_m = m[l];
                big_lo = lo[l];
                big_n = n[l];
                big_w = l == K / 2 ? A.w_center : A.w_other;
            }
        if (big_m > 0) {
            const int *B = SB + big_lo, *E = SE + big_lo;
            if (!last) khi = key<K, MODE>(A, B, E, big_n, (int)(((long long)(piece + 1) * big_m) >> lg), big_w);
            if (piece > 0) {
                const int klo = key<K, MODE>(A, B, E, big_n, (int)(((long long)piece * big_m) >> lg), big_w);
#pragma unroll
                for (int l = 0; l < K; ++l) {
                    const int w = l == K / 2 ? A.w_center : A.w_other;
                    int a = 0, b = m[l];
                    while (a < b) {
                        const int mid = (a + b) >> 1;
                        if (key<K, MODE>(A, SB + lo[l], SE + lo[l], n[l], mid, w) < klo) a = mid + 1; else b = mid;
                    }
                    p0[l] = a;
                }
            }
        }
    }
    int count = sweep<K, MODE, false>(A, SB, SE, lo, n, m, p0, khi, 0, pos, ce, open, bad);
    // the stretch after the last gap; a row of the domain without any gap is whole
    const int from = open ? ce : 0;
    const bool tail = MODE == SXB_ERODE && last && act && from < A.xhi;
    if (tail) ++count;
#pragma unroll
    for (int l = 0; l < K; ++l) {  // consecutive pieces of a row meet, and the last one ends with the row
        const int nxt = __shfl_down_sync(0xFFFFFFFFu, p0[l], 1);
        if (pos[l] != (last ? m[l] : nxt)) bad = true;
    }
    if (__any_sync(0xFFFFFFFFu, bad)) {
        flags |= SXF_CONTRACT;
        count = 0;
    }
    const bool write = !(flags & SXF_CONTRACT);
    int incl = count;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += v;
    }
    const int total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    // rows with runs, numbered through the tile by their last lanes
    const int before = __shfl_sync(0xFFFFFFFFu, incl - count, lane & ~((1 << lg) - 1));
    const bool kept = last && act && incl > before;
    const unsigned km = __ballot_sync(0xFFFFFFFFu, kept);
    int row_base;
    const int base = lookback(st, tile, total, __popc(km), flags, row_base);
    if (write) {
        const long long rank = (long long)base + incl - count;
        const int swept = sweep<K, MODE, true>(A, SB, SE, lo, n, m, p0, khi, rank, pos, ce, open, bad);
        if (MODE == SXB_ERODE) {
            if (tail && rank + swept < A.capacity) {
                A.out_begin[rank + swept] = from;
                A.out_end[rank + swept] = A.xhi;
            }
        } else if (last && open && (long long)base + incl - 1 < A.capacity) {
            A.out_end[(long long)base + incl - 1] = ce;
        }
    }
    if (A.out_rows) {
        if (kept) {
            const int r = row_base + __popc(km & ((1u << lane) - 1u));
            A.out_rows[r] = y;
            A.out_off[r + 1] = base + incl;
        }
    } else if (act && last) {
        A.out_off[i + 1] = base + incl;
    }
    if (tile == 0 && lane == 0) A.out_off[0] = 0;
    if (tile == tiles - 1 && lane == 0) {
        const long long all = (long long)base + total;
        A.result[0] = (int)all;
        A.result[1] = (int)(flags | (all > A.capacity ? SXF_CAPACITY : 0u));
        A.result[2] = row_base + __popc(km);
    }
}

// Lanes per row as in sx_union_shape, whose measurements hold here too.
int box_shape(const SxBoxArgs& A, size_t workspace_bytes)
{
    const long long per_row = A.row_count > 0 ? A.n / A.row_count : 0;
    int lg = 0;
    while (lg < 5 && ((long long)A.nrows << lg) < 148 * 700 && (per_row >> (lg + 1)) >= 2) ++lg;
    while (lg > 0 && sx_sweep_state_bytes((((long long)A.nrows << lg) + 31) / 32) > workspace_bytes) --lg;
    return lg;
}

template <int K, int MODE>
cudaError_t box_go(const SxBoxArgs& A, const SxSweepState& st, int tiles, int lg, cudaStream_t stream)
{
    // staged intervals per tile: 1.5 times the mean of the source rows under it
    const long long src_rows = MODE == SXB_RESTRICT ? (long long)(32 >> lg) * K : (32 >> lg) + K - 1;
    long long cap = (3 * (A.row_count > 0 ? A.n / A.row_count : 0) + 2) * src_rows / 2 + 32;
    if (cap > 6000) cap = 6000;
    const int bytes = SXB_WARPS * slice_words((int)cap) * (int)sizeof(int);
    cudaError_t err = cudaFuncSetAttribute(box_kernel<K, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           SXB_WARPS * slice_words(6000) * (int)sizeof(int));
    if (err != cudaSuccess) return err;
    const int blocks = (tiles + SXB_WARPS - 1) / SXB_WARPS;
    box_kernel<K, MODE><<<blocks, 32 * SXB_WARPS, bytes, stream>>>(A, st, tiles, lg, (int)cap);
    return cudaGetLastError();
}

}  // namespace

// mode 0 and 1: arg is hy; mode 2: arg is the ratio.
cudaError_t sx_box_launch(const SxBoxArgs& A, int mode, int arg, void* workspace, size_t workspace_bytes,
                          cudaStream_t stream)
{
    if (A.nrows <= 0) return cudaSuccess;
    const int lg = box_shape(A, workspace_bytes);
    const long long tiles = (((long long)A.nrows << lg) + 31) / 32;
    if (sx_sweep_state_bytes(tiles) > workspace_bytes) return cudaErrorInvalidValue;
    cudaError_t err = cudaMemsetAsync(workspace, 0, sx_sweep_state_bytes(tiles), stream);
    if (err != cudaSuccess) return err;
    const SxSweepState st = sx_sweep_state(workspace, tiles);
    const int t = (int)tiles;
    if (mode == SXB_RESTRICT) {
        switch (arg) {
            case 2: return box_go<2, SXB_RESTRICT>(A, st, t, lg, stream);
            case 3: return box_go<3, SXB_RESTRICT>(A, st, t, lg, stream);
            case 4: return box_go<4, SXB_RESTRICT>(A, st, t, lg, stream);
            default: return cudaErrorInvalidValue;
        }
    }
    if (mode == SXB_ERODE) {
        switch (arg) {
            case 0: return box_go<1, SXB_ERODE>(A, st, t, lg, stream);
            case 1: return box_go<3, SXB_ERODE>(A, st, t, lg, stream);
            case 2: return box_go<5, SXB_ERODE>(A, st, t, lg, stream);
            case 3: return box_go<7, SXB_ERODE>(A, st, t, lg, stream);
            case 4: return box_go<9, SXB_ERODE>(A, st, t, lg, stream);
            default: return cudaErrorInvalidValue;
        }
    }
    switch (arg) {
        case 0: return box_go<1, SXB_UNION>(A, st, t, lg, stream);
        case 1: return box_go<3, SXB_UNION>(A, st, t, lg, stream);
        case 2: return box_go<5, SXB_UNION>(A, st, t, lg, stream);
        case 3: return box_go<7, SXB_UNION>(A, st, t, lg, stream);
        case 4: return box_go<9, SXB_UNION>(A, st, t, lg, stream);
        default: return cudaErrorInvalidValue;
    }
}
