// batch_sell.cuh -- the execution layout of the mixed-precision batched CG:
// sorted slices of 32 rows, slot by slot (included by batched.cu).
//
// A system's columns are cut into windows of at most SELL_WIN columns (one
// window for n <= SELL_WIN), the slice of p a CTA keeps in shared memory.
// Per (system, window) the rows are sorted by their number of off-diagonal
// entries in the window, longest first (equal lengths in row order), and
// taken 32 at a time: one slice is one warp's work, lane l owns the l-th row
// of the slice and adds its entries one after another.  Entries are stored four
// slots at a time ("quads"): lane l's entries 4j .. 4j+3 are 16 consecutive
// bytes, a warp reads 512 consecutive bytes per quad, and no two lanes share
// a row, so a row sum needs neither shuffles nor a second pass.  Sorting
// keeps the padding small (rows of one slice differ by a few entries).  Rows
// of SELL_LONG entries or more are slices of their own, their entries dealt
// to the 32 lanes in turn.
//
// Four arrays share that geometry: cv (FP16 value bits << 16 | column in the
// window), v32 and v64 (FP32 and FP64 values) and c16 (column in the window).  Diagonal
// entries are left out: a row's FP32 diagonal and FP16 scale are part of its
// lane record {row, chunk, scale, diagonal}.
#pragma once
#include <cuda_fp16.h>

#include <cstdint>

namespace mf {
namespace {

constexpr int SELL_WIN = 55296;   // columns of a window: 216 KB of FP32 p beside the policy network's weights
constexpr int SELL_LONG = 256;    // rows from this length on are spread over a warp
constexpr int SELL_NT = 256;

// Windows of a system of n rows and their width (a multiple of 4 when there
// are several).
__host__ __device__ inline int sell_windows(int n) { return (n + SELL_WIN - 1) / SELL_WIN; }
__host__ __device__ inline int sell_width(int n)
{
    const int w = sell_windows(n);
    return w <= 1 ? n : (((n + w - 1) / w) + 3) & ~3;
}

struct SellView {
    const int *first;      // [windows + 1] first slice of each (system, window)
    const int *win0;       // [count] first window of each system
    const int2 *desc;      // per slice: first quad (of 128 words), quads | long << 31
    const int4 *rec;       // per slice and lane: row (-1 none), chunk, FP16 scale, FP32 diagonal
    const uint4 *cv;       // per quad and lane
    const float4 *v32;
    const uint2 *c16;
    const double2 *v64;    // two per quad and lane
    const double *diag64;  // per row
};

// What the build kernels read: the panel storage (columns of panel k at
// k * pw) and where each system's windows and rows are.
struct SellBuild {
    int count, pw;
    const int *n, *pan0, *win0;
    const long long *row0, *prow0, *pent0;
    const long long *len0;  // [windows] first of the window's n row lengths
    const int *sc, *crow;
    const int *prow;
    const uint16_t *col;
    const double *val;
    const __half *val16;
    const float *rscale, *diag32;
};

// The system of window w (win0 ascending).
__device__ __forceinline__ int sell_system(const SellBuild &a, int w)
{
    int lo = 0, hi = a.count - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (a.win0[mid] <= w) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// f(entry index in the panel arrays, column) over row i's entries with a
// column in [c0, c1), the diagonal left out, in panel and entry order
template <class F>
__device__ __forceinline__ void sell_entries(const SellBuild &a, int sys, int n, int i, int c0, int c1, F f)
{
    const int np = (n + a.pw - 1) / a.pw;
    for (int k = c0 / a.pw; k < np && k * a.pw < c1; k++) {
        const long long rpb = a.prow0[a.pan0[sys] + k], eb = a.pent0[a.pan0[sys] + k];
        for (int e = a.prow[rpb + i]; e < a.prow[rpb + i + 1]; e++) {
            const int c = (int)a.col[eb + e] + k * a.pw;
            if (c >= c0 && c < c1 && c != i) f(eb + e, c);
        }
    }
}

// Row lengths per window (grid y: blocks of one window).
__global__ void __launch_bounds__(SELL_NT) k_sell_lengths(SellBuild a, int windows, int *__restrict__ len)
{
    for (int w = blockIdx.x; w < windows; w += gridDim.x) {
        const int sys = sell_system(a, w), n = a.n[sys], W = sell_width(n);
        const int c0 = (w - a.win0[sys]) * W, c1 = min(n, c0 + W);
        int *l = len + a.len0[w];
        for (int i = blockIdx.y * SELL_NT + threadIdx.x; i < n; i += gridDim.y * SELL_NT) {
            int m = 0;
            sell_entries(a, sys, n, i, c0, c1, [&](long long, int) { m++; });
            l[i] = m;
        }
    }
}

// Per window (one block): the rows' histogram by length; slices[w] = long
// rows + ceil(the others / 32).
__global__ void __launch_bounds__(SELL_NT) k_sell_slices(SellBuild a, int windows, const int *__restrict__ len,
                                                         int *__restrict__ slices, int *__restrict__ nlong)
{
    __shared__ int s_long;
    for (int w = blockIdx.x; w < windows; w += gridDim.x) {
        const int n = a.n[sell_system(a, w)];
        const int *l = len + a.len0[w];
        if (threadIdx.x == 0) s_long = 0;
        __syncthreads();
        int m = 0;
        for (int i = threadIdx.x; i < n; i += SELL_NT) m += l[i] >= SELL_LONG;
        if (m) atomicAdd(&s_long, m);
        __syncthreads();
        if (threadIdx.x == 0) {
            nlong[w] = s_long;
            slices[w] = s_long + (n - s_long + 31) / 32;
        }
        __syncthreads();
    }
}

// Per window (one warp): a stable counting sort of the rows by length,
// longest first, and the slices' records and quad counts.
__global__ void __launch_bounds__(32) k_sell_sort(SellBuild a, int windows, const int *__restrict__ len,
                                                  const int *__restrict__ nlong, const int *__restrict__ first,
                                                  int4 *__restrict__ rec, int *__restrict__ quads)
{
    __shared__ int s_at[SELL_LONG + 1];  // next place of each length (SELL_LONG: all long rows)
    const int lane = threadIdx.x;
    for (int w = blockIdx.x; w < windows; w += gridDim.x) {
        const int sys = sell_system(a, w), n = a.n[sys];
        const long long r0 = a.row0[sys];
        const int *l = len + a.len0[w];
        const int f0 = first[w], nl = nlong[w], ns = first[w + 1] - f0;
        for (int k = lane; k <= SELL_LONG; k += 32) s_at[k] = 0;
        __syncwarp();
        for (int i = lane; i < n; i += 32) atomicAdd(&s_at[min(l[i], SELL_LONG)], 1);
        __syncwarp();
        if (lane == 0) {
            int at = 0;
            for (int k = SELL_LONG; k >= 0; k--) {
                const int c = s_at[k];
                s_at[k] = at;
                at += c;
            }
        }
        // empty lanes of the last slice, and its width
        for (int k = lane; k < 32 * ns; k += 32)
            if (k >= 32 * nl + (n - nl)) rec[(size_t)f0 * 32 + k] = make_int4(-1, 0, 0, 0);
        __syncwarp();
        int c = a.sc[sys];  // chunk of the current rows (rows ascend)
        for (int i0 = 0; i0 < n; i0 += 32) {
            const int i = i0 + lane;
            const bool in = i < n;
            const int m = in ? l[i] : -1, key = in ? min(m, SELL_LONG) : SELL_LONG + 1;
            const unsigned same = __match_any_sync(0xffffffffu, key);
            const int before = __popc(same & ((1u << lane) - 1u));
            int base = 0;
            if (in) base = s_at[key];
            __syncwarp();
            if (in && before == 0) s_at[key] = base + __popc(same);
            __syncwarp();
            int ci = c;
            if (in)
                while (a.crow[ci + 1 + sys] <= i) ci++;
            if (in) {
                const int at = base + before;
                const int4 v = make_int4(i, ci, __float_as_int(a.rscale[r0 + i]), __float_as_int(a.diag32[r0 + i]));
                if (key == SELL_LONG) {
                    for (int t = 0; t < 32; t++) rec[((size_t)f0 + at) * 32 + t] = v;
                    quads[f0 + at] = (m + 127) / 128;
                } else {
                    const int k = at - nl;  // place among the other rows
                    rec[((size_t)f0 + nl) * 32 + k] = v;
                    if ((k & 31) == 0) quads[f0 + nl + (k >> 5)] = (m + 3) / 4;  // the slice's longest row
                }
            }
            c = __shfl_sync(0xffffffffu, ci, 31);
        }
        __syncwarp();
    }
}

// One warp per slice: its descriptor and its entries (the arrays are zeroed
// before).
//
// The order of a row's entries is free, and it decides the shared-memory bank
// conflicts of the gathers: slot j of the 32 rows is one gather of 32 window
// elements, which in storage order falls on random banks (the fullest of 32
// banks then holds ~3.5 of 32 lanes).  So a slice of up to SELL_ORD slots is
// filled slot by slot: in rounds every lane without an entry for the slot
// looks through its remaining entries (at most SELL_SCAN of them) for one
// whose bank no lane has taken yet, the lowest lane that found a bank keeps
// it, the others look again; a lane that finds none takes its next entry.
// Deterministic: it depends on the matrix alone.
constexpr int SELL_ORD = 96;
constexpr int SELL_SCAN = 24;
constexpr int SELL_ROUNDS = 10;
constexpr int SELL_FNT = 128;

__global__ void __launch_bounds__(SELL_FNT)
k_sell_fill(SellBuild a, int windows, const int *__restrict__ first, const int *__restrict__ nlong,
            const int4 *__restrict__ rec, const int *__restrict__ quads, const int *__restrict__ quad0, int nslices,
            int2 *__restrict__ desc, uint32_t *__restrict__ cv, float *__restrict__ v32, uint16_t *__restrict__ c16,
            double *__restrict__ v64)
{
    // per warp and lane: banks of the entries still to place, their numbers,
    // and the slot of every entry
    __shared__ unsigned char s_bank[SELL_FNT / 32][SELL_ORD][32], s_id[SELL_FNT / 32][SELL_ORD][32],
        s_slot[SELL_FNT / 32][SELL_ORD][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    auto bank = s_bank[wid];
    auto id = s_id[wid];
    auto slot = s_slot[wid];
    for (int s = blockIdx.x * (SELL_FNT / 32) + wid; s < nslices; s += gridDim.x * (SELL_FNT / 32)) {
        int lo = 0, hi = windows - 1;  // the slice's window
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (first[mid] <= s) lo = mid;
            else hi = mid - 1;
        }
        const int w = lo, sys = sell_system(a, w), n = a.n[sys], W = sell_width(n);
        const int c0 = (w - a.win0[sys]) * W, c1 = min(n, c0 + W);
        const bool lng = s - first[w] < nlong[w];
        const int i = rec[(size_t)s * 32 + lane].x;
        const size_t base = (size_t)quad0[s] * 128;
        if (lane == 0) desc[s] = make_int2(quad0[s], quads[s] | (lng ? (int)0x80000000 : 0));
        const bool ordered = !lng && quads[s] * 4 <= SELL_ORD;
        if (ordered) {
            int m = 0;
            if (i >= 0)
                sell_entries(a, sys, n, i, c0, c1, [&](long long, int c) {
                    bank[m][lane] = (unsigned char)((c - c0) & 31);
                    id[m][lane] = (unsigned char)m;
                    m++;
                });
            const int most = __reduce_max_sync(0xffffffffu, m);
            for (int j = 0; j < most; j++) {
                int pick = -1;  // place of the chosen entry among the remaining ones
                for (int pass = 0; pass < 2; pass++) {  // the second pass lets every bank take one lane more
                    unsigned taken = 0;
                    bool open = j < m && pick < 0;  // this lane has no entry for the slot yet
                    for (int round = 0; round < SELL_ROUNDS && __any_sync(0xffffffffu, open); round++) {
                        int k = -1, b = 32 + lane;  // a bank of its own for lanes without a candidate
                        if (open) {
                            const int end = min(m, j + SELL_SCAN);
                            for (int t = j; t < end; t++) {
                                const int bt = bank[t][lane];
                                if (!((taken >> bt) & 1u)) {
                                    k = t;
                                    b = bt;
                                    break;
                                }
                            }
                        }
                        const unsigned same = __match_any_sync(0xffffffffu, b);
                        const bool won = k >= 0 && (same & ((1u << lane) - 1u)) == 0;
                        if (won) pick = k;
                        if (won || k < 0) open = false;
                        taken |= __reduce_or_sync(0xffffffffu, won ? 1u << b : 0u);
                    }
                }
                if (j < m) {
                    if (pick < 0) pick = j;
                    const unsigned char e = id[pick][lane];
                    slot[e][lane] = (unsigned char)j;
                    id[pick][lane] = id[j][lane];
                    bank[pick][lane] = bank[j][lane];
                }
            }
            __syncwarp();
        }
        if (i >= 0) {
            int j = 0;
            sell_entries(a, sys, n, i, c0, c1, [&](long long e, int c) {
                // long rows: entry j belongs to lane j % 32 (every lane walks
                // the row and keeps its own), else all entries are this lane's
                const int mine = lng ? ((j & 31) == lane ? j >> 5 : -1) : ordered ? (int)slot[j][lane] : j;
                if (mine >= 0) {
                    const size_t at = base + (size_t)(mine >> 2) * 128 + lane * 4 + (mine & 3);
                    cv[at] = ((uint32_t)__half_as_ushort(a.val16[e]) << 16) | (uint32_t)(c - c0);
                    v64[at] = a.val[e];
                    v32[at] = (float)a.val[e];
                    c16[at] = (uint16_t)(c - c0);
                }
                j++;
            });
        }
        __syncwarp();
    }
}

// Read-only matrix words: each is used once per product, so they do not
// take L1 space.
__device__ __forceinline__ uint4 ld_words(const uint4 *p)
{
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ uint2 ld_words(const uint2 *p)
{
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 ld_words(const float4 *p)
{
    const uint4 v = ld_words((const uint4 *)p);
    return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}

__device__ __forceinline__ double2 ld_words(const double2 *p)
{
    double2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}

__device__ __forceinline__ float half_hi(uint32_t w)
{
    return __half2float(__ushort_as_half((unsigned short)(w >> 16)));
}

// The three kinds of quad: its words as loaded, and its four terms added to
// a sum.  G: quads of a group; a group is loaded while the one before it is
// added (two groups of registers).
struct Quad16 {
    static constexpr int G = 4;
    const uint4 *cv;
    using T = uint4;
    __device__ __forceinline__ T ld(int q) const { return ld_words(cv + q * 32); }
    __device__ __forceinline__ float add(float acc, const T &w, const float *win) const
    {
        acc = fmaf(half_hi(w.x), win[w.x & 0xffffu], acc);
        acc = fmaf(half_hi(w.y), win[w.y & 0xffffu], acc);
        acc = fmaf(half_hi(w.z), win[w.z & 0xffffu], acc);
        return fmaf(half_hi(w.w), win[w.w & 0xffffu], acc);
    }
};

struct Quad32 {
    static constexpr int G = 2;
    const float4 *v32;
    const uint2 *c16;
    struct T {
        float4 v;
        uint2 c;
    };
    __device__ __forceinline__ T ld(int q) const { return T{ld_words(v32 + q * 32), ld_words(c16 + q * 32)}; }
    __device__ __forceinline__ float add(float acc, const T &w, const float *win) const
    {
        acc = fmaf(w.v.x, win[w.c.x & 0xffffu], acc);
        acc = fmaf(w.v.y, win[w.c.x >> 16], acc);
        acc = fmaf(w.v.z, win[w.c.y & 0xffffu], acc);
        return fmaf(w.v.w, win[w.c.y >> 16], acc);
    }
};

struct Quad64 {
    static constexpr int G = 2;
    const double2 *v64;  // two per quad and lane
    const uint2 *c16;
    struct T {
        double2 a, b;
        uint2 c;
    };
    __device__ __forceinline__ T ld(int q) const
    {
        return T{ld_words(v64 + q * 64), ld_words(v64 + q * 64 + 1), ld_words(c16 + q * 32)};
    }
    __device__ __forceinline__ double add(double acc, const T &w, const double *x) const
    {
        const double x0 = x[w.c.x & 0xffffu], x1 = x[w.c.x >> 16], x2 = x[w.c.y & 0xffffu], x3 = x[w.c.y >> 16];
        acc = fma(w.a.x, x0, acc);
        acc = fma(w.a.y, x1, acc);
        acc = fma(w.b.x, x2, acc);
        return fma(w.b.y, x3, acc);
    }
};

// One lane's sum over nq quads (the same count for the whole warp): the
// quads beyond a whole number of groups first, then group by group.
template <class Q, class S, class X>
__device__ __forceinline__ S sell_dot(const Q &src, int nq, const X *x)
{
    constexpr int G = Q::G;
    const int rem = nq % G, nf = nq / G;
    typename Q::T t[G], a[G];
    S acc = 0;
#pragma unroll
    for (int u = 0; u < G - 1; u++)
        if (u < rem) t[u] = src.ld(u);
    if (nf > 0)
#pragma unroll
        for (int u = 0; u < G; u++) a[u] = src.ld(rem + u);
#pragma unroll
    for (int u = 0; u < G - 1; u++)
        if (u < rem) acc = src.add(acc, t[u], x);
    if (nf == 0) return acc;
    int q = rem + G;
#pragma unroll 2
    for (int g = 1; g < nf; g++, q += G) {
        typename Q::T b[G];
#pragma unroll
        for (int u = 0; u < G; u++) b[u] = src.ld(q + u);
#pragma unroll
        for (int u = 0; u < G; u++) acc = src.add(acc, a[u], x);
#pragma unroll
        for (int u = 0; u < G; u++) a[u] = b[u];
    }
#pragma unroll
    for (int u = 0; u < G; u++) acc = src.add(acc, a[u], x);
    return acc;
}

}  // namespace
}  // namespace mf
