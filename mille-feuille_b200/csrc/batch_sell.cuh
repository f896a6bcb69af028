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
// The slices of a (system, window) are stored in the order of SELL_BINS bins:
// dealt longest first, slice t goes to bin bitrev(t mod SELL_BINS).  A warp
// takes a range of consecutive bins, and any power-of-two number of warps up
// to SELL_BINS gets equal shares: bit reversal spreads the bins with one slice
// more evenly over every such split.
//
// A row is summed in the order its entries are stored in: another rounding
// than the matrix's own order (FP32 in the products, FP64 in the refinement).
// Error of solves to 1e-14 against 64 bits, CSR order and this one: 24 systems
// of 1,000-4,000 rows 1.9e-12 and 2.5e-12, 256 of 1,000-32,000 rows 2.44e-12 and
// 2.42e-12.
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
constexpr int SELL_BINS = 512;    // most warps of a cluster

// Bit reversal of a bin number, and the place of dealt slice t (of ns) in
// storage: bins in order, a bin's slices in the order dealt.
__host__ __device__ inline int sell_bitrev(int v)
{
    int r = 0;
    for (int b = 1; b < SELL_BINS; b <<= 1, v >>= 1) r = (r << 1) | (v & 1);
    return r;
}
// slices in bins [0, b): bin c holds ns / BINS, one more when bitrev(c) < ns % BINS
__host__ __device__ inline int sell_before(int ns, int b)
{
    const int full = ns / SELL_BINS, extra = ns % SELL_BINS;
    int m = full * b;
    for (int c = 0; c < b; c++) m += sell_bitrev(c) < extra;
    return m;
}

// Windows of a system of n rows and their width (a multiple of 4 when there
// are several).
__host__ __device__ inline int sell_windows(int n) { return (n + SELL_WIN - 1) / SELL_WIN; }
__host__ __device__ inline int sell_width(int n)
{
    const int w = sell_windows(n);
    return w <= 1 ? n : (((n + w - 1) / w) + 3) & ~3;
}

struct SellView {
    const int *first;      // [windows * (SELL_BINS + 1)] first slice of every bin of each (system, window)
    const int *win0;       // [count] first window of each system
    const int2 *desc;      // per slice (+1 at the end): first quad (of 128 words), quads | long << 31
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
// longest first, and the slices' records and quad counts (long rows marked
// in the top bit), in storage order.
__global__ void __launch_bounds__(32) k_sell_sort(SellBuild a, int windows, const int *__restrict__ len,
                                                  const int *__restrict__ nlong, const int *__restrict__ first,
                                                  int4 *__restrict__ rec, int *__restrict__ quads,
                                                  int *__restrict__ bins)
{
    __shared__ int s_at[SELL_LONG + 1];  // next place of each length (SELL_LONG: all long rows)
    __shared__ int s_bin[SELL_BINS + 1]; // first slice of every bin
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
        for (int b = lane; b <= SELL_BINS; b += 32) {
            s_bin[b] = f0 + sell_before(ns, b);
            bins[w * (SELL_BINS + 1) + b] = s_bin[b];
        }
        __syncwarp();
        // where dealt slice t is stored
        auto place = [&](int t) { return (size_t)(s_bin[sell_bitrev(t % SELL_BINS)] + t / SELL_BINS); };
        // empty lanes of the last slice
        for (int k = 32 * nl + (n - nl) + lane; k < 32 * ns; k += 32) rec[place(ns - 1) * 32 + (k & 31)] = make_int4(-1, 0, 0, 0);
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
                    for (int t = 0; t < 32; t++) rec[place(at) * 32 + t] = v;
                    quads[place(at)] = (int)((unsigned)((m + 127) / 128) | 0x80000000u);
                } else {
                    const int k = at - nl;  // place among the other rows
                    rec[place(nl + (k >> 5)) * 32 + (k & 31)] = v;
                    if ((k & 31) == 0) quads[place(nl + (k >> 5))] = (m + 3) / 4;  // the slice's longest row
                }
            }
            c = __shfl_sync(0xffffffffu, ci, 31);
        }
        __syncwarp();
    }
}

// Quad counts without the long-row mark (to be scanned).
__global__ void __launch_bounds__(SELL_NT) k_sell_counts(int nslices, const int *__restrict__ quads, int *__restrict__ cnt)
{
    for (int s = blockIdx.x * SELL_NT + threadIdx.x; s <= nslices; s += gridDim.x * SELL_NT)
        cnt[s] = s < nslices ? (quads[s] & 0x7fffffff) : 0;
}

// One warp per slice: its descriptor and its entries (the arrays are zeroed
// before).
//
// The order of a row's entries is free, and it decides the shared-memory bank
// conflicts of the gathers: slot j of the 32 rows is one gather of 32 window
// elements, which in storage order falls on random banks (the fullest of 32
// banks then holds ~3.5 of 32 lanes).  So a slice of up to SELL_ORD slots is
// filled slot by slot: in rounds every lane without an entry for the slot
// looks through its remaining entries for one whose bank no lane has taken
// yet, the lowest lane that found a bank keeps it, the others look again;
// lanes left over go through a second pass in which every bank takes one
// more, and then take their next entry.  Rows of ~40 entries: the fullest
// bank holds 2.0 lanes instead of 3.4 (modelled).
// Deterministic: it depends on the matrix alone.
constexpr int SELL_ORD = 96;
constexpr int SELL_ROUNDS = 10;
constexpr int SELL_FNT = 128;

__global__ void __launch_bounds__(SELL_FNT)
k_sell_fill(SellBuild a, int windows, const int *__restrict__ first, const int4 *__restrict__ rec,
            const int *__restrict__ quads, const int *__restrict__ quad0, int nslices, int2 *__restrict__ desc,
            uint32_t *__restrict__ cv, float *__restrict__ v32, uint16_t *__restrict__ c16, double *__restrict__ v64)
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
        const bool lng = quads[s] < 0;
        const int i = rec[(size_t)s * 32 + lane].x;
        const size_t base = (size_t)quad0[s] * 128;
        if (lane == 0) desc[s] = make_int2(quad0[s], quads[s]);
        if (lane == 0 && s == nslices - 1) desc[nslices] = make_int2(quad0[nslices], 0);
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
                            for (int t = j; t < m; t++) {
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
// take L1 space.  Predicated inside the instruction: a branch around a load
// makes the compiler wait for it where the paths meet.
__device__ __forceinline__ void ld_words(uint4 &v, const uint4 *p, bool on)
{
    asm volatile(
        "{ .reg .pred q; setp.ne.u32 q, %5, 0; @q ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4]; }"
        : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)
        : "l"(p), "r"((unsigned)on));
}
__device__ __forceinline__ void ld_words(uint2 &v, const uint2 *p, bool on)
{
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %3, 0; @q ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2]; }"
                 : "+r"(v.x), "+r"(v.y)
                 : "l"(p), "r"((unsigned)on));
}
__device__ __forceinline__ void ld_words(float4 &v, const float4 *p, bool on)
{
    asm volatile(
        "{ .reg .pred q; setp.ne.u32 q, %5, 0; @q ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4]; }"
        : "+f"(v.x), "+f"(v.y), "+f"(v.z), "+f"(v.w)
        : "l"(p), "r"((unsigned)on));
}
__device__ __forceinline__ void ld_words(double2 &v, const double2 *p, bool on)
{
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %3, 0; @q ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2]; }"
                 : "+d"(v.x), "+d"(v.y)
                 : "l"(p), "r"((unsigned)on));
}

__device__ __forceinline__ float half_hi(uint32_t w)
{
    return __half2float(__ushort_as_half((unsigned short)(w >> 16)));
}

// The three kinds of quad: its words as loaded, and its four terms added to
// a sum.  N: quads loaded at once.
struct Quad16 {
    static constexpr int N = 3;
    const uint4 *cv;
    using T = uint4;
    __device__ __forceinline__ Quad16 at(int q) const { return Quad16{cv + (size_t)q * 32}; }
    __device__ __forceinline__ void ld(T &w, int q, bool on) const { ld_words(w, cv + q * 32, on); }
    __device__ __forceinline__ float add(float acc, const T &w, const float *win) const
    {
        acc = fmaf(half_hi(w.x), win[w.x & 0xffffu], acc);
        acc = fmaf(half_hi(w.y), win[w.y & 0xffffu], acc);
        acc = fmaf(half_hi(w.z), win[w.z & 0xffffu], acc);
        return fmaf(half_hi(w.w), win[w.w & 0xffffu], acc);
    }
};

struct Quad32 {
    static constexpr int N = 3;
    const float4 *v32;
    const uint2 *c16;
    struct T {
        float4 v;
        uint2 c;
    };
    __device__ __forceinline__ Quad32 at(int q) const { return Quad32{v32 + (size_t)q * 32, c16 + (size_t)q * 32}; }
    __device__ __forceinline__ void ld(T &w, int q, bool on) const
    {
        ld_words(w.v, v32 + q * 32, on);
        ld_words(w.c, c16 + q * 32, on);
    }
    __device__ __forceinline__ float add(float acc, const T &w, const float *win) const
    {
        acc = fmaf(w.v.x, win[w.c.x & 0xffffu], acc);
        acc = fmaf(w.v.y, win[w.c.x >> 16], acc);
        acc = fmaf(w.v.z, win[w.c.y & 0xffffu], acc);
        return fmaf(w.v.w, win[w.c.y >> 16], acc);
    }
};

struct Quad64 {
    static constexpr int N = 2;
    const double2 *v64;  // two per quad and lane
    const uint2 *c16;
    struct T {
        double2 a, b;
        uint2 c;
    };
    __device__ __forceinline__ Quad64 at(int q) const { return Quad64{v64 + (size_t)q * 64, c16 + (size_t)q * 32}; }
    __device__ __forceinline__ void ld(T &w, int q, bool on) const
    {
        ld_words(w.a, v64 + q * 64, on);
        ld_words(w.b, v64 + q * 64 + 1, on);
        ld_words(w.c, c16 + q * 32, on);
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

// One lane's sum over a slice's quads (the same count for the whole warp),
// N quads loaded at once, the next N after they are added: the latency is
// covered by the SM's 32 warps (3 quads per warp: 48 KB in flight).  More
// quads per warp with fewer warps was slower (16 warps, 12 quads: 357 ms
// against 322 for 256 systems), and so was a ring that reloads each quad as it
// is added (592 ms: the compiler waits for every load).  first() loads a slice's first quads (the
// matrix does not change, so it may run before the barrier that p waits
// for); sum() adds them and loads and adds the rest.
template <class Q>
struct SellSum {
    Q src;
    typename Q::T b[Q::N];

    __device__ __forceinline__ explicit SellSum(const Q &q) : src(q)
    {
#pragma unroll
        for (int u = 0; u < Q::N; u++) b[u] = typename Q::T{};
    }
    __device__ __forceinline__ void first(int q0, int nq)
    {
        const Q at = src.at(q0);
#pragma unroll
        for (int u = 0; u < Q::N; u++) at.ld(b[u], u, u < nq);
    }
    template <class S, class X>
    __device__ __forceinline__ S sum(int q0, int nq, const X *x)
    {
        S acc = 0;
        for (;;) {
            // two quads at a time: eight gathers in flight
#pragma unroll
            for (int u = 0; u + 1 < Q::N; u += 2) {
                if (u + 1 < nq) acc = src.add(src.add(acc, b[u], x), b[u + 1], x);
                else if (u < nq) acc = src.add(acc, b[u], x);
            }
            if (Q::N % 2 && Q::N - 1 < nq) acc = src.add(acc, b[Q::N - 1], x);
            nq -= Q::N;
            if (nq <= 0) return acc;
            q0 += Q::N;
            first(q0, nq);
        }
    }
};

}  // namespace
}  // namespace mf
