// tile_build.cu -- CSR -> 16x16 tile-CSR conversion on the GPU.
//
// Produces, bit-exact, the arrays of the reference Tile_create
// (src/csr2block.h:267-422): tiles of a tile-row in ascending column order,
// entries of a tile in CSR order, u8 in-tile row pointers (wrapping mod 256
// as the reference's unsigned char arithmetic does).  Then the derived
// arrays of the reference host drivers: the non-empty-row lists
// (src/main-cg.cu:1231-1288), the blockspmv_cpu row-block schedule
// (src/blockspmv_cpu.h:35-83), and the per-class payloads
// (src/main-cg-mixed.cu:2325-2342).
//
// Design (not the reference's): one warp per tile-row of up to 256 entries.
// It sorts the tile-row's entries by (tile column, CSR position) with a
// bitonic network on 32-bit keys in registers; after one scan of tile counts
// a second pass writes everything the tile-row's tiles have: because tiles
// are ordered by column and entries keep CSR order, an entry's destination is
// simply the tile-row's first CSR offset plus its sorted position, so the
// values, columns and payloads move once, coalesced; row counts and class
// flags of its tiles collect in shared memory, and the row pointers, classes
// and offsets follow from them.  Longer tile-rows (or more than 2^24 tile
// columns) take a CTA each: 64-bit keys in shared memory (global memory
// above SORT_CAP entries), then one pass per array.
//
// All arrays live in one allocation of the library's memory pool, sized by
// bounds known once the tiles are counted, so a build waits for the GPU three
// times and allocates once.  What the row slots (slots.cu) need to be allocated
// without another wait -- their number, the longest row, the farthest tile -- is
// summed up beside it.  Measured on a 96^3 Poisson matrix (6.1 M entries),
// create, one product, destroy: 11.3 -> 0.44 ms (create 6.3 -> 0.40, of which
// kernels 0.25 run one by one and cold; destroy 4.2 -> 0.01).
#include <cuda_fp16.h>

#include <algorithm>
#include <cstring>
#include <type_traits>

#include "mf_internal.h"

namespace mf {
namespace {

constexpr int BUILD_NT = 256;
constexpr int SORT_CAP = 4096;  // entries sorted in shared memory
constexpr unsigned long long KEY_PAD = ~0ull;
constexpr int WARP_CAP = 256;            // entries of a tile-row one warp handles
constexpr int WARP_TILEN = 1 << 24;      // tile columns its 32-bit keys can hold
constexpr int WS_NT = 256;               // threads of the warp sort
constexpr int WF_NT = 128;               // threads of the warp fill

// Ascending bitonic network over P (power of two) keys; only pairs whose
// partner index is above the lower index are compared, so virtual +inf
// padding beyond m never moves.  `keys` is shared or global memory.
__device__ void bitonic_sort(unsigned long long *keys, int m, int P)
{
    for (int k = 2; k <= P; k <<= 1) {
        const int half = k >> 1;
        for (int q = threadIdx.x; q < P / 2; q += blockDim.x) {
            int i = (q / half) * k + (q % half);
            int j = i ^ (k - 1);
            if (j < m) {
                unsigned long long a = keys[i], b = keys[j];
                if (a > b) { keys[i] = b; keys[j] = a; }
            }
        }
        __syncthreads();
        for (int jj = half >> 1; jj > 0; jj >>= 1) {
            for (int q = threadIdx.x; q < P / 2; q += blockDim.x) {
                int i = (q / jj) * (2 * jj) + (q % jj);
                int j = i + jj;
                if (j < m) {
                    unsigned long long a = keys[i], b = keys[j];
                    if (a > b) { keys[i] = b; keys[j] = a; }
                }
            }
            __syncthreads();
        }
    }
}

// Ascending bitonic sort of 32 R keys of a warp, element r * 32 + lane in
// key[r].
template <int R>
__device__ __forceinline__ void warp_sort(unsigned (&key)[R], int lane)
{
#pragma unroll
    for (int k = 2; k <= 32 * R; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                const bool up = ((r * 32 + lane) & k) == 0;
                if (j >= 32) {
                    const int o = r ^ (j / 32);
                    if (o > r) {
                        const unsigned a = min(key[r], key[o]), b = max(key[r], key[o]);
                        key[r] = up ? a : b;
                        key[o] = up ? b : a;
                    }
                } else {
                    const unsigned v = __shfl_xor_sync(0xffffffffu, key[r], j);
                    key[r] = ((lane & j) == 0) == up ? min(key[r], v) : max(key[r], v);
                }
            }
        }
    }
}

template <int R>
__device__ __forceinline__ int sort_tilerow(int m, const int *__restrict__ colidx, unsigned char *__restrict__ perm,
                                            int lane)
{
    unsigned key[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int k = r * 32 + lane;
        key[r] = k < m ? ((unsigned)(colidx[k] >> 4) << 8) | (unsigned)k : 0xffffffffu;
    }
    warp_sort(key, lane);
    int cnt = 0;
    unsigned last = 0xffffffffu;  // tile column before this register's first element
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int k = r * 32 + lane;
        const unsigned col = key[r] >> 8;
        unsigned before = __shfl_up_sync(0xffffffffu, col, 1);
        if (lane == 0) before = last;
        last = __shfl_sync(0xffffffffu, col, 31);
        cnt += __popc(__ballot_sync(0xffffffffu, k < m && (k == 0 || col != before)));
        if (k < m) perm[k] = (unsigned char)(key[r] & 255u);
    }
    return cnt;
}

// Pass 1 for tile-rows of at most `most` entries, a warp each: the entries'
// order (positions within the tile-row) and the number of distinct tile
// columns.
__global__ void __launch_bounds__(WS_NT)
k_sort_warps(int tilem, int rowA, int most, const int *__restrict__ rowptr, const int *__restrict__ colidx,
             unsigned char *__restrict__ perm, int *__restrict__ tilecnt)
{
    const int lane = threadIdx.x & 31, rp0 = rowptr[0];
    for (int bi = blockIdx.x * (WS_NT / 32) + (threadIdx.x >> 5); bi < tilem; bi += gridDim.x * (WS_NT / 32)) {
        const int rs = bi * MF_TILE, re = min(rowA, rs + MF_TILE);
        const int base = rowptr[rs], m = rowptr[re] - base;
        if (m > most) continue;
        const int *c = colidx + base;
        unsigned char *p = perm + (base - rp0);
        int cnt;
        if (m <= 32) cnt = sort_tilerow<1>(m, c, p, lane);
        else if (m <= 64) cnt = sort_tilerow<2>(m, c, p, lane);
        else if (m <= 128) cnt = sort_tilerow<4>(m, c, p, lane);
        else cnt = sort_tilerow<8>(m, c, p, lane);
        if (lane == 0) tilecnt[bi] = cnt;
    }
}

// The bits of a value's flags, and the value's payloads (see k_payloads).
constexpr unsigned FL_INT8 = 1, FL_IN16 = 2, FL_IN32 = 4, FL_FIN16 = 8, FL_NORM16 = 16, FL_ALL = 31;

__device__ __forceinline__ unsigned value_payload(double v, float low, uint16_t &f16, int8_t &i8)
{
    const half h = __float2half_rn(low);
    f16 = __half_as_ushort(h);
    const long long w = (fabs(v) < 2147483648.0) ? (long long)__double2int_rz(v) : (long long)INT_MIN;
    i8 = (int8_t)(unsigned char)(unsigned)(int)w;
    unsigned f = FL_ALL;
    if (!(v == trunc(v) && v >= -128.0 && v <= 127.0)) f &= ~FL_INT8;
    if ((double)(float)v != v) f &= ~FL_IN32;
    if ((double)__half2float(h) != v) f &= ~FL_IN16;
    if (__hisinf(h) || __hisnan(h)) f &= ~FL_FIN16;
    if (v != 0.0 && (f16 & 0x7C00u) == 0) f &= ~FL_NORM16;  // zero or subnormal from a nonzero value
    return f;
}

__device__ __forceinline__ unsigned char flags_class(unsigned f)
{
    return f & FL_INT8 ? MF_CLASS_INT8 : f & FL_IN16 ? MF_CLASS_FP16 : f & FL_IN32 ? MF_CLASS_FP32 : MF_CLASS_FP64;
}

__device__ __forceinline__ unsigned char flags_f16ok(unsigned f)
{
    return (unsigned char)((f & FL_FIN16 ? 1 : 0) | ((f & FL_FIN16) && (f & FL_NORM16) ? 2 : 0));
}

// What pass 2 writes.
struct TileOut {
    int *tile_columnidx, *tile_nnz, *tile_rowidx, *csrptr_offset, *nz_rows;
    unsigned char *blkptr, *blknnznnz, *col, *cls, *f16ok;
    double *val;
    float *low;
    uint16_t *f16;
    int8_t *i8;
    int *err, *class_count, *max_nz;
    int *slot_odd;  // bit 0: a tile's row pointers wrap (its rows are not the CSR's)
};

// Pass 2 for tile-rows of at most `most` entries, a warp each.
__global__ void __launch_bounds__(WF_NT)
k_fill_warps(int tilem, int rowA, int T, int most, const int *__restrict__ rowptr, const int *__restrict__ colidx,
             const double *__restrict__ val, const float *__restrict__ val_low, const unsigned char *__restrict__ perm,
             const int *__restrict__ tile_ptr, TileOut o)
{
    constexpr int NW = WF_NT / 32;
    __shared__ int s_rp[NW][MF_TILE + 1];
    __shared__ unsigned s_cnt[NW][WARP_CAP][MF_TILE / 2];  // entries per tile and row, 16 bits each
    __shared__ unsigned s_flag[NW][WARP_CAP];
    __shared__ int s_class[5], s_max;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x < 5) s_class[threadIdx.x] = 0;
    if (threadIdx.x == 5) s_max = 0;
    __syncthreads();
    const int rp0 = rowptr[0];
    const int last_begin = tile_ptr[tilem - 1], rowlen_last = rowA - (tilem - 1) * MF_TILE;
    if (blockIdx.x == 0 && threadIdx.x == 0) {  // the ends of the arrays with one entry more than tiles
        o.tile_nnz[T] = rowptr[rowA] - rp0;
        o.csrptr_offset[T] = T > last_begin ? last_begin * MF_TILE + (T - last_begin) * rowlen_last : T * MF_TILE;
        o.blknnznnz[T] = 0;
        o.nz_rows[T] = 0;
    }
    for (int bi = blockIdx.x * NW + w; bi < tilem; bi += gridDim.x * NW) {
        const int rs = bi * MF_TILE, rows = min(rowA - rs, MF_TILE);
        const int base = rowptr[rs], m = rowptr[rs + rows] - base;
        if (m > most) continue;
        const int t0 = tile_ptr[bi], nt = tile_ptr[bi + 1] - t0, d0 = base - rp0;
        if (lane <= rows) s_rp[w][lane] = rowptr[rs + lane] - base;
        for (int k = lane; k < nt * (MF_TILE / 2); k += 32) s_cnt[w][k / (MF_TILE / 2)][k % (MF_TILE / 2)] = 0;
        for (int k = lane; k < nt; k += 32) s_flag[w][k] = FL_ALL;
        __syncwarp();
        int carry = -1, last = -1;  // tile ordinal and tile column before this group of 32 entries
        for (int c0 = 0; c0 < m; c0 += 32) {
            const int k = c0 + lane;
            const bool in = k < m;
            const int p = in ? perm[d0 + k] : 0;
            const int col = in ? colidx[base + p] : -16;
            const double v = in ? val[base + p] : 0.0;
            const float low = in ? (val_low ? val_low[base + p] : (float)v) : 0.f;
            int row = 0;  // last r with s_rp[r] <= p
#pragma unroll
            for (int st = 8; st > 0; st >>= 1)
                if (row + st < rows && s_rp[w][row + st] <= p) row += st;
            const int jc = col >> 4;
            int before = __shfl_up_sync(0xffffffffu, jc, 1);
            if (lane == 0) before = last;
            last = __shfl_sync(0xffffffffu, jc, 31);
            const bool head = in && (k == 0 || jc != before);
            const unsigned heads = __ballot_sync(0xffffffffu, head);
            const int ord = carry + __popc(heads & (0xffffffffu >> (31 - lane)));
            carry += __popc(heads);
            if (in) {
                const int dst = d0 + k;
                if (head) {
                    o.tile_columnidx[t0 + ord] = jc;
                    o.tile_nnz[t0 + ord] = dst;
                    o.tile_rowidx[t0 + ord] = bi;
                }
                uint16_t f16;
                int8_t i8;
                const unsigned f = value_payload(v, low, f16, i8);
                o.val[dst] = v;
                o.low[dst] = low;
                o.col[dst] = (unsigned char)(col & 15);
                o.f16[dst] = f16;
                o.i8[dst] = i8;
                atomicAdd(&s_cnt[w][ord][row >> 1], row & 1 ? 0x10000u : 1u);
                if (f != FL_ALL) atomicAnd(&s_flag[w][ord], f);
            }
        }
        __syncwarp();
        for (int k = lane; k < nt; k += 32) {
            const int t = t0 + k;
            // row pointers: the counts' exclusive sums, mod 256 as the
            // reference's unsigned char arithmetic
            unsigned char p8[MF_TILE];
            int at = 0;
#pragma unroll
            for (int r = 0; r < MF_TILE; r += 2) {
                const unsigned c = s_cnt[w][k][r >> 1];
                p8[r] = (unsigned char)at;
                at += (int)(c & 0xffffu);
                p8[r + 1] = (unsigned char)at;
                at += (int)(c >> 16);
            }
            const int nz = at;
            if (nz > 256) atomicExch(o.err, (int)MF_ERR_UNSUPPORTED);
            if (nz == 256 && ((s_cnt[w][k][(rows - 1) >> 1] >> (16 * ((rows - 1) & 1))) & 0xffffu) == 0)
                atomicOr(o.slot_odd, 1);
            const int po = t < last_begin ? t * MF_TILE : last_begin * MF_TILE + (t - last_begin) * rowlen_last;
            int nonempty = 0;
            if (rows == MF_TILE) {
                uint4 q;
                unsigned *qw = reinterpret_cast<unsigned *>(&q);
#pragma unroll
                for (int r = 0; r < MF_TILE; r += 4)
                    qw[r / 4] = p8[r] | (unsigned)p8[r + 1] << 8 | (unsigned)p8[r + 2] << 16 | (unsigned)p8[r + 3] << 24;
                *reinterpret_cast<uint4 *>(o.blkptr + po) = q;
            }
#pragma unroll
            for (int r = 0; r < MF_TILE; r++) {
                if (r < rows) {
                    if (rows != MF_TILE) o.blkptr[po + r] = p8[r];
                    const int stop = (r == rows - 1) ? nz : (int)p8[r + 1 < MF_TILE ? r + 1 : r];
                    if (stop != (int)p8[r]) nonempty++;
                }
            }
            o.csrptr_offset[t] = po;
            o.blknnznnz[t] = (unsigned char)nz;
            o.nz_rows[t] = 1 + nonempty;
            const unsigned f = s_flag[w][k];
            const unsigned char c = flags_class(f);
            o.cls[t] = c;
            o.f16ok[t] = flags_f16ok(f);
            atomicAdd(&s_class[c], 1);
            atomicMax(&s_max, nz);
        }
        __syncwarp();
    }
    __syncthreads();
    if (threadIdx.x < 5 && s_class[threadIdx.x]) atomicAdd(&o.class_count[threadIdx.x], s_class[threadIdx.x]);
    if (threadIdx.x == 5 && s_max) atomicMax(o.max_nz, s_max);
}

// Pass 1 for tile-rows above `most` entries: sort by (tile column, CSR
// position); write the permutation and the number of distinct tile columns.
__global__ void __launch_bounds__(BUILD_NT)
k_sort_tilerows(int tilem, int rowA, int most, const int *__restrict__ rowptr, const int *__restrict__ colidx,
                int *__restrict__ perm, unsigned long long *__restrict__ big_keys, int *__restrict__ tilecnt)
{
    __shared__ unsigned long long s_keys[SORT_CAP];
    __shared__ int s_cnt[BUILD_NT / 32];
    for (int bi = blockIdx.x; bi < tilem; bi += gridDim.x) {
        const int rs = bi * MF_TILE, re = min(rowA, rs + MF_TILE);
        const int base = rowptr[rs], m = rowptr[re] - base;
        if (m <= most) continue;  // a warp has it
        int P = 1;
        while (P < m) P <<= 1;
        unsigned long long *keys = (m <= SORT_CAP) ? s_keys : (big_keys + base);
        if (m <= SORT_CAP) {
            for (int k = threadIdx.x; k < P; k += BUILD_NT)
                s_keys[k] = (k < m) ? (((unsigned long long)(colidx[base + k] >> 4) << 32) | (unsigned)k) : KEY_PAD;
        } else {
            for (int k = threadIdx.x; k < m; k += BUILD_NT)
                keys[k] = ((unsigned long long)(colidx[base + k] >> 4) << 32) | (unsigned)k;
        }
        __syncthreads();
        bitonic_sort(keys, m, P);
        int cnt = 0;
        for (int k = threadIdx.x; k < m; k += BUILD_NT) {
            unsigned long long key = keys[k];
            perm[base + k] = (int)(key & 0xffffffffull);
            if (k == 0 || (keys[k - 1] >> 32) != (key >> 32)) cnt++;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        if ((threadIdx.x & 31) == 0) s_cnt[threadIdx.x >> 5] = cnt;
        __syncthreads();
        if (threadIdx.x == 0) {
            int t = 0;
            for (int w = 0; w < BUILD_NT / 32; w++) t += s_cnt[w];
            tilecnt[bi] = t;
        }
        __syncthreads();
    }
}

// Pass 2 for tile-rows above `most` entries: scatter entries to tile order;
// tile columns, tile offsets, the first position of each non-empty (tile,row)
// run, tile row index.
__global__ void __launch_bounds__(BUILD_NT)
k_fill_tilerows(int tilem, int rowA, int most, int rp0, const int *__restrict__ rowptr, const int *__restrict__ colidx,
                const double *__restrict__ val, const float *__restrict__ val_low, const int *__restrict__ perm,
                const int *__restrict__ tile_ptr, int *__restrict__ tile_columnidx, int *__restrict__ tile_nnz,
                int *__restrict__ tile_rowidx, int *__restrict__ run_start, double *__restrict__ out_val,
                float *__restrict__ out_low, unsigned char *__restrict__ out_col)
{
    __shared__ int s_rp[MF_TILE + 1];
    __shared__ int s_warp[BUILD_NT / 32];
    __shared__ int s_carry;
    for (int bi = blockIdx.x; bi < tilem; bi += gridDim.x) {
        const int rs = bi * MF_TILE, re = min(rowA, rs + MF_TILE), rows = re - rs;
        if (threadIdx.x <= rows) s_rp[threadIdx.x] = rowptr[rs + threadIdx.x];
        if (threadIdx.x == 0) s_carry = 0;
        __syncthreads();
        const int base = s_rp[0], m = s_rp[rows] - base;
        if (m <= most) {  // a warp has it
            __syncthreads();
            continue;
        }
        const int t0 = tile_ptr[bi];
        for (int c0 = 0; c0 < m; c0 += BUILD_NT) {
            const int k = c0 + threadIdx.x;
            int src = 0, jc = -1, row = 0, head = 0, rowhead = 0;
            if (k < m) {
                src = base + perm[base + k];
                jc = colidx[src] >> 4;
                // row of src: last r with s_rp[r] <= src
                int lo = 0, hi = rows - 1;
                while (lo < hi) {
                    int mid = (lo + hi + 1) >> 1;
                    if (s_rp[mid] <= src) lo = mid; else hi = mid - 1;
                }
                row = lo;
                if (k == 0) {
                    head = 1;
                    rowhead = 1;
                } else {
                    int psrc = base + perm[base + k - 1];
                    int pjc = colidx[psrc] >> 4;
                    head = (pjc != jc);
                    if (head) rowhead = 1;
                    else {
                        int plo = 0, phi = rows - 1;
                        while (plo < phi) {
                            int mid = (plo + phi + 1) >> 1;
                            if (s_rp[mid] <= psrc) plo = mid; else phi = mid - 1;
                        }
                        rowhead = (plo != row);
                    }
                }
            }
            // inclusive scan of head flags across the CTA -> tile ordinal
            int x = head;
            const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (lane == 31) s_warp[w] = x;
            __syncthreads();
            int woff = 0, tot = 0;
            for (int i = 0; i < BUILD_NT / 32; i++) {
                if (i < w) woff += s_warp[i];
                tot += s_warp[i];
            }
            const int ord = s_carry + woff + x - 1;  // tile ordinal of this entry
            if (k < m) {
                const int t = t0 + ord;
                const int dst = base - rp0 + k;
                if (head) {
                    tile_columnidx[t] = jc;
                    tile_nnz[t] = dst;
                    tile_rowidx[t] = bi;
                }
                if (rowhead) run_start[(size_t)t * MF_TILE + row] = dst;  // absolute position
                out_val[dst] = val[src];
                out_low[dst] = val_low ? val_low[src] : (float)val[src];
                out_col[dst] = (unsigned char)(colidx[src] & 15);
            }
            __syncthreads();
            if (threadIdx.x == 0) s_carry += tot;
            __syncthreads();
        }
        __syncthreads();
    }
}

// Per tile of a tile-row above `most` entries: in-tile u8 row pointers from
// the first position of each non-empty row (empty rows take the start of the
// next non-empty row, as an exclusive scan of per-row counts does), u8 entry
// count, row-pointer offset, and the non-empty-row count with the reference's
// test (stop != start, src/main-cg.cu:1241-1245).
__global__ void k_tile_finish(int tilem, int rowA, int T, int most, const int *__restrict__ rowptr,
                              const int *__restrict__ tile_ptr, const int *__restrict__ run_start, TileOut o)
{
    const int last_row_tiles_begin = (tilem > 0) ? tile_ptr[tilem - 1] : 0;
    const int rowlen_last = rowA - (tilem - 1) * MF_TILE;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < T; t += gridDim.x * blockDim.x) {
        const int bi = o.tile_rowidx[t];
        if (rowptr[min(rowA, (bi + 1) * MF_TILE)] - rowptr[bi * MF_TILE] <= most) continue;
        const int off = o.tile_nnz[t];
        const int nz = o.tile_nnz[t + 1] - off;
        if (nz > 256) atomicExch(o.err, (int)MF_ERR_UNSUPPORTED);
        const int rowlen = (bi == tilem - 1) ? rowlen_last : MF_TILE;
        if (nz == 256 && run_start[(size_t)t * MF_TILE + rowlen - 1] < 0) atomicOr(o.slot_odd, 1);
        const int po = (t < last_row_tiles_begin) ? t * MF_TILE
                                                   : last_row_tiles_begin * MF_TILE + (t - last_row_tiles_begin) * rowlen_last;
        o.csrptr_offset[t] = po;
        o.blknnznnz[t] = (unsigned char)nz;
        int next = nz, nonempty = 0;
        unsigned char p8[MF_TILE];
        for (int r = rowlen - 1; r >= 0; r--) {
            const int st = run_start[(size_t)t * MF_TILE + r];
            if (st >= 0) next = st - off;
            if (r == 0) next = 0;
            p8[r] = (unsigned char)next;
        }
        for (int r = 0; r < rowlen; r++) {
            o.blkptr[po + r] = p8[r];
            const int stop = (r == rowlen - 1) ? nz : (int)p8[r + 1];
            if (stop != (int)p8[r]) nonempty++;
        }
        o.nz_rows[t] = 1 + nonempty;
    }
}

// Non-empty-row lists (src/main-cg.cu:1262-1288): per tile a sentinel
// (row 0, offset 0) then (row, u8 end offset) for every non-empty row.
__global__ void k_nonzero_lists(int tilem, int rowA, int T, const int *__restrict__ tile_rowidx,
                                const int *__restrict__ tile_nnz, const int *__restrict__ csrptr_offset,
                                const unsigned char *__restrict__ blkptr, const int *__restrict__ nzr,
                                unsigned char *__restrict__ rowid, unsigned char *__restrict__ ptrnew)
{
    const int rowlen_last = rowA - (tilem - 1) * MF_TILE;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < T; t += gridDim.x * blockDim.x) {
        const int rowlen = (tile_rowidx[t] == tilem - 1) ? rowlen_last : MF_TILE;
        const int nz = tile_nnz[t + 1] - tile_nnz[t];
        const int po = csrptr_offset[t];
        int o = nzr[t];
        rowid[o] = 0;
        ptrnew[o] = 0;
        o++;
        for (int r = 0; r < rowlen; r++) {
            int stop = (r == rowlen - 1) ? nz : blkptr[po + r + 1];
            if (stop != blkptr[po + r]) {
                rowid[o] = (unsigned char)r;
                ptrnew[o] = (unsigned char)stop;
                o++;
            }
        }
    }
}

// What the row slots (slots.cu) need: the sum over the strips of their longest
// row, the longest of all, the most tile columns between a tile and its strip;
// bit 1 of odd: a strip has more tiles than a slot's word can name.
struct SlotSizes {
    unsigned long long *total;
    int *kmax, *far, *odd;
};

// Row-block schedule of blockspmv_cpu (src/blockspmv_cpu.h:35-83), and the row
// slots' sizes.
__global__ void __launch_bounds__(BUILD_NT)
k_rbb_count(int tilem, int rowA, const int *__restrict__ rowptr, const int *__restrict__ tile_ptr,
            const int *__restrict__ tile_columnidx, int *__restrict__ cnt, int *__restrict__ block_signal, SlotSizes o)
{
    __shared__ int s_total[BUILD_NT / 32], s_kmax[BUILD_NT / 32], s_far[BUILD_NT / 32];
    int total = 0, kmax = 0, far = 0;  // a thread's few strips: far below 2^31
    for (int bi = blockIdx.x * BUILD_NT + threadIdx.x; bi <= tilem; bi += gridDim.x * BUILD_NT) {
        if (bi == tilem) {
            cnt[bi] = 0;
            block_signal[bi] = 0;
            continue;
        }
        const int t0 = tile_ptr[bi], t1 = tile_ptr[bi + 1], k = t1 - t0;
        int at[MF_TILE + 1], K = 0;  // all in flight together (rows past the last: empty)
#pragma unroll
        for (int r = 0; r <= MF_TILE; r++) at[r] = rowptr[min(bi * MF_TILE + r, rowA)];
        cnt[bi] = (k <= 4) ? 1 : (k + 3) / 4;
        block_signal[bi] = k;
#pragma unroll
        for (int r = 0; r < MF_TILE; r++) K = max(K, at[r + 1] - at[r]);
        total += K;
        kmax = max(kmax, K);
        if (k > 0) far = max(far, max(bi - tile_columnidx[t0], tile_columnidx[t1 - 1] - bi));
        if (k > SLOT_MAX_TILES) atomicOr(o.odd, 2);
    }
    const int w = threadIdx.x >> 5;
    unsigned long long sum = 0;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) total += __shfl_xor_sync(0xffffffffu, total, d);
    kmax = __reduce_max_sync(0xffffffffu, kmax);
    far = __reduce_max_sync(0xffffffffu, far);
    if ((threadIdx.x & 31) == 0) {
        s_total[w] = total;
        s_kmax[w] = kmax;
        s_far[w] = far;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int v = 0; v < BUILD_NT / 32; v++) {
        sum += s_total[v];
        kmax = max(kmax, s_kmax[v]);
        far = max(far, s_far[v]);
    }
    if (sum) atomicAdd(o.total, sum);
    if (kmax > *(volatile int *)o.kmax) atomicMax(o.kmax, kmax);
    if (far > *(volatile int *)o.far) atomicMax(o.far, far);
}

__global__ void k_rbb_fill(int tilem, const int *__restrict__ tile_ptr, const int *__restrict__ off,
                           unsigned *__restrict__ rowidx, int *__restrict__ cs, int *__restrict__ ce)
{
    for (int bi = blockIdx.x * blockDim.x + threadIdx.x; bi < tilem; bi += gridDim.x * blockDim.x) {
        int k = tile_ptr[bi + 1] - tile_ptr[bi];
        int e = off[bi];
        if (k <= 4) {
            rowidx[e] = (unsigned)bi;
            cs[e] = 0;
            ce[e] = 0;
            continue;
        }
        int parts = (k + 3) / 4;
        int len = (k + parts - 1) / parts;
        for (int p = 0; p < parts; p++) {
            rowidx[e + p] = (unsigned)bi | 0x80000000u;
            cs[e + p] = tile_ptr[bi] + p * len;
            ce[e + p] = (p == parts - 1) ? tile_ptr[bi] + k : tile_ptr[bi] + (p + 1) * len;
        }
    }
}

// Static (value-range) class per tile: the smallest format that holds every
// value of the tile exactly.
//   int8 : every value an integer in [-128, 127]
//   fp16 : every value exactly representable in binary16
//   fp32 : every value exactly representable in binary32
//   fp64 : otherwise
// Payloads: fp16 = (half)(float)v, int8 = (int8_t)v (low byte of the
// truncated 32-bit integer), as src/main-cg-mixed.cu:2333-2336 builds them.
// f16ok: bit 0 every FP16 payload value of the tile is finite (|v| within
// binary16's range), the condition for running an inexact tile in FP16;
// bit 1 every nonzero one is also normal (|v| >= 2^-14: no subnormal loss).
// (Here: the tiles of tile-rows above `most` entries.)
__global__ void k_payloads(int T, int rowA, int most, const int *__restrict__ rowptr, TileOut o)
{
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < T; t += gridDim.x * blockDim.x) {
        const int bi = o.tile_rowidx[t];
        if (rowptr[min(rowA, (bi + 1) * MF_TILE)] - rowptr[bi * MF_TILE] <= most) continue;
        const int a = o.tile_nnz[t], b = o.tile_nnz[t + 1];
        unsigned f = FL_ALL;
        for (int k = a; k < b; k++) {
            uint16_t f16;
            int8_t i8;
            f &= value_payload(o.val[k], o.low[k], f16, i8);
            o.f16[k] = f16;
            o.i8[k] = i8;
        }
        o.f16ok[t] = flags_f16ok(f);
        const unsigned char c = flags_class(f);
        o.cls[t] = c;
        atomicAdd(&o.class_count[c], 1);
        atomicMax(o.max_nz, b - a);
    }
}

// Also counts the tile-rows above `most` entries.
__global__ void k_validate(int rowA, int colA, int most, const int *__restrict__ rowptr,
                           const int *__restrict__ colidx, int *__restrict__ err, int *__restrict__ big)
{
    const int rp0 = rowptr[0], rpn = rowptr[rowA];
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < (long long)rowA + (rpn - rp0);
         i += (long long)gridDim.x * blockDim.x) {
        if (i < rowA) {
            if (rowptr[i + 1] < rowptr[i]) atomicExch(err, (int)MF_ERR_INVALID_ARG);
            if (i % MF_TILE == 0 && rowptr[i + min((long long)MF_TILE, rowA - i)] - rowptr[i] > most) atomicAdd(big, 1);
        } else {
            int c = colidx[rp0 + (i - rowA)];
            if (c < 0 || c >= colA) atomicExch(err, (int)MF_ERR_INVALID_ARG);
        }
    }
}

// Strip partition: split tile-rows into `ctas` contiguous ranges of about
// equal cost (entries + 8 per tile + 16 per tile-row).
__global__ void k_strip_cost(int tilem, const int *__restrict__ tile_ptr, const int *__restrict__ tile_nnz,
                             int *__restrict__ cost)
{
    for (int bi = blockIdx.x * blockDim.x + threadIdx.x; bi <= tilem; bi += gridDim.x * blockDim.x) {
        if (bi == tilem) { cost[bi] = 0; continue; }
        int t0 = tile_ptr[bi], t1 = tile_ptr[bi + 1];
        cost[bi] = (tile_nnz[t1] - tile_nnz[t0]) + 8 * (t1 - t0) + 16;
    }
}

__global__ void k_strip_split(int tilem, int ctas, const int *__restrict__ pref, int *__restrict__ part)
{
    const long long total = pref[tilem];
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g <= ctas; g += gridDim.x * blockDim.x) {
        if (g == 0) { part[0] = 0; continue; }
        if (g == ctas) { part[g] = tilem; continue; }
        long long target = total * g / ctas;
        int lo = 0, hi = tilem;  // first bi with pref[bi] >= target
        while (lo < hi) {
            int mid = (lo + hi) >> 1;
            if (pref[mid] < target) lo = mid + 1; else hi = mid;
        }
        part[g] = lo;
    }
}

int grid_for(long long work, int nt)
{
    long long g = (work + nt - 1) / nt;
    if (g < 1) g = 1;
    if (g > 148 * 32) g = 148 * 32;
    return (int)g;
}

}  // namespace

mf_status build_tiles(mf_matrix m, int rowA, int colA, const int *d_rowptr, const int *d_colidx,
                      const double *d_val, const float *d_val_low, cudaStream_t s)
{
    const int tilem = ceil_div(rowA, MF_TILE), tilen = ceil_div(colA, MF_TILE);
    const int most = tilen <= WARP_TILEN ? WARP_CAP : -1;  // entries of the tile-rows that go to warps
    // temporaries and status words, freed on every way out
    struct Temps {
        cudaStream_t s;
        void *p[8];
        int n = 0;
        ~Temps() { for (int k = 0; k < n; k++) cudaFreeAsync(p[k], s); }
        mf_status take(void **q, size_t bytes)
        {
            MF_CUDA(pool_malloc_async(q, bytes, s));
            p[n++] = *q;
            return MF_OK;
        }
    } tmp;
    tmp.s = s;
    // status words: [0] err, [1..5] tiles per class, [6] largest tile, [7] long
    // tile-rows, of the row slots [8, 9] number, [10] longest row, [11] farthest
    // tile, [12] odd
    constexpr int NSTAT = 16;
    int *d_err = nullptr;
    MF_TRY(tmp.take((void **)&d_err, sizeof(int) * NSTAT));
    MF_CUDA(cudaMemsetAsync(d_err, 0, sizeof(int) * NSTAT, s));
    if (rowA > 0) {
        k_validate<<<std::min(grid_for(rowA, 64), 148 * 16), 256, 0, s>>>(rowA, colA, most, d_rowptr, d_colidx, d_err,
                                                                         d_err + 7);
        note_launch();
        MF_CUDA(cudaGetLastError());
    }
    int h[8] = {0}, rp0 = 0, rpn = 0;
    MF_CUDA(cudaMemcpyAsync(&rp0, d_rowptr, sizeof(int), cudaMemcpyDeviceToHost, s));
    MF_CUDA(cudaMemcpyAsync(&rpn, d_rowptr + rowA, sizeof(int), cudaMemcpyDeviceToHost, s));
    MF_CUDA(cudaMemcpyAsync(h, d_err, sizeof(h), cudaMemcpyDeviceToHost, s));
    MF_CUDA(cudaStreamSynchronize(s));
    const int nnz = rpn - rp0;
    if (nnz < 0) { set_last_error("rowptr[rowA] < rowptr[0]"); return MF_ERR_INVALID_ARG; }
    if (h[0]) {
        set_last_error("CSR input invalid: rowptr not monotone or column outside [0, colA)");
        return MF_ERR_INVALID_ARG;
    }
    const bool big = h[7] > 0;

    // pass 1: the entries' order in every tile-row, tiles per tile-row
    unsigned char *d_perm8 = nullptr;
    int *d_perm = nullptr, *d_cnt = nullptr, *d_tp = nullptr;
    unsigned long long *d_big = nullptr;
    MF_TRY(tmp.take((void **)&d_perm8, (size_t)nnz + 16));
    MF_TRY(tmp.take((void **)&d_cnt, sizeof(int) * 2 * (size_t)(tilem + 1)));
    d_tp = d_cnt + tilem + 1;
    if (big) {
        MF_TRY(tmp.take((void **)&d_perm, sizeof(int) * ((size_t)nnz + rp0 + 1)));
        MF_TRY(tmp.take((void **)&d_big, sizeof(unsigned long long) * ((size_t)nnz + rp0 + 1)));
    }
    if (tilem > 0) {
        k_sort_warps<<<grid_for((long long)tilem * 32, WS_NT), WS_NT, 0, s>>>(tilem, rowA, most, d_rowptr, d_colidx,
                                                                               d_perm8, d_cnt);
        note_launch();
        if (big) {
            k_sort_tilerows<<<grid_for(tilem, 1), BUILD_NT, 0, s>>>(tilem, rowA, most, d_rowptr, d_colidx, d_perm, d_big,
                                                                     d_cnt);
            note_launch();
        }
        MF_CUDA(cudaGetLastError());
    }
    MF_CUDA(cudaMemsetAsync(d_cnt + tilem, 0, sizeof(int), s));
    MF_TRY(exclusive_scan_i32(d_cnt, d_tp, tilem + 1, s, nullptr));
    int T = 0, last_begin = 0;
    MF_CUDA(cudaMemcpyAsync(&T, d_tp + tilem, sizeof(int), cudaMemcpyDeviceToHost, s));
    if (tilem > 0) MF_CUDA(cudaMemcpyAsync(&last_begin, d_tp + tilem - 1, sizeof(int), cudaMemcpyDeviceToHost, s));
    MF_CUDA(cudaStreamSynchronize(s));
    // Blockcsr_Ptr size: T*16 minus the short last tile-row
    const int rowlen_last = rowA - (tilem - 1) * MF_TILE;
    const int ptrlen = (tilem > 0) ? last_begin * MF_TILE + (T - last_begin) * rowlen_last : 0;

    // every array: one allocation, each on a 256-byte boundary with 16 bytes of
    // slack for vector loads at its tail.  Not known yet: the non-empty rows
    // (at most one per entry, and a sentinel per tile) and the row blocks (at
    // most one per tile-row and one per four tiles).
    const size_t non_most = (size_t)T + nnz + 1, rbb_most = (size_t)tilem + T / 4 + 1;
    auto arrays = [&](auto take) {
        take(m->d_tile_ptr, tilem + 1);
        take(m->d_tile_columnidx, T);
        take(m->d_tile_nnz, T + 1);
        take(m->d_csrptr_offset, T + 1);
        take(m->d_blknnznnz, T + 1);
        take(m->d_tile_rowidx, T);
        take(m->d_val, nnz);
        take(m->d_val_low, nnz);
        take(m->d_col, nnz);
        take(m->d_cidx, (nnz + 1) / 2);
        take(m->d_nonzero_row_new, T + 1);
        take(m->d_ptr, ptrlen);
        take(m->d_blockrowid_new, non_most);
        take(m->d_blockcsr_ptr_new, non_most);
        take(m->d_block_signal, tilem + 1);
        take(m->d_rbb_rowidx, rbb_most);
        take(m->d_rbb_colstart, rbb_most);
        take(m->d_rbb_colstop, rbb_most);
        take(m->d_f16, nnz);
        take(m->d_i8, nnz);
        take(m->d_class, T);
        take(m->d_f16ok, T);
    };
    size_t total = 0;
    arrays([&](auto &p, size_t n) { total += (sizeof(*p) * (n > 0 ? n : 1) + 16 + 255) / 256 * 256; });
    MF_CUDA(pool_malloc_async(&m->tiles_mem, total, s));
    char *at = (char *)m->tiles_mem;
    arrays([&](auto &p, size_t n) {
        p = (std::remove_reference_t<decltype(p)>)at;
        at += (sizeof(*p) * (n > 0 ? n : 1) + 16 + 255) / 256 * 256;
    });
    MF_CUDA(cudaMemcpyAsync(m->d_tile_ptr, d_tp, sizeof(int) * (tilem + 1), cudaMemcpyDeviceToDevice, s));
    MF_CUDA(cudaMemsetAsync(m->d_cidx, 0, (size_t)(nnz + 1) / 2 + 1, s));
    TileOut o{m->d_tile_columnidx, m->d_tile_nnz, m->d_tile_rowidx, m->d_csrptr_offset, m->d_nonzero_row_new,
              m->d_ptr, m->d_blknnznnz, m->d_col, m->d_class, m->d_f16ok, m->d_val, m->d_val_low, m->d_f16, m->d_i8,
              d_err, d_err + 1, d_err + 6, d_err + 12};
    if (tilem == 0) MF_CUDA(cudaMemsetAsync(m->tiles_mem, 0, total, s));  // no tiles: every array ends at 0
    if (tilem > 0) {
        k_fill_warps<<<grid_for((long long)tilem * 32, WF_NT), WF_NT, 0, s>>>(
            tilem, rowA, T, most, d_rowptr, d_colidx, d_val, d_val_low, d_perm8, m->d_tile_ptr, o);
        note_launch();
        if (big) {
            int *d_run = nullptr;
            MF_TRY(tmp.take((void **)&d_run, sizeof(int) * (size_t)T * MF_TILE + 16));
            MF_CUDA(cudaMemsetAsync(d_run, 0xff, sizeof(int) * (size_t)T * MF_TILE + 16, s));
            k_fill_tilerows<<<grid_for(tilem, 1), BUILD_NT, 0, s>>>(
                tilem, rowA, most, rp0, d_rowptr, d_colidx, d_val, d_val_low, d_perm, m->d_tile_ptr, m->d_tile_columnidx,
                m->d_tile_nnz, m->d_tile_rowidx, d_run, m->d_val, m->d_val_low, m->d_col);
            k_tile_finish<<<grid_for(T, 256), 256, 0, s>>>(tilem, rowA, T, most, d_rowptr, m->d_tile_ptr, d_run, o);
            k_payloads<<<grid_for(T, 256), 256, 0, s>>>(T, rowA, most, d_rowptr, o);
            note_launch(3);
        }
    }
    MF_CUDA(cudaGetLastError());

    // non-empty-row lists
    MF_CUDA(cudaMemsetAsync(m->d_blockrowid_new, 0, non_most, s));
    MF_CUDA(cudaMemsetAsync(m->d_blockcsr_ptr_new, 0, non_most, s));
    MF_TRY(exclusive_scan_i32(m->d_nonzero_row_new, m->d_nonzero_row_new, T + 1, s, nullptr));
    if (T > 0) {
        k_nonzero_lists<<<grid_for(T, 256), 256, 0, s>>>(tilem, rowA, T, m->d_tile_rowidx, m->d_tile_nnz,
                                                         m->d_csrptr_offset, m->d_ptr, m->d_nonzero_row_new,
                                                         m->d_blockrowid_new, m->d_blockcsr_ptr_new);
        note_launch();
        MF_CUDA(cudaGetLastError());
    }

    // row-block schedule (d_cnt is free again)
    const SlotSizes slot_sizes{(unsigned long long *)(d_err + 8), d_err + 10, d_err + 11, d_err + 12};
    k_rbb_count<<<grid_for(tilem + 1, BUILD_NT), BUILD_NT, 0, s>>>(tilem, rowA, d_rowptr, m->d_tile_ptr,
                                                                    m->d_tile_columnidx, d_cnt, m->d_block_signal,
                                                                    slot_sizes);
    note_launch();
    MF_TRY(exclusive_scan_i32(d_cnt, d_cnt, tilem + 1, s, nullptr));
    if (tilem > 0) {
        k_rbb_fill<<<grid_for(tilem, 256), 256, 0, s>>>(tilem, m->d_tile_ptr, d_cnt, m->d_rbb_rowidx, m->d_rbb_colstart,
                                                        m->d_rbb_colstop);
        note_launch();
    }
    MF_CUDA(cudaGetLastError());

    int cnt_non = 0, rbb = 0, host_counts[NSTAT] = {0};
    MF_CUDA(cudaMemcpyAsync(&cnt_non, m->d_nonzero_row_new + T, sizeof(int), cudaMemcpyDeviceToHost, s));
    MF_CUDA(cudaMemcpyAsync(&rbb, d_cnt + tilem, sizeof(int), cudaMemcpyDeviceToHost, s));
    MF_CUDA(cudaMemcpyAsync(host_counts, d_err, sizeof(host_counts), cudaMemcpyDeviceToHost, s));
    MF_CUDA(cudaStreamSynchronize(s));
    if (host_counts[0]) {
        set_last_error("a 16x16 tile holds more than 256 entries (duplicate entries); u8 row pointers cannot describe it");
        return MF_ERR_UNSUPPORTED;
    }

    m->v.rows = rowA;
    m->v.cols = colA;
    m->v.nnz = nnz;
    m->v.tilem = tilem;
    m->v.tilen = tilen;
    m->v.tilenum = T;
    m->v.csrptrlen = ptrlen;
    m->v.rows_multiple_of_16 = (rowA % MF_TILE) == 0;
    m->v.tile_ptr = m->d_tile_ptr;
    m->v.tile_columnidx = m->d_tile_columnidx;
    m->v.tile_nnz = m->d_tile_nnz;
    m->v.csrptr_offset = m->d_csrptr_offset;
    m->v.val = m->d_val;
    m->v.val_low = m->d_val_low;
    m->v.col = m->d_col;
    m->v.ptr = m->d_ptr;
    m->v.val_f16 = m->d_f16;
    m->v.val_i8 = m->d_i8;
    m->v.tile_class = m->d_class;
    for (int c = 0; c < 5; c++) m->class_tiles[c] = host_counts[1 + c];
    m->max_tile_nnz = host_counts[6];
    m->nonzero_rows = cnt_non;
    m->last_tile_begin = last_begin;
    m->rowblkblock = rbb;
    m->device_bytes = total;
    unsigned long long slots = 0;
    memcpy(&slots, host_counts + 8, sizeof(slots));
    if (!(host_counts[12] & 1))  // else measured when the slots are built
        set_slot_sizes(m, host_counts[12] & 2 ? -1 : (long long)slots, host_counts[11], host_counts[10]);
    return MF_OK;
}

mf_status strip_partition(mf_matrix m, int ctas, cudaStream_t s)
{
    if (m->part_ctas == ctas && m->d_part) return MF_OK;
    handle_release(m->d_part);
    m->part_ctas = 0;
    const int tilem = m->v.tilem;
    MF_CUDA(handle_malloc(&m->d_part, sizeof(int) * (ctas + 1)));
    int *d_cost = nullptr;
    MF_CUDA(pool_malloc_async(&d_cost, sizeof(int) * (tilem + 1), s));
    k_strip_cost<<<grid_for(tilem + 1, 256), 256, 0, s>>>(tilem, m->d_tile_ptr, m->d_tile_nnz, d_cost);
    note_launch();
    MF_CUDA(cudaGetLastError());
    MF_TRY(exclusive_scan_i32(d_cost, d_cost, tilem + 1, s, nullptr));
    k_strip_split<<<grid_for(ctas + 1, 256), 256, 0, s>>>(tilem, ctas, d_cost, m->d_part);
    note_launch();
    MF_CUDA(cudaGetLastError());
    cudaFreeAsync(d_cost, s);
    m->part_ctas = ctas;
    return MF_OK;
}

}  // namespace mf
