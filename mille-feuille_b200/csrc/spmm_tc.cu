// spmm_tc.cu -- Y = A X for k <= 16 columns with the dense tiles on the
// tensor cores: FP16 inputs, FP32 accumulation (mf_spmm_f16).
//
// No reference counterpart: the reference runs one SpMV per vector
// (src/Mille-feuille-cg.h:97-166).  A 16x16 tile with at least `fill`
// entries is kept as a dense FP16 block (built once per matrix and fill
// threshold, duplicates added in FP32 before the rounding) in the order of the
// MMA's A fragments: 16 bytes per lane.  A warp owns a 16-row strip and
// multiplies each dense tile of it by the matching 16 rows of X with two
// mma.sync m16n8k16 instructions (columns 0-7 and 8-15), the accumulators held
// in the MMA fragment layout.  The strip's other entries are kept row by row
// (column and FP32 value) and added by the same threads into the same
// accumulators (each thread owns rows gid and gid + 8 and four columns): before
// each dense tile the entries of the tiles left of it, so that every output is
// summed tile by tile in column order, whatever kind its tiles are
// (deterministic).  X is first scaled per column by a power of two that maps
// its largest magnitude to [0.5, 1] and rounded to FP16, row-major with 16
// halves per row.  Y is rescaled and written in FP64.  Accuracy: FP16 rounding
// of A's dense tiles and of X (2^-11 relative each), FP32 sums.
//
// Bound by the latency of the entries' gathers of X: a row's entries are
// copied to shared memory with their X rows, 8 at a time and all in flight
// together (by cp.async; the next dense tile's X rows too), and then added from
// there.  16 columns of a 262,144-row block-structured matrix (about 4 dense
// and 64 sparse tiles per strip): 60 us a call, 36 of them in k_spmm_tc, 10 and
// 9 in the two passes over X; 284 us when the warp walked the strip's tiles one
// by one, the sparse ones among them.  With the window in registers instead of
// shared memory 88 us (2 entries of a row; 130 with 8, for fewer warps); with
// X a second time in B fragment order 68 us; with 4 entries in the window 78.
//
// The MMA is the warp-level form, which Blackwell runs on its tensor cores;
// a 16 x 16 x 16 block is far below the smallest tcgen05 tile (64 rows), so
// tcgen05 with TMEM accumulators would idle most of each instruction here.
#include <cuda_fp16.h>

#include <algorithm>
#include <climits>

#include "mf_internal.h"
#include "spmv_core.cuh"

namespace mf {
namespace {

constexpr int TC_NT = 256;  // 8 warps per CTA, one strip per warp at a time

int tc_grid(long long work, int nt)
{
    long long g = (work + nt - 1) / nt;
    return (int)(g < 1 ? 1 : g > 148 * 32 ? 148 * 32 : g);
}

__global__ void k_tc_mark(int T, const int *__restrict__ tile_nnz, const unsigned char *__restrict__ f16ok, int fill,
                          int *__restrict__ flag)
{
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < T; t += gridDim.x * blockDim.x)
        flag[t] = (tile_nnz[t + 1] - tile_nnz[t] >= fill && (f16ok[t] & 1)) ? 1 : 0;
}

// Per strip (16 threads, one per row): its dense tiles, and each row's sparse
// entries.  A zero closes each list for its scan.
__global__ void __launch_bounds__(TC_NT) k_tc_count(MfTiles A, const int *__restrict__ flag, int *__restrict__ nd,
                                                    int *__restrict__ ns)
{
    const int r = threadIdx.x & 15;
    for (int s = (blockIdx.x * TC_NT + threadIdx.x) >> 4; s <= A.tilem; s += (gridDim.x * TC_NT) >> 4) {
        if (s == A.tilem) {
            if (r == 0) nd[s] = ns[s * MF_TILE] = 0;
            continue;
        }
        const int rowlen = (s == A.tilem - 1) ? A.rows - s * MF_TILE : MF_TILE;
        int d = 0, c = 0;
        for (int t = A.tile_ptr[s]; t < A.tile_ptr[s + 1]; t++) {
            if (flag[t]) {
                d++;
            } else if (r < rowlen) {
                int lo, hi;
                tile_row_bounds(A, t, r, rowlen, 0, A.tile_nnz[t + 1] - A.tile_nnz[t], lo, hi);
                c += max(hi - lo, 0);
            }
        }
        ns[s * MF_TILE + r] = c;
        if (r == 0) nd[s] = d;
    }
}

// Per strip: the tile columns of its dense tiles, its rows' sparse entries, and
// where each tile's block is (index[t], -1 for a sparse tile).
__global__ void __launch_bounds__(TC_NT) k_tc_lists(MfTiles A, const int *__restrict__ flag,
                                                    const int *__restrict__ dptr, const int *__restrict__ rptr,
                                                    int *__restrict__ dcol, int2 *__restrict__ sent,
                                                    int *__restrict__ index)
{
    const int r = threadIdx.x & 15;
    for (int s = (blockIdx.x * TC_NT + threadIdx.x) >> 4; s < A.tilem; s += (gridDim.x * TC_NT) >> 4) {
        const int rowlen = (s == A.tilem - 1) ? A.rows - s * MF_TILE : MF_TILE;
        int d = dptr[s], at = rptr[s * MF_TILE + r];
        for (int t = A.tile_ptr[s]; t < A.tile_ptr[s + 1]; t++) {
            const int tc = A.tile_columnidx[t];
            if (flag[t]) {
                if (r == 0) {
                    dcol[d] = tc;
                    index[t] = d;
                }
                d++;
                continue;
            }
            if (r == 0) index[t] = -1;
            if (r >= rowlen) continue;
            const int off = A.tile_nnz[t];
            int lo, hi;
            tile_row_bounds(A, t, r, rowlen, off, A.tile_nnz[t + 1] - off, lo, hi);
            for (int e = off + lo; e < off + hi; e++)
                sent[at++] = make_int2(tc * MF_TILE + A.col[e], __float_as_int(A.val_low[e]));
        }
    }
}

// One warp per dense tile: lane r adds row r's entries (in entry order,
// duplicates summed) into a 16x16 FP32 block in shared memory, then the warp
// rounds it to FP16 in A fragment order: lane gid * 4 + tig holds rows gid and
// gid + 8 at columns 2 tig, 2 tig + 1 (registers 0, 1) and the same + 8
// (registers 2, 3).
__global__ void __launch_bounds__(TC_NT) k_tc_fill(MfTiles A, int T, const int *__restrict__ tile_strip,
                                                   const int *__restrict__ index, __half *__restrict__ dense)
{
    __shared__ float blk[TC_NT / 32][256];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float *b = blk[w];
    for (int t = blockIdx.x * (TC_NT / 32) + w; t < T; t += gridDim.x * (TC_NT / 32)) {
        const int di = index[t];
        if (di < 0) continue;  // uniform over the warp
        for (int i = lane; i < 256; i += 32) b[i] = 0.f;
        __syncwarp();
        const int bi = tile_strip[t];
        const int rowlen = (bi == A.tilem - 1) ? A.rows - bi * MF_TILE : MF_TILE;
        if (lane < rowlen) {
            const int off = A.tile_nnz[t], nz = A.tile_nnz[t + 1] - off;
            int lo, hi;
            tile_row_bounds(A, t, lane, rowlen, off, nz, lo, hi);
            for (int e = off + lo; e < off + hi; e++) b[lane * 16 + A.col[e]] += (float)A.val[e];
        }
        __syncwarp();
        const int gid = lane >> 2, c = 2 * (lane & 3);
        __half h[8];
#pragma unroll
        for (int g = 0; g < 4; g++) {
            const float *src = b + (gid + 8 * (g & 1)) * 16 + c + 8 * (g >> 1);
            h[2 * g] = __float2half_rn(src[0]);
            h[2 * g + 1] = __float2half_rn(src[1]);
        }
        *reinterpret_cast<uint4 *>(dense + (size_t)di * 256 + lane * 8) = *reinterpret_cast<const uint4 *>(h);
        __syncwarp();
    }
}

struct TcState {
    unsigned mx[16];
    float scale[16], inv[16];
    unsigned count;  // blocks finished
};

// Per column blockIdx.y: the largest |X[:, j]| as float bits (atomicMax, whose
// order does not matter); the last block sets the scales.
__global__ void __launch_bounds__(256) k_tc_colmax(int n, int k, const double *__restrict__ X, int ldx,
                                                   TcState *__restrict__ st)
{
    const double *x = X + (size_t)blockIdx.y * ldx;
    const int step = gridDim.x * 256;
    float m = 0.f;
    long long i = blockIdx.x * 256 + threadIdx.x;
    for (; i + 7LL * step < n; i += 8 * step) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) v[u] = x[i + u * step];
#pragma unroll
        for (int u = 0; u < 8; u++) m = fmaxf(m, fabsf((float)v[u]));
    }
    for (; i < n; i += step) m = fmaxf(m, fabsf((float)x[i]));
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ float s_m[8];
    __shared__ bool s_last;
    if ((threadIdx.x & 31) == 0) s_m[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) m = fmaxf(m, s_m[w]);
        atomicMax(&st->mx[blockIdx.y], __float_as_uint(m));
        __threadfence();
        s_last = atomicAdd(&st->count, 1u) == gridDim.x * gridDim.y - 1;
    }
    __syncthreads();
    // scale[j] = 2^-e with 2^(e-1) <= max|X[:, j]| < 2^e (1 for a zero column),
    // exact powers of two; inv[j] = 1 / scale[j]
    if (s_last && threadIdx.x < 16) {
        __threadfence();
        const int j = threadIdx.x;
        const float mm = j < k ? __uint_as_float(__ldcg(&st->mx[j])) : 0.f;
        int e = 0;
        if (mm > 0.f) frexpf(mm, &e);
        st->scale[j] = ldexpf(1.f, -e);
        st->inv[j] = ldexpf(1.f, e);
    }
}

// X scaled per column and rounded to FP16, row-major with 16 halves per row, up
// to the padded column count, columns >= k zero.  One thread per row
// (column-major X read coalesced column by column).
__global__ void __launch_bounds__(128) k_tc_xpack(int nrow_pad, int n, int k, const double *__restrict__ X, int ldx,
                                                  const TcState *__restrict__ st, __half *__restrict__ x16)
{
    const int r = blockIdx.x * 128 + threadIdx.x;
    if (r >= nrow_pad) return;
    unsigned w[8];
#pragma unroll
    for (int j = 0; j < 16; j++) {
        const float v = (j < k && r < n) ? (float)(X[(size_t)j * ldx + r] * (double)st->scale[j]) : 0.f;
        const unsigned h = __half_as_ushort(__float2half_rn(v));
        w[j / 2] = (j & 1) ? w[j / 2] | (h << 16) : h;
    }
    uint4 *d = reinterpret_cast<uint4 *>(x16 + (size_t)r * 16);
    d[0] = make_uint4(w[0], w[1], w[2], w[3]);
    d[1] = make_uint4(w[4], w[5], w[6], w[7]);
}

// D (16x8, FP32) += A (16x16, FP16, row-major fragments) * B (16x8, FP16)
__device__ __forceinline__ void mma_16816(float *d, unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0,
                                          unsigned b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

constexpr int TC_WARPS = 4, TC_MINB = 8;
constexpr int TC_S = 8;  // sparse entries of a row in shared memory at a time

// A warp's window on its strip's sparse entries, one more column than used so
// that the rows' reads fall into different banks.
struct TcWindow {
    uint4 x[MF_TILE][TC_S + 1][2];   // X row of each entry
    int2 e[MF_TILE][TC_S + 1];       // column (-1 none) and value bits
    uint4 xd[2][MF_TILE * 2];        // X rows of a dense tile and of the next one
};

__device__ __forceinline__ void tc_copy16(void *to, const void *from)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from)
                 : "memory");
}

// Row r's entries from `at` on, by its four threads (tig): the X rows are copied
// asynchronously.
__device__ __forceinline__ void tc_window(TcWindow &w, const int2 *__restrict__ sent, int at, int end, int r,
                                          const __half *__restrict__ x16, int tig)
{
    int2 c[TC_S / 4];
#pragma unroll
    for (int i = 0; i < TC_S / 4; i++) {
        const int k = at + 4 * i + tig;
        c[i] = k < end ? __ldcs(sent + k) : make_int2(-1, 0);
    }
#pragma unroll
    for (int i = 0; i < TC_S / 4; i++) {
        const int u = 4 * i + tig;
        w.e[r][u] = c[i];
        if (c[i].x >= 0) {
            const __half *x = x16 + (size_t)c[i].x * 16;
            tc_copy16(&w.x[r][u][0], x);
            tc_copy16(&w.x[r][u][1], x + 8);
        }
    }
}

__device__ __forceinline__ void tc_window_wait(unsigned mask)
{
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp(mask);
}

// One warp per strip.  Fragment layout of m16n8k16 (thread lane: gid =
// lane / 4, tig = lane % 4): A holds rows gid and gid + 8, columns 2 tig,
// 2 tig + 1 and the same + 8; B holds rows 2 tig, 2 tig + 1 (+ 8) of column
// gid; D holds rows gid, gid + 8 and columns 2 tig, 2 tig + 1.
template <bool TWO>
__global__ void __launch_bounds__(TC_WARPS * 32, TC_MINB) k_spmm_tc(int rows, int tilem, const int *__restrict__ dptr,
                                                      const int *__restrict__ dcol, const uint4 *__restrict__ dense,
                                                      const int *__restrict__ rptr, const int2 *__restrict__ sent,
                                                      const __half *__restrict__ x16, int k, const TcState *__restrict__ st, double *__restrict__ Y,
                                                      int ldy)
{
    __shared__ TcWindow s_w[TC_WARPS];
    TcWindow &w = s_w[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    const int bi = blockIdx.x * TC_WARPS + (threadIdx.x >> 5);
    if (bi >= tilem) return;
    const int d0 = dptr[bi], d1 = dptr[bi + 1];
    // rows gid and gid + 8: the window's first entry, the row's end, and where
    // in the window the row is
    int at[2], end[2], pos[2] = {0, 0};
#pragma unroll
    for (int h = 0; h < 2; h++) {
        at[h] = rptr[bi * MF_TILE + gid + 8 * h];
        end[h] = rptr[bi * MF_TILE + gid + 8 * h + 1];
        tc_window(w, sent, at[h], end[h], gid + 8 * h, x16, tig);
    }
    float a0[4] = {0.f, 0.f, 0.f, 0.f}, a1[4] = {0.f, 0.f, 0.f, 0.f};
    // the sparse entries of the columns before `limit` (an empty place's -1 is
    // after every limit)
    auto sparse = [&](unsigned limit) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int r = gid + 8 * h;
            for (;;) {
                for (; pos[h] < TC_S; pos[h]++) {
                    const int2 e = w.e[r][pos[h]];
                    if ((unsigned)e.x >= limit) break;
                    const float v = __int_as_float(e.y);
                    const __half2 *x = reinterpret_cast<const __half2 *>(&w.x[r][pos[h]][0]);
                    const float2 xa = __half22float2(x[tig]);
                    a0[2 * h] = fmaf(v, xa.x, a0[2 * h]);
                    a0[2 * h + 1] = fmaf(v, xa.y, a0[2 * h + 1]);
                    if (TWO) {
                        const float2 xb = __half22float2(x[4 + tig]);
                        a1[2 * h] = fmaf(v, xb.x, a1[2 * h]);
                        a1[2 * h + 1] = fmaf(v, xb.y, a1[2 * h + 1]);
                    }
                }
                if (pos[h] < TC_S || end[h] - at[h] <= TC_S) break;
                // the row's window is used up: the next one (its four threads)
                const unsigned quad = 0xFu << (lane & 28);
                __syncwarp(quad);
                at[h] += TC_S;
                pos[h] = 0;
                tc_window(w, sent, at[h], end[h], r, x16, tig);
                tc_window_wait(quad);
            }
        }
        __syncwarp();
    };
    // a dense tile's X rows, 16 bytes per lane, halves swapped in rows 4-7 and
    // 12-15 (the eight rows of an ldmatrix block in different banks)
    auto load_x = [&](int buf, int c) {
        const int r = lane >> 1, half = (lane & 1) ^ ((r >> 2) & 1);
        tc_copy16(&w.xd[buf][2 * r + half], x16 + (size_t)c * 256 + lane * 8);
    };
    int c = 0, buf = 0;
    uint4 a = make_uint4(0, 0, 0, 0);
    if (d0 < d1) {
        c = dcol[d0];
        a = dense[(size_t)d0 * 32 + lane];
        load_x(0, c);
    }
    tc_window_wait(0xffffffffu);
    for (int d = d0; d < d1; d++, buf ^= 1) {
        // the next dense tile loads under this one's sums
        int cn = 0;
        uint4 an = a;
        if (d + 1 < d1) {
            cn = dcol[d + 1];
            an = dense[(size_t)(d + 1) * 32 + lane];
            load_x(buf ^ 1, cn);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        sparse((unsigned)c * MF_TILE);
        // all but the copy just begun
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        // B fragments of columns 0-7 (rows 0-7, rows 8-15) and 8-15: lane l
        // gives the address of row l & 15 in column half l >> 4
        unsigned b[4];
        const int xr = lane & 15, xh = (lane >> 4) ^ ((xr >> 2) & 1);
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                     : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3])
                     : "r"((unsigned)__cvta_generic_to_shared(&w.xd[buf][2 * xr + xh]))
                     : "memory");
        mma_16816(a0, a.x, a.y, a.z, a.w, b[0], b[1]);
        if (TWO) mma_16816(a1, a.x, a.y, a.z, a.w, b[2], b[3]);
        __syncwarp();
        a = an;
        c = cn;
    }
    sparse(INT_MAX);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int i = bi * MF_TILE + gid + 8 * h;
        if (i >= rows) continue;
        const int c0 = 2 * tig, c1 = 2 * tig + 1, c2 = 8 + 2 * tig, c3 = 9 + 2 * tig;
        if (c0 < k) Y[(size_t)c0 * ldy + i] = (double)(a0[2 * h] * st->inv[c0]);
        if (c1 < k) Y[(size_t)c1 * ldy + i] = (double)(a0[2 * h + 1] * st->inv[c1]);
        if (TWO && c2 < k) Y[(size_t)c2 * ldy + i] = (double)(a1[2 * h] * st->inv[c2]);
        if (TWO && c3 < k) Y[(size_t)c3 * ldy + i] = (double)(a1[2 * h + 1] * st->inv[c3]);
    }
}

// The lists and dense blocks for threshold `fill` (kept on the handle;
// rebuilt when the threshold changes)
mf_status tc_prepare(mf_matrix m, int fill, cudaStream_t s)
{
    if (m->tc_mem && m->tc_fill == fill) return MF_OK;
    const int T = m->v.tilenum, tilem = m->v.tilem;
    handle_release(m->tc_mem);
    m->tc_fill = 0;
    m->tc_ndense = 0;
    // temporaries: flags and block index per tile; dense tiles per strip and
    // sparse entries per row, and their scans
    const size_t nr = (size_t)tilem * MF_TILE + 1;
    int *tmp = nullptr;
    MF_CUDA(pool_malloc_async(&tmp, sizeof(int) * (2 * ((size_t)T + 1) + 2 * ((size_t)tilem + 1) + 2 * nr), s));
    int *flag = tmp, *index = flag + T + 1, *nd = index + T + 1, *dp = nd + tilem + 1, *ns = dp + tilem + 1,
        *rp = ns + nr;
    mf_status st = MF_OK;
    int dense = 0, sparse = 0;
    do {
        const int grid = tc_grid((long long)(tilem + 1) * 16, TC_NT);
        if (T > 0) {
            k_tc_mark<<<tc_grid(T, 256), 256, 0, s>>>(T, m->d_tile_nnz, m->d_f16ok, fill, flag);
            note_launch();
        }
        k_tc_count<<<grid, TC_NT, 0, s>>>(m->v, flag, nd, ns);
        note_launch();
        if ((st = exclusive_scan_i32(nd, dp, tilem + 1, s, &dense)) != MF_OK) break;
        if ((st = exclusive_scan_i32(ns, rp, (int)nr, s, &sparse)) != MF_OK) break;
        auto pad = [](size_t v) { return (v + 255) / 256 * 256; };
        const size_t o_dptr = pad(sizeof(__half) * 256 * (size_t)dense),
                     o_rptr = o_dptr + pad(sizeof(int) * ((size_t)tilem + 1)), o_dcol = o_rptr + pad(sizeof(int) * nr),
                     o_sent = o_dcol + pad(sizeof(int) * (size_t)dense), bytes = o_sent + sizeof(int2) * (size_t)sparse;
        if (handle_malloc(&m->tc_mem, bytes) != cudaSuccess) {
            cudaGetLastError();
            set_last_error("mf_spmm_f16: no device memory for %d dense tiles and %d other entries", dense, sparse);
            st = MF_ERR_NO_MEMORY;
            break;
        }
        char *at = (char *)m->tc_mem;
        m->d_tc_dense = at;
        m->d_tc_dptr = (int *)(at + o_dptr);
        m->d_tc_rptr = (int *)(at + o_rptr);
        m->d_tc_dcol = (int *)(at + o_dcol);
        m->d_tc_sent = (int2 *)(at + o_sent);
        cudaMemcpyAsync(m->d_tc_dptr, dp, sizeof(int) * (tilem + 1), cudaMemcpyDeviceToDevice, s);
        cudaMemcpyAsync(m->d_tc_rptr, rp, sizeof(int) * nr, cudaMemcpyDeviceToDevice, s);
        if (tilem > 0) {
            k_tc_lists<<<grid, TC_NT, 0, s>>>(m->v, flag, dp, rp, m->d_tc_dcol, m->d_tc_sent, index);
            note_launch();
        }
        if (dense > 0) {
            k_tc_fill<<<tc_grid((long long)T * 32, TC_NT), TC_NT, 0, s>>>(m->v, T, m->d_tile_rowidx, index,
                                                                           (__half *)m->d_tc_dense);
            note_launch();
        }
        // waited for before anything tells that they are there: the next call
        // may come on another stream
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) {
            set_last_error("mf_spmm_f16: %s", cudaGetErrorString(e));
            st = MF_ERR_CUDA;
        }
    } while (false);
    cudaFreeAsync(tmp, s);
    MF_TRY(st);
    m->tc_fill = fill;
    m->tc_ndense = dense;
    return MF_OK;
}

}  // namespace
}  // namespace mf

using namespace mf;

extern "C" mf_status mf_spmm_f16(mf_matrix m, int k, const double *X, int ldx, double *Y, int ldy, int dense_fill,
                                 int *dense_tiles, void *stream)
{
    if (!m || k < 1 || k > 16 || dense_fill > 256 || (m->v.rows > 0 && (!X || !Y)) || ldx < m->v.cols ||
        ldy < m->v.rows) {
        set_last_error("mf_spmm_f16: null argument, k = %d outside 1..16, fill above 256 or a short leading dimension",
                       k);
        return MF_ERR_INVALID_ARG;
    }
    const int fill = dense_fill > 0 ? dense_fill : 64;
    cudaStream_t s = (cudaStream_t)stream;
    MF_TRY(tc_prepare(m, fill, s));
    if (dense_tiles) *dense_tiles = m->tc_ndense;
    if (m->v.rows == 0) return MF_OK;
    const int nrow_pad = m->v.tilen * MF_TILE;
    // X as halves (32 bytes per row), the state
    char *buf = nullptr;
    const size_t xb = 32 * (size_t)nrow_pad;
    MF_CUDA(pool_malloc_async(&buf, xb + sizeof(TcState), s));
    __half *x16 = (__half *)buf;
    TcState *st = (TcState *)(buf + xb);
    cudaMemsetAsync(st, 0, sizeof(TcState), s);
    // about a resident wave of blocks over all columns (8 blocks per SM)
    const dim3 cgrid(std::max(1, std::min(ceil_div(m->v.cols, 256), 148 * 8 / k)), k);
    k_tc_colmax<<<cgrid, 256, 0, s>>>(m->v.cols, k, X, ldx, st);
    k_tc_xpack<<<std::max(1, ceil_div(nrow_pad, 128)), 128, 0, s>>>(nrow_pad, m->v.cols, k, X, ldx, st, x16);
    const int grid = ceil_div(m->v.tilem, TC_WARPS);
    if (k > 8)
        k_spmm_tc<true><<<grid, TC_WARPS * 32, 0, s>>>(m->v.rows, m->v.tilem, m->d_tc_dptr, m->d_tc_dcol,
                                                       (const uint4 *)m->d_tc_dense, m->d_tc_rptr, m->d_tc_sent, x16,
                                                       k, st, Y, ldy);
    else
        k_spmm_tc<false><<<grid, TC_WARPS * 32, 0, s>>>(m->v.rows, m->v.tilem, m->d_tc_dptr, m->d_tc_dcol,
                                                        (const uint4 *)m->d_tc_dense, m->d_tc_rptr, m->d_tc_sent, x16,
                                                        k, st, Y, ldy);
    note_launch(3);
    const cudaError_t e = cudaGetLastError();
    cudaFreeAsync(buf, s);
    MF_CUDA(e);
    return MF_OK;
}
