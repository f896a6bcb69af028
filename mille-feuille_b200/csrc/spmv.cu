// spmv.cu -- standalone FP64 tiled SpMV (the role of the reference's
// stir_spmv_cuda_kernel_newcsr, src/Mille-feuille-cg.h:97-166, and of
// blockspmv_cpu, src/blockspmv_cpu.h:2-112).  Thread per row; no atomics;
// bit-identical to blockspmv_cpu.
//
// A handle's first product runs from the tiles; from the second on it runs
// from the row slots (slots.cu), built then: a strip's slots are read
// coalesced and a row's entries load eight at a time, where the tiles cost a
// chain of dependent loads per tile (128^3 Poisson 62.4 -> 37.9 us).
#include <climits>

#include "solver.h"
#include "spmv_core.cuh"

namespace mf {
namespace {

constexpr int SPMV_NT = 256;
constexpr int SPMV_MINB = 5;  // 48 registers, 40 warps per SM: 34.8 us (4: 38.9, 6: 35.2; 128^3 Poisson)

__global__ void __launch_bounds__(SPMV_NT) k_spmv_fp64(MfTiles A, const double *__restrict__ x, double *__restrict__ y)
{
    const int strips_per_cta = SPMV_NT / MF_TILE;
    for (int bi = blockIdx.x * strips_per_cta + (threadIdx.x >> 4); bi < A.tilem; bi += gridDim.x * strips_per_cta) {
        const int r = threadIdx.x & 15;
        const int rowlen = (bi == A.tilem - 1) ? A.rows - bi * MF_TILE : MF_TILE;
        if (r < rowlen) y[bi * MF_TILE + r] = row_fp64(A, bi, r, rowlen, x);
    }
}

// The next N entries of a row from the row slots: their columns and values,
// then their elements of x are in flight together; then the sums in
// blockspmv_cpu's order (a partial sum per tile, added when the tile column
// changes).  An empty entry (always after the row's others) adds a zero
// product: no sum here is ever -0.0, so that changes no bit.
template <int N, typename OT>
__device__ __forceinline__ void slot_sums(const OT *__restrict__ d0, const double *__restrict__ v0,
                                          const double *__restrict__ xi, int lane, int &prev, double &yd, double &part)
{
    constexpr OT EMPTY = (OT)(sizeof(OT) == 2 ? INT16_MIN : INT32_MIN);
    int d[N];
    double v[N], xv[N];
#pragma unroll
    for (int u = 0; u < N; u++) {
        d[u] = (int)__ldcs(d0 + u * MF_TILE);
        v[u] = __ldcs(v0 + u * MF_TILE);
    }
#pragma unroll
    for (int u = 0; u < N; u++) xv[u] = d[u] != (int)EMPTY ? xi[d[u]] : 0.0;
#pragma unroll
    for (int u = 0; u < N; u++) {
        const int t = (d[u] + lane) >> 4;  // tile column, counted from the strip's own
        if (t != (u == 0 ? prev : (d[u - 1] + lane) >> 4)) {
            yd = __dadd_rn(yd, part);
            part = 0.0;
        }
        part = __dadd_rn(part, __dmul_rn(xv[u], v[u]));
    }
    prev = (d[N - 1] + lane) >> 4;
}

// Thread per row over the row slots (slot k of a strip: the k-th entry of its
// 16 rows).
template <typename OT>
__global__ void __launch_bounds__(SPMV_NT, SPMV_MINB) k_spmv_slots(int rows, const int *__restrict__ sslot,
                                                           const OT *__restrict__ soff, const double *__restrict__ sval,
                                                           const double *__restrict__ x, double *__restrict__ y)
{
    const int i = blockIdx.x * SPMV_NT + threadIdx.x, s = i >> 4, lane = i & 15;
    if (i >= rows) return;
    const int k0 = sslot[s];
    int K = sslot[s + 1] - k0;
    const OT *d = soff + (size_t)k0 * MF_TILE + lane;
    const double *v = sval + (size_t)k0 * MF_TILE + lane, *xi = x + i;
    double yd = 0.0, part = 0.0;
    int prev = INT_MIN;
    for (; K > 8; K -= 8, d += 8 * MF_TILE, v += 8 * MF_TILE) slot_sums<8>(d, v, xi, lane, prev, yd, part);
    switch (K) {  // straight code for every remainder: no load is predicated
    case 8: slot_sums<8>(d, v, xi, lane, prev, yd, part); break;
    case 7: slot_sums<7>(d, v, xi, lane, prev, yd, part); break;
    case 6: slot_sums<6>(d, v, xi, lane, prev, yd, part); break;
    case 5: slot_sums<5>(d, v, xi, lane, prev, yd, part); break;
    case 4: slot_sums<4>(d, v, xi, lane, prev, yd, part); break;
    case 3: slot_sums<3>(d, v, xi, lane, prev, yd, part); break;
    case 2: slot_sums<2>(d, v, xi, lane, prev, yd, part); break;
    case 1: slot_sums<1>(d, v, xi, lane, prev, yd, part); break;
    default: break;
    }
    y[i] = __dadd_rn(yd, part);
}

// As k_spmv_fp64, with each entry's in-tile column read from the 4-bit
// packed array (two per byte, even positions in the high nibble), as
// blockspmv_cpu reads csr_compressedIdx (src/blockspmv_cpu.h:101-103).
__global__ void __launch_bounds__(SPMV_NT) k_spmv_fp64_cidx(MfTiles A, const unsigned char *__restrict__ cidx,
                                                             const double *__restrict__ x, double *__restrict__ y)
{
    const int strips_per_cta = SPMV_NT / MF_TILE;
    for (int bi = blockIdx.x * strips_per_cta + (threadIdx.x >> 4); bi < A.tilem; bi += gridDim.x * strips_per_cta) {
        const int r = threadIdx.x & 15;
        const int rowlen = (bi == A.tilem - 1) ? A.rows - bi * MF_TILE : MF_TILE;
        if (r >= rowlen) continue;
        double acc = 0.0;
        const int t0 = A.tile_ptr[bi], t1 = A.tile_ptr[bi + 1];
        int off = A.tile_nnz[t0];
        for (int t = t0; t < t1; t++) {
            const int nxt = A.tile_nnz[t + 1];
            const int xo = A.tile_columnidx[t] * MF_TILE;
            int lo, hi;
            tile_row_bounds(A, t, r, rowlen, off, nxt - off, lo, hi);
            double s = 0.0;
            for (int k = off + lo; k < off + hi; k++) {
                const unsigned char b = cidx[k >> 1];
                const int c = (k & 1) ? (b & 0x0F) : (b >> 4);
                s = __dadd_rn(s, __dmul_rn(x[xo + c], A.val[k]));
            }
            acc = __dadd_rn(acc, s);
            off = nxt;
        }
        y[bi * MF_TILE + r] = acc;
    }
}

}  // namespace

mf_status spmv_fp64_cidx(const MfTiles &A, const unsigned char *cidx, const double *x, double *y, cudaStream_t s)
{
    if (A.tilem == 0) return MF_OK;
    int grid = ceil_div(A.tilem, SPMV_NT / MF_TILE);
    k_spmv_fp64_cidx<<<grid, SPMV_NT, 0, s>>>(A, cidx, x, y);
    note_launch();
    MF_CUDA(cudaGetLastError());
    return MF_OK;
}

mf_status spmv_fp64(const MfTiles &A, const double *x, double *y, cudaStream_t s)
{
    if (A.tilem == 0) return MF_OK;
    int grid = ceil_div(A.tilem, SPMV_NT / MF_TILE);
    k_spmv_fp64<<<grid, SPMV_NT, 0, s>>>(A, x, y);
    note_launch();
    MF_CUDA(cudaGetLastError());
    return MF_OK;
}

// y = A x.  Building the slots costs as much as five products (128^3 Poisson: 0.18
// ms of kernels, against 25 us saved by each later product), so the first
// product of a handle, which may be its only one, does not; the second queues
// them in front of its own kernel.  Their sizes are known from the build of the
// tiles, so no call waits for the GPU.  A matrix whose slots would be more than
// half padding, or that they cannot describe, stays with the tiles, and so does a
// captured product while they are still on their way.
mf_status spmv(mf_matrix m, const double *x, double *y, cudaStream_t s)
{
    const MfTiles &A = m->v;
    if (A.tilem == 0) return MF_OK;
    const long long most = 2LL * A.nnz + 4096;
    bool slots = m->slots_state.load(std::memory_order_acquire) == 1, done = true;
    if (!slots && m->spmv_calls.load(std::memory_order_relaxed) >= 0) {
        const int calls = m->spmv_calls.fetch_add(1, std::memory_order_relaxed);
        if (m->slots_state.load() < 0 || m->nslots < 0 || m->nslots * MF_TILE > most) {
            m->spmv_calls.store(-1);  // never from slots that this call would have to build
        } else if (calls >= 1 && !capturing(s)) {
            RelaxedCapture relaxed;  // another thread's capture does not mind the allocations here
            mf_status st = build_slots(m, s, false);
            slots = m->slots_state.load(std::memory_order_acquire) == 1;
            if (st == MF_OK && slots) st = build_slots(m, s);  // another thread's: s waits for them
            if (st != MF_OK) {  // no memory for them: the tiles serve
                cudaGetLastError();
                m->spmv_calls.store(-1);
                slots = false;
            }
        }
    } else if (slots && !(slots_ready(m, done) && done)) {
        if (!capturing(s)) MF_TRY(build_slots(m, s));
        else slots = false;
    }
    if (!slots || m->nslots * MF_TILE > most) return spmv_fp64(A, x, y, s);
    const int grid = ceil_div(A.rows, SPMV_NT);
    if (m->soff_bytes == 2)
        k_spmv_slots<<<grid, SPMV_NT, 0, s>>>(A.rows, m->d_sslot, (const int16_t *)m->d_soff, m->d_sval, x, y);
    else
        k_spmv_slots<<<grid, SPMV_NT, 0, s>>>(A.rows, m->d_sslot, (const int32_t *)m->d_soff, m->d_sval, x, y);
    note_launch();
    MF_CUDA(cudaGetLastError());
    return MF_OK;
}

}  // namespace mf
