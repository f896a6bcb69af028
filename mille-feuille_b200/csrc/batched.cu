// batched.cu -- many independent CG solves of uneven size in one launch,
// with per-chunk precision classes chosen on the chip.
//
// No reference counterpart: the reference solves one system per launch.
// Design for B200: the systems are sorted by size and handed out by a device
// work queue to thread-block clusters; a cluster of C CTAs (one per SM)
// solves one system at a time.  A system's rows are cut into chunks and the
// chunks are split across the cluster's CTAs; every dot product is reduced
// through distributed shared memory with a hardware cluster barrier -- no
// grid-wide synchronisation, so small systems cost no more than their own
// iterations.
//
// Random column patterns make the SpMV gather-bound when the gathered vector
// comes from L1/L2: every lane's element is its own cache line, about one
// line per cycle per SM.  The mixed-precision kernel therefore keeps a window
// of p (FP32, up to 55,296 columns, 216 KB) in shared memory and streams the
// matrix in sorted slices of 32 rows (batch_sell.cuh): a lane owns a row, its
// words come as 16-byte loads straight from L2/HBM into registers, the
// gathers hit shared memory.  Systems whose window and vectors fit (up to
// ~22,000 rows with 2 CTAs) keep p, r, q and the correction on the chip, p
// and q going to the cluster's other CTAs by distributed shared memory.
// What bounds it: in the product the L1 data pipe (a warp's slot of 32 entries
// takes 5.1 wavefronts -- 2 for its words, ~2 for the gather, the rest for the
// row ends -- and 6.4 cycles); over a whole launch that pipe is busy 48 % of the
// time, the rest goes to the words' latency, the vectors and the three cluster
// barriers of an iteration.  The earlier form -- bulk copies into three shared-memory
// stages, products written back to shared memory, one lane per row adding
// them, vectors in global memory -- moved every entry through shared memory
// four times.  Measured on one B200: the 512-system benchmark batch (1,000 to
// 64,000 rows, 1e-10) 1,366 -> 665 ms learned, 1,419 -> 838 static; to 1e-14,
// 256 systems of 1,000-32,000 rows, learned, 630 -> 288 ms; 24 systems of
// 1,000-4,000 rows, static, 56.1 -> 28.4 ms.
//
// The panel storage (column panels of PW = 32768 columns, 16-bit column
// offsets within the panel, rows of each panel in CSR) is what the chunks,
// the exports and the FP64 kernel use.  A chunk is a range of rows with at
// most BCE entries in every panel.  The FP64 kernel (the FP64 policy and trace
// collection) stages (chunk, panel) passes in shared memory by bulk copies
// and gathers p from global memory.
//
// Values of the slices are held in FP64 (reliable updates), FP32, and FP16
// scaled per row by a power of two (the row's largest off-diagonal magnitude
// maps into [2^14, 2^15)), the diagonal kept apart.  A mixed-precision solve
// reads each chunk's rows in its working class -- FP32 (4 + 2 bytes per entry)
// or FP16 (one 4-byte word per entry: the value bits and the column offset) --
// and accumulates in FP32; FP64 dot products, FP64 reliable updates
// r = b - A x from the FP64 values, convergence judged on that FP64
// residual.
//
// Classes per chunk, decided inside the persistent kernel by the CTA that
// owns the chunk (no host round trip):
//   STATIC   the value-range class: FP16 when every value of the chunk is
//            exactly representable (scaled FP16 off-diagonals, FP32
//            diagonal), else FP32; fixed for the solve.
//   RULE     after every p update, the reference's partial-convergence
//            thresholds (src/main-cg-mixed.cu:415-460) on the chunk's own
//            rows: v = max |p_new - p_old| in FP64; v > 1e-6 (FP64 and FP32
//            decisions) -> FP32, else FP16 (the FP16, INT8 and BYPASS
//            decisions: rows cannot be skipped in a row-chunk layout, and
//            the values are not integers).
//   LEARNED  at the first iteration and at every reliable update, the MLP
//            (16 chunk features -> 32 -> 32 -> 4, BF16 weights, FP32
//            accumulation) of an attached mf_learned: FP16 where it is at
//            least 90 % sure the chunk's label is FP16 or narrower.
// RULE and LEARNED fall back to the static classes for the rest of a
// system's solve when a reliable update finds the FP64 residual above half
// of the previous one (the recurrence claimed a tenfold drop).
// A chunk whose rows' FP16 scales fall outside FP32's range stays FP32.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <numeric>
#include <thread>
#include <vector>

#include <type_traits>

#include "mf_internal.h"
#include "batch_sell.cuh"
#include "policy_net.cuh"
#include "tma.cuh"

namespace cg = cooperative_groups;

namespace mf {
namespace {
constexpr int PW = 32768;   // columns per storage panel (16-bit offsets)
#ifndef MF_BATCH_BCE
#define MF_BATCH_BCE 4096
#endif
#ifndef MF_BATCH_BCR
#define MF_BATCH_BCR 256
#endif
constexpr int BCE = MF_BATCH_BCE;   // entries of a (chunk, panel) stage
constexpr int BCR = MF_BATCH_BCR;   // rows of a chunk
}  // namespace
}  // namespace mf

// What a captured solve has fixed: two solves share a graph when all of it
// agrees.
struct BatchGraphKey {
    const double *b;
    double *x;
    int lanes, cluster, policy, maxiter;
    double tol, delta;
    const void *weights;  // LEARNED
    unsigned long long budget_ns;
    unsigned backoff_ns;
    bool operator==(const BatchGraphKey &o) const
    {
        return b == o.b && x == o.x && lanes == o.lanes && cluster == o.cluster && policy == o.policy &&
               maxiter == o.maxiter && tol == o.tol && delta == o.delta && weights == o.weights &&
               budget_ns == o.budget_ns && backoff_ns == o.backoff_ns;
    }
};

struct mf_batch_s {
    int count = 0;
    long long rows_total = 0, nnz_total = 0;
    int nchunks = 0, npanels = 0;
    std::vector<int> n;           // rows per system (caller order)
    std::vector<long long> row0;  // first row of each system (caller order)
    std::vector<long long> nz0;   // first entry of each system
    int *d_order = nullptr;       // systems by descending size
    long long *d_row0 = nullptr;
    int *d_n = nullptr, *d_pan0 = nullptr, *d_npan = nullptr;  // per system: first panel, panels
    long long *d_prow0 = nullptr; // per panel: first of its n+1 row pointers
    long long *d_pent0 = nullptr; // per panel (+1): first entry
    int *d_prow = nullptr;        // panel row pointers, relative to the panel's first entry
    uint16_t *d_col = nullptr;    // column offset within the panel
    double *d_val = nullptr;
    __half *d_val16 = nullptr;    // row-scaled, diagonal entries 0
    float *d_rscale = nullptr;    // per row: scale of the FP16 values
    float *d_diag32 = nullptr;    // per row: diagonal (sum of the row's diagonal entries)
    // row chunks of every system
    int *d_sc = nullptr;          // [count+1] first chunk of each system
    int *d_crow = nullptr;        // per system nch+1 chunk row starts (relative rows), at sc[s] + s
    int *d_cent = nullptr;        // the same chunks' entries over all panels (sc[s] + s, scanned)
    unsigned char *d_ccls = nullptr;         // [chunks] working class (0 FP32, 1 FP16)
    unsigned char *d_ccls_static = nullptr;  // [chunks] bit 0: FP16 exact, bit 1: FP16 allowed
    float *d_cstat = nullptr;     // [chunks][NCSTAT] static features
    float *d_cdyn = nullptr;      // [chunks][NCDYN] checkpoint statistics
    // per-system results
    int *d_iters = nullptr, *d_refs = nullptr, *d_status = nullptr;
    double *d_relres = nullptr;
    unsigned long long *d_sysstat = nullptr;  // [count][3] matrix bytes streamed, FP16 chunk passes, chunk passes
    void *arena = nullptr, *slices = nullptr, *words = nullptr;  // allocations the arrays above and below live in
    void *work = nullptr;
    size_t work_bytes = 0;
    int auto_cluster = 0;         // CTAs per system of untuned mixed solves (0: not found yet)
    int *d_queue = nullptr;
    // sorted slices of the mixed solves (batch_sell.cuh)
    int *d_sfirst = nullptr, *d_win0 = nullptr;
    int2 *d_sdesc = nullptr;
    int4 *d_srec = nullptr;
    uint32_t *d_scv = nullptr;
    float *d_sv32 = nullptr;
    double *d_sv64 = nullptr, *d_diag64 = nullptr;  // diag64: per row (sum of the row's diagonal entries)
    uint16_t *d_sc16 = nullptr;
    // CUDA graph of the last solve configuration
    cudaGraphExec_t graph = nullptr;
    BatchGraphKey graph_key = {};
    int tuned_lanes = 0, tuned_cluster = 0;
    int static_fp16_chunks = 0, fp16_allowed_chunks = 0;
    struct mf_policy_s *policy = nullptr;     // LEARNED solves
};

namespace mf {

mf_status policy_sample_buffers(struct mf_policy_s *p, long long max_samples, float **x, unsigned char **y,
                                long long *n);
mf_status policy_sample_commit(struct mf_policy_s *p, long long n_total);
const __nv_bfloat16 *policy_weights(struct mf_policy_s *p);

namespace {

constexpr int BNT = 512;
constexpr int BNW = BNT / 32;
#ifndef MF_BATCH_MNT
#define MF_BATCH_MNT 1024
#endif
constexpr int MNT = MF_BATCH_MNT;  // threads of a mixed-kernel CTA
constexpr int MNW = MNT / 32;
constexpr int NCSTAT = 6;   // static chunk features 0-4, and max |a| of the chunk
constexpr int NCDYN = 10;   // [0..3] raw maxima |r|, |p|, |dp|, |q|; [4..7] previous features 6..9; [8] label ratio
constexpr float LEARN_CONF = 0.9f;   // FP16 when P(label <= FP16) >= this
constexpr double LABEL_TAU = 0.015625;  // label FP16: ||dq_c|| <= 2^-6 ||q_c|| (FP16 perturbation of A p)

struct BatchArgs {
    int count;
    const int *order;
    const int *n, *pan0, *npan;
    const long long *row0, *prow0, *pent0;
    const int *prow;
    const uint16_t *col;
    const double *val;
    const __half *val16;
    const float *rscale, *diag32;
    SellView sell;                 // mixed solves: the sorted slices
    const double *b;
    double *x;
    void *r, *p0, *p1, *q, *xlo;  // workspace vectors (rows_total each)
    const int *sc, *crow, *cent;   // row chunks
    unsigned char *ccls;
    const unsigned char *ccls_static;
    const float *cstat;
    float *cdyn;
    int *queue;
    int *iters, *refs, *status;
    double *relres;
    unsigned long long *sysstat;
    int maxiter;
    double tol;
    double delta;
    unsigned long long budget_ns;  // bound of every shared-memory stage wait
    unsigned backoff_ns;           // sleep between retries of a stage wait
    int policy;
    const __nv_bfloat16 *mlp_w;    // LEARNED: the network's BF16 weights
    // trace collection (FP64 solves): samples every collect_every iterations
    int collect_every, collect_stride;
    unsigned collect_salt;
    float *cx;
    unsigned char *cy;
    unsigned long long *ccount;
    long long ccap;
};

// One system's view of the panel storage.
struct SysView {
    int n, npan, gp0;
    long long r0;
};

__device__ __forceinline__ SysView sys_view(const BatchArgs &a, int sys)
{
    SysView v;
    v.n = a.n[sys];
    v.npan = a.npan[sys];
    v.gp0 = a.pan0[sys];
    v.r0 = a.row0[sys];
    return v;
}

// Deterministic cluster-wide sum: each CTA reduces its threads in a fixed
// tree, publishes the value in its shared memory, and after the cluster
// barrier every CTA adds the CTAs' values in rank order.
template <int NT>
__device__ __forceinline__ double cluster_sum(cg::cluster_group &cl, double v, double *slot, double *s_warp)
{
    const double c = block_sum<NT>(v, s_warp);
    if (threadIdx.x == 0) *slot = c;
    cl.sync();
    double s = 0.0;
    const unsigned ncta = cl.num_blocks();
    for (unsigned k = 0; k < ncta; k++) s += *cl.map_shared_rank(slot, k);
    return s;
}

// Cluster-wide maximum of two non-negative values (exact, so any order).
template <int NT>
__device__ __forceinline__ void cluster_max2(cg::cluster_group &cl, float &a, float &b, float *slot2, float *s_warp2)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, o));
        b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, o));
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        s_warp2[2 * (threadIdx.x >> 5)] = a;
        s_warp2[2 * (threadIdx.x >> 5) + 1] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float ma = 0.f, mb = 0.f;
        for (int w = 0; w < NT / 32; w++) {
            ma = fmaxf(ma, s_warp2[2 * w]);
            mb = fmaxf(mb, s_warp2[2 * w + 1]);
        }
        slot2[0] = ma;
        slot2[1] = mb;
    }
    cl.sync();
    a = 0.f;
    b = 0.f;
    for (unsigned k = 0; k < cl.num_blocks(); k++) {
        const float *o = cl.map_shared_rank(slot2, k);
        a = fmaxf(a, o[0]);
        b = fmaxf(b, o[1]);
    }
}

// FP64 kernel: the header of a staged (chunk, panel) pair.
struct BHdr {
    int r0, r1, e0, direct;   // rows [r0, r1), first entry e0 (relative to the panel)
    int sh_rp, sh_col, sh_val, panel;
    long long ebase;          // the panel's first entry (global)
};

// FP64 kernel: shared-memory stages of (chunk, panel) pairs (row pointers,
// columns, values) in flight per CTA.
#ifndef MF_BATCH_STAGES_FP64
#define MF_BATCH_STAGES_FP64 3
#endif

struct Stage {
    static constexpr int NS = MF_BATCH_STAGES_FP64;
    static constexpr int OFF_RP = 0;
    static constexpr int OFF_COL = ((BCR + 1) * 4 + 32 + 15) & ~15;
    static constexpr int OFF_VAL = OFF_COL + ((BCE * 2 + 32 + 15) & ~15);
    static constexpr int SIZE = OFF_VAL + ((BCE * 8 + 32 + 15) & ~15);
    static_assert(OFF_COL % 16 == 0 && OFF_VAL % 16 == 0 && SIZE % 16 == 0, "stage regions 16-byte aligned");
    static_assert((BCR + 1) * 4 + 32 <= OFF_COL, "row pointers fit");
    static_assert(NS >= 1 && NS <= 8, "stage phases kept in a byte");
};

struct BSmem {
    unsigned char stage[Stage::NS][Stage::SIZE];
    BHdr hdr[Stage::NS];
    uint64_t bar[Stage::NS];    // stage full (the producer's copies landed)
    uint64_t empty[Stage::NS];  // stage released by every consumer warp
};
static_assert(sizeof(BSmem) <= 227 * 1024, "one CTA per SM");

// Dynamic shared memory of the mixed kernel: the window of p (its first
// element at the same 16-byte phase as in global memory), the policy
// network's weights as float, a feature row per warp.
struct MixSmem {
    static constexpr size_t W = ((size_t)SELL_WIN + 4) * 4;
    static constexpr size_t FEAT = W + sizeof(float) * ((PN_NPARAM + 3) & ~3);
    static constexpr size_t TOTAL = FEAT + sizeof(float) * MNW * PN_NF;
    static_assert(TOTAL <= 226 * 1024, "one CTA per SM, 1 KB for the static arrays");
};

__device__ __forceinline__ void b_add_range(unsigned char *dst, const unsigned char *src, long long a0, long long a1,
                                            uint64_t *bar, int &shift)
{
    const long long c0 = a0 & ~15ll, c1 = (a1 + 15) & ~15ll;
    shift = (int)(a0 - c0);
    if (c1 > c0) bulk_g2s_hint(dst, src + c0, (unsigned)(c1 - c0), bar, l2_policy_evict_first());
}

__device__ __forceinline__ unsigned b_range_bytes(long long a0, long long a1)
{
    return (unsigned)(((a1 + 15) & ~15ll) - (a0 & ~15ll));
}

// A (chunk, panel) pair: rows [r0, r1) of the system, entries [e0, e1) of
// the panel (relative to its first entry ebase).
struct BChunk {
    int r0, r1, e0, e1, panel;
    long long ebase, rpbase;
};

__device__ __forceinline__ BChunk b_chunk(const BatchArgs &a, int sys, const SysView &v, int c, int k)
{
    BChunk ch;
    ch.r0 = a.crow[c + sys];
    ch.r1 = a.crow[c + 1 + sys];
    ch.panel = k;
    ch.rpbase = a.prow0[v.gp0 + k];
    ch.ebase = a.pent0[v.gp0 + k];
    ch.e0 = a.prow[ch.rpbase + ch.r0];
    ch.e1 = a.prow[ch.rpbase + ch.r1];
    return ch;
}

// Algorithmic bytes of nr rows with ne entries over np panels: vb-byte
// values, 2-byte columns, row pointers, and for FP16 the rows' scales and
// diagonals.
__device__ __forceinline__ unsigned long long pass_bytes(long long ne, int nr, int np, int vb)
{
    return (unsigned long long)ne * (vb + 2) + (unsigned long long)np * ((unsigned)(nr + 1) * 4u + (vb == 2 ? nr * 8u : 0u));
}

// Thread 0: stage pair `ch` into stage k.
__device__ void b_issue(const BatchArgs &a, BSmem &S, const BChunk &ch, int k)
{
    BHdr &h = S.hdr[k];
    const int r0 = ch.r0, r1 = ch.r1, e0 = ch.e0, e1 = ch.e1;
    h.r0 = r0;
    h.r1 = r1;
    h.e0 = e0;
    h.direct = (e1 - e0 > BCE) ? 1 : 0;
    h.panel = ch.panel;
    h.ebase = ch.ebase;
    const long long z0 = ch.ebase;
    unsigned total = b_range_bytes(4 * (ch.rpbase + r0), 4 * (ch.rpbase + r1 + 1));
    if (!h.direct) total += b_range_bytes(8 * (z0 + e0), 8 * (z0 + e1)) + b_range_bytes(2 * (z0 + e0), 2 * (z0 + e1));
    fence_proxy_async_smem();
    mbar_arrive_expect_tx(&S.bar[k], total);
    unsigned char *st = S.stage[k];
    b_add_range(st + Stage::OFF_RP, (const unsigned char *)a.prow, 4 * (ch.rpbase + r0), 4 * (ch.rpbase + r1 + 1),
                &S.bar[k], h.sh_rp);
    if (h.direct) return;
    b_add_range(st + Stage::OFF_COL, (const unsigned char *)a.col, 2 * (z0 + e0), 2 * (z0 + e1), &S.bar[k], h.sh_col);
    b_add_range(st + Stage::OFF_VAL, (const unsigned char *)a.val, 8 * (z0 + e0), 8 * (z0 + e1), &S.bar[k], h.sh_val);
}

// L lanes per row: lanes stride over the row's entries (BU entries per lane
// loaded before any is used); the partials are combined with a fixed xor
// tree, so every run gives the same bits.  Two rows per lane group are in
// flight at once (a row with no entries: bounds 0, 0).
#ifndef MF_BATCH_BU
#define MF_BATCH_BU 4
#endif
constexpr int BU = MF_BATCH_BU;

struct RowPair {
    int a0, e0, a1, e1;
};

// FP64 sums of two rows from global memory.
template <int L, class Src>
__device__ __forceinline__ void row_dot2(const RowPair &rb, const uint16_t *__restrict__ col,
                                         const double *__restrict__ val, int lane, Src src, double &y0, double &y1)
{
    const int a0 = rb.a0, e0 = rb.e0, a1 = rb.a1, e1 = rb.e1;
    double s0 = 0, s1 = 0;
    const int n0 = e0 - a0, n1 = e1 - a1, nmax = n0 > n1 ? n0 : n1;
    for (int k = lane; k < nmax; k += L * BU) {
        int c0[BU], c1[BU];
        double v0[BU], v1[BU];
#pragma unroll
        for (int u = 0; u < BU; u++) {
            const int kk = k + u * L;
            const bool in0 = kk < n0, in1 = kk < n1;
            c0[u] = in0 ? (int)__ldcs(col + a0 + kk) : -1;
            c1[u] = in1 ? (int)__ldcs(col + a1 + kk) : -1;
            v0[u] = in0 ? __ldcs(val + a0 + kk) : 0.0;
            v1[u] = in1 ? __ldcs(val + a1 + kk) : 0.0;
        }
        double x0[BU], x1[BU];
#pragma unroll
        for (int u = 0; u < BU; u++) {
            x0[u] = c0[u] >= 0 ? src(c0[u]) : 0.0;
            x1[u] = c1[u] >= 0 ? src(c1[u]) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < BU; u++) {
            s0 = fma(v0[u], x0[u], s0);
            s1 = fma(v1[u], x1[u], s1);
        }
    }
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
        s0 += __shfl_xor_sync(0xffffffffu, s0, o, L);
        s1 += __shfl_xor_sync(0xffffffffu, s1, o, L);
    }
    y0 = s0;
    y1 = s1;
}

// One row's FP64 sum from a staged pass: lanes stride over the row's
// entries, BU per lane per trip, loaded without predicates -- columns past
// the row's end are read from the stage and masked into the panel, their
// weights are zero.  Lane sums combine in a fixed xor tree.
template <int L, class Src>
__device__ __forceinline__ double row_dot1_smem(int a, int e, const uint16_t *__restrict__ col,
                                                const double *__restrict__ val, int lane, Src src)
{
    double s = 0;
    const int n = e - a;
    for (int k = lane; k < n; k += L * BU) {
#pragma unroll
        for (int u = 0; u < BU; u++) {
            const int kk = k + u * L;
            const int c = (int)col[a + kk] & (PW - 1);
            const double v = kk < n ? val[a + kk] : 0.0;
            s = fma(v, src(c), s);
        }
    }
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, L);
    return s;
}

// FP64 row sums of rows i0, i1 (-1: none) of a system over all its panels,
// read from global memory, panels added in order; x in FP64.
template <int L>
__device__ __forceinline__ void row_dot2_fp64_all(const BatchArgs &a, const SysView &v, const double *xs, int i0,
                                                  int i1, int lane, double &y0, double &y1)
{
    y0 = 0.0;
    y1 = 0.0;
    for (int k = 0; k < v.npan; k++) {
        const long long rpb = a.prow0[v.gp0 + k], eb = a.pent0[v.gp0 + k];
        const int *rp = a.prow + rpb;
        RowPair rr;
        rr.a0 = i0 >= 0 ? rp[i0] : 0;
        rr.e0 = i0 >= 0 ? rp[i0 + 1] : 0;
        rr.a1 = i1 >= 0 ? rp[i1] : 0;
        rr.e1 = i1 >= 0 ? rp[i1 + 1] : 0;
        const double *xk = xs + (long long)k * PW;
        auto src = [=](int c) -> double { return xk[c]; };
        double t0, t1;
        row_dot2<L>(rr, a.col + eb, a.val + eb, lane, src, t0, t1);
        y0 += t0;
        y1 += t1;
    }
}

// ---- chunk classes ----------------------------------------------------------

__device__ __forceinline__ float slog10(float v) { return log10f(fmaxf(v, 1e-30f)); }

// The reference's thresholds on a chunk's largest |p_new - p_old| (FP64),
// mapped to the classes a row chunk can run in.
__device__ __forceinline__ int rule_chunk_class(double v, int stat)
{
    if (stat & 1) return 1;          // exact in FP16
    if (!(stat & 2)) return 0;       // FP16 scales out of range
    return v > 1e-6 ? 0 : 1;         // FP64 / FP32 decisions -> FP32; FP16 / INT8 / BYPASS -> FP16
}

// Checkpoint statistics of chunk c (rows [r0, r1) of a system): maxima of
// |r|, |p_new|, |p_new - p_old|, |q| by one warp, written to cdyn[c][0..3];
// with `label`, also the FP16 perturbation ratio ||dq|| / ||q|| of the
// chunk's rows (dq = A16 p - A p over the off-diagonal entries, in FP64),
// written to cdyn[c][8].  Lane results combine in a fixed tree.
template <typename VT>
__device__ void chunk_stats_warp(const BatchArgs &a, const SysView &v, int c, int r0, int r1, const VT *r,
                                 const VT *pn, const VT *po, const VT *q, const float *rscale, bool label, float &gr,
                                 float &gp)
{
    const int lane = threadIdx.x & 31;
    float mr = 0.f, mp = 0.f, mdp = 0.f, mq = 0.f;
    double num = 0.0, den = 0.0;
    for (int i = r0 + lane; i < r1; i += 32) {
        const double pv = (double)pn[i];
        mr = fmaxf(mr, (float)fabs((double)r[i]));
        mp = fmaxf(mp, (float)fabs(pv));
        mdp = fmaxf(mdp, (float)fabs(pv - (double)po[i]));
        // FP64 solves: q read past L1 (partial sums arrive by reductions in
        // L2); mixed solves: q may be in shared memory
        double qv;
        if constexpr (std::is_same<VT, double>::value) qv = __ldcg(q + i);
        else qv = (double)q[i];
        mq = fmaxf(mq, (float)fabs(qv));
        if (label) {
            const double s = (double)rscale[i];
            double dq = 0.0, qq = 0.0;
            for (int k = 0; k < v.npan; k++) {
                const long long rpb = a.prow0[v.gp0 + k], eb = a.pent0[v.gp0 + k];
                for (int e = a.prow[rpb + i]; e < a.prow[rpb + i + 1]; e++) {
                    const int j = (int)a.col[eb + e] + k * PW;
                    const double pj = (double)pn[j], av = a.val[eb + e];
                    qq = fma(av, pj, qq);
                    if (j != i) dq = fma((double)__half2float(a.val16[eb + e]) * s - av, pj, dq);
                }
            }
            num = fma(dq, dq, num);
            den = fma(qq, qq, den);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mr = fmaxf(mr, __shfl_xor_sync(0xffffffffu, mr, o));
        mp = fmaxf(mp, __shfl_xor_sync(0xffffffffu, mp, o));
        mdp = fmaxf(mdp, __shfl_xor_sync(0xffffffffu, mdp, o));
        mq = fmaxf(mq, __shfl_xor_sync(0xffffffffu, mq, o));
        num += __shfl_xor_sync(0xffffffffu, num, o);
        den += __shfl_xor_sync(0xffffffffu, den, o);
    }
    if (lane == 0) {
        float *d = a.cdyn + (size_t)c * NCDYN;
        d[0] = mr;
        d[1] = mp;
        d[2] = mdp;
        d[3] = mq;
        if (label) d[8] = den > 0.0 ? (float)(sqrt(num) / sqrt(den)) : (num > 0.0 ? 1e30f : 0.f);
    }
    gr = fmaxf(gr, mr);
    gp = fmaxf(gp, mp);
}

// The 16 features of chunk c (lane 0 writes them to x):
//   0-4 static: log10 max|a| / 10, log10 min|a| / 10, entries / 2048,
//       log10 max_i (S_i / m_i) / 10 (S_i the row's off-diagonal |a| sum,
//       m_i = a_ii - S_i its diagonal-dominance margin), log10 of the largest
//       off-diagonal dynamic range of a row / 10
//   5   log10(||r|| / ||b||) / 10
//   6   log10(max_c |r| / max |r|) / 10      7  log10(max_c |p| / max |p|) / 10
//   8   log10(max_c |dp| / max_c |p|) / 10   9  log10(max_c |q| / (max_c |p| max_c |a|)) / 10
//  10-13 features 6-9 at the previous checkpoint (the current ones at the first)
//  14  reliable updates so far / 16          15 1
__device__ __forceinline__ void chunk_features(const BatchArgs &a, int c, float relres, float gr, float gp, int refs,
                                               bool have_prev, float *x)
{
    const float *s = a.cstat + (size_t)c * NCSTAT;
    float *d = a.cdyn + (size_t)c * NCDYN;
    for (int k = 0; k < 5; k++) x[k] = s[k];
    x[5] = slog10(relres) * 0.1f;
    const float amax = s[5];
    x[6] = slog10(gr > 0.f ? d[0] / gr : 0.f) * 0.1f;
    x[7] = slog10(gp > 0.f ? d[1] / gp : 0.f) * 0.1f;
    x[8] = slog10(d[1] > 0.f ? d[2] / d[1] : 0.f) * 0.1f;
    x[9] = slog10(d[1] > 0.f && amax > 0.f ? d[3] / (d[1] * amax) : 0.f) * 0.1f;
    for (int k = 0; k < 4; k++) x[10 + k] = have_prev ? d[4 + k] : x[6 + k];
    x[14] = (float)refs * (1.f / 16.f);
    x[15] = 1.f;
}

// The policy's class for one chunk: one warp evaluates the network (lane j
// holds hidden unit j), in the same operation order as the host-launched
// classifier.  1 = FP16 when P(label <= FP16) >= LEARN_CONF.
__device__ __forceinline__ int learned_chunk_class(const float *w, const float *x, int stat)
{
    float o[PN_NO];
    pn_forward_warp(w, x, o);
    if (stat & 1) return 1;
    if (!(stat & 2)) return 0;
    float mx = o[0];
    for (int k = 1; k < PN_NO; k++) mx = fmaxf(mx, o[k]);
    float e[PN_NO], z = 0.f;
    for (int k = 0; k < PN_NO; k++) {
        e[k] = expf(o[k] - mx);
        z += e[k];
    }
    return (e[0] + e[1] >= LEARN_CONF * z) ? 1 : 0;
}

// The FP64 kernel (the FP64 policy and trace collection): one cluster per
// system; warp 0 stages (chunk, panel) passes, the other warps sum their
// rows, p gathered from global memory.
template <int L>
__global__ void __launch_bounds__(BNT, 1) k_batched_cg64(const __grid_constant__ BatchArgs a)
{
    constexpr int NS = Stage::NS;
    cg::cluster_group cl = cg::this_cluster();
    __shared__ double s_warp[BNW];
    __shared__ double s_slot[8];
    __shared__ float s_fslot[2];
    __shared__ float s_fwarp[2 * BNW];
    __shared__ float s_feat[BNW * PN_NF];
    __shared__ int s_sys;
    __shared__ int s_fail;
    extern __shared__ __align__(16) unsigned char b_smem_raw[];
    BSmem &S = *reinterpret_cast<BSmem *>(b_smem_raw);
    const bool collect = a.collect_every > 0;
    if (threadIdx.x == 0) {
        for (int k = 0; k < NS; k++) {
            mbar_init(&S.bar[k], 1);
            mbar_init(&S.empty[k], BNW - 1);  // the consumer warps
        }
        mbar_fence_init();
    }
    __syncthreads();
    // mbarrier phase parities, one bit per stage (registers: an array indexed
    // by the stage number would live in local memory).  Producer (thread 0):
    // fills of each stage so far (parity) and which stages were filled at
    // all.  Consumers: passes consumed per stage (parity).
    unsigned pfill = 0, pstarted = 0, cfull = 0;
    const unsigned rank = cl.block_rank(), ncta = cl.num_blocks();
    const int tid = threadIdx.x;
    const int wid = tid >> 5, wl = tid & 31;
    for (;;) {
        // after a wait that gave up (status word set) no cluster takes another
        // system: the stages' barrier phases of the failed CTA are not known
        if (rank == 0 && tid == 0) s_sys = ld_volatile_i32(a.queue + 1) != 0 ? a.count : atomicAdd(a.queue, 1);
        cl.sync();
        const int qi = *cl.map_shared_rank(&s_sys, 0);
        cl.sync();  // every CTA has read the index before rank 0 writes the next
        if (qi >= a.count) break;
        const int sys = a.order[qi];
        const SysView V = sys_view(a, sys);
        const long long r0 = V.r0;
        const double *b = a.b + r0;
        double *x = a.x + r0;
        const float *rscale = a.rscale + r0;
        double *r = (double *)a.r + r0, *q = (double *)a.q + r0;
        double *pb[2] = {(double *)a.p0 + r0, (double *)a.p1 + r0};
        // this CTA's chunks and rows
        const int sc0 = a.sc[sys], nch = a.sc[sys + 1] - sc0;
        const int cl0 = sc0 + (int)((long long)nch * rank / ncta), cl1 = sc0 + (int)((long long)nch * (rank + 1) / ncta);
        const int nchl = cl1 - cl0;
        const int ra = a.crow[cl0 + sys], rb = a.crow[cl1 + sys];
        const int npan = V.npan;
        const int J = nchl * npan;  // (chunk, panel) passes per SpMV, panel-major
        unsigned long long st_bytes = 0, st_pass = 0;  // thread 0: passes issued
        double lb = 0.0;
        for (int i = ra + tid; i < rb; i += BNT) {
            const double bv = b[i];
            x[i] = 0.0;
            r[i] = bv;
            pb[0][i] = 0.0;
            lb += bv * bv;
        }
        const double bb = cluster_sum<BNT>(cl, lb, &s_slot[0], s_warp);
        double rho = bb;
        const double nb = sqrt(bb) > 0.0 ? sqrt(bb) : 1.0;
        double beta = 0.0, relres = sqrt(rho) / nb;
        int it = 0, status = MF_OK;
        bool have_prev = false;
        while (true) {
            if (sqrt(rho) <= a.tol * nb) break;
            if (it >= a.maxiter) {
                status = MF_ERR_NOT_CONVERGED;
                break;
            }
            const double *pold = pb[it & 1];
            double *pnew = pb[(it & 1) ^ 1];
            // p = r + beta p over this CTA's rows, then a cluster barrier: the
            // SpMV needs all of p.  Four rows per thread in flight: loads
            // first, then the stores.
            {
                int i = ra + tid;
                for (; i + 3 * BNT < rb; i += 4 * BNT) {
                    double po4[4], r4[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        po4[u] = pold[i + u * BNT];
                        r4[u] = r[i + u * BNT];
                    }
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        pnew[i + u * BNT] = fma(beta, po4[u], r4[u]);
                        if (npan == 2) q[i + u * BNT] = 0.0;
                    }
                }
                for (; i < rb; i += BNT) {
                    pnew[i] = fma(beta, pold[i], r[i]);
                    if (npan == 2) q[i] = 0.0;
                }
            }
            cl.sync();
            double loc = 0.0;
            // SpMV.  Warp 0 produces: its lanes load the descriptors of 32
            // (chunk, panel) passes at a time and lane 0 issues their bulk
            // copies into NS shared-memory stages, each stage refilled once
            // the consumers have released it (empty barrier).  Warps 1..
            // consume: wait for a stage (full barrier), compute its rows,
            // release it -- no CTA-wide barrier per pass.  Every wait is
            // bounded; a failure is voted CTA-wide and cluster-wide below.
            bool fail = false;
            if (J > 0) {
                if (wid == 0) {
                    // descriptors of the next 32 passes load while the current
                    // ones are issued
                    BChunk dn;
                    memset(&dn, 0, sizeof(dn));
                    if (wl < J) dn = b_chunk(a, sys, V, cl0 + wl % nchl, wl / nchl);
                    for (int jb = 0; jb < J && !fail; jb += 32) {
                        const BChunk d = dn;
                        memset(&dn, 0, sizeof(dn));
                        if (jb + 32 + wl < J) dn = b_chunk(a, sys, V, cl0 + (jb + 32 + wl) % nchl, (jb + 32 + wl) / nchl);
                        const int cnt = min(32, J - jb);
                        for (int t = 0; t < cnt; t++) {
                            BChunk ch;
                            ch.r0 = __shfl_sync(0xffffffffu, d.r0, t);
                            ch.r1 = __shfl_sync(0xffffffffu, d.r1, t);
                            ch.e0 = __shfl_sync(0xffffffffu, d.e0, t);
                            ch.e1 = __shfl_sync(0xffffffffu, d.e1, t);
                            ch.panel = __shfl_sync(0xffffffffu, d.panel, t);
                            ch.ebase = __shfl_sync(0xffffffffu, d.ebase, t);
                            ch.rpbase = __shfl_sync(0xffffffffu, d.rpbase, t);
                            const int k = (jb + t) % NS;
                            int ok = 1;
                            if (wl == 0) {
                                if ((pstarted >> k) & 1u)
                                    ok = mbar_wait_sleep_bounded(&S.empty[k], ((pfill >> k) & 1u) ^ 1u, a.queue + 1,
                                                                 a.budget_ns, a.backoff_ns);
                                if (ok) {
                                    b_issue(a, S, ch, k);
                                    pfill ^= 1u << k;
                                    pstarted |= 1u << k;
                                    st_bytes += pass_bytes(ch.e1 - ch.e0, ch.r1 - ch.r0, 1, 8);
                                    st_pass++;
                                }
                            }
                            ok = __shfl_sync(0xffffffffu, ok, 0);
                            if (!ok) {
                                fail = true;
                                break;
                            }
                        }
                    }
                } else {
                    // consumer warps: all of them take every pass, so that a
                    // row's panels are added in panel order
                    constexpr int NCW = BNW - 1;
                    const int ct = (wid - 1) * 32 + wl;         // consumer thread
                    const int clane = ct % L, cgrp = ct / L;
                    constexpr int GPC = NCW * 32 / L;           // row groups
                    for (int j = 0; j < J; j++) {
                        const int k = j % NS;
                        bool w = mbar_wait_sleep_bounded(&S.bar[k], (cfull >> k) & 1u, a.queue + 1, a.budget_ns,
                                                         a.backoff_ns);
                        cfull ^= 1u << k;
                        if (!__all_sync(0xffffffffu, w)) {
                            fail = true;
                            break;
                        }
                        const BHdr &h = S.hdr[k];
                        const unsigned char *st = S.stage[k];
                        const int *rps = (const int *)(st + Stage::OFF_RP + h.sh_rp);  // panel row pointers of h.r0 ..
                        const int nr = h.r1 - h.r0;
                        const bool firstp = h.panel == 0;
                        const double *pk = pnew + (long long)h.panel * PW;
                        auto psrc = [=](int c) -> double { return pk[c]; };
                        const uint16_t *scol = (const uint16_t *)(st + Stage::OFF_COL + h.sh_col);
                        const double *sval = (const double *)(st + Stage::OFF_VAL + h.sh_val);
                        // one row per lane group; the trip count is the same
                        // for every lane of a warp (shuffles inside)
                        for (int qb = 0; qb < nr; qb += GPC) {
                            const int q0 = qb + cgrp;
                            const bool in = q0 < nr;
                            const int ra0 = in ? rps[q0] : 0, re0 = in ? rps[q0 + 1] : 0;
                            double y0;
                            if (h.direct) {
                                RowPair rr{ra0, re0, 0, 0};
                                double y1;
                                row_dot2<L>(rr, a.col + h.ebase, a.val + h.ebase, clane, psrc, y0, y1);
                            } else {
                                y0 = row_dot1_smem<L>(ra0 - h.e0, re0 - h.e0, scol, sval, clane, psrc);
                            }
                            if (clane == 0 && in) {
                                // One panel: the row sum is q; two panels: both
                                // partial sums are added to q (zeroed by the p
                                // update; two additions onto zero give the same
                                // bits in either order); more panels: added in
                                // panel order.
                                double *qi = q + h.r0 + q0;
                                if (npan == 1) *qi = y0;
                                else if (npan == 2) atomicAdd(qi, y0);
                                else *qi = firstp ? y0 : *qi + y0;
                            }
                        }
                        __syncwarp();
                        if (wl == 0) mbar_arrive(&S.empty[k]);
                    }
                }
            }
            // CTA-wide vote; on a failure the producing thread waits (bounded)
            // for the copies it issued that may still be landing
            fail = __syncthreads_or(fail) != 0;
            if (fail && tid == 0) {
                for (int k = 0; k < NS; k++)
                    if ((pstarted >> k) & 1u) mbar_drain(&S.bar[k], ((pfill >> k) & 1u) ^ 1u, a.queue + 1, a.budget_ns);
            }
            if (tid == 0) s_fail = fail ? 1 : 0;
            // p.q over this CTA's rows (q read past L1: partial sums arrive by
            // reductions in L2)
            if (!fail) {
                int i = ra + tid;
                for (; i + 3 * BNT < rb; i += 4 * BNT) {
                    double p4[4], q4[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        p4[u] = pnew[i + u * BNT];
                        q4[u] = __ldcg(q + i + u * BNT);
                    }
#pragma unroll
                    for (int u = 0; u < 4; u++) loc += p4[u] * q4[u];
                }
                for (; i < rb; i += BNT) loc += pnew[i] * __ldcg(q + i);
            }
            const double pq = cluster_sum<BNT>(cl, loc, &s_slot[2], s_warp);
            int any_fail = 0;
            for (unsigned kk = 0; kk < ncta; kk++) any_fail |= *cl.map_shared_rank(&s_fail, kk);
            if (any_fail) {
                status = MF_ERR_TIMEOUT;
                break;
            }
            if (!(pq != 0.0) || !isfinite(pq)) {
                status = MF_ERR_BREAKDOWN;
                break;
            }
            const double alpha = rho / pq;
            loc = 0.0;
            {
                // four rows per thread in flight (loads first)
                int i = ra + tid;
                for (; i + 3 * BNT < rb; i += 4 * BNT) {
                    double p4[4], q4[4], r4[4], x4[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        p4[u] = pnew[i + u * BNT];
                        q4[u] = __ldcg(q + i + u * BNT);
                        r4[u] = r[i + u * BNT];
                        x4[u] = x[i + u * BNT];
                    }
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        x[i + u * BNT] = fma(alpha, p4[u], x4[u]);
                        const double ri = fma(-alpha, q4[u], r4[u]);
                        r[i + u * BNT] = ri;
                        loc += ri * ri;
                    }
                }
                for (; i < rb; i += BNT) {
                    x[i] = fma(alpha, pnew[i], x[i]);
                    const double ri = fma(-alpha, __ldcg(q + i), r[i]);
                    r[i] = ri;
                    loc += ri * ri;
                }
            }
            const double rho_new = cluster_sum<BNT>(cl, loc, &s_slot[3], s_warp);
            it++;
            if (collect && (it % a.collect_every == 1 || a.collect_every == 1)) {
                // checkpoint statistics: one warp per chunk of this CTA, then
                // the system's maxima of |r| and |p| over the cluster
                float gr = 0.f, gp = 0.f;
                for (int c = cl0 + wid; c < cl1; c += BNW)
                    chunk_stats_warp<double>(a, V, c, a.crow[c + sys], a.crow[c + 1 + sys], r, pnew, pold, q, rscale,
                                             true, gr, gp);
                cluster_max2<BNT>(cl, gr, gp, s_fslot, s_fwarp);
                const float rel = (float)(sqrt(rho_new) / nb);
                float *xf = s_feat + wid * PN_NF;
                for (int c = cl0 + wid; c < cl1; c += BNW) {
                    if (wl == 0) {
                        chunk_features(a, c, rel, gr, gp, 0, have_prev, xf);
                        float *d = a.cdyn + (size_t)c * NCDYN;
                        const unsigned h = ((unsigned)c * 2654435761u) ^ (a.collect_salt + (unsigned)it * 0x9E3779B9u);
                        if ((h >> 8) % (unsigned)a.collect_stride == 0u) {
                            const unsigned long long slot = atomicAdd(a.ccount, 1ull);
                            if ((long long)slot < a.ccap) {
                                for (int k = 0; k < PN_NF; k++) a.cx[slot * PN_NF + k] = xf[k];
                                a.cy[slot] = (unsigned char)((double)d[8] <= LABEL_TAU ? 1 : 2);
                            }
                        }
                        for (int k = 0; k < 4; k++) d[4 + k] = xf[6 + k];
                    }
                    __syncwarp();
                }
                have_prev = true;
            }
            beta = rho_new / rho;
            rho = rho_new;
            relres = sqrt(rho) / nb;
        }
        if (tid == 0) {
            atomicAdd(&a.sysstat[3 * sys], st_bytes);
            atomicAdd(&a.sysstat[3 * sys + 2], st_pass);
        }
        if (rank == 0 && tid == 0) {
            a.iters[sys] = it;
            a.refs[sys] = 0;
            a.status[sys] = status;
            a.relres[sys] = relres;
        }
        cl.sync();  // the cluster's last writes land before the next system
    }
}

// The mixed kernel's dynamic shared memory: the window of p and, for a
// system on the chip, from the window's end the vectors r, q, xlo.
extern __shared__ __align__(16) unsigned char mix_smem[];
__device__ __forceinline__ float *mix_win() { return reinterpret_cast<float *>(mix_smem); }

// Distributed shared memory by address: `addr` (of this CTA) in CTA `rank`
// of the cluster, and plain stores to it.
__device__ __forceinline__ unsigned mix_remote(const void *p, int rank)
{
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void mix_put(unsigned addr, float v)
{
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void mix_put(unsigned addr, float4 v)
{
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}

// The mixed kernel's view of the system its cluster is solving.  The CTA's
// own rows are [ra, rb); r, xlo and q are indexed from ra4, ra rounded down
// to a multiple of four (16-byte words of the same rows in every vector).  On
// chip (CHIP below; systems whose window and vectors fit): p is the window
// itself, r, q and xlo follow from its end, p and q reach the other CTAs by
// distributed shared memory.  Otherwise the vectors are in global memory.
struct MixSys {
    int sys, n, ra, rb, ra4, npan;
    int most;               // entries of an on-chip vector (the CTA with most rows)
    bool xwin;              // on chip, and x fits in FP64 beside r and q (reliable updates)
    float *r, *xlo, *q;     // global vectors of this CTA's rows
    float *pnew, *pold;     // global p buffers, indexed by row (on chip: written for LEARNED only)
    int s0, s1;             // this warp's slices (one window)
};

template <bool CHIP>
__device__ __forceinline__ float *mix_r(const MixSys &M) { return CHIP ? mix_win() + SELL_WIN - M.most : M.r; }
template <bool CHIP>
__device__ __forceinline__ float *mix_q(const MixSys &M) { return CHIP ? mix_win() + SELL_WIN - 2 * M.most : M.q; }
template <bool CHIP>
__device__ __forceinline__ float *mix_xlo(const MixSys &M) { return CHIP ? mix_win() + SELL_WIN - 3 * M.most : M.xlo; }

// This warp's share of a window's slices: consecutive bins.
__device__ __forceinline__ void mix_share(const BatchArgs &a, int win, int rank, int ncta, MixSys &M)
{
    const int per = SELL_BINS / (MNW * ncta), b0 = (rank * MNW + (threadIdx.x >> 5)) * per;
    const int *first = a.sell.first + win * (SELL_BINS + 1);
    M.s0 = first[b0];
    M.s1 = first[b0 + per];
}
static_assert(SELL_BINS % (MNW * 16) == 0, "every cluster size deals whole bins");

// Sum over the cluster: warp tree, then warp 0 adds the warps' sums in a
// fixed tree and writes the CTA's value to every CTA's slots (remote
// stores), then after the cluster barrier all add the slots in rank order.
// Two barriers; `slots` is reused only after another cluster barrier.
__device__ __forceinline__ double mix_sum(cg::cluster_group &cl, double v, double *slots, double *s_warp)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int wid = threadIdx.x >> 5, wl = threadIdx.x & 31;
    const int rank = (int)cl.block_rank(), ncta = (int)cl.num_blocks();
    if (wl == 0) s_warp[wid] = v;
    __syncthreads();
    if (wid == 0) {
        double c = wl < MNW ? s_warp[wl] : 0.0;
#pragma unroll
        for (int o = MNW / 2; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        if (wl < ncta) *cl.map_shared_rank(slots + rank, wl) = c;  // lanes below MNW hold the sum
    }
    cl.sync();
    double s = slots[0];
    for (int k = 1; k < ncta; k++) s += slots[k];
    return s;
}
static_assert(MNW <= 32 && MNW >= 16, "a lane per warp in the second step, a lane with the sum per CTA of a cluster");

// The CTA that owns row i (rab: first row of every CTA).
__device__ __forceinline__ int mix_owner(const int *rab, int ncta, int i)
{
    int o = 0;
    for (int k = 1; k < ncta; k++) o += i >= rab[k];
    return o;
}

// q = A p over the sorted slices; returns this thread's part of p.q (one
// window; 0 for several).  mode: 0 every chunk FP32, 1 every chunk FP16, 2
// both kinds.  sync: the cluster barrier that p waits for is still to come
// (the first matrix words load before it).
template <int mode, bool CHIP>
__device__ __noinline__ double mix_spmv(const BatchArgs &a, MixSys M, const int *rab, bool sync)
{
    cg::cluster_group cl = cg::this_cluster();
    const int tid = threadIdx.x, wl = tid & 31;
    const int rank = (int)cl.block_rank(), ncta = (int)cl.num_blocks();
    const int nwin = CHIP ? 1 : sell_windows(M.n), W = sell_width(M.n);
    const int2 *desc = a.sell.desc;
    const int4 *recs = a.sell.rec + wl;
    float *win = mix_win();
    float *q = mix_q<CHIP>(M);
    double loc = 0.0;
    for (int k = 0; k < nwin; k++) {
        const int c0 = k * W, c1 = min(M.n, c0 + W);
        if (nwin > 1) mix_share(a, a.sell.win0[M.sys] + k, rank, ncta, M);
        int4 rec = __ldg(recs + (size_t)M.s0 * 32), recn = rec;
        int2 sd = __ldg(desc + M.s0), sdn = sd;
        // a row's sum: scale, diagonal, store
        auto row = [&](float acc, bool h16, bool lng) {
            if (lng) {  // a long row: its lanes' sums in a fixed tree
                double d = (double)acc;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
                acc = (float)d;
            }
            if (rec.x >= 0 && (!lng || wl == 0)) {
                const int i = rec.x;
                const bool own = i >= c0 && i < c1;  // the diagonal's window
                const float pi = own ? win[i - c0] : 0.f;
                const float y = fmaf(h16 ? __int_as_float(rec.z) : 1.f, acc, own ? __int_as_float(rec.w) * pi : 0.f);
                if (CHIP) {
                    const int o = mix_owner(rab, ncta, i), at = i - (rab[o] & ~3);
                    if (o == rank) q[at] = y;
                    else mix_put(mix_remote(q + at, o), y);
                } else {
                    float *qi = q + (i - M.ra4);
                    *qi = k == 0 ? y : __ldcg(qi) + y;
                }
                if (nwin == 1) loc += (double)pi * (double)y;
            }
        };
        auto window = [&]() {
            if (sync) cl.sync();
            sync = false;
            if (CHIP) return;
            // window: whole 16-byte words (up to three elements past the
            // window's end come from the vector's slack)
            const float4 *src = reinterpret_cast<const float4 *>(M.pnew + c0);
            float4 *dst = reinterpret_cast<float4 *>(win);
            const int nq4 = (c1 - c0 + 3) >> 2;
            int i = tid;
            for (; i + 7 * MNT < nq4; i += 8 * MNT) {
                float4 v[8];
#pragma unroll
                for (int u = 0; u < 8; u++) v[u] = __ldcg(src + i + u * MNT);
#pragma unroll
                for (int u = 0; u < 8; u++) dst[i + u * MNT] = v[u];
            }
            for (; i < nq4; i += MNT) dst[i] = __ldcg(src + i);
            __syncthreads();
        };
        // the warp's slices: the next slice's descriptor, record and first
        // words on their way while a slice is finished
        auto run = [&](auto sum) {
            sum.first(sd.x, M.s0 < M.s1 ? sd.y & 0x7fffffff : 0);
            window();
            for (int s = M.s0; s < M.s1; s++) {
                const int sn = min(s + 1, M.s1 - 1);
                sdn = __ldg(desc + sn);
                recn = __ldg(recs + (size_t)sn * 32);
                const float acc = sum.template sum<float>(sd.x, sd.y & 0x7fffffff, win);
                const bool lng = sd.y < 0;
                sd = sdn;
                sum.first(sd.x, s + 1 < M.s1 ? sd.y & 0x7fffffff : 0);
                row(acc, mode == 1, lng);
                rec = recn;
            }
        };
        if constexpr (mode == 1) {
            run(SellSum<Quad16>(Quad16{a.sell.cv + wl}));
        } else if constexpr (mode == 0) {
            run(SellSum<Quad32>(Quad32{a.sell.v32 + wl, a.sell.c16 + wl}));
        } else {
            window();
            SellSum<Quad16> s16(Quad16{a.sell.cv + wl});
            SellSum<Quad32> s32(Quad32{a.sell.v32 + wl, a.sell.c16 + wl});
            for (int s = M.s0; s < M.s1; s++) {
                rec = __ldg(recs + (size_t)s * 32);
                sd = __ldg(desc + s);
                const int nq = sd.y & 0x7fffffff;
                const bool h = rec.x >= 0 && __ldcg(a.ccls + rec.y) != 0;
                const unsigned m16 = __ballot_sync(0xffffffffu, h);
                const unsigned m32 = __ballot_sync(0xffffffffu, !h && rec.x >= 0);
                float a16 = 0.f, a32 = 0.f;
                if (m16) {
                    s16.first(sd.x, nq);
                    a16 = s16.template sum<float>(sd.x, nq, win);
                }
                if (m32) {
                    s32.first(sd.x, nq);
                    a32 = s32.template sum<float>(sd.x, nq, win);
                }
                row(h ? a16 : a32, h, sd.y < 0);
            }
        }
        // several windows: the next one's sums continue from every warp's
        // q, and the window is overwritten
        if (k + 1 < nwin) cl.sync();
    }
    return loc;
}

// f4(i) for every aligned group of four rows i .. i+3 inside [ra, rb), f1(i)
// for the rows at the two ends.
template <class F4, class F1>
__device__ __forceinline__ void mix_rows(int ra, int rb, F4 f4, F1 f1)
{
    const int tid = threadIdx.x, qa = (ra + 3) >> 2, qb = rb >> 2;
    if (qa < qb) {
        for (int j = qa + tid; j < qb; j += MNT) f4(4 * j);
        const int i = tid < 4 ? ra + tid : 4 * qb + tid - 4;
        if (tid < 4 ? i < 4 * qa : (tid < 8 && i < rb)) f1(i);
    } else {
        for (int i = ra + tid; i < rb; i += MNT) f1(i);
    }
}

// The rare steps, out of line so that the iteration keeps its registers.
// Reliable update: x += xlo, xlo = 0, then (cluster barrier) r = b - A x from
// the FP64 values; returns this thread's part of ||r||^2.  One window: over
// the slices as in the product, x gathered from shared memory where it fits
// beside r and q (the window of p gives way; this CTA's rows of p are kept in
// global memory meanwhile), else from L2 -- there every lane's element is a
// cache line of its own, ~10 times the time.  Several windows: lane groups
// over the rows of the panel storage.
template <int L, bool CHIP>
__device__ __noinline__ double mix_refine(const BatchArgs &a, SysView V, MixSys M, const int *rab, bool psaved)
{
    cg::cluster_group cl = cg::this_cluster();
    const int tid = threadIdx.x, wl = tid & 31;
    const int rank = (int)cl.block_rank(), ncta = (int)cl.num_blocks();
    const double *b = a.b + V.r0;
    double *x = a.x + V.r0;
    float *win = mix_win(), *r = mix_r<CHIP>(M), *xlo = mix_xlo<CHIP>(M);
    const bool xwin = CHIP && M.xwin;
    for (int i = M.ra + tid; i < M.rb; i += MNT) {
        x[i] += (double)xlo[i - M.ra4];
        if (xwin && !psaved) M.pnew[i] = win[i];
    }
    cl.sync();
    double loc = 0.0;
    if (CHIP || sell_windows(M.n) == 1) {
        const double *diag = a.sell.diag64 + V.r0;
        const int2 *desc = a.sell.desc;
        const int4 *recs = a.sell.rec + wl;
        double *xw = reinterpret_cast<double *>(mix_smem);
        if (xwin) {
            int i = tid;
            for (; i + 7 * MNT < M.n; i += 8 * MNT) {
                double v[8];
#pragma unroll
                for (int u = 0; u < 8; u++) v[u] = __ldcg(x + i + u * MNT);
#pragma unroll
                for (int u = 0; u < 8; u++) xw[i + u * MNT] = v[u];
            }
            for (; i < M.n; i += MNT) xw[i] = __ldcg(x + i);
            __syncthreads();
        }
        auto rows = [&](const double *xg) {
            SellSum<Quad64> sum(Quad64{a.sell.v64 + 2 * wl, a.sell.c16 + wl});
            for (int s = M.s0; s < M.s1; s++) {
                const int2 sd = __ldg(desc + s);
                const int i = __ldg(&recs[(size_t)s * 32].x), nq = sd.y & 0x7fffffff;
                sum.first(sd.x, nq);
                double y = sum.template sum<double>(sd.x, nq, xg);
                const bool lng = sd.y < 0;
                if (lng)
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
                if (i >= 0 && (!lng || wl == 0)) {
                    const float rv = (float)(b[i] - fma(diag[i], xg[i], y));
                    if (CHIP) {
                        const int o = mix_owner(rab, ncta, i), at = i - (rab[o] & ~3);
                        if (o == rank) r[at] = rv;
                        else mix_put(mix_remote(r + at, o), rv);
                    } else {
                        r[i - M.ra4] = rv;
                    }
                    loc += (double)rv * (double)rv;
                }
            }
        };
        if (xwin) {
            rows(xw);
            __syncthreads();  // x read
            for (int i = M.ra + tid; i < M.rb; i += MNT) win[i] = M.pnew[i];
        } else {
            rows(x);
        }
    } else {
        const int lane = tid % L, grp = tid / L;
        constexpr int GPB = MNT / L;  // row groups per CTA
        for (int base = M.ra; base < M.rb; base += 2 * GPB) {
            const int i0 = base + grp < M.rb ? base + grp : -1;
            const int i1 = base + GPB + grp < M.rb ? base + GPB + grp : -1;
            double y0, y1;
            row_dot2_fp64_all<L>(a, V, x, i0, i1, lane, y0, y1);
            if (lane == 0) {
                if (i0 >= 0) {
                    const float rv = (float)(b[i0] - y0);
                    r[i0 - M.ra4] = rv;
                    loc += (double)rv * (double)rv;
                }
                if (i1 >= 0) {
                    const float rv = (float)(b[i1] - y1);
                    r[i1 - M.ra4] = rv;
                    loc += (double)rv * (double)rv;
                }
            }
        }
    }
    for (int i = M.ra + tid; i < M.rb; i += MNT) xlo[i - M.ra4] = 0.f;
    return loc;
}

// LEARNED checkpoint: one warp per chunk of this CTA gathers its statistics,
// then, with the system's maxima of |r| and |p| over the cluster, its class.
template <bool CHIP>
__device__ __noinline__ void mix_checkpoint(const BatchArgs &a, SysView V, MixSys M, int cl0, int cl1, float relres,
                                            int refs, bool have_prev, const float *s_w, float *s_feat, float *s_fslot,
                                            float *s_fwarp)
{
    cg::cluster_group cl = cg::this_cluster();
    const int wid = threadIdx.x >> 5, wl = threadIdx.x & 31;
    float gr = 0.f, gp = 0.f;
    for (int c = cl0 + wid; c < cl1; c += MNW) {
        // chunk_stats_warp indexes all vectors alike: from the chunk's first row
        const int r0 = a.crow[c + M.sys], r1 = a.crow[c + 1 + M.sys], at = r0 - M.ra4;
        chunk_stats_warp<float>(a, V, c, 0, r1 - r0, mix_r<CHIP>(M) + at, M.pnew + r0, M.pold + r0, mix_q<CHIP>(M) + at,
                                nullptr, false, gr, gp);
    }
    cluster_max2<MNT>(cl, gr, gp, s_fslot, s_fwarp);
    float *xf = s_feat + wid * PN_NF;
    for (int c = cl0 + wid; c < cl1; c += MNW) {
        if (wl == 0) chunk_features(a, c, relres, gr, gp, refs, have_prev, xf);
        __syncwarp();
        const int cls = learned_chunk_class(s_w, xf, a.ccls_static[c]);
        if (wl == 0) {
            a.ccls[c] = (unsigned char)cls;
            float *d = a.cdyn + (size_t)c * NCDYN;
            for (int k = 0; k < 4; k++) d[4 + k] = xf[6 + k];
        }
        __syncwarp();
    }
}

// p = r + beta p over this CTA's rows, to the window of every CTA (on chip)
// or to global memory.  RULE: one warp per chunk, deciding the chunk's class
// from its own rows' change.
template <bool CHIP>
__device__ __forceinline__ void mix_direction(const BatchArgs &a, cg::cluster_group &cl, const MixSys &M, float bt,
                                              bool by_rule, bool keep, int cl0, int cl1)
{
    const int wid = threadIdx.x >> 5, wl = threadIdx.x & 31, ra4 = M.ra4;
    const int rank = (int)cl.block_rank(), ncta = (int)cl.num_blocks();
    float *win = mix_win();
    const float *po = CHIP ? win : M.pold, *r = mix_r<CHIP>(M);
    auto put1 = [&](int i, float pv) {
        if (CHIP) {
            win[i] = pv;
            for (int k = 1; k < ncta; k++)
                mix_put(mix_remote(win + i, rank + k < ncta ? rank + k : rank + k - ncta), pv);
            if (keep) M.pnew[i] = pv;
        } else {
            M.pnew[i] = pv;
        }
    };
    if (by_rule) {
        for (int c = cl0 + wid; c < cl1; c += MNW) {
            const int i0 = a.crow[c + M.sys], i1 = a.crow[c + 1 + M.sys];
            double v = 0.0;
            for (int i = i0 + wl; i < i1; i += 32) {
                const float old = po[i], pv = fmaf(bt, old, r[i - ra4]);
                put1(i, pv);
                v = fmax(v, fabs((double)pv - (double)old));
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
            if (wl == 0) a.ccls[c] = (unsigned char)rule_chunk_class(v, a.ccls_static[c]);
        }
        return;
    }
    mix_rows(
        M.ra, M.rb,
        [&](int i) {
            const float4 o = *(const float4 *)(po + i), rv = *(const float4 *)(r + (i - ra4));
            const float4 pv = make_float4(fmaf(bt, o.x, rv.x), fmaf(bt, o.y, rv.y), fmaf(bt, o.z, rv.z), fmaf(bt, o.w, rv.w));
            if (CHIP) {
                *(float4 *)(win + i) = pv;
                for (int k = 1; k < ncta; k++)
                    mix_put(mix_remote(win + i, rank + k < ncta ? rank + k : rank + k - ncta), pv);
                if (keep) *(float4 *)(M.pnew + i) = pv;
            } else {
                *(float4 *)(M.pnew + i) = pv;
            }
        },
        [&](int i) { put1(i, fmaf(bt, po[i], r[i - ra4])); });
}

// x += alpha p, r -= alpha q over this CTA's rows (x: the FP32 correction);
// returns this thread's part of ||r||^2.
template <bool CHIP>
__device__ __forceinline__ double mix_update(const MixSys &M, float af)
{
    const int ra4 = M.ra4;
    const float *pn = CHIP ? mix_win() : M.pnew, *q = mix_q<CHIP>(M);
    float *r = mix_r<CHIP>(M), *xlo = mix_xlo<CHIP>(M);
    double loc = 0.0;
    mix_rows(
        M.ra, M.rb,
        [&](int i) {
            const int o = i - ra4;
            const float4 p4 = *(const float4 *)(pn + i), q4 = *(const float4 *)(q + o);
            float4 r4 = *(const float4 *)(r + o), x4 = *(const float4 *)(xlo + o);
            x4 = make_float4(fmaf(af, p4.x, x4.x), fmaf(af, p4.y, x4.y), fmaf(af, p4.z, x4.z), fmaf(af, p4.w, x4.w));
            r4 = make_float4(fmaf(-af, q4.x, r4.x), fmaf(-af, q4.y, r4.y), fmaf(-af, q4.z, r4.z), fmaf(-af, q4.w, r4.w));
            *(float4 *)(xlo + o) = x4;
            *(float4 *)(r + o) = r4;
            loc += (double)r4.x * (double)r4.x;
            loc += (double)r4.y * (double)r4.y;
            loc += (double)r4.z * (double)r4.z;
            loc += (double)r4.w * (double)r4.w;
        },
        [&](int i) {
            const int o = i - ra4;
            xlo[o] = fmaf(af, pn[i], xlo[o]);
            const float ri = fmaf(-af, q[o], r[o]);
            r[o] = ri;
            loc += (double)ri * (double)ri;
        });
    return loc;
}

// Shared memory of a mixed CTA beside the window.
struct MixShared {
    double warp[MNW];
    double slot[4][16];
    float fslot[2];
    float fwarp[2 * MNW];
    int sys;
    int rab[17];  // first row of every CTA of the cluster
};

// One system, by the whole cluster.
template <int L, bool CHIP>
__device__ __noinline__ void mix_solve(const BatchArgs &a, MixShared &S, SysView V, MixSys M, int sc0, int nch)
{
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), ncta = (int)cl.num_blocks(), tid = threadIdx.x;
    float *s_w = reinterpret_cast<float *>(mix_smem + MixSmem::W), *s_feat = reinterpret_cast<float *>(mix_smem + MixSmem::FEAT);
    const bool learned = a.policy == MF_POLICY_LEARNED && a.mlp_w;
    const bool rule = a.policy == MF_POLICY_RULE;
    const double *b = a.b + V.r0;
    double *x = a.x + V.r0;
    const int sys = M.sys, nwin = CHIP ? 1 : sell_windows(V.n);
    const int ra = M.ra, rb = M.rb, ra4 = M.ra4;
    const int cl0 = sc0 + (int)((long long)nch * rank / ncta), cl1 = sc0 + (int)((long long)nch * (rank + 1) / ncta);
    unsigned long long st_bytes = 0, it_bytes = 0;  // this thread's chunks: in all, per iteration by the current classes
    unsigned it_lowp = 0, it_pass = 0;
    unsigned long long st_lowp = 0, st_pass = 0;
    double lb = 0.0, lr = 0.0;
    {
        float *r = mix_r<CHIP>(M), *xlo = mix_xlo<CHIP>(M);
        for (int i = ra + tid; i < rb; i += MNT) {
            const double bv = b[i];
            const float rv = (float)bv;
            x[i] = 0.0;
            r[i - ra4] = rv;
            xlo[i - ra4] = 0.f;
            M.pnew[i] = 0.f;  // p before the first iteration
            if (CHIP) mix_win()[i] = 0.f;
            lb += bv * bv;
            lr += (double)rv * (double)rv;
        }
    }
    for (int c = cl0 + tid; c < cl1; c += MNT) a.ccls[c] = (a.ccls_static[c] & 1) ? 1 : 0;
    const double bb = mix_sum(cl, lb, S.slot[0], S.warp);
    double rho = mix_sum(cl, lr, S.slot[1], S.warp);
    const double nb = sqrt(bb) > 0.0 ? sqrt(bb) : 1.0;
    double beta = 0.0, rmax = sqrt(rho), relres = sqrt(rho) / nb;
    int it = 0, refs = 0, status = MF_OK, mode = 0;
    bool lowp_off = false, have_prev = false, dirty = true;  // dirty: classes written since `mode` was found
    while (true) {
        if (sqrt(rho) <= a.tol * nb) break;
        if (it >= a.maxiter) {
            status = MF_ERR_NOT_CONVERGED;
            break;
        }
        {
            float *t = M.pold;
            M.pold = M.pnew;
            M.pnew = t;
        }
        const bool by_rule = rule && !lowp_off;
        mix_direction<CHIP>(a, cl, M, (float)beta, by_rule, learned, cl0, cl1);
        // a cluster barrier: the product needs all of p (mix_spmv has it
        // where the classes are known)
        const bool sync = !dirty && !by_rule;
        if (!sync) {
            cl.sync();
            // the classes of the system's chunks: all FP16, all FP32 or both
            bool c16 = true, c32 = true;
            it_bytes = 0;
            it_lowp = it_pass = 0;
            for (int c = sc0 + tid; c < sc0 + nch; c += MNT) {
                const bool h = __ldcg(a.ccls + c) != 0;
                c16 &= h;
                c32 &= !h;
                if (c >= cl0 && c < cl1) {
                    it_bytes += pass_bytes(a.cent[c + 1 + sys] - a.cent[c + sys], a.crow[c + 1 + sys] - a.crow[c + sys],
                                           M.npan, h ? 2 : 4);
                    it_lowp += h ? M.npan : 0;
                    it_pass += M.npan;
                }
            }
            mode = __syncthreads_and(c16) ? 1 : __syncthreads_and(c32) ? 0 : 2;
            dirty = false;
        }
        st_bytes += it_bytes;
        st_lowp += it_lowp;
        st_pass += it_pass;
        double loc = mode == 1   ? mix_spmv<1, CHIP>(a, M, S.rab, sync)
                     : mode == 0 ? mix_spmv<0, CHIP>(a, M, S.rab, sync)
                                 : mix_spmv<2, CHIP>(a, M, S.rab, sync);
        if (nwin > 1) {
            cl.sync();
            for (int i = ra + tid; i < rb; i += MNT) loc += (double)M.pnew[i] * (double)__ldcg(M.q + i - ra4);
        }
        const double pq = mix_sum(cl, loc, S.slot[2], S.warp);
        if (!(pq != 0.0) || !isfinite(pq)) {
            status = MF_ERR_BREAKDOWN;
            break;
        }
        const double alpha = rho / pq;
        loc = mix_update<CHIP>(M, (float)alpha);
        double rho_new = mix_sum(cl, loc, S.slot[3], S.warp);
        it++;
        bool checkpoint = learned && !lowp_off && it == 1;
        if (sqrt(rho_new) <= a.delta * rmax || sqrt(rho_new) <= a.tol * nb) {
            loc = mix_refine<L, CHIP>(a, V, M, S.rab, learned);
            rho_new = mix_sum(cl, loc, S.slot[1], S.warp);
            const double rt = sqrt(rho_new);
            // the low-precision classes stop where the FP64 residual did
            // not follow the recurrence (uniform: every CTA holds the same
            // cluster sums)
            if ((rule || learned) && !lowp_off && rt > 0.5 * rmax) {
                lowp_off = true;
                dirty = true;
                for (int c = cl0 + tid; c < cl1; c += MNT) a.ccls[c] = (a.ccls_static[c] & 1) ? 1 : 0;
            }
            rmax = rt;
            refs++;
            checkpoint = learned && !lowp_off;
        }
        if (checkpoint) {
            mix_checkpoint<CHIP>(a, V, M, cl0, cl1, (float)(sqrt(rho_new) / nb), refs, have_prev, s_w, s_feat, S.fslot,
                                 S.fwarp);
            have_prev = true;
            dirty = true;
        }
        beta = rho_new / rho;
        rho = rho_new;
        relres = sqrt(rho) / nb;
    }
    if (status != MF_OK) {
        const float *xlo = mix_xlo<CHIP>(M);
        for (int i = ra + tid; i < rb; i += MNT) x[i] += (double)xlo[i - ra4];
    }
    if (st_pass) {
        atomicAdd(&a.sysstat[3 * sys], st_bytes);
        atomicAdd(&a.sysstat[3 * sys + 1], st_lowp);
        atomicAdd(&a.sysstat[3 * sys + 2], st_pass);
    }
    if (rank == 0 && tid == 0) {
        a.iters[sys] = it;
        a.refs[sys] = refs;
        a.status[sys] = status;
        a.relres[sys] = relres;
    }
}

// The mixed kernel (STATIC, RULE, LEARNED): one cluster per system, FP32
// vectors.  The product q = A p runs over the sorted slices: every CTA holds
// the window of p in shared memory, the slices are dealt to the cluster's
// warps longest first (so all warps get nearly equal work whatever the row
// order), a lane sums one row from 16-byte words that stream from L2/HBM
// straight into registers, the gathers hit shared memory.  A system whose
// window and vectors fit keeps them on the chip for the whole solve.
template <int L>
__global__ void __launch_bounds__(MNT, 1) k_batched_cg(const __grid_constant__ BatchArgs a)
{
    cg::cluster_group cl = cg::this_cluster();
    __shared__ MixShared S;
    if (a.policy == MF_POLICY_LEARNED && a.mlp_w) {
        float *s_w = reinterpret_cast<float *>(mix_smem + MixSmem::W);
        for (int k = threadIdx.x; k < PN_NPARAM; k += MNT) s_w[k] = __bfloat162float(a.mlp_w[k]);
    }
    __syncthreads();
    const int rank = (int)cl.block_rank(), ncta = (int)cl.num_blocks(), tid = threadIdx.x;
    for (;;) {
        if (rank == 0 && tid == 0) S.sys = atomicAdd(a.queue, 1);
        cl.sync();
        const int qi = *cl.map_shared_rank(&S.sys, 0);
        cl.sync();  // every CTA has read the index before rank 0 writes the next
        if (qi >= a.count) break;
        const int sys = a.order[qi];
        const SysView V = sys_view(a, sys);
        // the CTAs' rows: whole chunks
        const int sc0 = a.sc[sys], nch = a.sc[sys + 1] - sc0;
        if (tid <= ncta) S.rab[tid] = a.crow[sc0 + (int)((long long)nch * tid / ncta) + sys];
        __syncthreads();
        int most = 0;
        for (int k = 0; k < ncta; k++) most = max(most, S.rab[k + 1] - (S.rab[k] & ~3));
        MixSys M;
        M.sys = sys;
        M.n = V.n;
        M.ra = S.rab[rank];
        M.rb = S.rab[rank + 1];
        M.ra4 = M.ra & ~3;
        M.npan = V.npan;
        M.most = (most + 3) & ~3;
        const int n4 = (V.n + 3) & ~3;
        const bool chip = n4 + 3 * M.most <= SELL_WIN;
        M.xwin = 2 * n4 + 2 * M.most <= SELL_WIN;
        M.s0 = M.s1 = 0;
        if (sell_windows(V.n) == 1) mix_share(a, a.sell.win0[sys], rank, ncta, M);
        // global vectors: every system starts on a 16-byte boundary
        const long long w0 = ((V.r0 + 4ll * sys) >> 2) << 2;
        M.pnew = (float *)a.p0 + w0;
        M.pold = (float *)a.p1 + w0;
        M.r = (float *)a.r + w0 + M.ra4;
        M.xlo = (float *)a.xlo + w0 + M.ra4;
        M.q = (float *)a.q + w0 + M.ra4;
        if (chip) mix_solve<L, true>(a, S, V, M, sc0, nch);
        else mix_solve<L, false>(a, S, V, M, sc0, nch);
        cl.sync();  // the cluster's last writes land before the next system
    }
}

// One CTA per system: the LEARNED classes for given FP64 vectors (the
// classifier of the solve, run outside it so that its decisions can be
// checked).  Every chunk of the system is classified.
__global__ void __launch_bounds__(BNT) k_batch_classify(BatchArgs a, const double *r, const double *pn,
                                                        const double *po, const double *q, const double *relres,
                                                        const int *refs, int have_prev, unsigned char *out,
                                                        float *feat_out)
{
    __shared__ float s_w[PN_NPARAM];
    __shared__ float s_feat[BNW * PN_NF];
    __shared__ float s_m[2 * BNW];
    for (int k = threadIdx.x; k < PN_NPARAM; k += BNT) s_w[k] = __bfloat162float(a.mlp_w[k]);
    __syncthreads();
    const int wid = threadIdx.x >> 5, wl = threadIdx.x & 31;
    for (int sys = blockIdx.x; sys < a.count; sys += gridDim.x) {
        const SysView V = sys_view(a, sys);
        const long long r0 = V.r0;
        const int sc0 = a.sc[sys], sc1 = a.sc[sys + 1];
        float gr = 0.f, gp = 0.f;
        for (int c = sc0 + wid; c < sc1; c += BNW)
            chunk_stats_warp<double>(a, V, c, a.crow[c + sys], a.crow[c + 1 + sys], r + r0, pn + r0, po + r0, q + r0,
                                     a.rscale + r0, false, gr, gp);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            gr = fmaxf(gr, __shfl_xor_sync(0xffffffffu, gr, o));
            gp = fmaxf(gp, __shfl_xor_sync(0xffffffffu, gp, o));
        }
        __syncthreads();
        if (wl == 0) {
            s_m[2 * wid] = gr;
            s_m[2 * wid + 1] = gp;
        }
        __syncthreads();
        gr = gp = 0.f;
        for (int w = 0; w < BNW; w++) {
            gr = fmaxf(gr, s_m[2 * w]);
            gp = fmaxf(gp, s_m[2 * w + 1]);
        }
        float *xf = s_feat + wid * PN_NF;
        for (int c = sc0 + wid; c < sc1; c += BNW) {
            if (wl == 0) chunk_features(a, c, (float)relres[sys], gr, gp, refs[sys], have_prev != 0, xf);
            __syncwarp();
            const int cls = learned_chunk_class(s_w, xf, a.ccls_static[c]);
            if (wl == 0) {
                out[c] = (unsigned char)cls;
                if (feat_out)
                    for (int k = 0; k < PN_NF; k++) feat_out[(size_t)c * PN_NF + k] = xf[k];
                float *d = a.cdyn + (size_t)c * NCDYN;
                for (int k = 0; k < 4; k++) d[4 + k] = xf[6 + k];
            }
            __syncwarp();
        }
        __syncthreads();
    }
}

// The kernel of a policy kind: entry point, threads, dynamic shared memory.
struct BatchKernel {
    void (*fn)(const BatchArgs);
    int threads;
    size_t smem;
};

BatchKernel batch_kernel(bool mixed, int lanes)
{
    switch (lanes) {
    case 4: return mixed ? BatchKernel{k_batched_cg<4>, MNT, MixSmem::TOTAL} : BatchKernel{k_batched_cg64<4>, BNT, sizeof(BSmem)};
    case 8: return mixed ? BatchKernel{k_batched_cg<8>, MNT, MixSmem::TOTAL} : BatchKernel{k_batched_cg64<8>, BNT, sizeof(BSmem)};
    case 16: return mixed ? BatchKernel{k_batched_cg<16>, MNT, MixSmem::TOTAL} : BatchKernel{k_batched_cg64<16>, BNT, sizeof(BSmem)};
    default: return mixed ? BatchKernel{k_batched_cg<32>, MNT, MixSmem::TOTAL} : BatchKernel{k_batched_cg64<32>, BNT, sizeof(BSmem)};
    }
}

int batched_ctas(bool mixed, int lanes, int count, int cluster)
{
    const BatchKernel k = batch_kernel(mixed, lanes);
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // clusters of 16 CTAs are above the portable size: allowed explicitly
    if (cluster > 8) cudaFuncSetAttribute(k.fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k.fn, k.threads, k.smem);
    int ctas = sms * (per > 0 ? per : 1);
    ctas = (ctas / cluster) * cluster;
    const int want = count * cluster;
    if (ctas > want) ctas = want;
    if (ctas < cluster) ctas = cluster;
    return ctas;
}

struct BatchConfig {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
};

void batch_config(BatchConfig &c, const BatchKernel &k, int cluster, int ctas, cudaStream_t s)
{
    memset(&c, 0, sizeof(c));
    c.attr[0].id = cudaLaunchAttributeClusterDimension;
    c.attr[0].val.clusterDim.x = cluster;
    c.attr[0].val.clusterDim.y = 1;
    c.attr[0].val.clusterDim.z = 1;
    c.cfg.blockDim = dim3(k.threads);
    c.cfg.dynamicSmemBytes = k.smem;
    c.cfg.stream = s;
    c.cfg.attrs = c.attr;
    c.cfg.numAttrs = 1;
    c.cfg.gridDim = dim3(ctas);
}

// ctas: computed before any stream capture (batched_ctas); enough clusters to
// fill the GPU (the work queue balances them)
mf_status launch_batched(bool mixed, int lanes, const BatchArgs &a, int cluster, int ctas, cudaStream_t s)
{
    const BatchKernel k = batch_kernel(mixed, lanes);
    BatchConfig c;
    batch_config(c, k, cluster, ctas, s);
    note_launch();
    MF_CUDA(cudaLaunchKernelEx(&c.cfg, k.fn, a));
    return MF_OK;
}

// One CTA per system: ||b - A x|| / ||b|| in FP64 (panels added in order
// per row).
__global__ void k_batch_resid(BatchArgs a, const double *b, const double *x, double *out)
{
    __shared__ double s_warp[8];
    for (int sys = blockIdx.x; sys < a.count; sys += gridDim.x) {
        const SysView V = sys_view(a, sys);
        double rr = 0.0, bb = 0.0;
        for (int i = threadIdx.x; i < V.n; i += blockDim.x) {
            double y = 0.0;
            for (int k = 0; k < V.npan; k++) {
                const long long rpb = a.prow0[V.gp0 + k], eb = a.pent0[V.gp0 + k];
                double t = 0.0;
                for (int e = a.prow[rpb + i]; e < a.prow[rpb + i + 1]; e++)
                    t += a.val[eb + e] * x[V.r0 + (long long)k * PW + a.col[eb + e]];
                y += t;
            }
            const double d = b[V.r0 + i] - y;
            rr += d * d;
            bb += b[V.r0 + i] * b[V.r0 + i];
        }
        rr = block_sum<256>(rr, s_warp);
        bb = block_sum<256>(bb, s_warp);
        if (threadIdx.x == 0) out[sys] = bb > 0 ? sqrt(rr) / sqrt(bb) : sqrt(rr);
        __syncthreads();
    }
}

// Per row of every system (one CTA per system): the row-scaled FP16 copy with
// the diagonal taken out, the row scale and the
// FP32 diagonal, and the row statistics the chunk features use.
// Row scale: 2^(e - 14) with e the exponent of the largest off-diagonal
// magnitude; rows whose scale leaves FP32's normal range, or whose diagonal
// does not fit FP32, are marked not FP16-capable.
__global__ void k_batch_rows(BatchArgs a, __half *val16, float *rscale, float *diag32, double *diag64,
                             float4 *rowstat, unsigned char *rowflag)
{
    for (int sys = blockIdx.x; sys < a.count; sys += gridDim.x) {
        const SysView V = sys_view(a, sys);
        for (int i = threadIdx.x; i < V.n; i += blockDim.x) {
            double offmax = 0.0, offmin = 0.0, S = 0.0, d = 0.0, amin = 0.0;
            for (int k = 0; k < V.npan; k++) {
                const long long rpb = a.prow0[V.gp0 + k], eb = a.pent0[V.gp0 + k];
                for (int e = a.prow[rpb + i]; e < a.prow[rpb + i + 1]; e++) {
                    const double v = a.val[eb + e], av = fabs(v);
                    if (av > 0.0 && (amin == 0.0 || av < amin)) amin = av;
                    if ((int)a.col[eb + e] + k * PW == i) {
                        d += v;
                    } else {
                        S += av;
                        if (av > offmax) offmax = av;
                        if (av > 0.0 && (offmin == 0.0 || av < offmin)) offmin = av;
                    }
                }
            }
            const int e = offmax > 0.0 ? ilogb(offmax) - 14 : 0;
            const bool ok = e >= -126 && e <= 127 && isfinite(d) && fabs(d) <= 3.0e38;
            bool exact = ok && (double)(float)d == d;
            for (int k = 0; k < V.npan; k++) {
                const long long rpb = a.prow0[V.gp0 + k], eb = a.pent0[V.gp0 + k];
                for (int q = a.prow[rpb + i]; q < a.prow[rpb + i + 1]; q++) {
                    const double v = a.val[eb + q];
                    __half h = __float2half_rn(0.f);
                    if (ok && (int)a.col[eb + q] + k * PW != i) {
                        h = __double2half(ldexp(v, -e));
                        if ((double)__half2float(h) * ldexp(1.0, e) != v) exact = false;
                    }
                    val16[eb + q] = h;
                }
            }
            rscale[V.r0 + i] = ok ? ldexpf(1.f, e) : 0.f;
            diag32[V.r0 + i] = (float)d;
            diag64[V.r0 + i] = d;
            const double margin = d - S;
            rowstat[V.r0 + i] = make_float4((float)fmax(offmax, fabs(d)), (float)amin,
                                            (float)(S / fmax(margin, 1e-30 * fmax(S, 1e-300))),
                                            offmin > 0.0 ? (float)(offmax / offmin) : 1.f);
            rowflag[V.r0 + i] = (unsigned char)((exact ? 1 : 0) | (ok ? 2 : 0));
        }
    }
}

__global__ void k_batch_cast32(long long n, const double *v, float *out)
{
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        out[e] = (float)v[e];
}

// Per chunk (one warp per chunk, one CTA per system): the static class byte
// (bit 0 every row exact in FP16, bit 1 every row FP16-capable) and the
// static features.
__global__ void k_batch_chunks(int count, const long long *row0, const int *sc, const int *crow, const int *cent,
                               const float4 *rowstat, const unsigned char *rowflag, unsigned char *ccls_static,
                               float *cstat)
{
    const int wid = threadIdx.x >> 5, wl = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int sys = blockIdx.x; sys < count; sys += gridDim.x) {
        const long long r0 = row0[sys];
        for (int c = sc[sys] + wid; c < sc[sys + 1]; c += nw) {
            const int c0 = crow[c + sys], c1 = crow[c + 1 + sys];
            float amax = 0.f, amin = 3e38f, dd = 0.f, rng = 1.f;
            unsigned flag = 3u;
            for (int i = c0 + wl; i < c1; i += 32) {
                const float4 st = rowstat[r0 + i];
                amax = fmaxf(amax, st.x);
                if (st.y > 0.f) amin = fminf(amin, st.y);
                dd = fmaxf(dd, st.z);
                rng = fmaxf(rng, st.w);
                flag &= rowflag[r0 + i];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
                amin = fminf(amin, __shfl_xor_sync(0xffffffffu, amin, o));
                dd = fmaxf(dd, __shfl_xor_sync(0xffffffffu, dd, o));
                rng = fmaxf(rng, __shfl_xor_sync(0xffffffffu, rng, o));
                flag &= __shfl_xor_sync(0xffffffffu, flag, o);
            }
            if (wl == 0) {
                ccls_static[c] = (unsigned char)flag;
                float *s = cstat + (size_t)c * NCSTAT;
                s[0] = slog10(amax) * 0.1f;
                s[1] = slog10(amin < 3e38f ? amin : 0.f) * 0.1f;
                s[2] = (float)(cent[c + 1 + sys] - cent[c + sys]) * (1.f / 2048.f);
                s[3] = slog10(dd) * 0.1f;
                s[4] = slog10(rng) * 0.1f;
                s[5] = amax;
            }
        }
    }
}

// Host: panel-major storage of one system.  Entries of row i in panel k
// (columns [k PW, (k+1) PW)) keep their order within the row; chunks are
// row ranges of at most BCR rows with at most BCE entries in every panel (a
// row with more is a chunk of its own).
struct HostSys {
    int np = 0;
    std::vector<int> prow;          // np x (n + 1)
    std::vector<long long> pnz;     // entries per panel
    std::vector<uint16_t> col;      // panel-major
    std::vector<double> val;
    std::vector<int> crow, cent;    // chunk row starts (n at the end), scanned entries
};

void host_panels(int n, const int *rp, const int *ci, const double *v, HostSys &h)
{
    const int np = (n + PW - 1) / PW;
    h.np = np;
    h.prow.assign((size_t)np * (n + 1), 0);
    h.pnz.assign(np, 0);
    for (int i = 0; i < n; i++)
        for (int k = rp[i]; k < rp[i + 1]; k++) h.prow[(size_t)(ci[k] / PW) * (n + 1) + i + 1]++;
    long long base = 0;
    std::vector<long long> pbase(np);
    for (int k = 0; k < np; k++) {
        int *p = &h.prow[(size_t)k * (n + 1)];
        for (int i = 0; i < n; i++) p[i + 1] += p[i];
        h.pnz[k] = p[n];
        pbase[k] = base;
        base += p[n];
    }
    h.col.resize((size_t)base);
    h.val.resize((size_t)base);
    std::vector<int> fill((size_t)np);
    for (int i = 0; i < n; i++) {
        for (int k = 0; k < np; k++) fill[k] = h.prow[(size_t)k * (n + 1) + i];
        for (int e = rp[i]; e < rp[i + 1]; e++) {
            const int k = ci[e] / PW;
            const long long at = pbase[k] + fill[k]++;
            h.col[(size_t)at] = (uint16_t)(ci[e] - k * PW);
            h.val[(size_t)at] = v[e];
        }
    }
    // chunks
    h.crow.clear();
    h.cent.clear();
    int r = 0;
    long long ent = 0;
    while (r < n) {
        h.crow.push_back(r);
        h.cent.push_back((int)ent);
        const int r_start = r;
        r++;
        auto fits = [&](int r1) {
            for (int k = 0; k < np; k++) {
                const int *p = &h.prow[(size_t)k * (n + 1)];
                if (p[r1] - p[r_start] > BCE) return false;
            }
            return true;
        };
        while (r < n && r - r_start < BCR && fits(r + 1)) r++;
        ent += rp[r] - rp[r_start];
    }
    h.crow.push_back(n);
    h.cent.push_back((int)ent);
}

}  // namespace
}  // namespace mf

using namespace mf;

namespace {

template <typename F>
void parallel_for(int count, F f)
{
    const int nt = std::max(1, std::min<int>(16, (int)std::thread::hardware_concurrency()));
    std::vector<std::thread> th;
    std::atomic<int> next{0};
    for (int t = 0; t < nt; t++)
        th.emplace_back([&]() {
            for (int s = next++; s < count; s = next++) f(s);
        });
    for (auto &t : th) t.join();
}

// The sorted slices of every system (after k_batch_rows): row lengths,
// slices per window, a stable sort, the slices' storage, the entries.
cudaError_t batch_slices(mf_batch bt)
{
    const int count = bt->count;
    std::vector<long long> len0;
    long long lens = 0;
    for (int s = 0; s < count; s++) {
        for (int k = 0; k < sell_windows(bt->n[s]); k++) {
            len0.push_back(lens);
            lens += bt->n[s];
        }
    }
    const int windows = (int)len0.size();
    cudaError_t e = cudaSuccess;
    // temporaries: len0 | row lengths | slices per window | long rows | first slices
    char *tmp = nullptr;
    int *quads = nullptr, *quad0 = nullptr;
    const size_t o_len = sizeof(long long) * windows, o_ns = o_len + sizeof(int) * (size_t)lens,
                 o_nl = o_ns + sizeof(int) * (windows + 1), o_f = o_nl + sizeof(int) * windows,
                 bytes = o_f + sizeof(int) * (windows + 1);
    int nslices = 0, nquads = 0;
    SellBuild B;
    memset(&B, 0, sizeof(B));
    auto pad = [](size_t v) { return (v + 255) / 256 * 256; };
    do {
        if ((e = pool_malloc_async(&tmp, bytes, 0)) != cudaSuccess) break;
        if ((e = cudaMemcpy(tmp, len0.data(), sizeof(long long) * windows, cudaMemcpyHostToDevice)) != cudaSuccess) break;
        int *len = (int *)(tmp + o_len), *ns = (int *)(tmp + o_ns), *nl = (int *)(tmp + o_nl), *first = (int *)(tmp + o_f);
        B.count = count;
        B.pw = PW;
        B.n = bt->d_n;
        B.pan0 = bt->d_pan0;
        B.win0 = bt->d_win0;
        B.row0 = bt->d_row0;
        B.prow0 = bt->d_prow0;
        B.pent0 = bt->d_pent0;
        B.len0 = (const long long *)tmp;
        B.sc = bt->d_sc;
        B.crow = bt->d_crow;
        B.prow = bt->d_prow;
        B.col = bt->d_col;
        B.val = bt->d_val;
        B.val16 = bt->d_val16;
        B.rscale = bt->d_rscale;
        B.diag32 = bt->d_diag32;
        const int gw = std::min(windows, 4096);
        k_sell_lengths<<<dim3(gw, 16), SELL_NT>>>(B, windows, len);
        k_sell_slices<<<gw, SELL_NT>>>(B, windows, len, ns, nl);
        note_launch(2);
        if ((e = cudaMemsetAsync(ns + windows, 0, sizeof(int), 0)) != cudaSuccess) break;
        if (exclusive_scan_i32(ns, first, windows + 1, 0, &nslices) != MF_OK) {
            e = cudaErrorUnknown;
            break;
        }
        // bins | descriptors | records
        const size_t o_desc = pad(sizeof(int) * (size_t)windows * (SELL_BINS + 1)),
                     o_rec = o_desc + pad(sizeof(int2) * ((size_t)nslices + 1)),
                     s_bytes = o_rec + sizeof(int4) * 32 * ((size_t)nslices + 2);
        if ((e = cudaMalloc(&bt->slices, s_bytes)) != cudaSuccess) break;
        bt->d_sfirst = (int *)bt->slices;
        bt->d_sdesc = (int2 *)((char *)bt->slices + o_desc);
        bt->d_srec = (int4 *)((char *)bt->slices + o_rec);
        if ((e = pool_malloc_async(&quads, sizeof(int) * 2 * ((size_t)nslices + 1), 0)) != cudaSuccess) break;
        quad0 = quads + nslices + 1;
        k_sell_sort<<<std::min(windows, 148 * 32), 32>>>(B, windows, len, nl, first, bt->d_srec, quads, bt->d_sfirst);
        k_sell_counts<<<std::min(nslices / SELL_NT + 1, 1184), SELL_NT>>>(nslices, quads, quad0);
        note_launch(2);
        if (exclusive_scan_i32(quad0, quad0, nslices + 1, 0, &nquads) != MF_OK) {
            e = cudaErrorUnknown;
            break;
        }
        // FP64 values | FP32 values | FP16 words | columns
        const size_t words = ((size_t)nquads + 1) * 128;
        if ((e = cudaMalloc(&bt->words, 18 * words)) != cudaSuccess) break;
        bt->d_sv64 = (double *)bt->words;
        bt->d_sv32 = (float *)(bt->d_sv64 + words);
        bt->d_scv = (uint32_t *)(bt->d_sv32 + words);
        bt->d_sc16 = (uint16_t *)(bt->d_scv + words);
        if ((e = cudaMemsetAsync(bt->words, 0, 18 * words, 0)) != cudaSuccess) break;
        k_sell_fill<<<std::min((nslices + SELL_FNT / 32 - 1) / (SELL_FNT / 32), 148 * 64), SELL_FNT>>>(
            B, windows, first, bt->d_srec, quads, quad0, nslices, bt->d_sdesc, bt->d_scv, bt->d_sv32, bt->d_sc16,
            bt->d_sv64);
        note_launch();
        e = cudaGetLastError();
    } while (false);
    if (tmp) cudaFreeAsync(tmp, 0);
    if (quads) cudaFreeAsync(quads, 0);
    // (not the device: that is not permitted while another thread captures)
    if (e == cudaSuccess) e = cudaStreamSynchronize(0);
    return e;
}

}  // namespace

extern "C" {

mf_status mf_batch_create(int count, const int *n, const int *const *rowptr, const int *const *colidx,
                          const double *const *val, mf_batch *out)
{
    if (!out || count <= 0 || !n || !rowptr || !colidx || !val) return MF_ERR_INVALID_ARG;
    *out = nullptr;
    mf_batch bt = new mf_batch_s();
    bt->count = count;
    bt->n.assign(n, n + count);
    std::vector<long long> row0(count), nz0(count);
    long long rows = 0, nz = 0;
    for (int s = 0; s < count; s++) {
        if (n[s] <= 0 || !rowptr[s] || rowptr[s][0] != 0) {
            delete bt;
            set_last_error("mf_batch_create: system %d has no rows or rowptr[0] != 0", s);
            return MF_ERR_INVALID_ARG;
        }
        row0[s] = rows;
        nz0[s] = nz;
        rows += n[s];
        nz += rowptr[s][n[s]];
    }
    bt->rows_total = rows;
    bt->nnz_total = nz;
    bt->row0 = row0;
    bt->nz0 = nz0;
    // validation
    for (int s = 0; s < count; s++) {
        for (int i = 0; i < n[s]; i++)
            if (rowptr[s][i + 1] < rowptr[s][i]) {
                delete bt;
                set_last_error("mf_batch_create: system %d row pointers decrease at row %d", s, i);
                return MF_ERR_INVALID_ARG;
            }
        const int e = rowptr[s][n[s]];
        for (int k = 0; k < e; k++) {
            const int c = colidx[s][k];
            if (c < 0 || c >= n[s]) {
                delete bt;
                set_last_error("mf_batch_create: system %d column %d outside [0, %d)", s, c, n[s]);
                return MF_ERR_INVALID_ARG;
            }
        }
    }
    // panel-major storage and chunks of every system (host threads)
    std::vector<HostSys> hs(count);
    parallel_for(count, [&](int s) { host_panels(n[s], rowptr[s], colidx[s], val[s], hs[s]); });
    std::vector<int> pan0(count), npan(count), sc(count + 1), crow, cent;
    std::vector<long long> prow0, pent0;
    long long prows = 0, pents = 0;
    int panels = 0;
    for (int s = 0; s < count; s++) {
        pan0[s] = panels;
        npan[s] = hs[s].np;
        for (int k = 0; k < hs[s].np; k++) {
            prow0.push_back(prows);
            pent0.push_back(pents);
            prows += n[s] + 1;
            pents += hs[s].pnz[k];
        }
        panels += hs[s].np;
        sc[s] = (int)(crow.size() - s);
        crow.insert(crow.end(), hs[s].crow.begin(), hs[s].crow.end());
        cent.insert(cent.end(), hs[s].cent.begin(), hs[s].cent.end());
    }
    prow0.push_back(prows);
    pent0.push_back(pents);
    sc[count] = (int)(crow.size() - count);
    const int nch = sc[count];
    bt->nchunks = nch;
    bt->npanels = panels;
    std::vector<int> order(count);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return n[a] > n[b]; });
    auto fail = [&](cudaError_t e) {
        set_last_error("mf_batch_create: %s", cudaGetErrorString(e));
        mf_batch_destroy(bt);
        return e == cudaErrorMemoryAllocation ? MF_ERR_NO_MEMORY : MF_ERR_CUDA;
    };
    float4 *rowstat = nullptr;
    unsigned char *rowflag = nullptr;
    cudaError_t e = cudaSuccess;
    // one allocation for all of them, every array on a 256-byte boundary (the
    // first pass adds up the sizes, the second hands out the addresses)
    auto arrays = [&](auto take) {
        take(bt->d_order, sizeof(int) * count);
        take(bt->d_win0, sizeof(int) * count);
        take(bt->d_n, sizeof(int) * count);
        take(bt->d_pan0, sizeof(int) * count);
        take(bt->d_npan, sizeof(int) * count);
        take(bt->d_row0, sizeof(long long) * count);
        take(bt->d_prow0, sizeof(long long) * (panels + 1));
        take(bt->d_pent0, sizeof(long long) * (panels + 1));
        take(bt->d_prow, sizeof(int) * (prows + 8));
        take(bt->d_sc, sizeof(int) * (count + 1));
        take(bt->d_crow, sizeof(int) * crow.size());
        take(bt->d_cent, sizeof(int) * cent.size());
        take(bt->d_col, sizeof(uint16_t) * (nz + 16));
        take(bt->d_val, sizeof(double) * (nz + 2));
        take(bt->d_val16, sizeof(__half) * (nz + 16));
        take(bt->d_rscale, sizeof(float) * (rows + 4));
        take(bt->d_diag32, sizeof(float) * (rows + 4));
        take(bt->d_diag64, sizeof(double) * (rows + 4));
        take(bt->d_ccls, (size_t)nch + 16);
        take(bt->d_ccls_static, (size_t)nch + 16);
        take(bt->d_cstat, sizeof(float) * NCSTAT * ((size_t)nch + 1));
        take(bt->d_cdyn, sizeof(float) * NCDYN * ((size_t)nch + 1));
        take(bt->d_iters, sizeof(int) * count);
        take(bt->d_refs, sizeof(int) * count);
        take(bt->d_status, sizeof(int) * count);
        take(bt->d_relres, sizeof(double) * count * 2);
        take(bt->d_sysstat, sizeof(unsigned long long) * 3 * count);
        take(bt->d_queue, sizeof(int) * 4);
    };
    size_t arena = 0;
    arrays([&](auto &, size_t bytes) { arena += (bytes + 255) / 256 * 256; });
    e = cudaMalloc(&bt->arena, arena);
    if (e == cudaSuccess) e = pool_malloc_async(&rowstat, sizeof(float4) * ((size_t)rows + 1), 0);
    if (e == cudaSuccess) e = pool_malloc_async(&rowflag, (size_t)rows + 16, 0);
    if (e == cudaSuccess) {
        char *at = (char *)bt->arena;
        arrays([&](auto &p, size_t bytes) {
            p = (std::remove_reference_t<decltype(p)>)at;
            at += (bytes + 255) / 256 * 256;
        });
    }
#define BT_COPY(dst, src, bytes) \
    if (e == cudaSuccess && (bytes) > 0) e = cudaMemcpy((dst), (src), (bytes), cudaMemcpyHostToDevice)
    std::vector<int> win0(count);
    for (int s = 1; s < count; s++) win0[s] = win0[s - 1] + sell_windows(n[s - 1]);
    BT_COPY(bt->d_order, order.data(), sizeof(int) * count);
    BT_COPY(bt->d_win0, win0.data(), sizeof(int) * count);
    BT_COPY(bt->d_n, n, sizeof(int) * count);
    BT_COPY(bt->d_pan0, pan0.data(), sizeof(int) * count);
    BT_COPY(bt->d_npan, npan.data(), sizeof(int) * count);
    BT_COPY(bt->d_row0, row0.data(), sizeof(long long) * count);
    BT_COPY(bt->d_prow0, prow0.data(), sizeof(long long) * (panels + 1));
    BT_COPY(bt->d_pent0, pent0.data(), sizeof(long long) * (panels + 1));
    BT_COPY(bt->d_sc, sc.data(), sizeof(int) * (count + 1));
    BT_COPY(bt->d_crow, crow.data(), sizeof(int) * crow.size());
    BT_COPY(bt->d_cent, cent.data(), sizeof(int) * cent.size());
    for (int s = 0; s < count && e == cudaSuccess; s++) {
        const long long pr = prow0[pan0[s]], pe = pent0[pan0[s]];
        BT_COPY(bt->d_prow + pr, hs[s].prow.data(), sizeof(int) * hs[s].prow.size());
        BT_COPY(bt->d_col + pe, hs[s].col.data(), sizeof(uint16_t) * hs[s].col.size());
        BT_COPY(bt->d_val + pe, hs[s].val.data(), sizeof(double) * hs[s].val.size());
    }
#undef BT_COPY
    hs.clear();
    if (e == cudaSuccess) e = cudaMemset(bt->d_cdyn, 0, sizeof(float) * NCDYN * ((size_t)nch + 1));
    if (e == cudaSuccess) {
        const int grid = std::min(count, 1184);
        BatchArgs a;
        memset(&a, 0, sizeof(a));
        a.count = count;
        a.n = bt->d_n;
        a.pan0 = bt->d_pan0;
        a.npan = bt->d_npan;
        a.row0 = bt->d_row0;
        a.prow0 = bt->d_prow0;
        a.pent0 = bt->d_pent0;
        a.prow = bt->d_prow;
        a.col = bt->d_col;
        a.val = bt->d_val;
        k_batch_rows<<<grid, 256>>>(a, bt->d_val16, bt->d_rscale, bt->d_diag32, bt->d_diag64, rowstat, rowflag);
        note_launch();
        e = cudaGetLastError();
        if (e == cudaSuccess) {
            k_batch_chunks<<<grid, 256>>>(count, bt->d_row0, bt->d_sc, bt->d_crow, bt->d_cent, rowstat, rowflag,
                                          bt->d_ccls_static, bt->d_cstat);
            note_launch();
            e = cudaGetLastError();
        }
    }
    if (e == cudaSuccess) e = batch_slices(bt);
    if (e == cudaSuccess) {
        std::vector<unsigned char> st((size_t)nch);
        e = cudaMemcpy(st.data(), bt->d_ccls_static, (size_t)nch, cudaMemcpyDeviceToHost);
        for (unsigned char v : st) {
            bt->static_fp16_chunks += v & 1;
            bt->fp16_allowed_chunks += (v >> 1) & 1;
        }
    }
    if (rowstat) cudaFreeAsync(rowstat, 0);
    if (rowflag) cudaFreeAsync(rowflag, 0);
    if (e != cudaSuccess) return fail(e);
    *out = bt;
    return MF_OK;
}

mf_status mf_batch_destroy(mf_batch bt)
{
    if (!bt) return MF_OK;
    if (bt->graph) cudaGraphExecDestroy(bt->graph);
    void *bufs[] = {bt->arena, bt->slices, bt->words, bt->work};
    for (void *p : bufs)
        if (p) cudaFree(p);
    delete bt;
    return MF_OK;
}

mf_status mf_batch_info(mf_batch bt, long long *rows_total, long long *nnz_total, const long long **row_offsets)
{
    if (!bt) return MF_ERR_INVALID_ARG;
    if (rows_total) *rows_total = bt->rows_total;
    if (nnz_total) *nnz_total = bt->nnz_total;
    if (row_offsets) *row_offsets = bt->row0.data();
    return MF_OK;
}

// five vectors of rows_total doubles, each followed by PW + 16 elements of
// slack (the FP64 kernel reads masked columns past a short last panel) and 4
// per system (the mixed kernel starts every system on a 16-byte boundary)
static size_t batch_vec_len(mf_batch bt) { return ((size_t)bt->rows_total + 4 * (size_t)bt->count + PW + 16 + 3) & ~(size_t)3; }

// The workspace, zeroed in the order of the stream that uses it first.
static mf_status batch_work(mf_batch bt, cudaStream_t s)
{
    const size_t need = batch_vec_len(bt) * 8 * 5 + 1024;
    if (bt->work_bytes >= need) return MF_OK;
    if (bt->work) cudaFree(bt->work);
    bt->work = nullptr;
    bt->work_bytes = 0;
    MF_CUDA(cudaMalloc(&bt->work, need));
    MF_CUDA(cudaMemsetAsync(bt->work, 0, need, s));
    bt->work_bytes = need;
    return MF_OK;
}

static BatchArgs batch_args(mf_batch bt, const double *b, double *x, const mf_solve_opts &o)
{
    const size_t rows = batch_vec_len(bt);
    char *w = (char *)bt->work;
    BatchArgs a;
    memset(&a, 0, sizeof(a));
    a.count = bt->count;
    a.order = bt->d_order;
    a.n = bt->d_n;
    a.pan0 = bt->d_pan0;
    a.npan = bt->d_npan;
    a.row0 = bt->d_row0;
    a.prow0 = bt->d_prow0;
    a.pent0 = bt->d_pent0;
    a.prow = bt->d_prow;
    a.col = bt->d_col;
    a.val = bt->d_val;
    a.val16 = bt->d_val16;
    a.sell = SellView{bt->d_sfirst, bt->d_win0, bt->d_sdesc, bt->d_srec, (const uint4 *)bt->d_scv,
                      (const float4 *)bt->d_sv32, (const uint2 *)bt->d_sc16, (const double2 *)bt->d_sv64,
                      bt->d_diag64};
    a.rscale = bt->d_rscale;
    a.diag32 = bt->d_diag32;
    a.b = b;
    a.x = x;
    a.r = w;
    a.p0 = w + rows * 8;
    a.p1 = w + rows * 16;
    a.q = w + rows * 24;
    a.xlo = w + rows * 32;
    a.sc = bt->d_sc;
    a.crow = bt->d_crow;
    a.cent = bt->d_cent;
    a.ccls = bt->d_ccls;
    a.ccls_static = bt->d_ccls_static;
    a.cstat = bt->d_cstat;
    a.cdyn = bt->d_cdyn;
    a.queue = bt->d_queue;
    a.iters = bt->d_iters;
    a.refs = bt->d_refs;
    a.status = bt->d_status;
    a.relres = bt->d_relres;
    a.sysstat = bt->d_sysstat;
    a.maxiter = o.maxiter;
    a.tol = o.tol;
    a.delta = (o.refine_delta > 0 && o.refine_delta < 1) ? o.refine_delta : 0.1;
    a.budget_ns = (unsigned long long)(o.wait_budget_s * 1e9);
    {
        const char *e = getenv("MF_BATCH_BACKOFF_NS");
        a.backoff_ns = e ? (unsigned)atoi(e) : 0u;
    }
    a.policy = o.policy;
    a.mlp_w = (o.policy == MF_POLICY_LEARNED && bt->policy) ? policy_weights(bt->policy) : nullptr;
    return a;
}

static int batch_ctas(mf_batch bt, bool mixed, int lanes, int cluster)
{
    return batched_ctas(mixed, lanes, bt->count, cluster);
}

// Enqueues one batched solve.  Nothing here allocates or queries the device:
// batch_work() and batch_ctas() run before (outside any stream capture).
static mf_status batch_enqueue(mf_batch bt, const BatchArgs &a, bool mixed, int lanes, int cluster, int ctas,
                               cudaStream_t s)
{
    MF_CUDA(cudaMemsetAsync(bt->d_queue, 0, sizeof(int) * 2, s));  // queue head, stage-wait status
    MF_CUDA(cudaMemsetAsync(bt->d_sysstat, 0, sizeof(unsigned long long) * 3 * bt->count, s));
    MF_TRY(launch_batched(mixed, lanes, a, cluster, ctas, s));
    k_batch_resid<<<std::min(bt->count, 1184), 256, 0, s>>>(a, a.b, a.x, bt->d_relres + bt->count);
    note_launch();
    MF_CUDA(cudaGetLastError());
    return MF_OK;
}

static mf_status batch_check_opts(mf_batch bt, const mf_solve_opts &o)
{
    if (o.tol <= 0 || o.maxiter <= 0 || o.wait_budget_s <= 0) {
        set_last_error("batched CG needs tol > 0, maxiter > 0 and a positive wait budget");
        return MF_ERR_INVALID_ARG;
    }
    if (o.policy < MF_POLICY_FP64 || o.policy > MF_POLICY_STATIC_FP16) {
        set_last_error("batched CG: unknown policy %d", o.policy);
        return MF_ERR_INVALID_ARG;
    }
    if (o.precond) {
        set_last_error("batched CG: no preconditioner");
        return MF_ERR_UNSUPPORTED;
    }
    if (o.policy == MF_POLICY_RULE_SCALED || o.policy == MF_POLICY_STATIC_FP16) {
        set_last_error("batched CG: the scaled rule and STATIC_FP16 are not available (RULE, LEARNED, STATIC, FP64 are;"
                       " its FP16 chunks are row-scaled)");
        return MF_ERR_UNSUPPORTED;
    }
    if (o.policy == MF_POLICY_LEARNED && !bt->policy) {
        set_last_error("batched CG: learned policy requested but none is attached (mf_batch_attach_policy)");
        return MF_ERR_UNSUPPORTED;
    }
    return MF_OK;
}

// CTAs per system of a mixed solve that nobody tuned: 2 where the systems
// fill the device, else the most (up to 16) at which every system still has a
// resident cluster and the largest at least 512 rows per CTA.  Measured (us
// per iteration): 24 systems of 1,000-4,000 rows 17.2 with 2 CTAs, 15.1 with
// 4, 15.1 with 8; 256 systems of 1,000-32,000 rows (1.7 waves of 2-CTA
// clusters) 322 ms a solve with 2, 362 with 4.
static int batch_auto_cluster(mf_batch bt, int lanes)
{
    if (bt->auto_cluster) return bt->auto_cluster;
    const BatchKernel k = batch_kernel(true, lanes);
    const int nmax = *std::max_element(bt->n.begin(), bt->n.end());
    int best = 2;
    for (int c = 4; c <= 16 && c * 512 <= nmax; c *= 2) {
        batched_ctas(true, lanes, bt->count, c);  // the kernel's attributes
        BatchConfig cfg;
        batch_config(cfg, k, c, c * bt->count, nullptr);
        int fit = 0;
        if (cudaOccupancyMaxActiveClusters(&fit, k.fn, &cfg.cfg) != cudaSuccess) {
            cudaGetLastError();
            break;
        }
        if (fit < bt->count) break;
        best = c;
    }
    bt->auto_cluster = best;
    return best;
}

static void batch_schedule(mf_batch bt, bool mixed, int &lanes, int &cluster)
{
    lanes = bt->tuned_lanes ? bt->tuned_lanes : 4;
    cluster = bt->tuned_cluster ? bt->tuned_cluster : mixed ? batch_auto_cluster(bt, lanes) : 2;
    if (const char *e = getenv("MF_BATCH_LANES")) lanes = atoi(e);
    if (const char *e = getenv("MF_BATCH_CLUSTER")) cluster = atoi(e);
    if (lanes != 4 && lanes != 8 && lanes != 16 && lanes != 32) lanes = 4;
    if (cluster != 1 && cluster != 2 && cluster != 4 && cluster != 8 && cluster != 16) cluster = 2;
}

mf_status mf_batch_cg_solve(mf_batch bt, const double *b, double *x, const mf_solve_opts *opts, int use_graph,
                            mf_batch_report *report, void *stream)
{
    if (!bt || !b || !x) return MF_ERR_INVALID_ARG;
    mf_solve_opts o;
    mf_solve_opts_default(&o);
    if (opts) o = *opts;
    MF_TRY(batch_check_opts(bt, o));
    cudaStream_t s = (cudaStream_t)stream;
    int lanes, cluster;
    const bool mixed = o.policy != MF_POLICY_FP64;
    batch_schedule(bt, mixed, lanes, cluster);
    MF_TRY(batch_work(bt, s));
    const int ctas = batch_ctas(bt, mixed, lanes, cluster);
    const BatchArgs a = batch_args(bt, b, x, o);
    cudaEvent_t e0, e1;
    MF_CUDA(cudaEventCreate(&e0));
    MF_CUDA(cudaEventCreate(&e1));
    MF_CUDA(cudaEventRecord(e0, s));
    const BatchGraphKey key = {b,     x,       lanes,   cluster,     o.policy,    o.maxiter,
                               o.tol, a.delta, a.mlp_w, a.budget_ns, a.backoff_ns};
    if (use_graph) {
        // one graph per (buffers, configuration): replayed on later calls
        if (!bt->graph || !(bt->graph_key == key)) {
            if (bt->graph) cudaGraphExecDestroy(bt->graph);
            bt->graph = nullptr;
            cudaStream_t cs;
            MF_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
            cudaGraph_t g;
            MF_CUDA(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
            mf_status st = batch_enqueue(bt, a, mixed, lanes, cluster, ctas, cs);
            cudaError_t ce = cudaStreamEndCapture(cs, &g);
            cudaStreamDestroy(cs);
            if (st != MF_OK || ce != cudaSuccess) {
                if (ce == cudaSuccess) cudaGraphDestroy(g);
                cudaGetLastError();
                if (st != MF_OK) return st;
                MF_CUDA(ce);
            }
            MF_CUDA(cudaGraphInstantiate(&bt->graph, g, 0));
            cudaGraphDestroy(g);
            bt->graph_key = key;
        }
        MF_CUDA(cudaGraphLaunch(bt->graph, s));
        note_launch(2);  // the graph's kernels: the batched CG and the residual check
    } else {
        MF_TRY(batch_enqueue(bt, a, mixed, lanes, cluster, ctas, s));
    }
    MF_CUDA(cudaEventRecord(e1, s));
    MF_CUDA(cudaEventSynchronize(e1));
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    const int count = bt->count;
    std::vector<int> it(count), rf(count), stt(count);
    std::vector<double> rr(count * 2);
    std::vector<unsigned long long> ss((size_t)count * 3);
    MF_CUDA(cudaMemcpy(it.data(), bt->d_iters, sizeof(int) * count, cudaMemcpyDeviceToHost));
    MF_CUDA(cudaMemcpy(rf.data(), bt->d_refs, sizeof(int) * count, cudaMemcpyDeviceToHost));
    MF_CUDA(cudaMemcpy(stt.data(), bt->d_status, sizeof(int) * count, cudaMemcpyDeviceToHost));
    MF_CUDA(cudaMemcpy(rr.data(), bt->d_relres, sizeof(double) * count * 2, cudaMemcpyDeviceToHost));
    MF_CUDA(cudaMemcpy(ss.data(), bt->d_sysstat, sizeof(unsigned long long) * 3 * count, cudaMemcpyDeviceToHost));
    mf_status worst = MF_OK;
    long long iters = 0, bytes = 0;
    unsigned long long lowp = 0, passes = 0;
    double maxrr = 0;
    int maxit = 0, refs = 0, failed = 0;
    for (int k = 0; k < count; k++) {
        iters += it[k];
        maxit = std::max(maxit, it[k]);
        refs += rf[k];
        maxrr = std::max(maxrr, rr[count + k]);
        lowp += ss[3 * k + 1];
        passes += ss[3 * k + 2];
        // matrix bytes streamed by the (chunk, panel) passes (counted in the
        // kernel), the vector streams of each iteration (p update: r, p_old
        // in, p out; SpMV: p read once, q out; x, r update: p, q, x, r in,
        // x, r out), and per reliable update an FP64 pass over the matrix
        // plus b, x in and r out
        const long long nn = bt->n[k];
        const long long nnz = (k + 1 < count ? bt->nz0[k + 1] : bt->nnz_total) - bt->nz0[k];
        const long long vb = mixed ? 4 : 8;
        bytes += (long long)ss[3 * k] + (long long)it[k] * 11 * vb * nn +
                 (long long)rf[k] * (nnz * (8 + 2) + 4 * (nn + 1) + 16 * nn + vb * nn);
        if (stt[k] != MF_OK) {
            failed++;
            if (worst == MF_OK) worst = (mf_status)stt[k];
        }
    }
    if (report) {
        report->systems = count;
        report->failed = failed;
        report->iterations_total = iters;
        report->iterations_max = maxit;
        report->refinements_total = refs;
        report->relres_true_max = maxrr;
        report->kernel_ms = ms;
        report->lanes_per_row = lanes;
        report->cluster_ctas = cluster;
        report->status = worst;
        report->bytes_moved = bytes;
        report->fp16_share = passes ? (double)lowp / (double)passes : 0.0;
    }
    if (worst != MF_OK) set_last_error("%d of %d systems did not converge", failed, count);
    return worst;
}

mf_status mf_batch_results(mf_batch bt, int *iterations, double *relres_true)
{
    if (!bt) return MF_ERR_INVALID_ARG;
    if (iterations) MF_CUDA(cudaMemcpy(iterations, bt->d_iters, sizeof(int) * bt->count, cudaMemcpyDeviceToHost));
    if (relres_true)
        MF_CUDA(cudaMemcpy(relres_true, bt->d_relres + bt->count, sizeof(double) * bt->count, cudaMemcpyDeviceToHost));
    return MF_OK;
}

mf_status mf_batch_chunk_count(mf_batch bt, int *chunks, int *static_fp16, int *fp16_capable)
{
    if (!bt) return MF_ERR_INVALID_ARG;
    if (chunks) *chunks = bt->nchunks;
    if (static_fp16) *static_fp16 = bt->static_fp16_chunks;
    if (fp16_capable) *fp16_capable = bt->fp16_allowed_chunks;
    return MF_OK;
}

mf_status mf_batch_export(mf_batch bt, const char *name, void *host_dst, size_t bytes)
{
    if (!bt || !name || (!host_dst && bytes)) return MF_ERR_INVALID_ARG;
    const void *src = nullptr;
    size_t need = 0;
    const size_t nz = (size_t)bt->nnz_total, rows = (size_t)bt->rows_total, nch = (size_t)bt->nchunks;
    if (!strcmp(name, "chunk_class")) src = bt->d_ccls, need = nch;
    else if (!strcmp(name, "chunk_static")) src = bt->d_ccls_static, need = nch;
    else if (!strcmp(name, "chunk_features_static")) src = bt->d_cstat, need = sizeof(float) * NCSTAT * nch;
    else if (!strcmp(name, "chunk_start")) src = bt->d_sc, need = sizeof(int) * (bt->count + 1);
    else if (!strcmp(name, "chunk_rows")) src = bt->d_crow, need = sizeof(int) * (nch + bt->count);
    else if (!strcmp(name, "chunk_ends")) src = bt->d_cent, need = sizeof(int) * (nch + bt->count);
    else if (!strcmp(name, "val16")) src = bt->d_val16, need = 2 * nz;
    else if (!strcmp(name, "val32")) need = 4 * nz;  // made from val below
    else if (!strcmp(name, "val")) src = bt->d_val, need = 8 * nz;
    else if (!strcmp(name, "col")) src = bt->d_col, need = 2 * nz;
    else if (!strcmp(name, "row_scale")) src = bt->d_rscale, need = 4 * rows;
    else if (!strcmp(name, "diag32")) src = bt->d_diag32, need = 4 * rows;
    else {
        set_last_error("mf_batch_export: unknown array %s", name);
        return MF_ERR_INVALID_ARG;
    }
    if (bytes != need) {
        set_last_error("mf_batch_export: %s has %zu bytes, %zu given", name, need, bytes);
        return MF_ERR_INVALID_ARG;
    }
    if (need && !src) {
        float *tmp = nullptr;
        MF_CUDA(cudaMalloc(&tmp, need));
        k_batch_cast32<<<(unsigned)std::min<size_t>((nz + 255) / 256, 148 * 32), 256>>>((long long)nz, bt->d_val, tmp);
        note_launch();
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpy(host_dst, tmp, need, cudaMemcpyDeviceToHost);
        cudaFree(tmp);
        MF_CUDA(e);
        return MF_OK;
    }
    if (need) MF_CUDA(cudaMemcpy(host_dst, src, need, cudaMemcpyDeviceToHost));
    return MF_OK;
}

mf_status mf_batch_attach_policy(mf_batch bt, mf_learned p)
{
    if (!bt) return MF_ERR_INVALID_ARG;
    bt->policy = p;
    if (bt->graph) cudaGraphExecDestroy(bt->graph);
    bt->graph = nullptr;
    return MF_OK;
}

mf_status mf_batch_policy_classify(mf_batch bt, const double *r, const double *p_new, const double *p_old,
                                   const double *q, const double *relres, const int *refinements, int have_prev,
                                   unsigned char *classes, float *features)
{
    if (!bt || !r || !p_new || !p_old || !q || !relres || !refinements || !classes) return MF_ERR_INVALID_ARG;
    if (!bt->policy) {
        set_last_error("mf_batch_policy_classify: no policy attached");
        return MF_ERR_UNSUPPORTED;
    }
    mf_solve_opts o;
    mf_solve_opts_default(&o);
    o.policy = MF_POLICY_LEARNED;
    BatchArgs a = batch_args(bt, nullptr, nullptr, o);
    k_batch_classify<<<std::min(bt->count, 1184), BNT>>>(a, r, p_new, p_old, q, relres, refinements, have_prev,
                                                         classes, features);
    note_launch();
    MF_CUDA(cudaGetLastError());
    MF_CUDA(cudaStreamSynchronize(0));
    return MF_OK;
}

// Plain FP64 batched solve of every system that adds (chunk features,
// label) samples every checkpoint_every iterations (about one chunk in
// sample_stride) to the policy's training set.  Label 1 (FP16) when the
// FP16 values perturb the chunk's A p by at most 2^-6 of it (2-norms over
// the chunk's rows), else 2 (FP32).
mf_status mf_batch_policy_collect(mf_learned p, mf_batch bt, const double *b, int checkpoint_every,
                                  int sample_stride, long long max_samples, long long *samples_out)
{
    if (!p || !bt || !b || checkpoint_every <= 0 || sample_stride <= 0 || max_samples <= 0)
        return MF_ERR_INVALID_ARG;
    float *cx = nullptr;
    unsigned char *cy = nullptr;
    long long have = 0;
    MF_TRY(policy_sample_buffers(p, max_samples, &cx, &cy, &have));
    MF_TRY(batch_work(bt, 0));
    double *x = nullptr;
    unsigned long long *cnt = nullptr;
    MF_CUDA(cudaMalloc(&x, sizeof(double) * (bt->rows_total + 1)));
    MF_CUDA(cudaMalloc(&cnt, sizeof(unsigned long long)));
    const unsigned long long start = (unsigned long long)have;
    MF_CUDA(cudaMemcpy(cnt, &start, sizeof(start), cudaMemcpyHostToDevice));
    mf_solve_opts o;
    mf_solve_opts_default(&o);
    o.policy = MF_POLICY_FP64;
    o.tol = 1e-10;
    o.maxiter = 100000;
    BatchArgs a = batch_args(bt, b, x, o);
    a.collect_every = checkpoint_every;
    a.collect_stride = sample_stride;
    a.collect_salt = (unsigned)(have * 2654435761ull);
    a.cx = cx;
    a.cy = cy;
    a.ccount = cnt;
    a.ccap = max_samples;
    const int lanes = 8, cluster = 2;
    const int ctas = batch_ctas(bt, false, lanes, cluster);
    mf_status st = batch_enqueue(bt, a, false, lanes, cluster, ctas, 0);
    unsigned long long end = start;
    if (st == MF_OK) {
        cudaError_t e = cudaMemcpy(&end, cnt, sizeof(end), cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) {
            set_last_error("mf_batch_policy_collect: %s", cudaGetErrorString(e));
            st = MF_ERR_CUDA;
        }
    }
    cudaFree(x);
    cudaFree(cnt);
    if (st != MF_OK) return st;
    const long long total = (long long)std::min<unsigned long long>(end, (unsigned long long)max_samples);
    MF_TRY(policy_sample_commit(p, total));
    if (samples_out) *samples_out = total;
    return MF_OK;
}

// Autotuner: times every (lanes per row, cluster size) pair on this batch
// and keeps the fastest; the choice is returned and kept on the handle.
mf_status mf_batch_tune(mf_batch bt, const double *b, double *x, const mf_solve_opts *opts, int *lanes_out,
                        int *cluster_out, void *stream)
{
    if (!bt || !b || !x) return MF_ERR_INVALID_ARG;
    mf_solve_opts o;
    mf_solve_opts_default(&o);
    if (opts) o = *opts;
    MF_TRY(batch_check_opts(bt, o));
    const int lanes_c[] = {4, 8, 16, 32};
    const int clus_c[] = {1, 2, 4, 8, 16};
    float best = 1e30f;
    int bl = 8, bc = 2;
    cudaStream_t s = (cudaStream_t)stream;
    const bool mixed = o.policy != MF_POLICY_FP64;
    MF_TRY(batch_work(bt, s));
    const BatchArgs a = batch_args(bt, b, x, o);
    for (int li : lanes_c)
        for (int ci : clus_c) {
            const int ctas = batch_ctas(bt, mixed, li, ci);
            cudaEvent_t e0, e1;
            MF_CUDA(cudaEventCreate(&e0));
            MF_CUDA(cudaEventCreate(&e1));
            MF_CUDA(cudaEventRecord(e0, s));
            mf_status st = batch_enqueue(bt, a, mixed, li, ci, ctas, s);
            MF_CUDA(cudaEventRecord(e1, s));
            MF_CUDA(cudaEventSynchronize(e1));
            float ms = 0;
            cudaEventElapsedTime(&ms, e0, e1);
            cudaEventDestroy(e0);
            cudaEventDestroy(e1);
            std::vector<int> stt(bt->count);
            MF_CUDA(cudaMemcpy(stt.data(), bt->d_status, sizeof(int) * bt->count, cudaMemcpyDeviceToHost));
            const bool ok = st == MF_OK && std::all_of(stt.begin(), stt.end(), [](int v) { return v == MF_OK; });
            if (ok && ms < best) {
                best = ms;
                bl = li;
                bc = ci;
            }
        }
    bt->tuned_lanes = bl;
    bt->tuned_cluster = bc;
    if (bt->graph) cudaGraphExecDestroy(bt->graph);
    bt->graph = nullptr;
    if (lanes_out) *lanes_out = bl;
    if (cluster_out) *cluster_out = bc;
    return MF_OK;
}

mf_status mf_batch_set_schedule(mf_batch bt, int lanes, int cluster)
{
    if (!bt || (lanes != 4 && lanes != 8 && lanes != 16 && lanes != 32) ||
        (cluster != 1 && cluster != 2 && cluster != 4 && cluster != 8 && cluster != 16))
        return MF_ERR_INVALID_ARG;
    bt->tuned_lanes = lanes;
    bt->tuned_cluster = cluster;
    if (bt->graph) cudaGraphExecDestroy(bt->graph);
    bt->graph = nullptr;
    return MF_OK;
}

}  // extern "C"
