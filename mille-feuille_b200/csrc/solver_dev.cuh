// solver_dev.cuh -- the persistent single-kernel CG / BiCGSTAB, the tile walks and
// the per-handle workspace, shared by solver.cu, solve_rows.cu and multi.cu (each
// instantiates its own kernels; everything here has internal linkage).
//
// One cooperative launch runs the whole solve (the reference's single-kernel
// design, Mille-feuille-cg.h:1113-1348 / main-cg-mixed.cu:1016-1385 /
// main-bicg-mixed.cu:122-723), re-designed for sm_100a:
//  * grid = SMs x resident blocks (cooperative launch guarantees co-residency);
//  * a half-warp owns a contiguous range of tile-rows (lane i = row 16R+i) for
//    every phase, so y rows are written by their owner only (no y atomics) and
//    every dot product is reduced in a fixed order (deterministic);
//  * the tile SpMV walks the half-warp's solver slices: one 16-byte header per
//    slice, the slice's tile words held one tile per lane (read with
//    __shfl_sync), the next slice's descriptor loaded while the current slice's
//    value + x loads are in flight;
//  * the grid barrier is a monotone counter: fence + relaxed arrive, relaxed
//    polls, one acquire fence, every wait bounded by %globaltimer (MF_ERR_TIMEOUT);
//  * dot products: warp shuffle tree -> per-block partial in a fixed slot ->
//    after the barrier each block sums the partials in the same order;
//  * matrix payload is streamed with evict-first loads so the vectors stay in L2.
#pragma once
#include "mf_internal.cuh"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <type_traits>

namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kRedKinds = 10;     // reduction slot groups
constexpr int kRedWidth = 4;      // doubles per group per block
constexpr int kDefaultLB = 2;     // default register-budget variant of the persistent kernel
constexpr int kVB = 4;            // tile-rows per step in the vector phases (loads in flight)
constexpr int kDemoteCool = 16;   // SpMVs without per-slice lookups after one that did not pay

enum { MODE_FP64 = 0, MODE_MIXED = 1, MODE_PARITY = 2 };

// ------------------------------------------------------------ bounds checks
// The bounds-checked build (-DMF_CHECK, libmillefeuille_check.so): every index
// the kernels take from stored data -- a half-warp's slice range, a tile word's
// column tile, a per-tile table entry, a slice's payload, a gathered vector
// position, an epilogue tile-row, a batch queue entry -- is compared with the
// extent of the array it addresses before the access.  A failed check keeps the
// first (site, index, limit) of the device in g_chk and the access is skipped
// (a load reads zero, a store or a slice is dropped); the entry point that
// launched the kernel returns MF_ERR_CHECK.  Nothing traps: the context stays
// usable.  In the normal build chk_in() is `true` and the checks compile away.
enum { CHK_SLICE = 1, CHK_TILE, CHK_PAYLOAD, CHK_X, CHK_ROWLEN, CHK_ROW, CHK_ITEM, CHK_NSITES };
#ifdef MF_CHECK
__device__ unsigned long long g_chk[3];   // site, index, limit of the first failed check

__device__ __noinline__ void chk_fail(int site, long long idx, long long lim)
{
    if (atomicCAS(&g_chk[0], 0ull, (unsigned long long)site) == 0ull) {
        g_chk[1] = (unsigned long long)idx;
        g_chk[2] = (unsigned long long)lim;
    }
}

__device__ __forceinline__ bool chk_in(int site, long long idx, long long lim)
{
    if (idx >= 0 && idx < lim) return true;
    chk_fail(site, idx, lim);
    return false;
}
#else
__device__ __forceinline__ bool chk_in(int, long long, long long) { return true; }
#endif

struct SolverParams {
    int n, tilem, vec_len;
    const int *rowptr;            // CSR row pointers (entry counts of the lean FP32 walk)
    const int *seg_ptr;
    const int4 *seg_hdr;
    const uint16_t *seg_rowlen;
    const unsigned char *meta;
    const double *v64;
    const float *v32;
    const __half *v16;
    const int8_t *v8, *v8ref;
    const int *tile_col;
    const int *seg_tile;          // [nseg*16] tile words: column-tile << 8 | caps
    const int *tile_off;          // csr_offset: tile payload offsets (tile nnz for the counters)
    const float *i8_scale;
    const unsigned char *tile_caps;
    const int *hw_begin;
    const double *b;
    double *x, *r, *p, *q, *rh, *s, *t;
    float *p32, *s32, *mag_p, *mag_s;
    float *mag_r;                 // CG with the SpMV on r: r's segment magnitudes
    __half *p16, *s16;
    int8_t *p8, *s8;
    signed char *lab_p, *lab_s;
    double *red;
    unsigned int *bar;
    int *err;
    double *out;
    unsigned long long *counts;
    unsigned long long *phase_ns;   // [8] block-0 time per phase: spmv, vecB, vecC, barrier, replacement
    int method, max_iter, fixed_iters, replace_every, use_lossless;
    int x0_given;                 // x holds the initial guess: r = b - A x at the start
    int lossless_any;             // use_lossless and enough tiles are exact in INT8 / FP16
    float min_demoted;            // mixed: a dynamic SpMV that runs fewer tiles than this below FP32
                                  // turns the operand's per-slice lookups off for kDemoteCool SpMVs
    float min_small;              // mixed: narrower tiles only when at least this many column
                                  // segments were small in the operand's previous update
    double tol;
    float demote16, demote8;
    unsigned long long timeout_ns;
    int stall_first_barrier;   // test hook: first barrier expects one extra arrival
    float relax_eta;           // mixed CG: relaxation factor of the matvec precision (0: off)
    int relax_int8;            // the relaxation may go down to scaled INT8 (else FP16 at most)
    int fp16_ok;               // every tile's values are within FP16's normal range
    int lean_f16;              // mixed, use_lossless: every tile is exact in FP16, so the lookup-free
                               // walk runs FP16 stored values (the lossless choice made once)
    // extents for the bounds-checked build: slices, tiles, payload entries, and
    // the operand length its gathers are checked against (vec_len, or less
    // through the test_check_limit hook)
    int nseg, ntiles, chk_xlen;
    long long n_payload;
    long long nnz;
    int cluster;               // > 0: the launch is one cluster of this many blocks
};

constexpr int kMaxCluster = 16;

// CL: a launch of one cluster (SolverParams::cluster blocks)
template <bool CL>
struct SharedT {
    static constexpr bool kCluster = CL;
    double part[CL ? kRedKinds : 1][kRedWidth][kMaxCluster];   // every block's partials
    double wred[kWarps][kRedWidth];
    double bcast[kRedWidth];
    int flag;
    unsigned cnt[kWarps * 2][10];   // per-half-warp tile / entry counters per precision (mixed / parity)
    unsigned whole[4];              // block 0: products of the whole matrix in one precision (spmv_rows)
    unsigned long long clk_t, clk_acc[5];   // block 0 phase clock
};

// ------------------------------------------------------------ grid barrier
// One-cluster solves: the hardware's cluster barrier, with release / acquire of
// everything the blocks wrote.  It waits for the threads of the cluster that
// have not exited, and all of them run through the same barriers, so it needs no
// limit of its own.  `aligned` asks for whole warps: their lanes meet first.
__device__ __forceinline__ void cluster_barrier()
{
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A double into another block's copy of `p` (shared memory of the cluster's block `rank`).
// Another block's shared memory may be accessed only between that block's start and
// its exit.  Start: k_solve passes a cluster_barrier before its first reduction, and
// no block leaves that barrier before all have arrived.  Exit: every store here is
// followed by a cluster_barrier that the target passes too (solve_barrier, before the
// partials are read), and a block returns only after its last one.
__device__ __forceinline__ void cluster_store(double *p, int rank, double v)
{
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
    unsigned ra;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(ra), "d"(v) : "memory");
}

template <class SH>
__device__ bool grid_barrier(const SolverParams &P, unsigned &epoch, SH &sh)
{
    __syncthreads();
    epoch += 1;
    if (threadIdx.x == 0) {
        const bool timed = blockIdx.x == 0 && P.phase_ns;
        const unsigned long long tw0 = timed ? mf_globaltimer() : 0ull;
        const unsigned target = epoch * gridDim.x + ((P.stall_first_barrier && epoch == 1) ? 1u : 0u);
        // fence-release pattern: the block's writes (ordered before by bar.sync) are
        // visible at gpu scope before the arrival; polls are relaxed loads and one
        // acquire fence follows (an acquire load per poll costs like a fence)
        __threadfence();
        mf_red_relaxed_add_u32(P.bar, 1u);
        bool ok = true;
        const unsigned long long t0 = mf_globaltimer();
        unsigned spins = 0;
        for (;;) {
            unsigned v = mf_ld_relaxed_u32(P.bar);
            if ((int)(v - target) >= 0) break;
            if (*(volatile int *)P.err) { ok = false; break; }
            if ((++spins & 63u) == 0u && mf_globaltimer() - t0 > P.timeout_ns) {
                atomicCAS(P.err, 0, MF_ERR_TIMEOUT);
                ok = false;
                break;
            }
        }
        mf_fence_acq_rel_gpu();
        sh.flag = ok ? 1 : 0;
        if (timed) P.phase_ns[5] += mf_globaltimer() - tw0;   // block 0 spin time
    }
    __syncthreads();
    return sh.flag != 0;
}

// The barrier of a solve: the cluster's or the grid's.
template <bool CL>
__device__ __forceinline__ bool solve_barrier(const SolverParams &P, unsigned &epoch, SharedT<CL> &sh)
{
    if constexpr (CL) {
        cluster_barrier();
        return true;
    } else {
        return grid_barrier(P, epoch, sh);
    }
}

// Block partial of up to 4 sums (mask bit k set -> max instead of sum) written
// to red[kind][k][block] (value-major, so a collect reads consecutive blocks).
template <bool CL>
__device__ void block_partial(const SolverParams &P, SharedT<CL> &sh, int kind, double v0, double v1, double v2,
                              double v3, int nv, unsigned maxmask)
{
    double v[kRedWidth] = {v0, v1, v2, v3};
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < kRedWidth; k++) {
        if (k >= nv) break;
        double a = v[k];
        const bool mx = (maxmask >> k) & 1u;
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            double b = __shfl_xor_sync(0xffffffffu, a, o);
            a = mx ? fmax(a, b) : a + b;
        }
        if (lane == 0) sh.wred[wib][k] = a;
    }
    __syncthreads();
    if (wib < nv) {                       // warp k reduces value k
        const int k = wib;
        const bool mx = (maxmask >> k) & 1u;
        double a = (lane < kWarps) ? sh.wred[lane][k] : (mx ? -1.0e300 : 0.0);
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            double b = __shfl_xor_sync(0xffffffffu, a, o);
            a = mx ? fmax(a, b) : a + b;
        }
        if (CL) {
            if (lane < P.cluster) cluster_store(&sh.part[CL ? kind : 0][k][blockIdx.x], lane, a);
        } else if (lane == 0) P.red[((long long)kind * kRedWidth + k) * gridDim.x + blockIdx.x] = a;
    }
}

// After the barrier: every block sums the partials of `kind` in the same order
// (lane c takes blocks c, c + 32, ... in turn, then a shuffle tree).  Partials
// sit value-major (red[kind][k][block]), warp k reduces value k, and each lane
// issues all its loads before the first add, so the collect costs one L2 round
// trip instead of one per partial.  No trailing barrier: the next writer of
// sh.bcast is the next collect, which every thread reaches only through the
// barriers of block_partial and grid_barrier, after it has read bcast here.
template <bool CL>
__device__ void grid_collect(const SolverParams &P, SharedT<CL> &sh, int kind, int nv, unsigned maxmask,
                             double *outv)
{
    if constexpr (CL) {
        // every block holds all partials: each thread sums them as the grid's shuffle
        // tree does (blocks 8 apart first, then 4, 2, 1)
#pragma unroll
        for (int k = 0; k < kRedWidth; k++) {
            if (k >= nv) break;
            const bool mx = (maxmask >> k) & 1u;
            double t[kMaxCluster];
#pragma unroll
            for (int c = 0; c < kMaxCluster; c++)
                t[c] = c < P.cluster ? sh.part[CL ? kind : 0][k][c] : (mx ? -1.0e300 : 0.0);
#pragma unroll
            for (int o = kMaxCluster / 2; o; o >>= 1)
#pragma unroll
                for (int c = 0; c < kMaxCluster / 2; c++)
                    if (c < o) t[c] = mx ? fmax(t[c], t[c + o]) : t[c] + t[c + o];
            outv[k] = t[0];
        }
        return;
    }
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    if (wib < nv) {
        const bool mx = (maxmask >> wib) & 1u;
        const double id = mx ? -1.0e300 : 0.0;
        const int G = (int)gridDim.x;
        const double *src = P.red + ((long long)kind * kRedWidth + wib) * G;
        constexpr int kU = 10;              // 320 blocks per pass: the grid of 148 SMs x 2 in one
        double a = id;
        for (int c0 = 0; c0 < G; c0 += 32 * kU) {
            double t[kU];
#pragma unroll
            for (int j = 0; j < kU; j++) {
                const int cb = c0 + lane + 32 * j;
                t[j] = cb < G ? src[cb] : id;
            }
#pragma unroll
            for (int j = 0; j < kU; j++) a = mx ? fmax(a, t[j]) : a + t[j];
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const double b = __shfl_xor_sync(0xffffffffu, a, o);
            a = mx ? fmax(a, b) : a + b;
        }
        if (lane == 0) sh.bcast[wib] = a;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kRedWidth; k++)
        if (k < nv) outv[k] = sh.bcast[k];
}

// ------------------------------------------------------------ tile SpMV
// Reference-rule label code (d_vis) -> entry precision.
__device__ __forceinline__ int parity_prec(int code)
{
    return code == 0 ? MF_P64 : code == 4 ? MF_P32 : code == 3 ? MF_P16 : code == 2 ? MF_P8 : MF_PSKIP;
}

// The x operands of one SpMV: the FP64 vector (FP64 and mixed modes multiply
// every stored precision against it), and in parity mode its FP32 / FP16 /
// INT8 shadows; mag / lab are the per-column-segment statistics the precision
// choice reads.
struct XVec {
    const double *x64;
    const float *x32;
    const __half *x16;
    const int8_t *x8;
    const float *mag;
    const signed char *lab;
    float invM;
    int force_pr;            // >= 0: every tile in this precision
    int dyn;                 // mixed: 0 = no tile can leave the base precision (no precision lookups)
    int lean_pr;             // mixed: the base precision of the lookup-free walk (FP32, or FP16 when
                             // every tile is exact in FP16)
};

// Tile table of a slice, one tile per lane (lane i holds slot i).
struct TileReg {
    int xb;       // column-tile * 16
    int pr;       // entry precision of the tile (the slice runs at the half's minimum)
};

__device__ __forceinline__ int hdr_kp(int4 h) { return h.z & 0xFFFF; }
__device__ __forceinline__ int hdr_nt(int4 h) { return (h.z >> 16) & 0xFF; }
__device__ __forceinline__ bool hdr_last(int4 h) { return (h.z >> 24) & 1; }
__device__ __forceinline__ long long hdr_off(int4 h) { return (long long)h.w << 7; }

// The precision statistic of lane i's tile (tile word tw = column-tile << 8 |
// caps): the column segment's magnitude (mixed mode) or its reference label
// (parity mode).  Issued one slice ahead so its latency overlaps a slice.
template <int MODE, bool F64>
__device__ __forceinline__ float load_stat(const XVec &X, int tw, int i, int nt)
{
    if (F64 || MODE == MODE_FP64 || i >= nt || X.force_pr >= 0 || (MODE == MODE_MIXED && !X.dyn)) return 0.0f;
    const int jc = tw >> 8;
    if (MODE == MODE_MIXED) return X.mag[jc];
    return (float)X.lab[jc];
}

// Entry precision of lane i's tile from its tile word and statistic.
template <int MODE, bool F64>
__device__ __forceinline__ int tile_prec(const SolverParams &P, int tw, float st, const XVec &X)
{
    if (F64 || MODE == MODE_FP64) return MF_P64;
    if (X.force_pr >= 0) return X.force_pr;
    if (MODE == MODE_PARITY) return parity_prec((int)st);
    if (!X.dyn) return MF_P32;
    const unsigned cap = (unsigned)tw & 0xFFu;
    const float rel = st * X.invM;
    int pr = MF_P32;
    if (rel <= P.demote8) pr = MF_P8;
    else if (rel <= P.demote16 && (cap & MF_CAP_FP16_OK)) pr = MF_P16;
    if (P.use_lossless) {
        if (cap & MF_CAP_EXACT_I8) pr = MF_P8;
        else if ((cap & MF_CAP_EXACT_F16) && pr == MF_P32) pr = MF_P16;
    }
    return pr;
}

// Lane i's 8 stored values of the chunk whose payload starts at entry cb (a
// multiple of 128), in precision PR: 128-bit loads of the row's 16-byte groups
// (4 for FP64, 2 for FP32, 1 for FP16; an 8-byte load for INT8), each issued
// only when its first entry lies inside the row (nact entries of the row fall
// in this chunk; the stored padding past a row's end is zero).  FP32 / FP16 /
// INT8 values come back as float (INT8 unscaled).
template <int PR>
__device__ __forceinline__ void load_chunk(const SolverParams &P, long long cb, int i, int nact,
                                           double (&v64)[8], float (&v)[8])
{
    if (PR == MF_P64) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            double2 d = make_double2(0.0, 0.0);
            if (2 * q < nact) d = __ldcs((const double2 *)(P.v64 + cb + 32 * q) + i);
            v64[2 * q] = d.x;
            v64[2 * q + 1] = d.y;
        }
    } else if (PR == MF_P32) {
#pragma unroll
        for (int q = 0; q < 2; q++) {
            float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
            if (4 * q < nact) f = __ldcs((const float4 *)(P.v32 + cb + 64 * q) + i);
            v[4 * q] = f.x;
            v[4 * q + 1] = f.y;
            v[4 * q + 2] = f.z;
            v[4 * q + 3] = f.w;
        }
    } else if (PR == MF_P16) {
        uint4 u = make_uint4(0u, 0u, 0u, 0u);
        if (nact > 0) u = __ldcs((const uint4 *)(P.v16 + cb) + i);
        const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int q = 0; q < 4; q++) {
            v[2 * q] = __half2float(__ushort_as_half((unsigned short)(w[q] & 0xFFFFu)));
            v[2 * q + 1] = __half2float(__ushort_as_half((unsigned short)(w[q] >> 16)));
        }
    } else {
        uint2 u = make_uint2(0u, 0u);
        if (nact > 0) u = __ldcs((const uint2 *)(P.v8 + cb) + i);
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = (float)(int8_t)(((j < 4 ? u.x : u.y) >> (8 * (j & 3))) & 0xFFu);
    }
}

// Uniform-precision chunk loop: every entry of the slice is stored in
// precision PR (FP64, FP32, FP16 or scaled INT8); the value is widened to FP64
// in registers and multiplied with the FP64 x, so the row sum is FP64 and only
// the stored values are rounded.  The kernel waits on memory, not on the FP64
// pipe: against FP32 products with an FP32 copy of x this measured 6 % fewer
// iterations on the 128^3 variable-coefficient system at the same time per
// iteration, and needs no FP32 copy of the operand.
// A slice is kp/8 chunks of 16 rows x 8 entries.  Per chunk the value loads
// are issued first (they need only the slice offset, known at the top of the
// slice), then the index word, then the gathered x; pre() issues the next
// slice's dependent loads once the first chunk is in flight.
// No row lengths: a row's padding entries are stored as value 0 with index
// byte 0 (slot 0, column 0), so a lane loads and gathers all kp entries of its
// row and the padding adds 0 * x.  Against loads and gathers predicated on
// per-lane row-length words this measured 15 % faster on the 128^3 FP64 solve.
template <int PR, typename Pre>
__device__ __forceinline__ double slice_dot_uniform(const SolverParams &P, int4 h, long long off, int i,
                                                    unsigned hmask, const TileReg &T, const XVec &X, Pre &pre)
{
    const int kp = hdr_kp(h);
    float sc = 0.0f;
    if (PR == MF_P8) sc = (i < hdr_nt(h) && chk_in(CHK_TILE, h.x + i, P.ntiles)) ? P.i8_scale[h.x + i] : 0.0f;
    // (uniform over the half-warp: the slice is skipped by all 16 lanes)
    if (!chk_in(CHK_PAYLOAD, off + (long long)kp * MF_BS - 1, P.n_payload)) return 0.0;
    double acc = 0.0;
    for (int k0 = 0; k0 < kp; k0 += 8) {
        const long long cb = off + (long long)(k0 >> 3) * 128;
        double v64[8];
        float v[8];
        load_chunk<PR>(P, cb, i, 8, v64, v);
        const unsigned long long m8 = __ldcs((const unsigned long long *)(P.meta + cb) + i);
        double xv[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const unsigned mm = (unsigned)(m8 >> (8 * j)) & 0xFFu;
            const int slot = (int)(mm >> 4);
            const int xi = __shfl_sync(hmask, T.xb, slot, 16) + (int)(mm & 15u);
            xv[j] = chk_in(CHK_X, xi, P.chk_xlen) ? X.x64[xi] : 0.0;
            if (PR == MF_P8) v[j] *= __shfl_sync(hmask, sc, slot, 16);
        }
        if (k0 == 0) pre();
#pragma unroll
        for (int j = 0; j < 8; j++) acc = fma(PR == MF_P64 ? v64[j] : (double)v[j], xv[j], acc);
    }
    return acc;
}

// Row i of one slice times x.  The 8 entries of a chunk are loaded together
// (value + gathered x), then accumulated; occupancy (32 warps per SM at 64
// registers) hides part of the memory latency.  Variants with more loads in
// flight per thread (two chunks, or 3-4 blocks per SM at 32-42 registers)
// spilled and were slower.  In mixed mode a slice runs in one precision, the
// most conservative of its tiles' labels (no per-entry dispatch).
template <int MODE, bool F64, typename Pre>
__device__ __forceinline__ double slice_dot(const SolverParams &P, int4 h, int i, unsigned hmask, long long off,
                                            const TileReg &T, const XVec &X, unsigned *cnt, Pre &pre)
{
    // precision codes order FP64 < FP32 < FP16 < INT8: the minimum is the most precise
    int pr = MF_P64;
    if (!(MODE == MODE_FP64 || F64)) {
        pr = __reduce_min_sync(hmask, (i < hdr_nt(h)) ? T.pr : MF_P8);
    }
    if (cnt && i == 0 && chk_in(CHK_TILE, (long long)h.x + hdr_nt(h), (long long)P.ntiles + 1)) {
        // the half-warp's own counter slots (lane 0 writes, no atomics): tile
        // products and entries of the executed precision (the slice's tiles
        // are consecutive, so its entries are a difference of tile payload
        // offsets); a half-warp's counts stay far below 2^32 per solve
        cnt[pr] += (unsigned)hdr_nt(h);
        cnt[5 + pr] += (unsigned)(P.tile_off[h.x + hdr_nt(h)] - P.tile_off[h.x]);
    }
    if (MODE == MODE_FP64 || F64) return slice_dot_uniform<MF_P64>(P, h, off, i, hmask, T, X, pre);
    if (pr == MF_P32) return slice_dot_uniform<MF_P32>(P, h, off, i, hmask, T, X, pre);
    if (pr == MF_P64) return slice_dot_uniform<MF_P64>(P, h, off, i, hmask, T, X, pre);
    if (pr == MF_P16) return slice_dot_uniform<MF_P16>(P, h, off, i, hmask, T, X, pre);
    return slice_dot_uniform<MF_P8>(P, h, off, i, hmask, T, X, pre);
}

// Parity mode: the reference's tile arithmetic (main-cg-mixed.cu:1130-1214):
// per (tile,row) two partial sums (even / odd entry positions, the lane pair of
// the reference), each in the tile's precision -- FP64 fma, FP32 fmaf, FP16
// __hfma on half x, INT8 in int8 on truncated x -- bypass tiles skipped; the
// partials are added to the FP64 row sum, even then odd.
__device__ __forceinline__ void parity_flush(double &acc, int pr, const double *a64, const float *a32,
                                             const __half *a16, const int8_t *a8)
{
    for (int q = 0; q < 2; q++) {
        if (pr == MF_P64) acc += a64[q];
        else if (pr == MF_P32) acc += (double)a32[q];
        else if (pr == MF_P16) acc += (double)__half2float(a16[q]);
        else if (pr == MF_P8) acc += (double)a8[q];
    }
}

__device__ __forceinline__ double slice_dot_parity(const SolverParams &P, int4 h, int i, unsigned hmask, int len,
                                                   const TileReg &T, const XVec &X)
{
    const int kp = hdr_kp(h);
    const long long off = hdr_off(h);
    if (!chk_in(CHK_PAYLOAD, off + (long long)kp * MF_BS - 1, P.n_payload)) return 0.0;
    double acc = 0.0;
    double a64[2] = {0.0, 0.0};
    float a32[2] = {0.0f, 0.0f};
    __half a16[2] = {__float2half_rn(0.0f), __float2half_rn(0.0f)};
    int8_t a8[2] = {0, 0};
    int cur_slot = -1, cur_pr = MF_PSKIP, pos = 0;
    for (int k = 0; k < kp; k++) {
        const bool act = k < len;
        const unsigned mm = act ? (unsigned)P.meta[mf_slot<1>(off, k, i)] : 0u;
        const int slot = (int)(mm >> 4);
        const int xi = __shfl_sync(hmask, T.xb, slot, 16) + (int)(mm & 15u);
        const int pr = __shfl_sync(hmask, T.pr, slot, 16);
        if (!act || !chk_in(CHK_X, xi, P.chk_xlen)) continue;
        if (slot != cur_slot) {
            parity_flush(acc, cur_pr, a64, a32, a16, a8);
            a64[0] = a64[1] = 0.0;
            a32[0] = a32[1] = 0.0f;
            a16[0] = a16[1] = __float2half_rn(0.0f);
            a8[0] = a8[1] = 0;
            cur_slot = slot;
            cur_pr = pr;
            pos = 0;
        }
        const int q = pos & 1;
        if (pr == MF_P64) a64[q] = fma(X.x64[xi], P.v64[mf_slot<8>(off, k, i)], a64[q]);
        else if (pr == MF_P32) a32[q] = fmaf(X.x32[xi], P.v32[mf_slot<4>(off, k, i)], a32[q]);
        else if (pr == MF_P16) a16[q] = __hfma(X.x16[xi], P.v16[mf_slot<2>(off, k, i)], a16[q]);
        else if (pr == MF_P8) a8[q] = (int8_t)((int)a8[q] + (int)X.x8[xi] * (int)P.v8ref[mf_slot<1>(off, k, i)]);
        pos++;
    }
    parity_flush(acc, cur_pr, a64, a32, a16, a8);
    return acc;
}

// Lane i's tile word and row length of slice s (header h).  The bounds-checked
// build checks the tile word's column tile against the operand length and the
// row length against the slice width; a word that fails reads as 0 (column
// tile 0, an empty row).
__device__ __forceinline__ int load_tw(const SolverParams &P, int s, int i)
{
    const int tw = P.seg_tile[(long long)s * MF_BS + i];
    return chk_in(CHK_TILE, (long long)(tw >> 8) * MF_BS, P.chk_xlen) ? tw : 0;
}

__device__ __forceinline__ int load_len(const SolverParams &P, int s, int i, int4 h)
{
    const int len = P.seg_rowlen[(long long)s * MF_BS + i];
    return chk_in(CHK_ROWLEN, len, hdr_kp(h) + 1) ? len : 0;
}

// One chunk of the lean walk: lane i's 8 stored values of a uniform-precision
// slice (FP64: four 16-byte loads; FP32: two; FP16: one) and its index word,
// loaded unpredicated (the stored padding past a row's end is zero).
template <int PR> struct LeanChunk;

template <> struct LeanChunk<MF_P64> {
    double2 d[4];
    unsigned long long m;
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int q = 0; q < 4; q++) d[q] = make_double2(0.0, 0.0);
        m = 0ull;
    }
    // LEN: entries of the longest row; groups past it hold padding only
    template <int LEN = 8>
    __device__ __forceinline__ void load(const SolverParams &P, long long cb, int i)
    {
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (2 * q < LEN) d[q] = __ldcs((const double2 *)(P.v64 + cb + 32 * q) + i);
        m = __ldcs((const unsigned long long *)(P.meta + cb) + i);
    }
    __device__ __forceinline__ void values(double (&v)[8]) const
    {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            v[2 * q] = d[q].x;
            v[2 * q + 1] = d[q].y;
        }
    }
};

template <> struct LeanChunk<MF_P32> {
    float4 a, b;
    unsigned long long m;
    __device__ __forceinline__ void zero()
    {
        a = b = make_float4(0.f, 0.f, 0.f, 0.f);
        m = 0ull;
    }
    template <int LEN = 8>
    __device__ __forceinline__ void load(const SolverParams &P, long long cb, int i)
    {
        a = __ldcs((const float4 *)(P.v32 + cb) + i);
        if (LEN > 4) b = __ldcs((const float4 *)(P.v32 + cb + 64) + i);
        m = __ldcs((const unsigned long long *)(P.meta + cb) + i);
    }
    __device__ __forceinline__ void values(double (&v)[8]) const
    {
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
};

template <> struct LeanChunk<MF_P16> {
    uint4 u;
    unsigned long long m;
    __device__ __forceinline__ void zero()
    {
        u = make_uint4(0u, 0u, 0u, 0u);
        m = 0ull;
    }
    template <int LEN = 8>
    __device__ __forceinline__ void load(const SolverParams &P, long long cb, int i)
    {
        u = __ldcs((const uint4 *)(P.v16 + cb) + i);
        m = __ldcs((const unsigned long long *)(P.meta + cb) + i);
    }
    __device__ __forceinline__ void values(double (&v)[8]) const
    {
        const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int q = 0; q < 4; q++) {
            v[2 * q] = (double)__half2float(__ushort_as_half((unsigned short)(w[q] & 0xFFFFu)));
            v[2 * q + 1] = (double)__half2float(__ushort_as_half((unsigned short)(w[q] >> 16)));
        }
    }
};

// The lean walk: every slice of the range runs stored precision PR (the FP64
// mode; mixed mode when no tile can leave the base precision in this SpMV --
// FP32, or FP16 when every tile is exact in FP16; the standalone SpMVs), no
// per-slice precision reduction; the range's tile and entry totals go to the
// counters once, at the end (entries from the CSR row pointers of the range's
// tile-rows).
// The walk reads no row lengths: a row's padding entries are stored as value
// 0 with index byte 0 (slot 0, column 0), so for them a lane gathers x at the
// slice's first tile column and adds 0 * x.  Without the per-lane row-length
// words (and their predicates) the 128^3 mixed solve measured 10 % faster.
// The walk is software-pipelined by one chunk.  A half-warp's slices are
// stored back to back, so its chunks (kp / 8 per slice) form one contiguous
// stream and chunk c + 1 starts 128 entries after chunk c whatever slice it
// belongs to: its values and index word are requested as soon as chunk c's x
// gathers are issued, so their DRAM trip overlaps chunk c's gathers, sum and
// tile-row epilogue instead of following them.  Sums are formed in the same
// order as slice_dot_uniform (per slice from 0, added to the tile-row's sum).
template <int PR, typename Epi>
__device__ __forceinline__ void spmv_range_lean(const SolverParams &P, int sb, int se, int i, unsigned hmask,
                                                const XVec &X, unsigned *cnt, Epi &epi)
{
    int4 h = P.seg_hdr[sb];
    const int4 hl = P.seg_hdr[se - 1];
    const long long off0 = hdr_off(h);
    const int nch = (int)((hdr_off(hl) + (long long)hdr_kp(hl) * MF_BS - off0) >> 7);
    if (!chk_in(CHK_PAYLOAD, off0, P.n_payload) || !chk_in(CHK_PAYLOAD, off0 + (long long)nch * 128 - 1, P.n_payload))
        return;
    const int R0 = h.y;
    int tw = load_tw(P, sb, i);
    LeanChunk<PR> cur;
    cur.load(P, off0, i);
    int4 hn = make_int4(0, 0, 0, 0);
    int twn = 0;
    int s = sb, kc = 0, kchunks = hdr_kp(h) >> 3;
    unsigned ntiles = 0;
    double acc = 0.0, sacc = 0.0;
    for (int c = 0; c < nch; c++) {
        if (kc == 0 && s + 1 < se) {       // the next slice's words, one slice ahead
            hn = P.seg_hdr[s + 1];
            twn = load_tw(P, s + 1, i);
        }
        const int xb = (tw >> 8) * MF_BS;
        double xv[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const unsigned mm = (unsigned)(cur.m >> (8 * j)) & 0xFFu;
            const int xi = __shfl_sync(hmask, xb, (int)(mm >> 4), 16) + (int)(mm & 15u);
            xv[j] = chk_in(CHK_X, xi, P.chk_xlen) ? X.x64[xi] : 0.0;
        }
        LeanChunk<PR> nxt;
        nxt.zero();
        if (c + 1 < nch) nxt.load(P, off0 + (long long)(c + 1) * 128, i);
        double v[8];
        cur.values(v);
#pragma unroll
        for (int j = 0; j < 8; j++) sacc = fma(v[j], xv[j], sacc);
        if (++kc == kchunks) {             // the slice is done
            ntiles += (unsigned)hdr_nt(h);
            acc += sacc;
            sacc = 0.0;
            if (hdr_last(h)) {
                if (chk_in(CHK_ROW, h.y, P.tilem)) epi(h.y, acc);
                acc = 0.0;
            }
            s++;
            h = hn;
            tw = twn;
            kc = 0;
            kchunks = hdr_kp(h) >> 3;
        }
        cur = nxt;
    }
    if (cnt && i == 0 && chk_in(CHK_ROW, R0, P.tilem) && chk_in(CHK_ROW, hl.y, P.tilem)) {
        cnt[PR] += ntiles;
        cnt[5 + PR] += (unsigned)(P.rowptr[min(P.n, (hl.y + 1) * MF_BS)] - P.rowptr[R0 * MF_BS]);
    }
}

// The walk of a matrix whose every tile-row is one slice of one chunk (rows of
// up to 8 entries in up to 15 tiles: the 5- and 7-point stencils): tile-row R's
// payload starts at entry 128 R and its tile words at 16 R, so there are no
// headers, no slice or chunk counters and nothing to wait for but the chunk.
//
// LEN: no row is longer (5, 7 or 8, a template argument).  Entries past it are
// padding in every row: they are neither loaded (FP64: three of four 16-byte
// groups with 5), nor gathered, nor multiplied.  A run-time length instead put a
// branch between the gathers and cost more than it saved (whole 128^3 FP32
// iterations: 29.4 us with all 8 entries, 34.9 with `j < len`).
//
// A block's half-warps take the block's tile-rows in turn (first, first + stride,
// ... < end): a warp's halves gather from neighbouring rows, and a block sweeps
// matrix and vectors as one stream instead of 32.  Turns over the whole launch
// cost 5 % on 128^3: then the update phase touches a row from another SM than
// the product did.
//
// What bounds it: DRAM for vectors larger than L2 (2048^2 FP64: 485 MB in 79 us,
// 6.1 TB/s, a copy's speed), the gathers' trips to L2 otherwise (128^3 mixed: L2
// 34 % busy, long_scoreboard first among the stalls).  Keeping more in flight was
// tried in whole iterations and did not help: a TMA ring with mbarriers, copies of
// the epilogue's operands with cp.async, gathers one step ahead, 3 or 4 blocks per
// SM; none was faster than this walk with the next chunk in registers.
template <int PR, int LEN, typename Epi>
__device__ __forceinline__ void spmv_rows(const SolverParams &P, int R, int end, int stride, int i, unsigned hmask,
                                          const double *x64, Epi &epi)
{
    if (R >= end) return;
    if (!chk_in(CHK_PAYLOAD, (long long)end * 128 - 1, P.n_payload)) return;
    int tw = load_tw(P, R, i);
    LeanChunk<PR> cur;
    cur.zero();
    cur.template load<LEN>(P, (long long)R * 128, i);
    for (;;) {
        const int xb = (tw >> 8) * MF_BS;
        double xv[LEN];
#pragma unroll
        for (int j = 0; j < LEN; j++) {
            const unsigned mm = (unsigned)(cur.m >> (8 * j)) & 0xFFu;
            const int xi = __shfl_sync(hmask, xb, (int)(mm >> 4), 16) + (int)(mm & 15u);
            xv[j] = chk_in(CHK_X, xi, P.chk_xlen) ? x64[xi] : 0.0;
        }
        const int Rn = R + stride;
        LeanChunk<PR> nxt;
        nxt.zero();
        if (Rn < end) {
            nxt.template load<LEN>(P, (long long)Rn * 128, i);
            tw = load_tw(P, Rn, i);
        }
        double v[8];
        cur.values(v);
        double acc = 0.0;
#pragma unroll
        for (int j = 0; j < LEN; j++) acc = fma(v[j], xv[j], acc);
        epi(R, acc);
        if (Rn >= end) return;
        R = Rn;
        cur = nxt;
    }
}

// The same walk with the precision chosen per slice (or forced to scaled INT8),
// as slice_dot does.
template <int LEN, typename Epi>
__device__ __forceinline__ void spmv_rows_dyn(const SolverParams &P, int R, int end, int stride, int i,
                                              unsigned hmask, const XVec &X, unsigned *cnt, Epi &epi)
{
    if (R < end && !chk_in(CHK_PAYLOAD, (long long)end * 128 - 1, P.n_payload)) return;
    for (; R < end; R += stride) {
        const int4 h = P.seg_hdr[R];
        const int nt = hdr_nt(h);
        const int tw = load_tw(P, R, i);
        const float st = load_stat<MODE_MIXED, false>(X, tw, i, nt);
        const int pr = __reduce_min_sync(hmask, i < nt ? tile_prec<MODE_MIXED, false>(P, tw, st, X) : MF_P8);
        if (cnt && i == 0 && chk_in(CHK_TILE, (long long)h.x + nt, (long long)P.ntiles + 1)) {
            cnt[pr] += (unsigned)nt;
            cnt[5 + pr] += (unsigned)(P.tile_off[h.x + nt] - P.tile_off[h.x]);
        }
        double v64[8];
        float v[8];
        const long long cb = (long long)R * 128;
        if (pr == MF_P32) load_chunk<MF_P32>(P, cb, i, LEN, v64, v);
        else if (pr == MF_P16) load_chunk<MF_P16>(P, cb, i, LEN, v64, v);
        else load_chunk<MF_P8>(P, cb, i, LEN, v64, v);
        const float sc =
            (pr == MF_P8 && i < nt && chk_in(CHK_TILE, h.x + i, P.ntiles)) ? P.i8_scale[h.x + i] : 1.0f;
        const unsigned long long m8 = __ldcs((const unsigned long long *)(P.meta + cb) + i);
        double acc = 0.0;
#pragma unroll
        for (int j = 0; j < LEN; j++) {
            const unsigned mm = (unsigned)(m8 >> (8 * j)) & 0xFFu;
            const int slot = (int)(mm >> 4);
            const int xi = __shfl_sync(hmask, (tw >> 8) * MF_BS, slot, 16) + (int)(mm & 15u);
            const float s8 = __shfl_sync(hmask, sc, slot, 16);     // 1 unless the slice runs INT8
            const double xv = chk_in(CHK_X, xi, P.chk_xlen) ? X.x64[xi] : 0.0;
            acc = fma((double)(v[j] * s8), xv, acc);
        }
        epi(R, acc);
    }
}

// y = A x over the half-warp's slices [sb, se); epi(R, y) is called once per
// tile-row (after its last slice) with the row sum of lane i.
// F64: every tile in FP64 (the FP64 residual replacement and the FP64 SpMV).
//
// Descriptor pipeline: a half-warp's slices are stored back to back, so slice
// s+1 starts where slice s ends (offset + 16 * kp).  The words indexed by the
// slice number alone (header, lane i's tile word, and in parity mode its row
// length) are loaded one slice ahead, at the top of the previous slice,
// together with that slice's own loads; the precision statistic (mixed /
// parity) is loaded one slice ahead once the tile word is in.  A slice then
// waits for two round trips: values + index word, then the gathered x.
// LEN > 0: a one-chunk matrix with rows of up to LEN entries (spmv_rows; the
// range is then the block's own tile-rows in a solve, all of them in turn in the
// standalone product, and sb, se are not used).
// TURN: the half-warps take the block's tile-rows in turn; without it each walks
// its own range, so dot products are summed as by the general walk.  BiCGSTAB
// does: its recurrences amplify the rounding of their order (two orders of the sums
// were 1.9e-9 apart after 20 iterations on a 48^3 upwind system, with FP64's own
// error at 3.7e-9), and turns gave it 3 %.
template <int MODE, bool F64, int LEN, bool TURN, typename Epi>
__device__ __forceinline__ void spmv_range(const SolverParams &P, int sb, int se, int i, unsigned hmask,
                                           const XVec &X, unsigned *cnt, Epi epi, unsigned *whole = nullptr)
{
    if constexpr (LEN > 0) {
        const int h = (int)(threadIdx.x >> 4);
        const int *hb = P.hw_begin ? P.hw_begin + blockIdx.x * kWarps * 2 : nullptr;
        const int R = !hb ? (int)blockIdx.x * kWarps * 2 + h : TURN ? hb[0] + h : hb[h];
        const int end = !hb ? P.tilem : TURN ? hb[kWarps * 2] : hb[h + 1];
        const int stride = !hb ? (int)gridDim.x * kWarps * 2 : TURN ? kWarps * 2 : 1;
        if constexpr (MODE == MODE_FP64 || F64) {
            spmv_rows<MF_P64, LEN>(P, R, end, stride, i, hmask, X.x64, epi);
        } else {
            const int pr = (X.force_pr < 0 && !X.dyn) ? X.lean_pr : X.force_pr;
            if (pr == MF_P32) spmv_rows<MF_P32, LEN>(P, R, end, stride, i, hmask, X.x64, epi);
            else if (pr == MF_P16) spmv_rows<MF_P16, LEN>(P, R, end, stride, i, hmask, X.x64, epi);
            else spmv_rows_dyn<LEN>(P, R, end, stride, i, hmask, X, cnt, epi);
            if (whole && (pr == MF_P32 || pr == MF_P16) && blockIdx.x == 0 && threadIdx.x == 0) whole[pr]++;
        }
        return;
    }
    if (sb >= se) return;
    if (!chk_in(CHK_SLICE, sb, P.nseg) || !chk_in(CHK_SLICE, se - 1, P.nseg)) return;
    // the FP64 mode takes the pipelined walk too (128^3 FP64 CG 62.0 -> 60.3 ms);
    // the mixed mode's FP64 replacement SpMVs do not: in that kernel the extra
    // code cost the mixed solve more (61.3 -> 62.0 ms) than it saved
    if (MODE == MODE_FP64) {
        spmv_range_lean<MF_P64>(P, sb, se, i, hmask, X, cnt, epi);
        return;
    }
    if (MODE == MODE_MIXED && !F64) {
        const int lean = (X.force_pr < 0 && !X.dyn) ? X.lean_pr : X.force_pr;
        if (lean == MF_P32) {
            spmv_range_lean<MF_P32>(P, sb, se, i, hmask, X, cnt, epi);
            return;
        }
        if (lean == MF_P16) {
            spmv_range_lean<MF_P16>(P, sb, se, i, hmask, X, cnt, epi);
            return;
        }
    }
    // row lengths: parity mode only (its tile arithmetic walks real entries)
    constexpr bool kLen = (MODE == MODE_PARITY && !F64);
    int4 h = P.seg_hdr[sb];
    int tw = load_tw(P, sb, i);
    int len = kLen ? load_len(P, sb, i, h) : 0;
    float st = load_stat<MODE, F64>(X, tw, i, hdr_nt(h));
    long long off = hdr_off(h);
    double acc = 0.0;
    for (int s = sb; s < se; s++) {
        const bool more = s + 1 < se;
        int4 hn = make_int4(0, 0, 0, 0);
        int twn = 0, lenn = 0;
        if (more) {
            hn = P.seg_hdr[s + 1];
            twn = load_tw(P, s + 1, i);
            lenn = kLen ? load_len(P, s + 1, i, hn) : 0;
        }
        float stn = 0.0f;
        auto pre = [&]() {
            if (more) stn = load_stat<MODE, F64>(X, twn, i, hdr_nt(hn));
        };
        TileReg T;
        T.xb = (tw >> 8) * MF_BS;
        T.pr = tile_prec<MODE, F64>(P, tw, st, X);
        if (MODE == MODE_PARITY && !F64) {
            pre();
            if (cnt && i < hdr_nt(h) && chk_in(CHK_TILE, h.x + i, P.ntiles)) {
                const int t = h.x + i;
                atomicAdd(&cnt[T.pr], 1u);
                atomicAdd(&cnt[5 + T.pr], (unsigned)(P.tile_off[t + 1] - P.tile_off[t]));
            }
            acc += slice_dot_parity(P, h, i, hmask, len, T, X);
        } else {
            acc += slice_dot<MODE, F64>(P, h, i, hmask, off, T, X, cnt, pre);
        }
        if (hdr_last(h)) {
            if (chk_in(CHK_ROW, h.y, P.tilem)) epi(h.y, acc);
            acc = 0.0;
        }
        off += (long long)hdr_kp(h) * MF_BS;
        h = hn;
        tw = twn;
        len = lenn;
        st = stn;
    }
}

// ------------------------------------------------------------ phases
struct Ctx {
    int lane, wib, half, i, rbeg, rend, sbeg, send;
    unsigned hmask;
};

__device__ __forceinline__ Ctx make_ctx(const SolverParams &P)
{
    Ctx c;
    c.lane = threadIdx.x & 31;
    c.wib = threadIdx.x >> 5;
    c.half = c.lane >> 4;
    c.i = c.lane & 15;
    c.hmask = 0xFFFFu << (16 * c.half);
    const int hw = (blockIdx.x * kWarps + c.wib) * 2 + c.half;
    c.rbeg = P.hw_begin[hw];
    c.rend = P.hw_begin[hw + 1];
    c.sbeg = P.seg_ptr[c.rbeg];
    c.send = P.seg_ptr[c.rend];
    return c;
}

// max over the 16 lanes of a half-warp; hmask names exactly those lanes (the
// two halves of a warp walk different tile-row ranges, so they never reduce
// together).  One redux.sync instead of a shuffle tree.  half_max takes
// magnitudes (v >= 0), whose IEEE order is the order of their bit patterns.
__device__ __forceinline__ float half_max(float v, unsigned hmask)
{
    return __int_as_float(__reduce_max_sync(hmask, __float_as_int(v)));
}
__device__ __forceinline__ int half_max_i(int v, unsigned hmask)
{
    return __reduce_max_sync(hmask, v);
}

// reference label rank of |dp| (main-cg-mixed.cu:1334-1351): 4 FP64, 3 FP32, 2 FP16, 1 INT8, 0 none
__device__ __forceinline__ int ref_rank(double dp)
{
    if (dp <= 1e-7 && dp > 1e-8) return 1;
    if (dp <= 1e-6 && dp > 1e-7) return 2;
    if (dp <= 1e-5 && dp > 1e-6) return 3;
    if (dp > 1e-5) return 4;
    return 0;
}
__device__ __forceinline__ signed char rank_to_vis(int rank)
{
    // 0 -> bypass(1), 1 -> int8(2), 2 -> fp16(3), 3 -> fp32(4), 4 -> fp64(0)
    return (signed char)(rank == 0 ? 1 : rank == 1 ? 2 : rank == 2 ? 3 : rank == 3 ? 4 : 0);
}

// (int8_t) of a double as the x86-64 host compiler emits it (truncate to int32,
// 0x80000000 when NaN / out of range, keep the low byte) -- the reference
// converts p this way (main-cg-mixed.cu:435).
__device__ __forceinline__ int8_t trunc_i8(double v)
{
    int w;
    if (!(v == v) || v >= 2147483648.0 || v < -2147483648.0) w = (int)0x80000000u;
    else w = (int)v;
    return (int8_t)(unsigned char)(w & 0xFF);
}

// Write a direction vector's shadows and segment statistics for the rows of
// tile-row R (all 16 lanes of the half-warp call this together).
template <int MODE>
__device__ __forceinline__ void publish_dir(int R, int row, bool valid, double vnew, double vold, float *v32,
                                            __half *v16, int8_t *v8, float *mag, signed char *lab, float &bmax,
                                            unsigned hmask, bool labels, float *bmin = nullptr,
                                            float small_thr = -1.0f, float *nsmall = nullptr)
{
    if (MODE == MODE_PARITY && valid) v32[row] = (float)vnew;
    if (MODE == MODE_MIXED) {
        float m = half_max(valid ? (float)fabs(vnew) : 0.0f, hmask);
        bmax = fmaxf(bmax, m);
        if (bmin) *bmin = fminf(*bmin, m);
        // segments at or below small_thr (demote_fp16 x the operand's previous maximum)
        if (nsmall && (threadIdx.x & 15) == 0 && m <= small_thr) *nsmall += 1.0f;
        if ((threadIdx.x & 15) == 0) mag[R] = m;
    } else if (MODE == MODE_PARITY) {
        if (valid) {
            v16[row] = __double2half(vnew);
            v8[row] = trunc_i8(vnew);
        }
        if (labels) {
            // reference rule: label of the next SpMV's tile column from |v_new - v_old|
            int rk = half_max_i(valid ? ref_rank(fabs(vnew - vold)) : 0, hmask);
            if ((threadIdx.x & 15) == 0) lab[R] = rank_to_vis(rk);
        }
    }
}

__device__ __forceinline__ XVec make_x(const double *x64, const float *x32, const __half *x16, const int8_t *x8,
                                       const float *mag, const signed char *lab, float invM, int dyn = 1)
{
    XVec X;
    X.x64 = x64;
    X.x32 = x32;
    X.x16 = x16;
    X.x8 = x8;
    X.mag = mag;
    X.lab = lab;
    X.invM = invM;
    X.force_pr = -1;
    X.dyn = dyn;
    X.lean_pr = MF_P32;
    return X;
}

__device__ __forceinline__ XVec fp64_x(const double *x64)
{
    XVec X = make_x(x64, nullptr, nullptr, nullptr, nullptr, nullptr, 0.f);
    X.force_pr = MF_P64;
    return X;
}

// LB = minimum resident blocks per SM the register budget is sized for:
// 1 -> up to 128 registers (no spills, 16 warps / SM), 2 -> 64 registers (32 warps / SM).
// Block 0 / thread 0 splits its wall time into phases (%globaltimer deltas);
// the state lives in shared memory so the other threads spend no registers on it.
template <class SH>
struct PhaseClock {
    SH *sh;
    __device__ bool on() const { return blockIdx.x == 0 && threadIdx.x == 0; }
    __device__ void start(SH *s)
    {
        sh = s;
        if (on()) {
            sh->clk_t = mf_globaltimer();
            for (int j = 0; j < 5; j++) sh->clk_acc[j] = 0ull;
        }
    }
    __device__ void lap(int ph)
    {
        if (on()) {
            const unsigned long long n = mf_globaltimer();
            sh->clk_acc[ph] += n - sh->clk_t;
            sh->clk_t = n;
        }
    }
};
enum { PH_SPMV = 0, PH_VECB = 1, PH_VECC = 2, PH_BAR = 3, PH_REPL = 4 };

// After an FP64 residual replacement r = b - A x: keep the CG direction only
// while the recursive residual still told the truth.  When the replacement
// follows a failed convergence check (the recursive residual claimed
// convergence, the true one did not) or the two squared norms differ by more
// than 4x, the recursive residual has drifted to the accuracy floor of the
// low-precision products; beta = r_true.r_true / r_old.r_old would then be
// meaningless (huge when r_old has collapsed), so CG restarts from the true
// residual (beta = 0, which also makes q = A p consistent again).
__device__ __forceinline__ bool restart_after_replacement(bool failed_check, double rr_true, double rr_rec)
{
    return failed_check || rr_true > 4.0 * rr_rec || 4.0 * rr_true < rr_rec;
}

// Relaxed matvec precision (mixed CG): inexact Krylov theory (van den Eshof &
// Sleijpen, SIAM J. Matrix Anal. Appl. 26(1), 2004; Bouras & Fraysse, SIAM J.
// Matrix Anal. Appl. 26(3), 2005) lets the relative error of the product at
// iteration k grow like eps_k = eta * tol / (||r_k|| / ||b||): the further the
// solve has converged, the coarser the operator may be.  The whole SpMV then
// runs in the narrowest stored precision whose rounding stays below eps_k:
// FP16 (unit roundoff 2^-11) when every tile fits FP16's normal range and,
// when allowed, scaled INT8 (half a step of the tile's largest magnitude /
// 127, below 2^-8 of it).  The FP64 residual replacement and the convergence
// test on the FP64 true residual keep the final accuracy either way.
constexpr double kRoundF16 = 1.0 / 2048.0;
constexpr double kRoundI8 = 1.0 / 256.0;
__device__ __forceinline__ int relaxed_precision(const SolverParams &P, double rr, double bb)
{
    if (P.relax_eta <= 0.0f || !(bb > 0.0) || !(rr > 0.0)) return MF_P32;
    const double eps = (double)P.relax_eta * P.tol / sqrt(rr / bb);
    if (P.relax_int8 && eps >= kRoundI8) return MF_P8;
    if (eps >= kRoundF16 && P.fp16_ok) return MF_P16;
    return MF_P32;
}

// METH: MF_METHOD_CG or MF_METHOD_BICGSTAB.  One instantiation per method, so
// each gets its own register allocation: the kernel sits at the 64-register
// limit of two 512-thread blocks per SM, and code in one method's branch
// moves spills into the other's hot loop.
enum { kVarGrid = 0, kVarResident = 1, kVarCluster = 2, kVarCluster2 = 3 };
// LEN > 0: for one-chunk matrices with rows of up to LEN entries (spmv_rows); these
// instantiations hold none of the general walks.
// VAR: kVarGrid the whole chip; kVarResident a grid with no more tile-rows than
// half-warps (CG iterations stay in registers); kVarCluster and kVarCluster2 one
// cluster with up to one and two tile-rows per half-warp in registers (four did
// not fit 128 registers: 32,768 rows took 8.0 us an iteration against 6.9 on the
// grid).  Instantiations of their own: the resident loop and the cluster's
// reduction inside the large kernels raised their spills from 0 - 68 to 250 - 300
// bytes.
template <int MODE, int LB, int METH, int LEN, int VAR>
__global__ void __launch_bounds__(kThreads, LB) k_solve(SolverParams P)
{
    constexpr bool CL = VAR >= kVarCluster;
    __shared__ SharedT<CL> sh;
    if constexpr (CL) cluster_barrier();       // every block has started: see cluster_store
    const Ctx c = make_ctx(P);
    unsigned epoch = 0;
    // tile-use counters: FP64 mode needs none (every tile of every SpMV is FP64;
    // the host derives the totals from the SpMV count)
    unsigned *cnt = (MODE == MODE_FP64) ? nullptr : sh.cnt[c.wib * 2 + c.half];
    if (cnt && c.i < 10) cnt[c.i] = 0u;
    if (threadIdx.x < 4) sh.whole[threadIdx.x] = 0u;
    int nspmv = 0;
    __syncwarp();
    PhaseClock<SharedT<CL>> clk;
    clk.start(&sh);
    const int n = P.n;
    constexpr bool bicg = (METH == MF_METHOD_BICGSTAB);

    // ---- init: x = 0 (owned rows), r = b, p = r (rh = r) ----
    // With an initial guess: r = b - A x in FP64, and |b|^2 reduced on its own
    // first (it scales the convergence test).
    double pb = 0.0, bb0 = 0.0;
    float bmax = 0.0f, bmin = 3.0e38f, nsm = 0.0f;   // no previous maximum: nothing counts as small
    if (P.x0_given) {
        double pbb = 0.0;
        for (int R = c.rbeg; R < c.rend; R++) {
            const int row = R * MF_BS + c.i;
            if (row < n) pbb += P.b[row] * P.b[row];
        }
        block_partial(P, sh, 8, pbb, 0, 0, 0, 1, 0u);
        if (!solve_barrier(P, epoch, sh)) return;
        double vb[4] = {0.0, 0.0, 0.0, 0.0};
        grid_collect(P, sh, 8, 1, 0u, vb);
        bb0 = vb[0];
        auto init_row = [&](int R, double y) {
            const int row = R * MF_BS + c.i;
            const bool valid = row < n;
            const double rv = valid ? P.b[row] - y : 0.0;
            if (valid) {
                P.r[row] = rv;
                P.p[row] = rv;
                if (bicg) P.rh[row] = rv;
                else P.q[row] = 0.0;               // the first q = w + 0 q
            }
            publish_dir<MODE>(R, row, valid, rv, 0.0, P.p32, P.p16, P.p8, P.mag_p, P.lab_p, bmax, c.hmask, false,
                              &bmin);
            pb += rv * rv;
        };
        spmv_range<MODE, true, LEN, !bicg>(P, c.sbeg, c.send, c.i, c.hmask, fp64_x(P.x), nullptr, init_row);
        for (int R = c.rbeg; LEN == 0 && R < c.rend; R++)
            if (P.seg_ptr[R] == P.seg_ptr[R + 1]) init_row(R, 0.0);
        nspmv++;
    } else {
        for (int R = c.rbeg; R < c.rend; R++) {
            const int row = R * MF_BS + c.i;
            const bool valid = row < n;
            const double bv = valid ? P.b[row] : 0.0;
            if (valid) {
                P.x[row] = 0.0;
                P.r[row] = bv;
                P.p[row] = bv;
                if (bicg) P.rh[row] = bv;
                else P.q[row] = 0.0;               // the first q = w + 0 q
            }
            // parity mode: labels start all FP64 (cudaMemset(d_vis, 0), main-cg-mixed.cu:2828)
            publish_dir<MODE>(R, row, valid, bv, 0.0, P.p32, P.p16, P.p8, P.mag_p, P.lab_p, bmax, c.hmask, false,
                              &bmin);
            pb += bv * bv;
        }
    }
    // the smallest segment magnitude (carried as -min) matters only to the mixed
    // mode's SpMV; FP64 and parity reduce (sum, max) as before
    // (sum, max, -min, small segments) in mixed mode, (sum, max) in parity mode; FP64
    // reads no magnitudes and reduces the sum alone
    constexpr int kNvSeg = (MODE == MODE_MIXED) ? 4 : (MODE == MODE_PARITY) ? 2 : 1;
    constexpr int kNvSegB = (MODE == MODE_MIXED) ? 3 : (MODE == MODE_PARITY) ? 1 : 0;   // without a sum
    block_partial(P, sh, 0, pb, (double)bmax, -(double)bmin, (double)nsm, kNvSeg, 0x6u);
    if (!solve_barrier(P, epoch, sh)) return;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    grid_collect(P, sh, 0, kNvSeg, 0x6u, v);
    // mixed: can any tile of the next SpMV leave FP32 at all?  Not when the
    // smallest column segment is within demote_fp16 of the largest and no tile
    // is exact in a narrower type: then the SpMV skips its precision lookups.
    // And narrower tiles are considered only when enough segments were small
    // (demote_min_fraction): a few demoted tiles save fewer bytes than the
    // lookups cost in a latency-bound SpMV.
    auto dyn_of = [&](double mx, double neg_mn, double nsmall) -> int {
        return (P.lossless_any ||
                ((mx <= 0.0 || -neg_mn <= (double)P.demote16 * mx) && nsmall >= (double)P.min_small)) ? 1 : 0;
    };
    int dynA = (MODE == MODE_MIXED) ? dyn_of(v[1], v[2], v[3]) : 0;
    // Feedback on the per-slice lookups (mixed BiCGSTAB): each SpMV's reduction
    // also carries how many tiles it ran below FP32.  A dynamic SpMV that
    // demoted fewer than min_demoted (demote_min_fraction of the tiles) did
    // not pay for its lookups, and the same operand's next kDemoteCool SpMVs
    // run the lean walk.  (A slice demotes only when all of its tiles'
    // segments are small: on the 96^3 BiCGSTAB system 1.3 % of the tile
    // products ran below FP32 while the lookups cost 7 % of the solve.)  CG
    // goes without it: the extra reduction value and counters cost its mixed
    // 128^3 solve 3.5 % although its lookups never engage there.
    constexpr bool kFb = (MODE == MODE_MIXED) && bicg;
    constexpr int kNvFb = kFb ? 2 : 1;
    auto demoted = [&]() -> unsigned { return (kFb && c.i == 0) ? cnt[MF_P16] + cnt[MF_P8] : 0u; };
    auto next_cool = [&](int cool, bool was_dyn, double dem) -> int {
        return cool > 0 ? cool - 1 : (was_dyn && dem < (double)P.min_demoted) ? kDemoteCool : 0;
    };
    int coolA = 0, coolS = 0;
    // the base precision of the lookup-free walk (FP16 when every tile is exact in it)
    auto lean_base = [&](XVec X) -> XVec {
        if (P.lean_f16) X.lean_pr = MF_P16;
        return X;
    };
    // mixed CG: the x / r update records r's per-segment magnitudes (one
    // half-warp max reduction and one store per tile-row, 4.5 % of the 128^3
    // solve) only while enough segments were small in the last update that the
    // next SpMV may demote tiles; otherwise it keeps just r's maximum and the
    // count of small segments (a vote per tile-row, on every 4th update only:
    // 1.5 % of the solve when taken on every one), and the next SpMV runs
    // all-FP32.  Demotion then starts up to four updates after the small
    // segments do.
    const float half_small = 0.5f * fmaxf(1.0f, P.min_small);
    int magB = (MODE == MODE_MIXED) ? ((P.lossless_any || v[3] >= (double)half_small) ? 1 : 0) : 1;
            clk.lap(PH_BAR);
    const double bb = P.x0_given ? bb0 : v[0];
    double rr = v[0], r1 = v[0];
    float invM = v[1] > 0.0 ? (float)(1.0 / v[1]) : 0.0f;
    float invMs = 0.0f;
    const double thr2 = P.tol * P.tol * bb;
    int k = 0, conv = 0, repl = 0, status = 0, last_true = 0;
    double rr_true = rr;
    if (!P.fixed_iters && rr <= thr2) { conv = 1; last_true = 1; }

    // tile-rows without slices (all-zero rows) get no SpMV epilogue
    bool has_empty = false;
    if (LEN == 0)
        for (int R = c.rbeg; R < c.rend && !has_empty; R++) has_empty = P.seg_ptr[R] == P.seg_ptr[R + 1];
    double beta2 = 0.0;
    // mixed CG: uniform reduced precision of the next SpMV (relaxed_precision)
    int prA = (MODE == MODE_MIXED) ? relaxed_precision(P, rr, bb) : MF_P32;

    // ---- resident iterations (CG, one-chunk matrices, up to kKR tile-rows per half-warp) ----
    // With no more tile-rows than that (kKR = 1 on the grid: 151,552 rows on 148 SMs)
    // everything a lane needs of its rows stays in registers from one iteration to
    // the next: values, gather positions, p, q, x and r.  An iteration is then the
    // gather of r from L2, two reductions and one store of r.  Without it an
    // iteration of the 256^2 Laplacian spent 2.2 us (FP64) on loads that depend on
    // one another (tile word and values, gathered r, then p and q; x, p, r, q in the
    // update).
    // The loop leaves for the general iteration's tail (`tail`) when a residual
    // replacement or a convergence check is due, at the end, and in mixed mode when
    // enough segments are small that narrower tiles may be chosen; x, p and q
    // are written back then, and a barrier makes them visible.
    constexpr bool kRes = VAR != kVarGrid && MODE != MODE_PARITY && !bicg && LEN > 0;
    constexpr int kKR = VAR == kVarCluster2 ? 2 : 1;
    constexpr int kLen = LEN > 0 ? LEN : 1;
    const int resR = (int)(blockIdx.x * kWarps * 2 + (threadIdx.x >> 4)), resS = (int)gridDim.x * kWarps * 2;
    const bool resident = kRes && P.tilem <= kKR * resS && P.relax_eta <= 0.0f;

    while (!conv && k < P.max_iter) {
        bool tail = false;
        double rr_tail = 0.0;
        float rthr = invM > 0.0f ? P.demote16 / invM : -1.0f;
        if constexpr (kRes) {
            if (resident && !dynA && (MODE == MODE_FP64 || !magB)) {
                typename std::conditional<MODE == MODE_FP64, double, float>::type val[kKR][kLen];
                int at[kKR][kLen];
                double xr[kKR], pr[kKR], qr[kKR], rv[kKR];
                bool own[kKR], valid[kKR];
#pragma unroll
                for (int u = 0; u < kKR; u++) {
                    const int R = resR + u * resS, row = R * MF_BS + c.i;
                    own[u] = R < P.tilem;                       // uniform over the half-warp
                    valid[u] = own[u] && row < n;
#pragma unroll
                    for (int j = 0; j < kLen; j++) {
                        val[u][j] = 0;
                        at[u][j] = 0;
                    }
                    const long long cb = (long long)R * 128;
                    if (own[u] && chk_in(CHK_PAYLOAD, cb + 127, P.n_payload)) {
                        const int xb = (load_tw(P, R, c.i) >> 8) * MF_BS;
                        const unsigned long long m8 = *((const unsigned long long *)(P.meta + cb) + c.i);
#pragma unroll
                        for (int j = 0; j < LEN; j++) {
                            const unsigned mm = (unsigned)(m8 >> (8 * j)) & 0xFFu;
                            const int xi = __shfl_sync(c.hmask, xb, (int)(mm >> 4), 16) + (int)(mm & 15u);
                            if (!chk_in(CHK_X, xi, P.chk_xlen)) continue;
                            at[u][j] = xi;
                            if (MODE == MODE_FP64) val[u][j] = P.v64[mf_slot<8>(cb, j, c.i)];
                            else val[u][j] = P.lean_f16 ? __half2float(P.v16[mf_slot<2>(cb, j, c.i)])
                                                        : P.v32[mf_slot<4>(cb, j, c.i)];
                        }
                    }
                    xr[u] = valid[u] ? P.x[row] : 0.0;
                    pr[u] = valid[u] ? P.p[row] : 0.0;
                    qr[u] = valid[u] ? P.q[row] : 0.0;
                    rv[u] = valid[u] ? P.r[row] : 0.0;
                }
                unsigned done = 0;
                for (;;) {
                    double ppq = 0.0;
                    {
                        double xv[kKR][kLen];
#pragma unroll
                        for (int u = 0; u < kKR; u++)
                            if (own[u]) {
#pragma unroll
                                for (int j = 0; j < LEN; j++) xv[u][j] = P.r[at[u][j]];
                            }
#pragma unroll
                        for (int u = 0; u < kKR; u++) {
                            double w = 0.0;
                            if (own[u]) {
#pragma unroll
                                for (int j = 0; j < LEN; j++) w = fma((double)val[u][j], xv[u][j], w);
                            }
                            pr[u] = rv[u] + beta2 * pr[u];
                            qr[u] = w + beta2 * qr[u];
                            if (valid[u]) ppq += pr[u] * qr[u];
                        }
                    }
                    done++;
                    clk.lap(PH_SPMV);
                    block_partial(P, sh, 1, ppq, 0, 0, 0, 1, 0u);
                    if (!solve_barrier(P, epoch, sh)) return;
                    grid_collect(P, sh, 1, 1, 0u, v);
                    clk.lap(PH_BAR);
                    const double alpha2 = rr / v[0];
                    if (!isfinite(alpha2)) { status = MF_ERR_BREAKDOWN; break; }
                    rthr = invM > 0.0f ? P.demote16 / invM : -1.0f;
                    const bool voteB = (k & 3) == 0;
                    double prr = 0.0;
                    float rmax = 0.0f, rsm = 0.0f;
#pragma unroll
                    for (int u = 0; u < kKR; u++) {
                        xr[u] += alpha2 * pr[u];
                        rv[u] = valid[u] ? rv[u] - alpha2 * qr[u] : 0.0;
                        if (valid[u]) P.r[(resR + u * resS) * MF_BS + c.i] = rv[u];
                        prr += rv[u] * rv[u];
                        const float m = (float)fabs(rv[u]);
                        rmax = fmaxf(rmax, m);
                        if (MODE == MODE_MIXED && voteB && own[u] && __all_sync(c.hmask, m <= rthr) && c.i == 0)
                            rsm += 1.0f;
                    }
                    clk.lap(PH_VECB);
                    // (without counted segments only r's norm and maximum are read)
                    const int nvB = (MODE == MODE_MIXED && !voteB) ? 2 : kNvSeg;
                    block_partial(P, sh, 2, prr, (double)rmax, -(double)3.0e38f, (double)rsm, nvB, 0x6u);
                    if (!solve_barrier(P, epoch, sh)) return;
                    grid_collect(P, sh, 2, nvB, 0x6u, v);
                    clk.lap(PH_BAR);
                    invM = v[1] > 0.0 ? (float)(1.0 / v[1]) : 0.0f;
                    if (MODE == MODE_MIXED && voteB) magB = (P.lossless_any || v[3] >= (double)half_small) ? 1 : 0;
                    if ((!P.fixed_iters && v[0] <= thr2) || (P.replace_every > 0 && (k + 1) % P.replace_every == 0) ||
                        k + 1 >= P.max_iter || (MODE == MODE_MIXED && magB))
                        break;
                    beta2 = v[0] / rr;
                    rr = v[0];
                    k++;
                    last_true = 0;
                }
                rr_tail = v[0];
                tail = true;
                nspmv += (int)done;
                if (MODE == MODE_MIXED && blockIdx.x == 0 && threadIdx.x == 0)
                    sh.whole[P.lean_f16 ? MF_P16 : MF_P32] += done;
#pragma unroll
                for (int u = 0; u < kKR; u++)
                    if (valid[u]) {
                        const int row = (resR + u * resS) * MF_BS + c.i;
                        P.x[row] = xr[u];
                        P.p[row] = pr[u];
                        P.q[row] = qr[u];
                    }
                if (!solve_barrier(P, epoch, sh)) return;
                if (status) break;
            }
        }
        if (MODE != MODE_PARITY && !bicg) {
            double rr_new = rr_tail;
            float rmax = 0.0f, rmin = 3.0e38f, rsm = 0.0f;
            if (!tail) {
            // CG with two grid syncs per iteration.  The SpMV is applied to r:
            // w = A r, then p = r + beta p and q = A p = w + beta q, so p never
            // needs a halo of its own; alpha = r.r / p.q and beta = r'.r' / r.r
            // are the textbook CG scalars (main-cg-mixed.cu:1224-1382 keeps the
            // same formulas with the SpMV on p and a third sync).
            // ---- A: w = A r; p = r + beta p; q = w + beta q; p.q ----
            // (mixed: with a relaxed precision prA the whole SpMV runs in it)
            double ppq = 0.0;
            XVec XA = make_x(P.r, nullptr, nullptr, nullptr, P.mag_r, nullptr, invM, dynA);
            if (MODE == MODE_MIXED && prA != MF_P32) XA.force_pr = prA;
            if (P.lean_f16) XA.lean_pr = MF_P16;
            spmv_range<MODE, false, LEN, !bicg>(P, c.sbeg, c.send, c.i, c.hmask, XA, cnt, [&](int R, double y) {
                const int row = R * MF_BS + c.i;
                if (row < n) {
                    const double pn = P.r[row] + beta2 * P.p[row];
                    const double qn = y + beta2 * P.q[row];
                    P.p[row] = pn;
                    P.q[row] = qn;
                    ppq += pn * qn;
                }
            }, sh.whole);
            if (has_empty) {
                for (int R = c.rbeg; LEN == 0 && R < c.rend; R++) {
                    if (P.seg_ptr[R] != P.seg_ptr[R + 1]) continue;
                    const int row = R * MF_BS + c.i;
                    if (row < n) {
                        const double pn = P.r[row] + beta2 * P.p[row];
                        const double qn = beta2 * P.q[row];
                        P.p[row] = pn;
                        P.q[row] = qn;
                        ppq += pn * qn;
                    }
                }
            }
            nspmv++;
            clk.lap(PH_SPMV);
            block_partial(P, sh, 1, ppq, 0, 0, 0, 1, 0u);
            if (!solve_barrier(P, epoch, sh)) return;
            grid_collect(P, sh, 1, 1, 0u, v);
            clk.lap(PH_BAR);
            const double alpha2 = rr / v[0];
            if (!isfinite(alpha2)) { status = MF_ERR_BREAKDOWN; break; }
            // ---- B: x += alpha p; r -= alpha q; r.r; r's shadow ----
            double prr = 0.0;
            const bool voteB = magB || (k & 3) == 0;     // this update counts small segments
            // kVB tile-rows per step: all loads first, so kVB round trips overlap
            for (int R0 = c.rbeg; R0 < c.rend; R0 += kVB) {
                double xv[kVB], pv[kVB], rv[kVB], qv[kVB];
#pragma unroll
                for (int u = 0; u < kVB; u++) {
                    const int row = (R0 + u) * MF_BS + c.i;
                    const bool valid = R0 + u < c.rend && row < n;
                    xv[u] = valid ? P.x[row] : 0.0;
                    pv[u] = valid ? P.p[row] : 0.0;
                    rv[u] = valid ? P.r[row] : 0.0;
                    qv[u] = valid ? P.q[row] : 0.0;
                }
#pragma unroll
                for (int u = 0; u < kVB; u++) {
                    const int R = R0 + u;
                    if (R >= c.rend) break;      // uniform over the half-warp
                    const int row = R * MF_BS + c.i;
                    const bool valid = row < n;
                    const double rn = valid ? rv[u] - alpha2 * qv[u] : 0.0;
                    if (valid) {
                        P.x[row] = xv[u] + alpha2 * pv[u];
                        P.r[row] = rn;
                        prr += rn * rn;
                    }
                    if (MODE != MODE_MIXED || magB) {
                        publish_dir<MODE>(R, row, valid, rn, 0.0, nullptr, nullptr, nullptr, P.mag_r, nullptr, rmax,
                                          c.hmask, false, &rmin, rthr, &rsm);
                    } else {
                        const float m = valid ? (float)fabs(rn) : 0.0f;
                        rmax = fmaxf(rmax, m);
                        if (voteB && __all_sync(c.hmask, m <= rthr) && c.i == 0) rsm += 1.0f;
                    }
                }
            }
            clk.lap(PH_VECB);
            block_partial(P, sh, 2, prr, (double)rmax, -(double)rmin, (double)rsm, kNvSeg, 0x6u);
            if (!solve_barrier(P, epoch, sh)) return;
            grid_collect(P, sh, 2, kNvSeg, 0x6u, v);
            clk.lap(PH_BAR);
            rr_new = v[0];
            invM = v[1] > 0.0 ? (float)(1.0 / v[1]) : 0.0f;
            if (MODE == MODE_MIXED) {
                dynA = magB ? dyn_of(v[1], v[2], v[3]) : 0;
                if (voteB) magB = (P.lossless_any || v[3] >= (double)half_small) ? 1 : 0;
            }
            }
            const double rr_rec = rr_new;       // recursive r.r of this iteration
            k++;
            last_true = 0;
            const bool want_check = !P.fixed_iters && rr_new <= thr2;
            const bool want_repl = P.replace_every > 0 && (k % P.replace_every) == 0;
            bool restart = false;
            if (want_check || want_repl) {
                // ---- FP64 true residual r = b - A x (x is current), r's shadow ----
                double prt = 0.0;
                rmax = 0.0f;
                rmin = 3.0e38f;
                rsm = 0.0f;
                spmv_range<MODE, true, LEN, !bicg>(P, c.sbeg, c.send, c.i, c.hmask, fp64_x(P.x), nullptr,
                                       [&](int R, double y) {
                                           const int row = R * MF_BS + c.i;
                                           const bool valid = row < n;
                                           double rv = 0.0;
                                           if (valid) {
                                               rv = P.b[row] - y;
                                               P.r[row] = rv;
                                               prt += rv * rv;
                                           }
                                           publish_dir<MODE>(R, row, valid, rv, 0.0, nullptr, nullptr, nullptr,
                                                             P.mag_r, nullptr, rmax, c.hmask, false, &rmin,
                                                             rthr, &rsm);
                                       });
                if (has_empty) {
                    for (int R = c.rbeg; LEN == 0 && R < c.rend; R++) {
                        if (P.seg_ptr[R] != P.seg_ptr[R + 1]) continue;
                        const int row = R * MF_BS + c.i;
                        const bool valid = row < n;
                        const double rv = valid ? P.b[row] : 0.0;
                        if (valid) {
                            P.r[row] = rv;
                            prt += rv * rv;
                        }
                        publish_dir<MODE>(R, row, valid, rv, 0.0, nullptr, nullptr, nullptr, P.mag_r, nullptr, rmax,
                                          c.hmask, false, &rmin, rthr, &rsm);
                    }
                }
                clk.lap(PH_REPL);
                block_partial(P, sh, 5, prt, (double)rmax, -(double)rmin, (double)rsm, kNvSeg, 0x6u);
                if (!solve_barrier(P, epoch, sh)) return;
                grid_collect(P, sh, 5, kNvSeg, 0x6u, v);
                clk.lap(PH_BAR);
                rr_new = v[0];
                invM = v[1] > 0.0 ? (float)(1.0 / v[1]) : 0.0f;
                if (MODE == MODE_MIXED) {
                    dynA = dyn_of(v[1], v[2], v[3]);     // the replacement records every segment
                    magB = (P.lossless_any || v[3] >= (double)half_small) ? 1 : 0;
                }
                rr_true = rr_new;
                repl++;
                last_true = 1;
                if (!P.fixed_iters && rr_new <= thr2) { rr = rr_new; conv = 1; break; }
                restart = restart_after_replacement(want_check, rr_new, rr_rec);
            }
            beta2 = restart ? 0.0 : rr_new / rr;
            rr = rr_new;
            if (MODE == MODE_MIXED) prA = relaxed_precision(P, rr, bb);
            continue;
        }
        double alpha = 0.0, omega = 0.0;
        if (!bicg) {
            // ---- A: q = A p, p.q ----
            double ppq = 0.0;
            spmv_range<MODE, false, LEN, !bicg>(P, c.sbeg, c.send, c.i, c.hmask,
                             make_x(P.p, P.p32, P.p16, P.p8, P.mag_p, P.lab_p, invM), cnt,
                             [&](int R, double y) {
                                 const int row = R * MF_BS + c.i;
                                 if (row < n) {
                                     P.q[row] = y;
                                     ppq += P.p[row] * y;
                                 }
                             });
            nspmv++;
            clk.lap(PH_SPMV);
            block_partial(P, sh, 1, ppq, 0, 0, 0, 1, 0u);
            if (!solve_barrier(P, epoch, sh)) return;
            grid_collect(P, sh, 1, 1, 0u, v);
            clk.lap(PH_BAR);
            alpha = rr / v[0];
            if (!isfinite(alpha)) { status = MF_ERR_BREAKDOWN; break; }
            // ---- B: r -= alpha q, r.r  (x is updated with p in phase C) ----
            double prr = 0.0;
            for (int R0 = c.rbeg; R0 < c.rend; R0 += kVB) {
                double rv[kVB], qv[kVB];
#pragma unroll
                for (int u = 0; u < kVB; u++) {
                    const int row = (R0 + u) * MF_BS + c.i;
                    const bool valid = R0 + u < c.rend && row < n;
                    rv[u] = valid ? P.r[row] : 0.0;
                    qv[u] = valid ? P.q[row] : 0.0;
                }
#pragma unroll
                for (int u = 0; u < kVB; u++) {
                    const int row = (R0 + u) * MF_BS + c.i;
                    if (R0 + u < c.rend && row < n) {
                        const double rn = rv[u] - alpha * qv[u];
                        P.r[row] = rn;
                        prr += rn * rn;
                    }
                }
            }
            clk.lap(PH_VECB);
            block_partial(P, sh, 2, prr, 0, 0, 0, 1, 0u);
            if (!solve_barrier(P, epoch, sh)) return;
            grid_collect(P, sh, 2, 1, 0u, v);
            clk.lap(PH_BAR);
        } else {
            // ---- BiCGSTAB A1: v = A p, alpha = r1 / (rh.v) ----
            double prv = 0.0;
            const int useA = (kFb && coolA > 0) ? 0 : dynA;
            const unsigned d0A = demoted();
            spmv_range<MODE, false, LEN, !bicg>(P, c.sbeg, c.send, c.i, c.hmask,
                             lean_base(make_x(P.p, P.p32, P.p16, P.p8, P.mag_p, P.lab_p, invM, useA)), cnt,
                             [&](int R, double y) {
                                 const int row = R * MF_BS + c.i;
                                 if (row < n) {
                                     P.q[row] = y;
                                     prv += P.rh[row] * y;
                                 }
                             }, sh.whole);
            nspmv++;
            clk.lap(PH_SPMV);
            block_partial(P, sh, 1, prv, (double)(demoted() - d0A), 0, 0, kNvFb, 0u);
            if (!solve_barrier(P, epoch, sh)) return;
            grid_collect(P, sh, 1, kNvFb, 0u, v);
            clk.lap(PH_BAR);
            if (kFb) coolA = next_cool(coolA, useA != 0, v[1]);
            alpha = r1 / v[0];
            if (!isfinite(alpha)) { status = MF_ERR_BREAKDOWN; break; }
            // ---- B1: s = r - alpha v ----
            float smax = 0.0f, smin = 3.0e38f, ssm = 0.0f;
            const float sthr = invMs > 0.0f ? P.demote16 / invMs : -1.0f;
            for (int R = c.rbeg; R < c.rend; R++) {
                const int row = R * MF_BS + c.i;
                const bool valid = row < n;
                double sold = 0.0, sn = 0.0;
                if (valid) {
                    sold = P.s[row];
                    sn = P.r[row] - alpha * P.q[row];
                    P.s[row] = sn;
                }
                publish_dir<MODE>(R, row, valid, sn, sold, P.s32, P.s16, P.s8, P.mag_s, P.lab_s, smax, c.hmask,
                                  true, &smin, sthr, &ssm);
            }
            clk.lap(PH_VECB);
            // (max, -min) of s's segment magnitudes; only the mixed mode uses the minimum
            block_partial(P, sh, 2, (double)smax, -(double)smin, (double)ssm, 0, kNvSegB, 0x3u);
            if (!solve_barrier(P, epoch, sh)) return;
            grid_collect(P, sh, 2, kNvSegB, 0x3u, v);
            clk.lap(PH_BAR);
            invMs = v[0] > 0.0 ? (float)(1.0 / v[0]) : 0.0f;
            const int dynS = (MODE == MODE_MIXED) ? dyn_of(v[0], v[1], v[2]) : 1;
            // ---- A2: t = A s, omega = (t.s)/(t.t) ----
            double pts = 0.0, ptt = 0.0;
            const int useS = (kFb && coolS > 0) ? 0 : dynS;
            const unsigned d0S = demoted();
            spmv_range<MODE, false, LEN, !bicg>(P, c.sbeg, c.send, c.i, c.hmask,
                             lean_base(make_x(P.s, P.s32, P.s16, P.s8, P.mag_s, P.lab_s, invMs, useS)), cnt,
                             [&](int R, double y) {
                                 const int row = R * MF_BS + c.i;
                                 if (row < n) {
                                     P.t[row] = y;
                                     pts += y * P.s[row];
                                     ptt += y * y;
                                 }
                             }, sh.whole);
            nspmv++;
            clk.lap(PH_SPMV);
            block_partial(P, sh, 3, pts, ptt, (double)(demoted() - d0S), 0, kNvFb + 1, 0u);
            if (!solve_barrier(P, epoch, sh)) return;
            grid_collect(P, sh, 3, kNvFb + 1, 0u, v);
            clk.lap(PH_BAR);
            if (kFb) coolS = next_cool(coolS, useS != 0, v[2]);
            omega = (v[1] != 0.0) ? v[0] / v[1] : 0.0;
            // ---- B2: x += alpha p + omega s; r = s - omega t ----
            double prr = 0.0, prh = 0.0;
#pragma unroll 2
            for (int R = c.rbeg; R < c.rend; R++) {
                const int row = R * MF_BS + c.i;
                if (row < n) {
                    const double sv = P.s[row];
                    P.x[row] = P.x[row] + alpha * P.p[row] + omega * sv;
                    const double rv = sv - omega * P.t[row];
                    P.r[row] = rv;
                    prr += rv * rv;
                    prh += rv * P.rh[row];
                }
            }
            clk.lap(PH_VECB);
            block_partial(P, sh, 4, prr, prh, 0, 0, 2, 0u);
            if (!solve_barrier(P, epoch, sh)) return;
            grid_collect(P, sh, 4, 2, 0u, v);
            clk.lap(PH_BAR);
        }
        double rr_new = v[0], r1_new = bicg ? v[1] : 0.0;
        const double rr_rec = rr_new;    // recursive r.r of this iteration
        k++;
        last_true = 0;
        bool x_done = bicg;      // CG defers x += alpha p to phase C
        const bool want_check = !P.fixed_iters && rr_new <= thr2;
        const bool want_repl = P.replace_every > 0 && (k % P.replace_every) == 0;
        bool restart = false;
        if (want_check || want_repl) {
            if (!x_done) {
                // the FP64 residual needs the current x: apply this iteration's step first
                for (int R = c.rbeg; R < c.rend; R++) {
                    const int row = R * MF_BS + c.i;
                    if (row < n) P.x[row] += alpha * P.p[row];
                }
                x_done = true;
                if (!solve_barrier(P, epoch, sh)) return;
            }
            // ---- FP64 true residual: r = b - A x ----
            double prt = 0.0, prth = 0.0;
            spmv_range<MODE, true, LEN, !bicg>(P, c.sbeg, c.send, c.i, c.hmask, fp64_x(P.x), nullptr, [&](int R, double y) {
                const int row = R * MF_BS + c.i;
                if (row < n) {
                    const double rv = P.b[row] - y;
                    P.r[row] = rv;
                    prt += rv * rv;
                    if (bicg) prth += rv * P.rh[row];
                }
            });
            // rows of tile-rows without tiles (A row = 0): r = b there
            for (int R = c.rbeg; LEN == 0 && R < c.rend; R++) {
                if (P.seg_ptr[R] != P.seg_ptr[R + 1]) continue;
                const int row = R * MF_BS + c.i;
                if (row < n) {
                    const double rv = P.b[row];
                    P.r[row] = rv;
                    prt += rv * rv;
                    if (bicg) prth += rv * P.rh[row];
                }
            }
            clk.lap(PH_REPL);
            block_partial(P, sh, 5, prt, prth, 0, 0, 2, 0u);
            if (!solve_barrier(P, epoch, sh)) return;
            grid_collect(P, sh, 5, 2, 0u, v);
            clk.lap(PH_BAR);
            rr_new = v[0];
            r1_new = v[1];
            rr_true = rr_new;
            repl++;
            last_true = 1;
            if (!P.fixed_iters && rr_new <= thr2) { rr = rr_new; conv = 1; break; }
            restart = restart_after_replacement(want_check, rr_new, rr_rec);
        }
        // ---- C: (CG: x += alpha p,) p = r + beta p  /  p = r + beta (p - omega v) ----
        // A restart (see restart_after_replacement) takes p = r; BiCGSTAB also
        // takes the true residual as its new shadow residual (rh = r, r1 = r.r).
        double beta;
        if (restart) {
            beta = 0.0;
            if (bicg) r1 = rr_new;
        } else if (!bicg) {
            beta = rr_new / rr;
        } else {
            beta = (r1_new * alpha) / (r1 * omega);
            r1 = r1_new;
            if (!isfinite(beta)) { rr = rr_new; status = MF_ERR_BREAKDOWN; break; }
        }
        rr = rr_new;
        bmax = 0.0f;
        float pmin = 3.0e38f, psm = 0.0f;
        const float pthr = invM > 0.0f ? P.demote16 / invM : -1.0f;
        for (int R0 = c.rbeg; R0 < c.rend; R0 += kVB) {
            double pv[kVB], rv[kVB], xq[kVB];    // xq: x (CG, x not yet updated) or v (BiCGSTAB)
#pragma unroll
            for (int u = 0; u < kVB; u++) {
                const int row = (R0 + u) * MF_BS + c.i;
                const bool valid = R0 + u < c.rend && row < n;
                pv[u] = valid ? P.p[row] : 0.0;
                rv[u] = valid ? P.r[row] : 0.0;
                xq[u] = (valid && (bicg || !x_done)) ? (bicg ? P.q[row] : P.x[row]) : 0.0;
            }
#pragma unroll
            for (int u = 0; u < kVB; u++) {
                const int R = R0 + u;
                if (R >= c.rend) break;          // uniform over the half-warp
                const int row = R * MF_BS + c.i;
                const bool valid = row < n;
                const double pold = pv[u];
                const double pn = bicg ? rv[u] + beta * (pold - omega * xq[u]) : rv[u] + beta * pold;
                if (valid) {
                    if (!bicg && !x_done) P.x[row] = xq[u] + alpha * pold;
                    P.p[row] = pn;
                    if (bicg && restart) P.rh[row] = rv[u];
                }
                publish_dir<MODE>(R, row, valid, valid ? pn : 0.0, pold, P.p32, P.p16, P.p8, P.mag_p, P.lab_p,
                                  bmax, c.hmask, true, &pmin, pthr, &psm);
            }
        }
        clk.lap(PH_VECC);
        block_partial(P, sh, 6, (double)bmax, -(double)pmin, (double)psm, 0, kNvSegB, 0x3u);
        if (!solve_barrier(P, epoch, sh)) return;
        grid_collect(P, sh, 6, kNvSegB, 0x3u, v);
            clk.lap(PH_BAR);
        invM = v[0] > 0.0 ? (float)(1.0 / v[0]) : 0.0f;
        if (MODE == MODE_MIXED) dynA = dyn_of(v[0], v[1], v[2]);
    }
    // ---- final FP64 true residual when the last one was not already formed ----
    if (!last_true) {
        double prt = 0.0;
        spmv_range<MODE, true, LEN, !bicg>(P, c.sbeg, c.send, c.i, c.hmask, fp64_x(P.x), nullptr, [&](int R, double y) {
            const int row = R * MF_BS + c.i;
            if (row < n) {
                const double d = P.b[row] - y;
                prt += d * d;
            }
        });
        for (int R = c.rbeg; LEN == 0 && R < c.rend; R++) {
            if (P.seg_ptr[R] != P.seg_ptr[R + 1]) continue;
            const int row = R * MF_BS + c.i;
            if (row < n) prt += P.b[row] * P.b[row];
        }
        block_partial(P, sh, 7, prt, 0, 0, 0, 1, 0u);
        if (!solve_barrier(P, epoch, sh)) return;
        grid_collect(P, sh, 7, 1, 0u, v);
            clk.lap(PH_BAR);
        rr_true = v[0];
    }
    // tile-use counters
    __syncwarp();
    if (cnt && c.i < 10 && cnt[c.i]) atomicAdd(&P.counts[c.i], (unsigned long long)cnt[c.i]);
    if (cnt && blockIdx.x == 0 && threadIdx.x == 0) {
        for (int pr = 0; pr < 4; pr++) {
            if (!sh.whole[pr]) continue;
            atomicAdd(&P.counts[pr], (unsigned long long)sh.whole[pr] * (unsigned long long)P.ntiles);
            atomicAdd(&P.counts[5 + pr], (unsigned long long)sh.whole[pr] * (unsigned long long)P.nnz);
        }
    }
    if (clk.on() && P.phase_ns)
        for (int j = 0; j < 5; j++) P.phase_ns[j] = sh.clk_acc[j];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        P.out[0] = (double)k;
        P.out[1] = (double)conv;
        P.out[2] = bb > 0 ? sqrt(rr_true / bb) : 0.0;
        P.out[3] = bb > 0 ? sqrt(rr / bb) : 0.0;
        P.out[4] = sqrt(rr);
        P.out[5] = (double)repl;
        P.out[6] = (double)status;
        P.out[7] = (double)nspmv;
    }
}

// ------------------------------------------------------------ workspace
// What a solve leaves for the host.
struct Readback {
    int err, pad[31];
    double out[16];
    unsigned long long counts[16];
    unsigned long long phase_ns[8];
};
constexpr size_t kCtlBytes = 128 + sizeof(Readback);

struct Workspace {
    int G;                 // grid blocks of the persistent kernel
    int lb;                // register-budget variant (blocks per SM it was built for)
    int cluster;           // blocks of a one-cluster launch (0: none), and its partition
    int *hw_begin_cl;
    int nsm;
    // every solver vector lives in one block, ordered so that one L2
    // access-policy window can cover any number of the vectors a solve reuses
    // most (vec_window):
    //   x | p | q | r | s | t | rh | p32 | s32 | p16 | s16 | p8 | s8
    // (CG, FP64 / mixed: x..r; BiCGSTAB, FP64 / mixed: x..rh; parity mode: all)
    char *vecs;
    size_t vec_bytes, all_bytes;   // one FP64 vector; the whole block
    double *r, *p, *q, *rh, *s, *t, *x;
    float *p32, *s32, *mag_p, *mag_s;
    __half *p16, *s16;
    int8_t *p8, *s8;
    signed char *lab_p, *lab_s;
    double *red;
    // one block zeroed before a solve and read back after it: the barrier counter
    // (a 128-byte line of its own), then Readback
    char *ctl;
    unsigned int *bar;
    int *err;
    double *out;
    unsigned long long *counts;
    unsigned long long *phase_ns;
    int *hw_begin;
    int nhw;
    cudaEvent_t e0, e1;
    // several right-hand sides (k_solve_multi): interleaved vectors for NR columns
    int m_nr, m_G;
    double *m_vec;         // B | X | R | P | Q, each vec_len * NR
    float *m_mag;
    double *m_red, *m_out; // m_out: one result record per column group of a call (m_groups of them)
    int *m_err;            // one error word per column group
    int *m_hw_begin;
    int m_groups;          // column-group slots of m_out / m_err / m_ev
    cudaEvent_t *m_ev;     // two timing events per column group
};

#define MF_TRY(expr)                        \
    do {                                    \
        int _rc = (expr);                   \
        if (_rc != MF_SUCCESS) return _rc;  \
    } while (0)

// count[0]: tiles exact in INT8 or FP16; count[1]: tiles within FP16's normal range
__global__ void k_count_exact(const unsigned char *caps, int n, unsigned long long *count)
{
    unsigned c = 0, h = 0, f = 0;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        if (caps[t] & (MF_CAP_EXACT_I8 | MF_CAP_EXACT_F16)) c++;
        if (caps[t] & MF_CAP_FP16_OK) h++;
        if (caps[t] & MF_CAP_EXACT_F16) f++;
    }
    c = __reduce_add_sync(0xffffffffu, c);
    h = __reduce_add_sync(0xffffffffu, h);
    f = __reduce_add_sync(0xffffffffu, f);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, (unsigned long long)c);
    if ((threadIdx.x & 31) == 0 && h) atomicAdd(count + 1, (unsigned long long)h);
    if ((threadIdx.x & 31) == 0 && f) atomicAdd(count + 2, (unsigned long long)f);
}

// Tiles exact in INT8 or FP16 (the lossless classes), tiles within FP16's
// normal range, and tiles exact in FP16, counted once per matrix through
// `scratch` (three unsigned long long of device memory).
int exact_tiles(mf_matrix_s *A, unsigned long long *scratch, cudaStream_t s)
{
    if (!A->n_exact_known) {
        unsigned long long h[3] = {0, 0, 0};
        MF_CUDA_TRY(cudaMemsetAsync(scratch, 0, sizeof(h), s));
        if (A->tilenum > 0) k_count_exact<<<256, 256, 0, s>>>(A->d_tile_caps, A->tilenum, scratch);
        MF_CUDA_TRY(cudaGetLastError());
        MF_CUDA_TRY(cudaMemcpyAsync(h, scratch, sizeof(h), cudaMemcpyDeviceToHost, s));
        MF_CUDA_TRY(cudaStreamSynchronize(s));
        A->n_exact = (long long)h[0];
        A->n_fp16_ok = (long long)h[1];
        A->n_exact_f16 = (long long)h[2];
        A->n_exact_known = 1;
    }
    return MF_SUCCESS;
}

// Lossless classes apply when asked for and enough tiles are exact in a narrower
// type (the same fraction that gates demotion by magnitude).
inline int lossless_on(int use_lossless, double min_fraction, long long n_exact, int tilenum)
{
    return (use_lossless && n_exact > 0 && (double)n_exact >= min_fraction * (double)tilenum) ? 1 : 0;
}

void fill_params(SolverParams &P, mf_matrix_s *A, Workspace *w)
{
    memset(&P, 0, sizeof(P));
    P.n = A->n_rows;
    P.tilem = A->tilem;
    P.vec_len = A->vec_len;
    P.rowptr = A->d_rowptr;
    P.seg_ptr = A->d_seg_ptr;
    P.seg_hdr = A->d_seg_hdr;
    P.seg_rowlen = A->d_seg_rowlen;
    P.meta = A->d_meta;
    P.v64 = A->d_v64;
    P.v32 = A->d_v32;
    P.v16 = A->d_v16;
    P.v8 = A->d_v8;
    P.v8ref = A->d_v8ref;
    P.tile_col = A->d_tile_columnidx;
    P.seg_tile = A->d_seg_tile;
    P.tile_off = A->d_csr_offset;
    P.i8_scale = A->d_i8_scale;
    P.tile_caps = A->d_tile_caps;
    P.nseg = A->nseg;
    P.ntiles = A->tilenum;
    P.chk_xlen = A->vec_len;
    P.n_payload = A->slice_entries;
    P.nnz = A->nnz;
    if (w) {
        P.hw_begin = w->hw_begin;
        P.x = w->x; P.r = w->r; P.p = w->p; P.q = w->q; P.rh = w->rh; P.s = w->s; P.t = w->t;
        P.p32 = w->p32; P.s32 = w->s32; P.p16 = w->p16; P.s16 = w->s16; P.p8 = w->p8; P.s8 = w->s8;
        P.mag_p = w->mag_p; P.mag_s = w->mag_s; P.lab_p = w->lab_p; P.lab_s = w->lab_s;
        // CG in the FP64 / mixed modes multiplies r, not p: r's shadow takes p's slots
        P.mag_r = w->mag_p;
        P.red = w->red; P.bar = w->bar; P.err = w->err; P.out = w->out; P.counts = w->counts;
        P.phase_ns = w->phase_ns;
    }
}

// The first failed bounds check of the device since the last call (bounds-
// checked build): printed as site, index and limit, cleared, and returned as
// MF_ERR_CHECK.  Called after the entry point's own stream synchronisation.
// The normal build has no checks: MF_SUCCESS.
int chk_take()
{
#ifdef MF_CHECK
    unsigned long long h[3] = {0ull, 0ull, 0ull};
    if (cudaMemcpyFromSymbol(h, g_chk, sizeof(h)) != cudaSuccess) return MF_ERR_CUDA;
    if (h[0] == 0ull) return MF_SUCCESS;
    static const char *const kSite[CHK_NSITES] = {"",
                                                  "slice range",
                                                  "tile word / tile table",
                                                  "slice payload",
                                                  "gathered vector entry",
                                                  "row length",
                                                  "epilogue tile-row",
                                                  "batch queue entry"};
    fprintf(stderr, "millefeuille: bounds check failed: %s, index %lld, limit %lld\n",
            h[0] < (unsigned long long)CHK_NSITES ? kSite[h[0]] : "?", (long long)h[1], (long long)h[2]);
    const unsigned long long z[3] = {0ull, 0ull, 0ull};
    if (cudaMemcpyToSymbol(g_chk, z, sizeof(z)) != cudaSuccess) return MF_ERR_CUDA;
    return MF_ERR_CHECK;
#else
    return MF_SUCCESS;
#endif
}

// Partition tile-rows over half-warps by the cost prefix (lower bound).
__global__ void k_partition(const long long *__restrict__ cost, int tilem, int nhw, int *__restrict__ hw_begin)
{
    for (int h = blockIdx.x * blockDim.x + threadIdx.x; h <= nhw; h += gridDim.x * blockDim.x) {
        if (h == nhw) { hw_begin[h] = tilem; continue; }
        const long long total = cost[tilem];
        const long long target = (long long)((double)total * (double)h / (double)nhw);
        int lo = 0, hi = tilem;
        while (lo < hi) {
            int mid = (lo + hi) >> 1;
            if (cost[mid] < target) lo = mid + 1; else hi = mid;
        }
        hw_begin[h] = lo;
    }
}

// column block g of B (nrhs x n, one column after another) -> interleaved [row * NR + k]
__global__ void k_interleave(const double *B, int n, int L, int nrhs, int g, int NR, double *Bi)
{
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < (long long)L * NR;
         t += (long long)gridDim.x * blockDim.x) {
        const int row = (int)(t / NR), k = (int)(t % NR), col = g * NR + k;
        Bi[t] = (row < n && col < nrhs) ? B[(long long)col * n + row] : 0.0;
    }
}
__global__ void k_deinterleave(const double *Xi, int n, int nrhs, int g, int NR, double *X)
{
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < (long long)n * NR;
         t += (long long)gridDim.x * blockDim.x) {
        const int row = (int)(t / NR), k = (int)(t % NR), col = g * NR + k;
        if (col < nrhs) X[(long long)col * n + row] = Xi[t];
    }
}

}  // namespace
