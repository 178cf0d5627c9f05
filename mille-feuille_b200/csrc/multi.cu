// multi.cu -- CG on several right-hand sides at once and batches of uneven
// systems (mf_solve_multi, mf_batch_*).
#include "solver_dev.cuh"

#include <vector>

namespace {

// ------------------------------------------------------------ several right-hand sides
// CG on NR right-hand sides at once (FP64 and mixed modes): the vectors are
// interleaved (row i's NR values contiguous), so every matrix entry is read
// once per SpMV for all NR columns and one grid sync serves every column; the
// scalars alpha_k, beta_k and the convergence state are per column.  Same
// two-sync schedule as the single-column kernel (SpMV on R; P = R + beta P,
// Q = W + beta Q; then X += alpha P, R -= alpha Q).
constexpr int kMaxNR = 8;
constexpr int kRedWidthM = kMaxNR + 2;    // NR dot products + segment max / -min

struct SharedM {
    double wred[kWarps][kRedWidthM];
    double bcast[kRedWidthM];
    double alpha[kMaxNR], beta[kMaxNR], rr[kMaxNR], thr2[kMaxNR], bb[kMaxNR];
    int active[kMaxNR], pending[kMaxNR], iters[kMaxNR], conv[kMaxNR];
    int brk;                  // some column broke down (a scalar became non-finite)
    int flag;                 // grid_barrier's result
};

struct MultiParams {
    const double *B;          // [vec_len * NR] interleaved right-hand sides (zero columns past nr)
    double *X, *R, *Pv, *Q;   // interleaved
    float *mag;               // per tile-row: max over its rows and columns of |R|
    double *red;              // [kinds][kRedWidthM][blocks]: a collect reads consecutive blocks
    double *out;              // per column: iterations, converged, true rel. residual, recursive; then k, status
    int nr;                   // columns in use
};

// Block partial of NV values (maxmask bit k: max instead of sum) into
// red[kind][*][bidx] of an nblk-block group (the grid, or a batched item's team).
// The half-warps of a warp come from loops over tile-row ranges of different
// lengths: they meet here before the shuffles and the barriers.
template <int NV>
__device__ void block_partial_m(const MultiParams &M, SharedM &sh, int kind, const double (&v)[NV], unsigned maxmask,
                                int nblk, int bidx)
{
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < NV; k++) {
        double a = v[k];
        const bool mx = (maxmask >> k) & 1u;
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const double b = __shfl_xor_sync(0xffffffffu, a, o);
            a = mx ? fmax(a, b) : a + b;
        }
        if (lane == 0) sh.wred[wib][k] = a;
    }
    __syncthreads();
    // warp w reduces value w (fixed order)
    if (wib < NV) {
        const bool mx = (maxmask >> wib) & 1u;
        double a = (lane < kWarps) ? sh.wred[lane][wib] : (mx ? -1.0e300 : 0.0);
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const double b = __shfl_xor_sync(0xffffffffu, a, o);
            a = mx ? fmax(a, b) : a + b;
        }
        if (lane == 0) M.red[((long long)kind * kRedWidthM + wib) * nblk + bidx] = a;
    }
}

// After the sync: every block of the group sums the nblk partials of `kind` in
// the same order, into sh.bcast, where they stay until the next collect.
template <int NV>
__device__ void grid_collect_m(const MultiParams &M, SharedM &sh, int kind, unsigned maxmask, double (&out)[NV],
                               int nblk)
{
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    if (wib < NV) {
        const bool mx = (maxmask >> wib) & 1u;
        const double id = mx ? -1.0e300 : 0.0;
        const double *src = M.red + ((long long)kind * kRedWidthM + wib) * nblk;
        double a = id;
        // lane c takes blocks c, c + 32, ...; a pass issues all its loads first
        constexpr int kU = 5;               // 160 blocks per pass (one block per SM on 148 SMs)
        for (int c0 = 0; c0 < nblk; c0 += 32 * kU) {
            double t[kU];
#pragma unroll
            for (int j = 0; j < kU; j++) {
                const int cb = c0 + lane + 32 * j;
                t[j] = cb < nblk ? src[cb] : id;
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
    for (int k = 0; k < NV; k++) out[k] = sh.bcast[k];
    __syncthreads();
}

// One chunk of the NR-column walk: lane i's stored values of the chunk at
// entry offset cb in precision PR (FP32 / FP16 / scaled INT8 widened to FP64
// against the FP64 operand rows, as the single-column walk: no FP32 copy of
// R), each times its gathered NR-wide operand row.  The values are loaded one
// at a time next to their use: the NR-wide accumulators and operand rows take
// the registers, and these solves wait on the operand rows, not the values.
template <int PR, int NR>
__device__ __forceinline__ void multi_chunk(const SolverParams &P, long long cb, int i, unsigned hmask, int xb, int k0,
                                            int len, float sc, const double *X64, double (&acc)[NR])
{
    const unsigned long long m8 = __ldcs((const unsigned long long *)(P.meta + cb) + i);
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const unsigned mm = (unsigned)(m8 >> (8 * j)) & 0xFFu;
        const int slot = (int)(mm >> 4);
        const int xi = __shfl_sync(hmask, xb, slot, 16) + (int)(mm & 15u);
        const float s8 = (PR == MF_P8) ? __shfl_sync(hmask, sc, slot, 16) : 0.0f;
        if ((NR < 8 || k0 + j < len) && chk_in(CHK_X, xi, P.chk_xlen)) {
            double a;
            if (PR == MF_P64) a = __ldcs(P.v64 + mf_slot<8>(cb, j, i));
            else if (PR == MF_P32) a = (double)__ldcs(P.v32 + mf_slot<4>(cb, j, i));
            else if (PR == MF_P16) a = (double)__half2float(P.v16[mf_slot<2>(cb, j, i)]);
            else a = (double)((float)P.v8[mf_slot<1>(cb, j, i)] * s8);
            if constexpr (NR == 1) {
                acc[0] = fma(a, X64[xi], acc[0]);
            } else {
                const double2 *xr = (const double2 *)(X64 + (long long)xi * NR);
#pragma unroll
                for (int q = 0; q < NR / 2; q++) {
                    const double2 d = xr[q];
                    acc[2 * q] = fma(a, d.x, acc[2 * q]);
                    acc[2 * q + 1] = fma(a, d.y, acc[2 * q + 1]);
                }
            }
        }
    }
}

// Y = A X for NR interleaved columns over the half-warp's slices; epi(R, acc)
// once per tile-row with lane i's NR row sums.  Precision per slice as in
// slice_dot (mixed: from the column segments' max over rows and columns).
// Up to 4 columns the walk reads no row lengths (padding is value 0 with
// index byte 0, as in slice_dot_uniform: measured 10 % faster on the
// 512-system batch); with 8 columns a padding entry would gather 64 bytes of
// X, and the row-length predicate measured 6 % faster on the 512^2 system.
template <int MODE, int NR, bool F64, typename Epi>
__device__ __forceinline__ void spmv_multi(const SolverParams &P, int sb, int se, int i, unsigned hmask,
                                           const double *X64, const float *mag, float invM,
                                           int dyn, Epi epi)
{
    constexpr bool kMixed = (MODE == MODE_MIXED) && !F64;
    constexpr bool kLen = NR >= 8;
    XVec X = make_x(X64, nullptr, nullptr, nullptr, mag, nullptr, invM, dyn);
    double acc[NR];
#pragma unroll
    for (int k = 0; k < NR; k++) acc[k] = 0.0;
    if (sb >= se) return;
    if (!chk_in(CHK_SLICE, sb, P.nseg) || !chk_in(CHK_SLICE, se - 1, P.nseg)) return;
    int4 h = P.seg_hdr[sb];
    int tw = load_tw(P, sb, i);
    int len = kLen ? load_len(P, sb, i, h) : 0;
    for (int s = sb; s < se; s++) {
        const bool more = s + 1 < se;
        int4 hn = make_int4(0, 0, 0, 0);
        int twn = 0, lenn = 0;
        if (more) {
            hn = P.seg_hdr[s + 1];
            twn = load_tw(P, s + 1, i);
            lenn = kLen ? load_len(P, s + 1, i, hn) : 0;
        }
        const int xb = (tw >> 8) * MF_BS;
        int pr = MF_P64;
        if (kMixed && !dyn) {
            pr = MF_P32;                 // no tile can leave FP32 in this SpMV: no lookups
        } else if (kMixed) {
            const float st = (i < hdr_nt(h)) ? mag[tw >> 8] : 0.0f;
            pr = __reduce_min_sync(hmask, (i < hdr_nt(h)) ? tile_prec<MODE, false>(P, tw, st, X) : MF_P8);
        }
        float sc = 0.0f;
        if (kMixed && pr == MF_P8)
            sc = (i < hdr_nt(h) && chk_in(CHK_TILE, h.x + i, P.ntiles)) ? P.i8_scale[h.x + i] : 0.0f;
        const int kp = hdr_kp(h);
        const long long off = hdr_off(h);
        const int kpc = chk_in(CHK_PAYLOAD, off + (long long)kp * MF_BS - 1, P.n_payload) ? kp : 0;
        for (int k0 = 0; k0 < kpc; k0 += 8) {
            const long long cb = off + (long long)(k0 >> 3) * 128;
            // one instantiation per stored precision, so only that precision's
            // values are live across the chunk's gathers
            if (!kMixed || pr == MF_P64) multi_chunk<MF_P64, NR>(P, cb, i, hmask, xb, k0, len, sc, X64, acc);
            else if (pr == MF_P32) multi_chunk<MF_P32, NR>(P, cb, i, hmask, xb, k0, len, sc, X64, acc);
            else if (pr == MF_P16) multi_chunk<MF_P16, NR>(P, cb, i, hmask, xb, k0, len, sc, X64, acc);
            else multi_chunk<MF_P8, NR>(P, cb, i, hmask, xb, k0, len, sc, X64, acc);
        }
        if (hdr_last(h)) {
            if (chk_in(CHK_ROW, h.y, P.tilem)) epi(h.y, acc);
#pragma unroll
            for (int k = 0; k < NR; k++) acc[k] = 0.0;
        }
        h = hn;
        tw = twn;
        len = lenn;
    }
}

// Largest / smallest segment magnitude of the SpMV operand (mixed mode).
struct SegMM {
    float mx, mn;
};

// R's segment magnitude (max over the tile-row's rows and all columns) for
// tile-row R; all 16 lanes of the half-warp call it together.
template <int MODE, int NR>
__device__ __forceinline__ void publish_multi(const MultiParams &M, int R, int row, bool valid, const double (&rv)[NR],
                                              SegMM &st, unsigned hmask)
{
    if (MODE != MODE_MIXED) return;
    float m = 0.0f;
    if (valid) {
#pragma unroll
        for (int q = 0; q < NR; q++) m = fmaxf(m, fabsf((float)rv[q]));
    }
    m = half_max(m, hmask);
    st.mx = fmaxf(st.mx, m);
    st.mn = fminf(st.mn, m);
    if ((threadIdx.x & 15) == 0) M.mag[R] = m;
}

template <int NR>
__device__ __forceinline__ void load_row(const double *v, int row, double (&out)[NR])
{
    if constexpr (NR == 1) {
        out[0] = v[row];
        return;
    }
    const double2 *p = (const double2 *)(v + (long long)row * NR);
#pragma unroll
    for (int q = 0; q < NR / 2; q++) {
        const double2 d = p[q];
        out[2 * q] = d.x;
        out[2 * q + 1] = d.y;
    }
}
template <int NR>
__device__ __forceinline__ void store_row(double *v, int row, const double (&in)[NR])
{
    if constexpr (NR == 1) {
        v[row] = in[0];
        return;
    }
    double2 *p = (double2 *)(v + (long long)row * NR);
#pragma unroll
    for (int q = 0; q < NR / 2; q++) p[q] = make_double2(in[2 * q], in[2 * q + 1]);
}

// The CG iterations on NR columns, generic in how the threads that share a
// system synchronise: the whole grid (k_solve_multi) or one block (k_batch).
template <int MODE, int NR, class Sync>
__device__ void cg_multi_body(const SolverParams &P, const MultiParams &M, const Ctx &c, SharedM &sh, Sync &sy)
{
    const int n = P.n;
    bool has_empty = false;
    for (int R = c.rbeg; R < c.rend && !has_empty; R++) has_empty = P.seg_ptr[R] == P.seg_ptr[R + 1];
    const unsigned mm2 = 3u << NR;          // the two trailing max slots

    // ---- init: X = 0, R = B, P = Q = 0; |b_k|^2; R's segment magnitudes ----
    // With an initial guess (x0_given): |b_k|^2 reduced first (it scales the
    // convergence test), then R = B - A X in FP64.
    double pb[NR + 2], bb0[NR];
#pragma unroll
    for (int k = 0; k < NR + 2; k++) pb[k] = 0.0;
    SegMM st = {0.0f, 3.0e38f};
    if (P.x0_given) {
        double pbb[NR];
#pragma unroll
        for (int k = 0; k < NR; k++) pbb[k] = 0.0;
        for (int R = c.rbeg; R < c.rend; R++) {
            const int row = R * MF_BS + c.i;
            if (row < n) {
                double bv[NR];
                load_row<NR>(M.B, row, bv);
#pragma unroll
                for (int k = 0; k < NR; k++) pbb[k] += bv[k] * bv[k];
            }
        }
        if (!sy.template reduce<NR>(8, pbb, 0u, bb0)) return;
        auto init_r = [&](int R, const double (&y)[NR]) {
            const int row = R * MF_BS + c.i;
            const bool valid = row < n;
            double rv[NR], z[NR];
#pragma unroll
            for (int k = 0; k < NR; k++) { rv[k] = 0.0; z[k] = 0.0; }
            if (valid) {
                load_row<NR>(M.B, row, rv);
#pragma unroll
                for (int k = 0; k < NR; k++) rv[k] -= y[k];
                store_row<NR>(M.R, row, rv);
                store_row<NR>(M.Pv, row, z);
                store_row<NR>(M.Q, row, z);
#pragma unroll
                for (int k = 0; k < NR; k++) pb[k] += rv[k] * rv[k];
            }
            publish_multi<MODE, NR>(M, R, row, valid, rv, st, c.hmask);
        };
        spmv_multi<MODE, NR, true>(P, c.sbeg, c.send, c.i, c.hmask, M.X, nullptr, 0.0f, 1, init_r);
        if (has_empty) {
            double zy[NR];
#pragma unroll
            for (int k = 0; k < NR; k++) zy[k] = 0.0;
            for (int R = c.rbeg; R < c.rend; R++)
                if (P.seg_ptr[R] == P.seg_ptr[R + 1]) init_r(R, zy);
        }
    } else {
        for (int R = c.rbeg; R < c.rend; R++) {
            const int row = R * MF_BS + c.i;
            const bool valid = row < n;
            double rv[NR], z[NR];
#pragma unroll
            for (int k = 0; k < NR; k++) { rv[k] = 0.0; z[k] = 0.0; }
            if (valid) {
                load_row<NR>(M.B, row, rv);
                store_row<NR>(M.X, row, z);
                store_row<NR>(M.R, row, rv);
                store_row<NR>(M.Pv, row, z);
                store_row<NR>(M.Q, row, z);
#pragma unroll
                for (int k = 0; k < NR; k++) pb[k] += rv[k] * rv[k];
            }
            publish_multi<MODE, NR>(M, R, row, valid, rv, st, c.hmask);
        }
    }
    pb[NR] = st.mx;
    pb[NR + 1] = -st.mn;
    double v[NR + 2];
    if (!sy.template reduce<NR + 2>(0, pb, mm2, v)) return;
    if (threadIdx.x == 0) {
        for (int k = 0; k < NR; k++) {
            sh.bb[k] = P.x0_given ? bb0[k] : v[k];
            sh.rr[k] = v[k];
            sh.thr2[k] = P.tol * P.tol * sh.bb[k];
            sh.beta[k] = 0.0;
            sh.pending[k] = 0;
            sh.iters[k] = 0;
            sh.conv[k] = (k < M.nr && !P.fixed_iters && v[k] <= sh.thr2[k]) ? 1 : 0;
            sh.active[k] = (k < M.nr && !sh.conv[k]) ? 1 : 0;
        }
        sh.brk = 0;
    }
    __syncthreads();
    float invM = v[NR] > 0.0 ? (float)(1.0 / v[NR]) : 0.0f;
    // mixed: some tile may leave FP32 only if the smallest segment is below
    // demote_fp16 of the largest or lossless classes apply (see dyn in XVec)
    auto dyn_of = [&](double mx, double neg_mn) -> int {
        return (P.lossless_any || mx <= 0.0 || -neg_mn <= (double)P.demote16 * mx) ? 1 : 0;
    };
    int dyn = dyn_of(v[NR], v[NR + 1]);
    int k = 0, status = 0, repl = 0, last_true = 0;
    double rt[NR];
#pragma unroll
    for (int j = 0; j < NR; j++) rt[j] = v[j];

    for (;;) {
        int any = 0;
#pragma unroll
        for (int j = 0; j < NR; j++) any |= sh.active[j];
        if (!any || k >= P.max_iter) break;
        // ---- A: W = A R; P = R + beta P; Q = W + beta Q; P.Q per column ----
        double ppq[NR];
#pragma unroll
        for (int j = 0; j < NR; j++) ppq[j] = 0.0;
        auto upd_a = [&](int R, const double (&w)[NR]) {
            const int row = R * MF_BS + c.i;
            if (row < n) {
                double r[NR], p[NR], q[NR];
                load_row<NR>(M.R, row, r);
                load_row<NR>(M.Pv, row, p);
                load_row<NR>(M.Q, row, q);
#pragma unroll
                for (int j = 0; j < NR; j++) {
                    p[j] = r[j] + sh.beta[j] * p[j];
                    q[j] = w[j] + sh.beta[j] * q[j];
                    ppq[j] += p[j] * q[j];
                }
                store_row<NR>(M.Pv, row, p);
                store_row<NR>(M.Q, row, q);
            }
        };
        spmv_multi<MODE, NR, false>(P, c.sbeg, c.send, c.i, c.hmask, M.R, M.mag, invM, dyn, upd_a);
        if (has_empty) {
            double zw[NR];
#pragma unroll
            for (int j = 0; j < NR; j++) zw[j] = 0.0;
            for (int R = c.rbeg; R < c.rend; R++)
                if (P.seg_ptr[R] == P.seg_ptr[R + 1]) upd_a(R, zw);
        }
        double pq[NR];
        if (!sy.template reduce<NR>(1, ppq, 0u, pq)) return;
        if (threadIdx.x == 0) {
            for (int j = 0; j < NR; j++) {
                double a = sh.active[j] ? sh.rr[j] / pq[j] : 0.0;
                if (!isfinite(a)) {      // breakdown of this column: it stops where it is
                    a = 0.0;
                    sh.active[j] = 0;
                    sh.brk = 1;
                }
                sh.alpha[j] = a;
            }
        }
        __syncthreads();
        if (sh.brk) status = MF_ERR_BREAKDOWN;
        // ---- B: X += alpha P; R -= alpha Q; R.R; R's shadow ----
        double prr[NR + 2];
#pragma unroll
        for (int j = 0; j < NR + 2; j++) prr[j] = 0.0;
        st = SegMM{0.0f, 3.0e38f};
        for (int R = c.rbeg; R < c.rend; R++) {
            const int row = R * MF_BS + c.i;
            const bool valid = row < n;
            double r[NR];
#pragma unroll
            for (int j = 0; j < NR; j++) r[j] = 0.0;
            if (valid) {
                double x[NR], p[NR], q[NR];
                load_row<NR>(M.X, row, x);
                load_row<NR>(M.Pv, row, p);
                load_row<NR>(M.R, row, r);
                load_row<NR>(M.Q, row, q);
#pragma unroll
                for (int j = 0; j < NR; j++) {
                    x[j] += sh.alpha[j] * p[j];
                    r[j] -= sh.alpha[j] * q[j];
                    prr[j] += r[j] * r[j];
                }
                store_row<NR>(M.X, row, x);
                store_row<NR>(M.R, row, r);
            }
            publish_multi<MODE, NR>(M, R, row, valid, r, st, c.hmask);
        }
        prr[NR] = st.mx;
        prr[NR + 1] = -st.mn;
        if (!sy.template reduce<NR + 2>(2, prr, mm2, v)) return;
        invM = v[NR] > 0.0 ? (float)(1.0 / v[NR]) : 0.0f;
        dyn = dyn_of(v[NR], v[NR + 1]);
        k++;
        last_true = 0;
        bool want_repl = P.replace_every > 0 && (k % P.replace_every) == 0;
#pragma unroll
        for (int j = 0; j < NR; j++)
            if (sh.active[j] && !P.fixed_iters && v[j] <= sh.thr2[j]) want_repl = true;
        double rnew[NR], rrec[NR];
#pragma unroll
        for (int j = 0; j < NR; j++) rnew[j] = rrec[j] = v[j];
        if (want_repl) {
            // ---- FP64 R = B - A X, R's shadow, true residual norms ----
            double prt[NR + 2];
#pragma unroll
            for (int j = 0; j < NR + 2; j++) prt[j] = 0.0;
            st = SegMM{0.0f, 3.0e38f};
            auto upd_r = [&](int R, const double (&y)[NR]) {
                const int row = R * MF_BS + c.i;
                const bool valid = row < n;
                double r[NR];
#pragma unroll
                for (int j = 0; j < NR; j++) r[j] = 0.0;
                if (valid) {
                    load_row<NR>(M.B, row, r);
#pragma unroll
                    for (int j = 0; j < NR; j++) {
                        r[j] -= y[j];
                        prt[j] += r[j] * r[j];
                    }
                    store_row<NR>(M.R, row, r);
                }
                publish_multi<MODE, NR>(M, R, row, valid, r, st, c.hmask);
            };
            spmv_multi<MODE, NR, true>(P, c.sbeg, c.send, c.i, c.hmask, M.X, nullptr, 0.0f, 1, upd_r);
            if (has_empty) {
                double zy[NR];
#pragma unroll
                for (int j = 0; j < NR; j++) zy[j] = 0.0;
                for (int R = c.rbeg; R < c.rend; R++)
                    if (P.seg_ptr[R] == P.seg_ptr[R + 1]) upd_r(R, zy);
            }
            prt[NR] = st.mx;
            prt[NR + 1] = -st.mn;
            if (!sy.template reduce<NR + 2>(5, prt, mm2, v)) return;
            invM = v[NR] > 0.0 ? (float)(1.0 / v[NR]) : 0.0f;
            dyn = dyn_of(v[NR], v[NR + 1]);
            repl++;
            last_true = 1;
#pragma unroll
            for (int j = 0; j < NR; j++) {
                rt[j] = v[j];
                rnew[j] = v[j];
            }
        }
        if (threadIdx.x == 0) {
            for (int j = 0; j < NR; j++) {
                if (sh.active[j] && last_true && !P.fixed_iters && rnew[j] <= sh.thr2[j]) {
                    sh.active[j] = 0;            // converged on the FP64 true residual
                    sh.conv[j] = 1;
                    sh.iters[j] = k;
                }
                const bool restart = last_true &&
                                     restart_after_replacement(!P.fixed_iters && rrec[j] <= sh.thr2[j], rnew[j], rrec[j]);
                sh.beta[j] = (sh.active[j] && !restart) ? rnew[j] / sh.rr[j] : 0.0;
                if (sh.active[j] || !sh.conv[j]) sh.rr[j] = rnew[j];
            }
        }
        __syncthreads();
    }
    // ---- final FP64 true residuals when the last step did not form them ----
    if (!last_true) {
        double prt[NR];
#pragma unroll
        for (int j = 0; j < NR; j++) prt[j] = 0.0;
        auto acc_r = [&](int R, const double (&y)[NR]) {
            const int row = R * MF_BS + c.i;
            if (row < n) {
                double b[NR];
                load_row<NR>(M.B, row, b);
#pragma unroll
                for (int j = 0; j < NR; j++) prt[j] += (b[j] - y[j]) * (b[j] - y[j]);
            }
        };
        spmv_multi<MODE, NR, true>(P, c.sbeg, c.send, c.i, c.hmask, M.X, nullptr, 0.0f, 1, acc_r);
        if (has_empty) {
            double zy[NR];
#pragma unroll
            for (int j = 0; j < NR; j++) zy[j] = 0.0;
            for (int R = c.rbeg; R < c.rend; R++)
                if (P.seg_ptr[R] == P.seg_ptr[R + 1]) acc_r(R, zy);
        }
        double w[NR];
        if (!sy.template reduce<NR>(7, prt, 0u, w)) return;
#pragma unroll
        for (int j = 0; j < NR; j++) rt[j] = w[j];
    }
    if (sy.writer()) {
        for (int j = 0; j < NR; j++) {
            const double bb = sh.bb[j];
            M.out[4 * j + 0] = (double)(sh.conv[j] ? sh.iters[j] : k);
            M.out[4 * j + 1] = (double)sh.conv[j];
            M.out[4 * j + 2] = bb > 0 ? sqrt(rt[j] / bb) : 0.0;
            M.out[4 * j + 3] = bb > 0 ? sqrt(sh.rr[j] / bb) : 0.0;
        }
        M.out[4 * NR + 0] = (double)k;
        M.out[4 * NR + 1] = (double)status;
        M.out[4 * NR + 2] = (double)repl;
    }
}

// Grid-wide synchronisation: block partials, the counter barrier, a fixed-order collect.
struct GridSync {
    const SolverParams &P;
    const MultiParams &M;
    SharedM &sh;
    unsigned epoch;
    template <int NV>
    __device__ bool reduce(int kind, const double (&v)[NV], unsigned maxmask, double (&out)[NV])
    {
        block_partial_m<NV>(M, sh, kind, v, maxmask, (int)gridDim.x, (int)blockIdx.x);
        if (!grid_barrier(P, epoch, sh)) return false;
        grid_collect_m<NV>(M, sh, kind, maxmask, out, (int)gridDim.x);
        return true;
    }
    __device__ bool writer() const { return blockIdx.x == 0 && threadIdx.x == 0; }
};

template <int MODE, int NR>
__global__ void __launch_bounds__(kThreads, 1) k_solve_multi(SolverParams P, MultiParams M)
{
    __shared__ SharedM sh;
    const Ctx c = make_ctx(P);
    GridSync sy{P, M, sh, 0u};
    cg_multi_body<MODE, NR>(P, M, c, sh, sy);
}

// ------------------------------------------------------------ batched systems
// Many independent systems in one persistent launch of one or two 512-thread
// blocks per SM (k_batch<MODE, LB>).  Work items are (system, up to 8 of its
// right-hand sides).
//  * Team items: an item whose estimated cost exceeds a fair share of the
//    launch (total cost / blocks) is solved by a team of k blocks, sized by its
//    cost; the host list-schedules team items onto blocks (the k blocks that
//    are free first) and gives every block its ordered list.  Team members
//    synchronise through a counter of their own (bounded waits) and reduce in
//    a fixed order over the k block partials.
//  * Queue items: everything else sits in a device work queue, largest
//    estimated cost first; a block that has finished its list takes the next
//    queue item and solves it alone with block-level syncs.
// The launch is cooperative, so every block is resident and a team never waits
// on a block that cannot run; the lists are sorted by the same global order
// (scheduled start, then item), so no two teams wait on each other.
constexpr int kHalvesPerBlock = kWarps * 2;
constexpr int kMinTeamRows = 64;  // tile-rows per team block at least (2 per half-warp)
// Team size = round(kTeamGrain x cost / fair share): a team's members finish an
// item in about 1 / kTeamGrain of a fair share, so no single item sets the
// launch's end.  A team costs a few microseconds per sync, small against the
// milliseconds a large item's iteration takes on one block.
// Measured on the 512-system batch: grain 1, 2, 4 -> 20.2, 18.7, 17.8 s.
constexpr double kTeamGrain = 4.0;

struct BatchItem {
    const int *seg_ptr;
    const int4 *seg_hdr;
    const int *seg_tile;
    const uint16_t *seg_rowlen;
    const unsigned char *meta;
    const double *v64;
    const float *v32;
    const __half *v16;
    const int8_t *v8;
    const float *i8_scale;
    const long long *row_cost;    // tile-row cost prefix [tilem + 1]
    MultiParams M;                // the item's interleaved vectors and report words (M.nr columns used);
                                  // team items: M.red holds the team's partials [kinds][team][kRedWidthM]
    unsigned *ctr;                // team items: the team's barrier counter (zeroed before the launch)
    long long n_exact;            // tiles exact in INT8 / FP16
    int n, tilem, nr;             // nr: interleave width (1, 2, 4 or 8)
    int tilenum;
    int team;                     // blocks solving the item (1: queue item)
    int nrhs, group;              // the system's right-hand sides, and which group of nr the item holds
    int nseg, vec_len;            // extents for the bounds-checked build
    long long n_payload;
};

struct BatchParams {
    const BatchItem *items;
    const int *order;             // queue items, largest estimated cost first
    int n_items;                  // queue items
    int n_all;                    // entries of `items` (queue and team items)
    unsigned *head;               // next position in `order` (zeroed before the launch)
    const int *bptr;              // [grid + 1] each block's list of team entries
    const int2 *blist;            // (item, rank in its team)
    int *err;                     // first error of a team wait (zeroed before the launch)
    unsigned long long timeout_ns, arrive_timeout_ns;
    int stall_first;              // test hook: a team's first barrier expects one extra arrival
    int x0_given;                 // every item's X holds its initial guess
    int max_iter, fixed_iters, replace_every, use_lossless;
    double tol, min_fraction;
    float demote16, demote8;
};

// One block's synchronisation: warp shuffles, shared memory, fixed order.
struct BlockSync {
    SharedM &sh;
    template <int NV>
    __device__ bool reduce(int, const double (&v)[NV], unsigned maxmask, double (&out)[NV])
    {
        const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
        __syncwarp();                      // as in block_partial_m
#pragma unroll
        for (int k = 0; k < NV; k++) {
            double a = v[k];
            const bool mx = (maxmask >> k) & 1u;
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                const double b = __shfl_xor_sync(0xffffffffu, a, o);
                a = mx ? fmax(a, b) : a + b;
            }
            if (lane == 0) sh.wred[wib][k] = a;
        }
        __syncthreads();
        if (wib < NV) {
            const bool mx = (maxmask >> wib) & 1u;
            double a = (lane < kWarps) ? sh.wred[lane][wib] : (mx ? -1.0e300 : 0.0);
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                const double b = __shfl_xor_sync(0xffffffffu, a, o);
                a = mx ? fmax(a, b) : a + b;
            }
            if (lane == 0) sh.bcast[wib] = a;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < NV; k++) out[k] = sh.bcast[k];
        __syncthreads();
        return true;
    }
    __device__ bool writer() const { return threadIdx.x == 0; }
};

// Barrier of the k blocks of one team: a monotone counter with the pattern of
// grid_barrier (fence, relaxed add, relaxed polls, one acquire fence), bounded
// by `limit_ns`; a timeout, or an error set elsewhere, returns false and the
// first error is kept in *err.
__device__ bool team_barrier(unsigned *ctr, unsigned k, unsigned &epoch, int *err, unsigned long long limit_ns,
                             SharedM &sh, int stall = 0)
{
    __syncthreads();
    epoch += 1;
    if (threadIdx.x == 0) {
        const unsigned target = epoch * k + ((stall && epoch == 1) ? 1u : 0u);
        __threadfence();
        mf_red_relaxed_add_u32(ctr, 1u);
        bool ok = true;
        const unsigned long long t0 = mf_globaltimer();
        unsigned spins = 0;
        for (;;) {
            const unsigned v = mf_ld_relaxed_u32(ctr);
            if ((int)(v - target) >= 0) break;
            if (*(volatile int *)err) { ok = false; break; }
            if ((++spins & 63u) == 0u && mf_globaltimer() - t0 > limit_ns) {
                atomicCAS(err, 0, MF_ERR_TIMEOUT);
                ok = false;
                break;
            }
        }
        mf_fence_acq_rel_gpu();
        sh.flag = ok ? 1 : 0;
    }
    __syncthreads();
    return sh.flag != 0;
}

// The synchronisation of a team item: block partials into the team's slots,
// the team barrier, then every member sums the k partials in the same order.
// The first barrier (every member arriving at the item) may wait for members
// still finishing earlier list entries, so it gets the longer limit.  The team's
// words are read from the item, which nothing writes during the launch: a warp
// that lags cannot see another item's.
struct TeamSync {
    const BatchParams &B;
    const BatchItem &it;
    SharedM &sh;
    int r;                        // this block's rank in the team
    unsigned epoch;
    template <int NV>
    __device__ bool reduce(int kind, const double (&v)[NV], unsigned maxmask, double (&out)[NV])
    {
        MultiParams R;
        R.red = it.M.red;
        const int k = it.team;
        block_partial_m<NV>(R, sh, kind, v, maxmask, k, r);
        const unsigned long long limit = epoch == 0 ? B.arrive_timeout_ns : B.timeout_ns;
        if (!team_barrier(it.ctr, (unsigned)k, epoch, B.err, limit, sh, B.stall_first)) return false;
        grid_collect_m<NV>(R, sh, kind, maxmask, out, k);
        return true;
    }
    __device__ bool writer() const { return r == 0 && threadIdx.x == 0; }
};

// The half-warps of a team of k blocks (this block: rank r) split a system's
// tile-rows by the cost prefix (k = 1: one block).
__device__ __forceinline__ Ctx team_ctx(const BatchItem &it, int r, int k)
{
    Ctx c;
    c.lane = threadIdx.x & 31;
    c.wib = threadIdx.x >> 5;
    c.half = c.lane >> 4;
    c.i = c.lane & 15;
    c.hmask = 0xFFFFu << (16 * c.half);
    const int halves = kHalvesPerBlock * k;
    const int hw = r * kHalvesPerBlock + c.wib * 2 + c.half;
    const long long total = it.row_cost[it.tilem];
    auto split = [&](int h) -> int {
        if (h >= halves) return it.tilem;
        const long long target = (long long)((double)total * (double)h / (double)halves);
        int lo = 0, hi = it.tilem;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (it.row_cost[mid] < target) lo = mid + 1;
            else hi = mid;
        }
        return lo;
    };
    c.rbeg = split(hw);
    c.rend = split(hw + 1);
    c.sbeg = it.seg_ptr[c.rbeg];
    c.send = it.seg_ptr[c.rend];
    return c;
}

// The fields of SolverParams the CG body and the slice walk read, for one item.
__device__ __forceinline__ SolverParams item_params(const BatchItem &it, const BatchParams &B)
{
    SolverParams P;
    P.n = it.n;
    P.tilem = it.tilem;
    P.seg_ptr = it.seg_ptr;
    P.seg_hdr = it.seg_hdr;
    P.seg_tile = it.seg_tile;
    P.seg_rowlen = it.seg_rowlen;
    P.meta = it.meta;
    P.v64 = it.v64;
    P.v32 = it.v32;
    P.v16 = it.v16;
    P.v8 = it.v8;
    P.i8_scale = it.i8_scale;
    P.max_iter = B.max_iter;
    P.x0_given = B.x0_given;
    P.fixed_iters = B.fixed_iters;
    P.replace_every = B.replace_every;
    P.use_lossless = B.use_lossless;
    P.lossless_any = (B.use_lossless && it.n_exact > 0 && (double)it.n_exact >= B.min_fraction * (double)it.tilenum)
                         ? 1 : 0;
    P.tol = B.tol;
    P.demote16 = B.demote16;
    P.demote8 = B.demote8;
    P.nseg = it.nseg;
    P.ntiles = it.tilenum;
    P.chk_xlen = it.vec_len;
    P.n_payload = it.n_payload;
    return P;
}

// MAXNR: the widest interleave the launch was built for (8 with one block per
// SM; 4 with two, whose items never exceed 4 columns).
template <int MODE, int MAXNR, class Sync>
__device__ __forceinline__ void item_solve(const SolverParams &P, const MultiParams &M, int nr, const Ctx &c,
                                           SharedM &sh, Sync &sy)
{
    switch (nr) {
    case 1: cg_multi_body<MODE, 1>(P, M, c, sh, sy); break;
    case 2: cg_multi_body<MODE, 2>(P, M, c, sh, sy); break;
    case 4: cg_multi_body<MODE, 4>(P, M, c, sh, sy); break;
    default:
        if constexpr (MAXNR >= 8) cg_multi_body<MODE, 8>(P, M, c, sh, sy);
        break;
    }
}

// LB: resident blocks per SM the launch is built for (1: up to 128 registers a
// thread, the widest items without spills; 2: 64 registers, twice the warps to
// hide latency, for items of up to 4 columns).  The tuner picks.
template <int MODE, int LB>
__global__ void __launch_bounds__(kThreads, LB) k_batch(const __grid_constant__ BatchParams B)
{
    __shared__ SharedM sh;
    __shared__ int next, stop;
    // this block's team entries, in the global schedule order
    for (int e = B.bptr[blockIdx.x]; e < B.bptr[blockIdx.x + 1]; e++) {
        const int2 ent = B.blist[e];
        if (!chk_in(CHK_ITEM, ent.x, B.n_all)) continue;
        const BatchItem &it = B.items[ent.x];
        const SolverParams P = item_params(it, B);
        const Ctx c = team_ctx(it, ent.y, it.team);
        const MultiParams M = it.M;
        const unsigned long long t0 = mf_globaltimer();
        TeamSync sy{B, it, sh, ent.y, 0u};
        item_solve<MODE, (LB == 1 ? 8 : 4)>(P, M, it.nr, c, sh, sy);
        if (threadIdx.x == 0) stop = *(volatile int *)B.err;
        __syncthreads();
        if (ent.y == 0 && threadIdx.x == 0) {         // the item's start and end, for the report
            M.out[4 * it.nr + 3] = (double)t0;
            M.out[4 * it.nr + 4] = (double)mf_globaltimer();
        }
        if (stop) return;      // a team wait gave up: the launch reports it (one answer for the whole block)
    }
    for (;;) {
        if (threadIdx.x == 0) next = (int)atomicAdd(B.head, 1u);
        __syncthreads();
        const int pos = next;
        __syncthreads();
        if (pos >= B.n_items) break;
        if (!chk_in(CHK_ITEM, B.order[pos], B.n_all)) continue;
        const BatchItem &it = B.items[B.order[pos]];
        const SolverParams P = item_params(it, B);
        const Ctx c = team_ctx(it, 0, 1);
        BlockSync sy{sh};
        const MultiParams M = it.M;
        const unsigned long long t0 = mf_globaltimer();
        item_solve<MODE, (LB == 1 ? 8 : 4)>(P, M, it.nr, c, sh, sy);
        __syncthreads();
        if (threadIdx.x == 0) {
            M.out[4 * it.nr + 3] = (double)t0;
            M.out[4 * it.nr + 4] = (double)mf_globaltimer();
        }
    }
}

}  // namespace

// ------------------------------------------------------------ several right-hand sides (host)
namespace {

const void *multi_kernel(int mode, int nr)
{
    if (mode == MODE_FP64)
        return nr == 2 ? (const void *)k_solve_multi<MODE_FP64, 2>
               : nr == 4 ? (const void *)k_solve_multi<MODE_FP64, 4> : (const void *)k_solve_multi<MODE_FP64, 8>;
    return nr == 2 ? (const void *)k_solve_multi<MODE_MIXED, 2>
           : nr == 4 ? (const void *)k_solve_multi<MODE_MIXED, 4> : (const void *)k_solve_multi<MODE_MIXED, 8>;
}

// The multi-column workspace for NR columns (grid: one block of 512 threads per SM).
int ws_multi(mf_matrix_s *A, Workspace *w, int mode, int nr, cudaStream_t s)
{
    if (w->m_nr == nr && w->m_vec) return MF_SUCCESS;
    void *old[] = {w->m_vec, w->m_mag, w->m_red, w->m_hw_begin};
    if (w->m_vec) mf_handle_wait(A);
    mf_pool_give_back(old, 4);
    w->m_vec = nullptr; w->m_mag = nullptr; w->m_red = nullptr;
    w->m_hw_begin = nullptr;
    w->m_nr = 0;
    int dev = 0, nsm = 0, occ = 0;
    MF_CUDA_TRY(cudaGetDevice(&dev));
    MF_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    for (int m = MODE_FP64; m <= MODE_MIXED; m++) {
        int o = 0;
        MF_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, multi_kernel(m, nr), kThreads, 0));
        occ = (m == MODE_FP64 || o < occ) ? o : occ;
    }
    if (occ < 1) return MF_ERR_UNSUPPORTED;
    int G = nsm * (occ > 1 ? 1 : occ);
    const int need = (A->tilem + kWarps * 2 - 1) / (kWarps * 2);
    if (need < G) G = need > 0 ? need : 1;
    const long long L = A->vec_len, S = std::max(A->tilem, A->tilen) + 1;
    MF_TRY(mf_pool_array(&w->m_vec, 5 * L * nr, s));
    MF_TRY(mf_pool_array(&w->m_mag, S, s));
    MF_TRY(mf_pool_array(&w->m_red, (long long)kRedKinds * G * kRedWidthM, s));
    MF_TRY(mf_pool_array(&w->m_hw_begin, (long long)G * kWarps * 2 + 1, s));
    MF_CUDA_TRY(cudaMemsetAsync(w->m_vec, 0, (size_t)5 * L * nr * sizeof(double), s));
    MF_CUDA_TRY(cudaMemsetAsync(w->m_mag, 0, (size_t)S * sizeof(float), s));
    const int nhw = G * kWarps * 2;
    k_partition<<<(nhw + 256) / 256, 256, 0, s>>>(A->d_row_cost, A->tilem, nhw, w->m_hw_begin);
    MF_CUDA_TRY(cudaGetLastError());
    w->m_G = G;
    w->m_nr = nr;
    return MF_SUCCESS;
}

constexpr int kOutM = 4 * kMaxNR + 8;    // doubles per column group's result record

// Result slots for `groups` column groups (grown, never shrunk).
int ws_multi_groups(const mf_matrix_s *A, Workspace *w, int groups, cudaStream_t s)
{
    if (w->m_groups >= groups) return MF_SUCCESS;
    if (w->m_out) mf_handle_wait(A);
    void *old[] = {w->m_out, w->m_err};
    mf_pool_give_back(old, 2);
    w->m_out = nullptr;
    w->m_err = nullptr;
    for (int k = 0; k < 2 * w->m_groups; k++) cudaEventDestroy(w->m_ev[k]);
    delete[] w->m_ev;
    w->m_ev = nullptr;
    w->m_groups = 0;
    MF_TRY(mf_pool_array(&w->m_out, (long long)groups * kOutM, s));
    MF_TRY(mf_pool_array(&w->m_err, groups, s));
    w->m_ev = new cudaEvent_t[2 * groups];
    for (int k = 0; k < 2 * groups; k++) MF_CUDA_TRY(cudaEventCreate(&w->m_ev[k]));
    w->m_groups = groups;
    return MF_SUCCESS;
}

}  // namespace

int mf_solver_multi_run(mf_matrix_s *A, int nrhs, const double *d_B, double *d_X, const mf_options *opt,
                        mf_report *reps, cudaStream_t s)
{
    if (opt->method != MF_METHOD_CG || opt->precision == MF_PREC_PARITY) return MF_ERR_UNSUPPORTED;
    const int mode = opt->precision == MF_PREC_FP64 ? MODE_FP64 : MODE_MIXED;
    Workspace *w = nullptr;
    MF_TRY(mf_ws_get(A, opt->blocks_per_sm, (void **)&w, s));
    const int nr = nrhs >= 8 ? 8 : nrhs >= 4 ? 4 : 2;   // columns per launch
    MF_TRY(ws_multi(A, w, mode, nr, s));
    const long long L = A->vec_len;
    const int n = A->n_rows;
    SolverParams P;
    fill_params(P, A, w);
    P.hw_begin = w->m_hw_begin;
    P.method = MF_METHOD_CG;
    P.x0_given = opt->x0_given ? 1 : 0;
    P.max_iter = opt->max_iter;
    P.fixed_iters = opt->fixed_iters;
    P.replace_every = opt->replace_every;
    P.use_lossless = opt->use_lossless;
    P.lossless_any = lossless_on(opt->use_lossless, opt->demote_min_fraction, A->n_exact, A->tilenum);
    P.min_small = (float)(opt->demote_min_fraction * (double)A->tilem);
    P.min_demoted = (float)(opt->demote_min_fraction * (double)A->tilenum);
    P.tol = opt->tol;
    P.demote16 = (float)opt->demote_fp16;
    P.demote8 = (float)opt->demote_int8;
    const double to = opt->wait_timeout_s > 0 ? opt->wait_timeout_s : 10.0;
    P.timeout_ns = (unsigned long long)(to * 1e9);
    P.stall_first_barrier = opt->test_stall_barrier ? 1 : 0;
    MultiParams M;
    M.B = w->m_vec;
    M.X = w->m_vec + L * nr;
    M.R = w->m_vec + 2 * L * nr;
    M.Pv = w->m_vec + 3 * L * nr;
    M.Q = w->m_vec + 4 * L * nr;
    M.mag = w->m_mag;
    M.red = w->m_red;
    const int groups = (nrhs + nr - 1) / nr;
    MF_TRY(ws_multi_groups(A, w, groups, s));
    MF_CUDA_TRY(cudaMemsetAsync(w->m_out, 0, (size_t)groups * kOutM * sizeof(double), s));
    MF_CUDA_TRY(cudaMemsetAsync(w->m_err, 0, (size_t)groups * sizeof(int), s));
    // every column group is enqueued back to back (the interleaved buffers are
    // reused in stream order); the host reads the results once, at the end
    for (int g = 0; g < groups; g++) {
        M.nr = std::min(nr, nrhs - g * nr);
        M.out = w->m_out + (size_t)g * kOutM;
        P.err = w->m_err + g;
        k_interleave<<<592, 256, 0, s>>>(d_B, n, (int)L, nrhs, g, nr, (double *)M.B);
        if (opt->x0_given) k_interleave<<<592, 256, 0, s>>>(d_X, n, (int)L, nrhs, g, nr, M.X);
        MF_CUDA_TRY(cudaGetLastError());
        MF_CUDA_TRY(cudaMemsetAsync(w->bar, 0, sizeof(unsigned int), s));
        void *args[] = {&P, &M};
        MF_CUDA_TRY(cudaEventRecord(w->m_ev[2 * g], s));
        MF_CUDA_TRY(cudaLaunchCooperativeKernel(multi_kernel(mode, nr), dim3(w->m_G), dim3(kThreads), args, 0, s));
        MF_CUDA_TRY(cudaEventRecord(w->m_ev[2 * g + 1], s));
        k_deinterleave<<<592, 256, 0, s>>>(M.X, n, nrhs, g, nr, d_X);
        MF_CUDA_TRY(cudaGetLastError());
    }
    std::vector<double> out((size_t)groups * kOutM);
    std::vector<int> err(groups);
    MF_CUDA_TRY(cudaMemcpyAsync(out.data(), w->m_out, out.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
    MF_CUDA_TRY(cudaMemcpyAsync(err.data(), w->m_err, err.size() * sizeof(int), cudaMemcpyDeviceToHost, s));
    MF_CUDA_TRY(cudaStreamSynchronize(s));
    int first_err = chk_take();
    for (int g = 0; g < groups; g++) {
        const double *o = out.data() + (size_t)g * kOutM;
        float ms = 0.f;
        MF_CUDA_TRY(cudaEventElapsedTime(&ms, w->m_ev[2 * g], w->m_ev[2 * g + 1]));
        const int status = err[g] ? err[g] : (int)o[4 * nr + 1];
        if (status != MF_SUCCESS && first_err == MF_SUCCESS) first_err = status;
        if (reps) {
            for (int k = 0; k < std::min(nr, nrhs - g * nr); k++) {
                mf_report *r = &reps[g * nr + k];
                memset(r, 0, sizeof(*r));
                r->status = status;
                r->iterations = (int)o[4 * k + 0];
                r->converged = (int)o[4 * k + 1];
                r->relres_true = o[4 * k + 2];
                r->relres_rec = o[4 * k + 3];
                r->time_ms = ms;
                r->replacements = (int)o[4 * nr + 2];
                r->grid_blocks = w->m_G;
                r->threads_per_block = kThreads;
            }
        }
    }
    return first_err;
}

// ------------------------------------------------------------ batched systems (host)
namespace {

struct BatchImpl {
    MfContext ctx = {nullptr, 0};
    int dev = 0, cap = 8, lb = 1, nitems = 0, nsm = 0;
    int max_res[3] = {0, 0, 0};        // co-resident blocks of the k_batch<*, lb> launch, lb = 1, 2
    std::vector<mf_matrix_s *> sys;
    std::vector<int> nrhs;
    // items: system, first column, columns, interleave width, team size
    std::vector<int> it_sys, it_col0, it_ncol, it_nr, it_team;
    std::vector<BatchItem> h_items;
    BatchItem *d_items = nullptr;
    int *d_order = nullptr;            // queue items, largest estimated cost first
    int nqueue = 0;
    int grid = 1;                      // blocks of the launch
    int *d_bptr = nullptr;             // [grid + 1] team entries per block
    int2 *d_blist = nullptr;
    unsigned *d_ctl = nullptr;         // queue head | error word | one barrier counter per team item
    size_t ctl_bytes = 0;
    char *d_pool = nullptr;
    size_t pool_bytes = 0;
    cudaStream_t own = nullptr;        // used when the caller passes the default stream
    cudaGraphExec_t graph = nullptr;
    std::vector<const void *> graph_key;
    int graph_mode = -1;
    cudaEvent_t e0 = nullptr, e1 = nullptr, e_in = nullptr;
    double last_ms = 0.0;
    bool unsynced = false;             // a call failed half-way: its work may still run

    // Ends a call: where it failed, the batch and its systems wait for the device
    // before they give memory back.
    int ended(int rc)
    {
        if (rc == MF_SUCCESS) return rc;
        unsynced = true;
        for (mf_matrix_s *A : sys) A->unsynced = 1;
        return rc;
    }

    void release_items()
    {
        MfDeviceGuard guard(dev);
        if (!mf_context_gone(ctx)) {
            if (graph) cudaGraphExecDestroy(graph);
            void *p[] = {d_items, d_order, d_bptr, d_blist, d_ctl, d_pool};
            if (unsynced) mf_device_wait();
            mf_pool_give_back(p, 6);
        }
        unsynced = false;
        graph = nullptr;
        graph_key.clear();
        d_items = nullptr; d_order = nullptr; d_bptr = nullptr; d_blist = nullptr; d_ctl = nullptr;
        d_pool = nullptr;
    }
};

inline size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }
constexpr int kOutWords = 4 * kMaxNR + 8;

// Team sizes and the list schedule of team items.  fair = total cost / blocks;
// an item gets k = round(kTeamGrain x cost / fair) blocks, at most the launch and at most
// one block per kMinTeamRows tile-rows; k >= 2 makes it a team item.  Team
// items, largest first, go to the k blocks that are free first (ties: lower
// block), start = the latest of their free times, and those blocks are busy
// for cost / k.  Each block's list is sorted by (start, item).
void batch_schedule(const std::vector<double> &cost, const std::vector<int> &tilem, int grid, std::vector<int> &team,
                    std::vector<int> &bptr, std::vector<int2> &blist, std::vector<int> &queue)
{
    const int ni = (int)cost.size();
    double total = 0.0;
    for (double c : cost) total += c;
    const double fair = total / (double)std::max(1, grid);
    team.assign(ni, 1);
    std::vector<int> order(ni);
    for (int t = 0; t < ni; t++) order[t] = t;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return cost[a] > cost[b]; });
    std::vector<double> free_at(grid, 0.0);
    std::vector<std::vector<std::pair<double, int2>>> lists(grid);
    queue.clear();
    for (int t : order) {
        int k = 1;
        if (fair > 0.0 && grid > 1) {
            const double want = std::floor(kTeamGrain * cost[t] / fair + 0.5);
            k = (int)std::min<double>(want, (double)std::min(grid, std::max(1, tilem[t] / kMinTeamRows)));
            k = std::max(k, 1);
        }
        if (k < 2) {
            queue.push_back(t);
            continue;
        }
        team[t] = k;
        std::vector<int> blk(grid);
        for (int q = 0; q < grid; q++) blk[q] = q;
        std::stable_sort(blk.begin(), blk.end(), [&](int a, int b) { return free_at[a] < free_at[b]; });
        blk.resize(k);
        std::sort(blk.begin(), blk.end());
        double start = 0.0;
        for (int q : blk) start = std::max(start, free_at[q]);
        const double end = start + cost[t] / (double)k;
        for (int r = 0; r < k; r++) {
            free_at[blk[r]] = end;
            lists[blk[r]].push_back({start, make_int2(t, r)});
        }
    }
    bptr.assign(grid + 1, 0);
    blist.clear();
    for (int q = 0; q < grid; q++) {
        std::stable_sort(lists[q].begin(), lists[q].end(), [](const std::pair<double, int2> &a,
                                                             const std::pair<double, int2> &b) {
            return a.first < b.first || (a.first == b.first && a.second.x < b.second.x);
        });
        for (auto &e : lists[q]) blist.push_back(e.second);
        bptr[q + 1] = (int)blist.size();
    }
}

// Items for column cap `cap`: each system's right-hand sides in groups of <= cap,
// interleave width the next power of two (1, 2, 4, 8); team sizes and the
// schedule; all vectors in one pool.
int batch_build_items(BatchImpl &B, int cap, int lb, cudaStream_t s)
{
    B.release_items();
    B.cap = cap;
    B.lb = lb;
    B.it_sys.clear(); B.it_col0.clear(); B.it_ncol.clear(); B.it_nr.clear();
    for (int k = 0; k < (int)B.sys.size(); k++)
        for (int c0 = 0; c0 < B.nrhs[k]; c0 += cap) {
            const int g = std::min(cap, B.nrhs[k] - c0);
            B.it_sys.push_back(k);
            B.it_col0.push_back(c0);
            B.it_ncol.push_back(g);
            B.it_nr.push_back(mf_batch_width(g));
        }
    B.nitems = (int)B.it_sys.size();
    {
        // exact-tile counts of the systems (once per matrix)
        unsigned long long *scratch = nullptr;
        MF_TRY(mf_pool_array(&scratch, 3, s));
        int rc = MF_SUCCESS;
        for (mf_matrix_s *A : B.sys)
            if (rc == MF_SUCCESS) rc = exact_tiles(A, scratch, s);
        mf_pool_free(scratch, s);
        MF_TRY(rc);
    }
    std::vector<double> cost(B.nitems);
    std::vector<int> tilem(B.nitems);
    for (int t = 0; t < B.nitems; t++) {
        const mf_matrix_s *A = B.sys[B.it_sys[t]];
        cost[t] = mf_batch_item_cost(A->nnz, A->n_rows, B.it_nr[t]);
        tilem[t] = A->tilem;
    }
    // lb blocks per SM (all resident: the launch is cooperative)
    B.grid = std::max(1, std::min(B.max_res[lb], lb * B.nsm));
    std::vector<int> bptr, queue;
    std::vector<int2> blist;
    batch_schedule(cost, tilem, B.grid, B.it_team, bptr, blist, queue);
    if (blist.empty()) {
        // no team: one block per item at most
        B.grid = std::max(1, std::min(B.grid, B.nitems));
        bptr.assign(B.grid + 1, 0);
    }
    B.nqueue = (int)queue.size();
    // per item: B | X | R | P | Q (doubles), segment magnitudes, team partials
    std::vector<size_t> off(B.nitems), red_off(B.nitems, 0);
    // the report words of all items first, so one copy reads them back
    size_t total = align256((size_t)B.nitems * kOutWords * sizeof(double));
    for (int t = 0; t < B.nitems; t++) {
        const mf_matrix_s *A = B.sys[B.it_sys[t]];
        const size_t L = (size_t)A->vec_len, nr = (size_t)B.it_nr[t];
        off[t] = total;
        total += align256(5 * L * nr * sizeof(double)) + align256((size_t)(A->tilem + 1) * sizeof(float));
        if (B.it_team[t] > 1) {
            red_off[t] = total;
            total += align256((size_t)kRedKinds * B.it_team[t] * kRedWidthM * sizeof(double));
        }
    }
    B.pool_bytes = total;
    MF_TRY(mf_pool_alloc((void **)&B.d_pool, total > 0 ? total : 256, s));
    MF_CUDA_TRY(cudaMemsetAsync(B.d_pool, 0, total > 0 ? total : 256, s));
    int nteam = 0;
    std::vector<int> ctr_of(B.nitems, -1);
    for (int t = 0; t < B.nitems; t++)
        if (B.it_team[t] > 1) ctr_of[t] = nteam++;
    B.ctl_bytes = sizeof(unsigned) * (size_t)(2 + nteam);
    MF_TRY(mf_pool_alloc((void **)&B.d_ctl, B.ctl_bytes, s));
    B.h_items.resize(B.nitems);
    for (int t = 0; t < B.nitems; t++) {
        const mf_matrix_s *A = B.sys[B.it_sys[t]];
        const size_t L = (size_t)A->vec_len, nr = (size_t)B.it_nr[t];
        BatchItem &it = B.h_items[t];
        memset(&it, 0, sizeof(it));
        it.seg_ptr = A->d_seg_ptr; it.seg_hdr = A->d_seg_hdr; it.seg_tile = A->d_seg_tile;
        it.seg_rowlen = A->d_seg_rowlen; it.meta = A->d_meta; it.v64 = A->d_v64; it.v32 = A->d_v32;
        it.v16 = A->d_v16; it.v8 = A->d_v8; it.i8_scale = A->d_i8_scale; it.row_cost = A->d_row_cost;
        it.n = A->n_rows; it.tilem = A->tilem; it.nr = (int)nr; it.team = B.it_team[t];
        it.nrhs = B.nrhs[B.it_sys[t]]; it.group = B.it_col0[t] / it.nr;
        it.n_exact = A->n_exact; it.tilenum = A->tilenum;
        it.nseg = A->nseg; it.vec_len = A->vec_len; it.n_payload = A->slice_entries;
        char *base = B.d_pool + off[t];
        double *v = (double *)base;
        it.M.B = v; it.M.X = v + L * nr; it.M.R = v + 2 * L * nr; it.M.Pv = v + 3 * L * nr; it.M.Q = v + 4 * L * nr;
        it.M.mag = (float *)(base + align256(5 * L * nr * sizeof(double)));
        it.M.red = it.team > 1 ? (double *)(B.d_pool + red_off[t]) : nullptr;
        it.M.out = (double *)B.d_pool + (size_t)t * kOutWords;
        it.M.nr = B.it_ncol[t];
        it.ctr = it.team > 1 ? B.d_ctl + 2 + ctr_of[t] : nullptr;
    }
    MF_TRY(mf_pool_array(&B.d_items, B.nitems, s));
    MF_TRY(mf_pool_array(&B.d_order, B.nqueue, s));
    MF_TRY(mf_pool_array(&B.d_bptr, B.grid + 1, s));
    MF_TRY(mf_pool_array(&B.d_blist, (long long)blist.size(), s));
    if (B.nitems > 0)
        MF_CUDA_TRY(cudaMemcpyAsync(B.d_items, B.h_items.data(), sizeof(BatchItem) * B.nitems,
                                    cudaMemcpyHostToDevice, s));
    if (B.nqueue > 0)
        MF_CUDA_TRY(cudaMemcpyAsync(B.d_order, queue.data(), sizeof(int) * B.nqueue, cudaMemcpyHostToDevice, s));
    MF_CUDA_TRY(cudaMemcpyAsync(B.d_bptr, bptr.data(), sizeof(int) * (B.grid + 1), cudaMemcpyHostToDevice, s));
    if (!blist.empty())
        MF_CUDA_TRY(cudaMemcpyAsync(B.d_blist, blist.data(), sizeof(int2) * blist.size(), cudaMemcpyHostToDevice, s));
    MF_CUDA_TRY(cudaStreamSynchronize(s));
    return MF_SUCCESS;
}

// Every item's columns between the caller's arrays (one column after another)
// and the interleaved vectors: up to kMoveItems items per launch (blockIdx.y),
// their arrays passed as arguments.  (A launch per item and direction, and a
// read-back per item, took 1.5 of the 7.9 ms of a 40-system solve.)
constexpr int kMoveItems = 64;
enum { kMoveB = 0, kMoveX0 = 1, kMoveX = 2 };       // B in, X in, X out
struct MoveArgs {
    double *p[kMoveItems];
    int first, what;
};

__global__ void k_batch_move(const BatchItem *items, MoveArgs a)
{
    const BatchItem &it = items[a.first + blockIdx.y];
    double *flat = a.p[blockIdx.y];
    const int NR = it.nr, sh = __ffs(NR) - 1, n = it.n;
    double *mix = a.what == kMoveB ? const_cast<double *>(it.M.B) : it.M.X;
    const long long end = (long long)(a.what == kMoveX ? n : it.vec_len) * NR;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < end;
         t += (long long)gridDim.x * blockDim.x) {
        const int row = (int)(t >> sh), col = it.group * NR + (int)(t & (NR - 1));
        const bool real = row < n && col < it.nrhs;
        if (a.what != kMoveX) mix[t] = real ? flat[(long long)col * n + row] : 0.0;
        else if (real) flat[(long long)col * n + row] = mix[t];
    }
}

int batch_move(BatchImpl &B, const double *const *arrays, int what, cudaStream_t s)
{
    for (int t0 = 0; t0 < B.nitems; t0 += kMoveItems) {
        MoveArgs a;
        memset(&a, 0, sizeof(a));
        a.first = t0;
        a.what = what;
        const int count = std::min(kMoveItems, B.nitems - t0);
        for (int k = 0; k < count; k++) a.p[k] = const_cast<double *>(arrays[B.it_sys[t0 + k]]);
        k_batch_move<<<dim3(64, count), 256, 0, s>>>(B.d_items, a);
        MF_CUDA_TRY(cudaGetLastError());
    }
    return MF_SUCCESS;
}

// Enqueue one batched solve on s: interleave every item's columns, reset the
// queue head, error word and team counters, the cooperative persistent launch,
// de-interleave.  No host synchronisation.
int batch_enqueue(BatchImpl &B, const double *const *Bd, double *const *Xd, const BatchParams &bp0, int mode,
                  cudaStream_t s)
{
    MF_TRY(batch_move(B, Bd, kMoveB, s));
    if (bp0.x0_given) MF_TRY(batch_move(B, Xd, kMoveX0, s));     // the initial guesses: R = B - A X is formed in the launch
    MF_CUDA_TRY(cudaMemsetAsync(B.d_ctl, 0, B.ctl_bytes, s));
    BatchParams bp = bp0;
    bp.items = B.d_items;
    bp.order = B.d_order;
    bp.n_items = B.nqueue;
    bp.n_all = B.nitems;
    bp.head = B.d_ctl;
    bp.err = (int *)(B.d_ctl + 1);
    bp.bptr = B.d_bptr;
    bp.blist = B.d_blist;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(B.grid);
    cfg.blockDim = dim3(kThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (B.lb == 2) {
        if (mode == MODE_FP64) MF_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_batch<MODE_FP64, 2>, bp));
        else MF_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_batch<MODE_MIXED, 2>, bp));
    } else {
        if (mode == MODE_FP64) MF_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_batch<MODE_FP64, 1>, bp));
        else MF_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_batch<MODE_MIXED, 1>, bp));
    }
    MF_TRY(batch_move(B, Xd, kMoveX, s));
    return MF_SUCCESS;
}

}  // namespace

// The batch's team sizes and list schedule for given item costs (host only).
int mf_batch_schedule_impl(int nitems, const double *cost, const int *tilem, int grid, int *team, int *bptr,
                           int *blist, int *queue, int *nqueue)
{
    std::vector<double> c(cost, cost + nitems);
    std::vector<int> tm(tilem, tilem + nitems), tv, bp, q;
    std::vector<int2> bl;
    batch_schedule(c, tm, grid, tv, bp, bl, q);
    for (int t = 0; t < nitems; t++) team[t] = tv[t];
    for (int b = 0; b <= grid; b++) bptr[b] = bp[b];
    for (size_t e = 0; e < bl.size(); e++) {
        blist[2 * e] = bl[e].x;
        blist[2 * e + 1] = bl[e].y;
    }
    for (size_t k = 0; k < q.size(); k++) queue[k] = q[k];
    *nqueue = (int)q.size();
    return MF_SUCCESS;
}

struct mf_batch_s {
    BatchImpl impl;
};

int mf_batch_create_impl(mf_batch_s **out, int nsys, mf_matrix_s *const *systems, const int *nrhs, cudaStream_t s)
{
    mf_batch_s *b = new mf_batch_s();
    BatchImpl &B = b->impl;
    int rc = MF_SUCCESS;
    if (cudaGetDevice(&B.dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&B.nsm, cudaDevAttrMultiProcessorCount, B.dev) != cudaSuccess)
        rc = MF_ERR_CUDA;
    B.ctx = mf_context();
    if (rc == MF_SUCCESS) {
        // co-resident blocks of the cooperative launch (both precisions, both register budgets)
        int o[4] = {0, 0, 0, 0};
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o[0], k_batch<MODE_FP64, 1>, kThreads, 0) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o[1], k_batch<MODE_MIXED, 1>, kThreads, 0) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o[2], k_batch<MODE_FP64, 2>, kThreads, 0) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o[3], k_batch<MODE_MIXED, 2>, kThreads, 0) != cudaSuccess ||
            std::min(o[0], o[1]) < 1)
            rc = MF_ERR_CUDA;
        B.max_res[1] = std::min(o[0], o[1]) * B.nsm;
        B.max_res[2] = std::min(o[2], o[3]) * B.nsm;   // 0 if two blocks do not fit: never chosen
    }
    for (int k = 0; rc == MF_SUCCESS && k < nsys; k++) {
        if (!systems[k] || nrhs[k] < 1 || systems[k]->n_rows != systems[k]->n_cols || systems[k]->dev != B.dev) {
            rc = MF_ERR_INVALID;
            break;
        }
        B.sys.push_back(systems[k]);
        B.nrhs.push_back(nrhs[k]);
    }
    if (rc == MF_SUCCESS &&
        (cudaEventCreate(&B.e0) != cudaSuccess || cudaEventCreate(&B.e1) != cudaSuccess ||
         cudaEventCreateWithFlags(&B.e_in, cudaEventDisableTiming) != cudaSuccess ||
         cudaStreamCreateWithFlags(&B.own, cudaStreamNonBlocking) != cudaSuccess))
        rc = MF_ERR_CUDA;
    if (rc == MF_SUCCESS) rc = batch_build_items(B, 8, 1, s ? s : B.own);
    if (rc != MF_SUCCESS) {
        B.ended(rc);
        mf_batch_destroy_impl(b);
        return rc;
    }
    *out = b;
    return MF_SUCCESS;
}

void mf_batch_destroy_impl(mf_batch_s *b)
{
    if (!b) return;
    BatchImpl &B = b->impl;
    B.release_items();
    MfDeviceGuard guard(B.dev);
    if (!mf_context_gone(B.ctx)) {
        if (B.e0) cudaEventDestroy(B.e0);
        if (B.e1) cudaEventDestroy(B.e1);
        if (B.e_in) cudaEventDestroy(B.e_in);
        if (B.own) cudaStreamDestroy(B.own);
        mf_pool_settle(B.dev);
    }
    delete b;
}

// Solve every system's right-hand sides.  Bd[k] / Xd[k]: device arrays of
// nrhs[k] x n_k doubles.  With use_graph the sequence is captured into a CUDA
// graph on first use and replayed while pointers, options and items stay the same.
static int batch_solve(mf_batch_s *b, const double *const *Bd, double *const *Xd, const mf_options *opt,
                       mf_report *reps, int use_graph, cudaStream_t s)
{
    BatchImpl &B = b->impl;
    if (opt->method != MF_METHOD_CG || opt->precision == MF_PREC_PARITY) return MF_ERR_UNSUPPORTED;
    const int mode = opt->precision == MF_PREC_FP64 ? MODE_FP64 : MODE_MIXED;
    BatchParams bp;
    memset(&bp, 0, sizeof(bp));
    bp.max_iter = opt->max_iter;
    bp.fixed_iters = opt->fixed_iters;
    bp.replace_every = opt->replace_every;
    bp.use_lossless = opt->use_lossless;
    bp.tol = opt->tol;
    bp.min_fraction = opt->demote_min_fraction;
    bp.x0_given = opt->x0_given ? 1 : 0;
    bp.demote16 = (float)opt->demote_fp16;
    bp.demote8 = (float)opt->demote_int8;
    // team waits: within an item the members run in step (the normal bound);
    // arriving at an item may wait for members finishing earlier list entries
    const double to = opt->wait_timeout_s > 0 ? opt->wait_timeout_s : 10.0;
    bp.timeout_ns = (unsigned long long)(to * 1e9);
    bp.arrive_timeout_ns = (unsigned long long)(std::max(to * 30.0, 300.0) * 1e9);
    if (opt->test_stall_barrier) {
        // test hook: every team's first barrier waits for an arrival that never
        // comes and gives up after wait_timeout_s (MF_ERR_TIMEOUT, no fault)
        bp.stall_first = 1;
        bp.arrive_timeout_ns = bp.timeout_ns;
    }
    cudaStream_t run = s ? s : B.own;
    if (!s) {
        // the batch's own stream does not synchronise with the default stream on
        // its own: order it after the work already queued there (inputs, zeroing)
        MF_CUDA_TRY(cudaEventRecord(B.e_in, 0));
        MF_CUDA_TRY(cudaStreamWaitEvent(B.own, B.e_in, 0));
    }
    if (use_graph) {
        // the graph bakes in pointers, options and items: rebuilt when any changes
        std::vector<const void *> key;
        for (size_t k = 0; k < B.sys.size(); k++) {
            key.push_back(Bd[k]);
            key.push_back(Xd[k]);
        }
        const double opts[] = {opt->tol, (double)opt->max_iter, (double)opt->fixed_iters, (double)opt->replace_every,
                               opt->demote_fp16, opt->demote_int8, (double)opt->use_lossless, (double)B.cap,
                               (double)B.lb,
                               opt->wait_timeout_s, (double)opt->test_stall_barrier, opt->demote_min_fraction,
                               (double)opt->x0_given};
        for (double v : opts) {
            unsigned long long u;
            memcpy(&u, &v, sizeof(u));
            key.push_back((const void *)(uintptr_t)u);
        }
        if (!B.graph || key != B.graph_key || B.graph_mode != mode) {
            if (B.graph) cudaGraphExecDestroy(B.graph);
            B.graph = nullptr;
            cudaGraph_t g = nullptr;
            MF_CUDA_TRY(cudaStreamBeginCapture(run, cudaStreamCaptureModeThreadLocal));
            const int rc = batch_enqueue(B, Bd, Xd, bp, mode, run);
            const cudaError_t ce = cudaStreamEndCapture(run, &g);
            if (rc != MF_SUCCESS) {
                if (g) cudaGraphDestroy(g);
                return rc;
            }
            MF_CUDA_TRY(ce);
            const cudaError_t ie = cudaGraphInstantiate(&B.graph, g, 0);
            cudaGraphDestroy(g);
            MF_CUDA_TRY(ie);
            B.graph_key = key;
            B.graph_mode = mode;
        }
        MF_CUDA_TRY(cudaEventRecord(B.e0, run));
        MF_CUDA_TRY(cudaGraphLaunch(B.graph, run));
        MF_CUDA_TRY(cudaEventRecord(B.e1, run));
    } else {
        MF_CUDA_TRY(cudaEventRecord(B.e0, run));
        MF_TRY(batch_enqueue(B, Bd, Xd, bp, mode, run));
        MF_CUDA_TRY(cudaEventRecord(B.e1, run));
    }
    std::vector<double> outs((size_t)B.nitems * kOutWords);
    MF_CUDA_TRY(cudaMemcpyAsync(outs.data(), B.d_pool, outs.size() * sizeof(double), cudaMemcpyDeviceToHost, run));
    int team_err = 0;
    MF_CUDA_TRY(cudaMemcpyAsync(&team_err, B.d_ctl + 1, sizeof(int), cudaMemcpyDeviceToHost, run));
    MF_CUDA_TRY(cudaStreamSynchronize(run));
    const int chk = chk_take();
    if (chk) team_err = chk;
    float ms = 0.f;
    MF_CUDA_TRY(cudaEventElapsedTime(&ms, B.e0, B.e1));
    B.last_ms = ms;
    int status = team_err;
    double t_first = 0.0;                  // the launch's first item start (globaltimer ns)
    for (int t = 0; t < B.nitems; t++) {
        const double ts = outs[(size_t)t * kOutWords + 4 * B.it_nr[t] + 3];
        if (ts > 0.0 && (t_first == 0.0 || ts < t_first)) t_first = ts;
    }
    std::vector<int> first(B.sys.size() + 1, 0);
    for (size_t k = 0; k < B.sys.size(); k++) first[k + 1] = first[k] + B.nrhs[k];
    for (int t = 0; t < B.nitems; t++) {
        const double *o = outs.data() + (size_t)t * kOutWords;
        const int nr = B.it_nr[t];
        if ((int)o[4 * nr + 1] != MF_SUCCESS && status == MF_SUCCESS) status = (int)o[4 * nr + 1];
        if (!reps) continue;
        for (int c = 0; c < B.it_ncol[t]; c++) {
            mf_report *r = &reps[first[B.it_sys[t]] + B.it_col0[t] + c];
            memset(r, 0, sizeof(*r));
            r->iterations = (int)o[4 * c + 0];
            r->converged = (int)o[4 * c + 1];
            r->relres_true = o[4 * c + 2];
            r->relres_rec = o[4 * c + 3];
            r->status = team_err ? team_err : (int)o[4 * nr + 1];
            r->replacements = (int)o[4 * nr + 2];
            r->time_ms = ms;
            r->phase_ms[0] = o[4 * nr + 3] > 0.0 ? (o[4 * nr + 3] - t_first) * 1e-6 : 0.0;
            r->phase_ms[1] = o[4 * nr + 4] > 0.0 ? (o[4 * nr + 4] - t_first) * 1e-6 : 0.0;
            r->phase_ms[2] = (double)B.it_team[t];
            r->grid_blocks = B.grid;
            r->threads_per_block = kThreads;
        }
    }
    return status;
}

int mf_batch_solve_impl(mf_batch_s *b, const double *const *Bd, double *const *Xd, const mf_options *opt,
                        mf_report *reps, int use_graph, cudaStream_t s)
{
    return b->impl.ended(batch_solve(b, Bd, Xd, opt, reps, use_graph, s));
}

// Right-hand sides per work item chosen by timing: each candidate cap runs
// `iters` fixed iterations of the real batch with all-ones right-hand sides.
// A given (columns per item, blocks per SM), e.g. what mf_batch_tune chose for
// a batch of the same systems' shapes: the same item build, no timing runs.
int mf_batch_configure_impl(mf_batch_s *b, int cap, int lb, cudaStream_t s)
{
    BatchImpl &B = b->impl;
    if (cap != 1 && cap != 2 && cap != 4 && cap != 8) return MF_ERR_INVALID;
    // two blocks per SM only for items of up to 4 columns, as the tuner's candidates
    if (lb != 1 && !(lb == 2 && cap <= 4 && B.max_res[2] >= 1)) return MF_ERR_INVALID;
    return B.ended(batch_build_items(B, cap, lb, s ? s : B.own));
}

void mf_batch_config_impl(const mf_batch_s *b, int *cap, int *lb)
{
    if (cap) *cap = b->impl.cap;
    if (lb) *lb = b->impl.lb;
}

int mf_batch_tune_impl(mf_batch_s *b, int precision, int iters, int *chosen, cudaStream_t s)
{
    BatchImpl &B = b->impl;
    cudaStream_t run = s ? s : B.own;
    std::vector<double *> bufB(B.sys.size(), nullptr), bufX(B.sys.size(), nullptr);
    int rc = MF_SUCCESS;
    for (size_t k = 0; k < B.sys.size() && rc == MF_SUCCESS; k++) {
        const size_t e = (size_t)B.nrhs[k] * B.sys[k]->n_rows;
        if ((rc = mf_pool_array(&bufB[k], (long long)(2 * e), run)) != MF_SUCCESS) break;
        if (cudaStreamSynchronize(run) != cudaSuccess) rc = MF_ERR_CUDA;   // the copy below is not on this stream
        bufX[k] = bufB[k] + e;
        std::vector<double> ones(e, 1.0);
        if (cudaMemcpy(bufB[k], ones.data(), e * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess)
            rc = MF_ERR_CUDA;
    }
    mf_options o;
    mf_options_default(&o);
    o.precision = precision;
    o.fixed_iters = 1;
    o.max_iter = iters;
    o.replace_every = 0;
    // (columns per item, blocks per SM): two blocks per SM only for items of up
    // to 4 columns (8-column items need the 128-register budget)
    const int cand[][2] = {{8, 1}, {4, 1}, {2, 1}, {4, 2}, {2, 2}};
    int best = 8, best_lb = 1;
    double best_ms = 1e300;
    for (const auto &cl : cand) {
        if (rc != MF_SUCCESS) break;
        if (cl[1] == 2 && B.max_res[2] < 1) continue;
        if ((rc = batch_build_items(B, cl[0], cl[1], run)) != MF_SUCCESS) break;
        // the first run warms up; the faster of the next two counts (one timed
        // run of 20 iterations picked two blocks per SM where one was 7 %
        // faster over the whole 512-system batch)
        double ms = 1e300;
        for (int rep = 0; rep < 3 && rc == MF_SUCCESS; rep++) {
            rc = mf_batch_solve_impl(b, bufB.data(), bufX.data(), &o, nullptr, 0, run);
            if (rep > 0) ms = std::min(ms, B.last_ms);
        }
        // Two blocks per SM (64 registers, the multi-column walk spills) win the
        // short probe, where every item is active, but lose a full solve, whose
        // end is a tail of a few long items run at per-block speed: on the
        // 512-system batch the probe measured 315 ms (4 columns, 2 blocks)
        // against 344 ms (4 columns, 1 block), and the whole solve 13.2 s
        // against 11.2 s.  They count 15 % slower than measured.
        const double score = cl[1] == 2 ? 1.15 * ms : ms;
        if (rc == MF_SUCCESS && score < best_ms) {
            best_ms = score;
            best = cl[0];
            best_lb = cl[1];
        }
    }
    for (size_t k = 0; k < B.sys.size(); k++)
        mf_pool_free(bufB[k], run);
    if (rc == MF_SUCCESS) rc = batch_build_items(B, best, best_lb, run);
    if (chosen) *chosen = best;
    return B.ended(rc);
}
