// solver.cu -- host side of the single solves and the standalone products; the
// kernels of matrices without a one-chunk form (solver_dev.cuh).
#include "solver_dev.cuh"

#include <atomic>
#include <chrono>
#include <mutex>
#include <vector>

namespace {

// ------------------------------------------------------------ standalone SpMV
// y = A x, one half-warp per tile-row range (same pipeline as the solver), or
// tile-rows in turn when every tile-row is one chunk.
template <int MODE, int LB, int LEN>
__global__ void __launch_bounds__(kThreads, LB) k_spmv(SolverParams P, int force_pr, double *y, int rows_per_hw)
{
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, half = lane >> 4, i = lane & 15;
    const unsigned hmask = 0xFFFFu << (16 * half);
    XVec X = make_x(P.x, P.p32, nullptr, nullptr, nullptr, nullptr, 0.f);
    X.force_pr = force_pr;
    const int n = P.n;
    auto store = [&](int R, double v) {
        const int row = R * MF_BS + i;
        if (row < n) y[row] = v;
    };
    int rb = 0, re = 0;
    if (LEN == 0) {
        const int hw = (blockIdx.x * kWarps + wib) * 2 + half;
        rb = min(P.tilem, hw * rows_per_hw);
        re = min(P.tilem, rb + rows_per_hw);
        if (rb >= re) return;
    }
    spmv_range<MODE, MODE == MODE_FP64, LEN, true>(P, P.seg_ptr[rb], P.seg_ptr[re], i, hmask, X, nullptr, store);
    for (int R = rb; R < re; R++)            // tile-rows without tiles: y = 0
        if (P.seg_ptr[R] == P.seg_ptr[R + 1]) store(R, 0.0);
}

__global__ void k_ref_labels(const double *pold, const double *pnew, int nseg, int *vis)
{
    const int lane = threadIdx.x & 31;
    const int half = lane >> 4, i = lane & 15;
    const int seg = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 2 + half;
    const bool valid = seg < nseg;
    const int rk = valid ? ref_rank(fabs(pnew[(long long)seg * MF_BS + i] - pold[(long long)seg * MF_BS + i])) : 0;
    const int m = half_max_i(rk, 0xFFFFu << (16 * half));
    if (valid && i == 0) vis[seg] = rank_to_vis(m);
}

template <int METH>
const void *solve_kernel_m(int mode, int lb)
{
    if (lb == 2) {
        if (mode == MODE_FP64) return (const void *)k_solve<MODE_FP64, 2, METH, 0, kVarGrid>;
        if (mode == MODE_MIXED) return (const void *)k_solve<MODE_MIXED, 2, METH, 0, kVarGrid>;
        return (const void *)k_solve<MODE_PARITY, 2, METH, 0, kVarGrid>;
    }
    if (mode == MODE_FP64) return (const void *)k_solve<MODE_FP64, 1, METH, 0, kVarGrid>;
    if (mode == MODE_MIXED) return (const void *)k_solve<MODE_MIXED, 1, METH, 0, kVarGrid>;
    return (const void *)k_solve<MODE_PARITY, 1, METH, 0, kVarGrid>;
}

const void *solve_kernel(int mode, int lb, int method)
{
    return method == MF_METHOD_BICGSTAB ? solve_kernel_m<MF_METHOD_BICGSTAB>(mode, lb)
                                        : solve_kernel_m<MF_METHOD_CG>(mode, lb);
}

int ws_get(mf_matrix_s *A, int blocks_per_sm, Workspace **out, cudaStream_t s)
{
    // blocks_per_sm: 0 = default variant, 1 or 2 = that register-budget variant
    const int lb = (blocks_per_sm == 2) ? 2 : (blocks_per_sm == 1) ? 1 : kDefaultLB;
    // the workspace of an earlier call with the same variant (its grid depends on
    // the handle and the device alone)
    Workspace *w = (Workspace *)A->ws;
    if (w && w->lb == lb) {
        *out = w;
        return MF_SUCCESS;
    }
    int dev = 0;
    MF_CUDA_TRY(cudaGetDevice(&dev));
    int nsm = 0;
    MF_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    int coop = 0;
    MF_CUDA_TRY(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop) return MF_ERR_UNSUPPORTED;
    // one grid size for every precision mode, so the cached workspace is shared
    int occ = 1 << 20;
    for (int m = MODE_FP64; m <= MODE_PARITY; m++) {
        for (int meth = MF_METHOD_CG; meth <= MF_METHOD_BICGSTAB; meth++) {
            int o = 0;
            MF_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, solve_kernel(m, lb, meth), kThreads, 0));
            occ = o < occ ? o : occ;
        }
    }
    if (occ < 1) return MF_ERR_UNSUPPORTED;
    if (occ > lb) occ = lb;
    int G = nsm * occ;
    // small systems: no more blocks than needed for one tile-row per half-warp
    const int need = (A->tilem + kWarps * 2 - 1) / (kWarps * 2);
    if (need < G) G = need > 0 ? need : 1;
    if (w) {
        mf_handle_wait(A);
        mf_solver_free_ws(A);
    }
    w = new Workspace();
    memset(w, 0, sizeof(*w));
    w->G = G;
    w->lb = lb;
    w->nsm = nsm;
    const long long L = A->vec_len;
    const long long S = std::max(A->tilem, A->tilen) + 1;
    {
        const size_t f = (size_t)L * sizeof(float), d = (size_t)L * sizeof(double), h = (size_t)L * sizeof(__half);
        w->vec_bytes = d;
        w->all_bytes = 7 * d + 2 * f + 2 * h + 2 * (size_t)L;
        MF_TRY(mf_pool_alloc((void **)&w->vecs, w->all_bytes, s));
        char *c = w->vecs;
        w->x = (double *)c; c += d;
        w->p = (double *)c; c += d;
        w->q = (double *)c; c += d;
        w->r = (double *)c; c += d;
        w->s = (double *)c; c += d;
        w->t = (double *)c; c += d;
        w->rh = (double *)c; c += d;
        w->p32 = (float *)c; c += f;
        w->s32 = (float *)c; c += f;
        w->p16 = (__half *)c; c += h;
        w->s16 = (__half *)c; c += h;
        w->p8 = (int8_t *)c; c += L;
        w->s8 = (int8_t *)c;
        // zeros past n_rows: a matrix with more columns than rows gathers there
        MF_CUDA_TRY(cudaMemsetAsync(w->vecs, 0, w->all_bytes, s));
    }
    MF_TRY(mf_pool_array(&w->mag_p, S, s)); MF_TRY(mf_pool_array(&w->mag_s, S, s));
    MF_TRY(mf_pool_array(&w->lab_p, S, s)); MF_TRY(mf_pool_array(&w->lab_s, S, s));
    MF_TRY(mf_pool_array(&w->red, (long long)kRedKinds * G * kRedWidth, s));
    MF_TRY(mf_pool_array(&w->ctl, (long long)kCtlBytes, s));
    {
        Readback *rb = (Readback *)(w->ctl + 128);
        w->bar = (unsigned int *)w->ctl;
        w->err = &rb->err;
        w->out = rb->out;
        w->counts = rb->counts;
        w->phase_ns = rb->phase_ns;
    }
    // column segments past the tile-rows keep magnitude 0 (a matrix with more columns than rows)
    MF_CUDA_TRY(cudaMemsetAsync(w->mag_p, 0, (size_t)S * sizeof(float), s));
    MF_CUDA_TRY(cudaMemsetAsync(w->mag_s, 0, (size_t)S * sizeof(float), s));
    MF_TRY(exact_tiles(A, w->counts, s));    // counts: scratch before the first solve zeroes it
    // Small systems run as one cluster of up to 16 blocks, where the device can place
    // it.  One-chunk matrices up to two tile-rows per half-warp (1,024): us per
    // iteration, one cluster against the grid, 8,281 / 16,384 rows of the 2D
    // Laplacian 3.2 / 3.4 against 6.2 / 6.1 (CG, FP64), 9,261 rows in 3D 4.2 against
    // 7.0 (CG), 12.9 against 18.6 (BiCGSTAB); 32,768 rows 8.0 against 6.9.  Others
    // have more to stream through 16 SMs: 27-point 9,261 rows 9.0 against 11.2,
    // 32,768 rows 18.9 against 12.5; irregular 16,000 rows 11.3 against 11.5.
    if (A->tilem <= (A->one_chunk ? 2 * kMaxCluster * kWarps * 2 : 768)) {
        const void *fn = mf_solve_cluster_kernel(MODE_FP64, MF_METHOD_CG, 0, 1);
        const int C = std::min(G, kMaxCluster);
        cudaLaunchConfig_t cfg;
        memset(&cfg, 0, sizeof(cfg));
        cfg.gridDim = dim3(C);
        cfg.blockDim = dim3(kThreads);
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = C;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int fit = 0;
        if (cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&fit, fn, &cfg) != cudaSuccess)
            cudaGetLastError();
        if (fit > 0) {
            const int nhw = C * kWarps * 2;
            w->cluster = C;
            MF_TRY(mf_pool_array(&w->hw_begin_cl, nhw + 1, s));
            k_partition<<<(nhw + 256) / 256, 256, 0, s>>>(A->d_row_cost, A->tilem, nhw, w->hw_begin_cl);
            MF_CUDA_TRY(cudaGetLastError());
        }
    }
    w->nhw = G * kWarps * 2;
    MF_TRY(mf_pool_array(&w->hw_begin, w->nhw + 1, s));
    MF_CUDA_TRY(cudaEventCreate(&w->e0));
    MF_CUDA_TRY(cudaEventCreate(&w->e1));
    k_partition<<<(w->nhw + 256) / 256, 256, 0, s>>>(A->d_row_cost, A->tilem, w->nhw, w->hw_begin);
    MF_CUDA_TRY(cudaGetLastError());
    A->ws = w;
    *out = w;
    return MF_SUCCESS;
}

// Persisting L2 access-policy window on a stream for the duration of a solve.
struct L2Window {
    bool active = false;
    size_t old_limit = 0;
    cudaStreamAttrValue old_attr;
    void set(cudaStream_t s, void *base, size_t bytes)
    {
        int dev = 0, max_persist = 0, max_win = 0;
        if (cudaGetDevice(&dev) != cudaSuccess) return;
        if (cudaDeviceGetAttribute(&max_persist, cudaDevAttrMaxPersistingL2CacheSize, dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&max_win, cudaDevAttrMaxAccessPolicyWindowSize, dev) != cudaSuccess ||
            max_persist <= 0 || max_win <= 0) {
            cudaGetLastError();
            return;
        }
        if (cudaStreamGetAttribute(s, cudaStreamAttributeAccessPolicyWindow, &old_attr) != cudaSuccess ||
            cudaDeviceGetLimit(&old_limit, cudaLimitPersistingL2CacheSize) != cudaSuccess) {
            cudaGetLastError();
            return;
        }
        const size_t win = bytes < (size_t)max_win ? bytes : (size_t)max_win;
        const size_t lim = win < (size_t)max_persist ? win : (size_t)max_persist;
        if (cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, lim) != cudaSuccess) {
            cudaGetLastError();
            return;
        }
        cudaStreamAttrValue a;
        memset(&a, 0, sizeof(a));
        a.accessPolicyWindow.base_ptr = base;
        a.accessPolicyWindow.num_bytes = win;
        a.accessPolicyWindow.hitRatio = (float)((double)lim / (double)win);
        a.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
        a.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
        if (cudaStreamSetAttribute(s, cudaStreamAttributeAccessPolicyWindow, &a) != cudaSuccess) {
            cudaGetLastError();
            cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, old_limit);
            return;
        }
        active = true;
    }
    void reset(cudaStream_t s)
    {
        if (!active) return;
        cudaStreamSetAttribute(s, cudaStreamAttributeAccessPolicyWindow, &old_attr);
        cudaCtxResetPersistingL2Cache();
        cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, old_limit);
        cudaGetLastError();
        active = false;
    }
};

// The part of the vector block to keep in L2 for a solve (0 bytes: no window).
//  * Nothing when the vectors and the matrix stream fit in three quarters of L2
//    together: the window changed no solve time below that (96^3 CG and
//    BiCGSTAB, 256^2: within 1 %) and setting it up and back costs 50 us a call.
//  * Whole vectors only, as many as fit in 7/8 of the persisting set-aside
//    (72 of 83 MB): a window wider than the set-aside marks part of its lines
//    streaming, and those thrash (2048^2 CG with all four vectors, 134 MB:
//    20.5 ms per 100 iterations, 10.5 without a window; 160^3: 3.5 against 3.1).
//    CG takes r first (read by the SpMV and the update, written by the update),
//    then q, p and x; BiCGSTAB p, q, r, s, t, rh, then x.
//    Measured per 24 CG iterations, no window -> this rule: 128^3 1.41 -> 1.23,
//    144^3 2.18 -> 1.98 (p, q, r), 160^3 3.13 -> 2.82 (q, r), 2048^2 3.22 ->
//    2.97 (q, r), 2500^2 4.81 -> 4.37 ms (r); 112^3 BiCGSTAB 1.22 -> 1.17.
struct VecWindow {
    void *base;
    size_t bytes;
};

VecWindow vec_window(const Workspace *w, int mode, int method, size_t matrix_bytes)
{
    int dev = 0, l2 = 0, persist = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&persist, cudaDevAttrMaxPersistingL2CacheSize, dev) != cudaSuccess) {
        cudaGetLastError();
        return {w->vecs, 0};
    }
    const size_t room = (size_t)(persist > 0 ? persist : 0) / 8 * 7, d = w->vec_bytes;
    const bool bicg = method == MF_METHOD_BICGSTAB;
    const size_t used = bicg ? 7 : 4;
    if (mode == MODE_PARITY) return {w->vecs, w->all_bytes <= room ? w->all_bytes : 0};
    if (used * d + matrix_bytes <= (size_t)l2 / 4 * 3) return {w->vecs, 0};
    const size_t k = std::min(used, d > 0 ? room / d : 0);
    char *base = k == used ? w->vecs : bicg ? (char *)w->p : (char *)(w->r + d / sizeof(double)) - k * d;
    return {base, k * d};
}

}  // namespace

// (after mf_handle_wait)
void mf_solver_free_ws(mf_matrix_s *A, bool gone)
{
    Workspace *w = (Workspace *)A->ws;
    if (!w) return;
    if (!gone) {
        void *ptrs[] = {w->vecs, w->mag_p, w->mag_s, w->lab_p, w->lab_s, w->red, w->ctl, w->hw_begin, w->hw_begin_cl,
                        w->m_vec, w->m_mag, w->m_red, w->m_out, w->m_err, w->m_hw_begin};
        mf_pool_give_back(ptrs, (int)(sizeof(ptrs) / sizeof(ptrs[0])));
        for (int k = 0; k < 2 * w->m_groups; k++) cudaEventDestroy(w->m_ev[k]);
        cudaEventDestroy(w->e0);
        cudaEventDestroy(w->e1);
    }
    delete[] w->m_ev;
    delete w;
    A->ws = nullptr;
}

int mf_ws_get(mf_matrix_s *A, int blocks_per_sm, void **out, cudaStream_t s)
{
    return ws_get(A, blocks_per_sm, (Workspace **)out, s);
}

int mf_solver_run(mf_matrix_s *A, const double *d_b, double *d_x, const mf_options *opt, mf_report *rep,
                  cudaStream_t s)
{
    const int mode = opt->precision == MF_PREC_FP64 ? MODE_FP64
                     : opt->precision == MF_PREC_PARITY ? MODE_PARITY : MODE_MIXED;
    if (opt->method != MF_METHOD_CG && opt->method != MF_METHOD_BICGSTAB) return MF_ERR_INVALID;
    const auto t_begin = std::chrono::steady_clock::now();
    Workspace *w = nullptr;
    MF_TRY(ws_get(A, opt->blocks_per_sm, &w, s));
    const long long L = A->vec_len;
    const long long S = std::max(A->tilem, A->tilen) + 1;
    // The kernel writes every entry below n_rows before it reads it, and the tails
    // stay zero from the workspace's creation; parity mode's shadows and labels
    // start from zero each time.  (Seven fills of whole vectors, and one per result
    // array, went before each solve: 60 us of launches, and five read-backs after.)
    if (opt->x0_given)
        MF_CUDA_TRY(cudaMemcpyAsync(w->x, d_x, (size_t)A->n_rows * sizeof(double), cudaMemcpyDeviceToDevice, s));
    if (mode == MODE_PARITY) {
        MF_CUDA_TRY(cudaMemsetAsync(w->s, 0, L * sizeof(double), s));
        MF_CUDA_TRY(cudaMemsetAsync(w->p32, 0, w->all_bytes - 7 * w->vec_bytes, s));   // p32 .. s8
        MF_CUDA_TRY(cudaMemsetAsync(w->lab_p, 0, S, s));
        MF_CUDA_TRY(cudaMemsetAsync(w->lab_s, 0, S, s));
    }
    MF_CUDA_TRY(cudaMemsetAsync(w->ctl, 0, kCtlBytes, s));
    SolverParams P;
    fill_params(P, A, w);
    P.b = d_b;
    P.method = opt->method;
    P.x0_given = opt->x0_given ? 1 : 0;
    P.max_iter = opt->max_iter;
    P.fixed_iters = opt->fixed_iters;
    P.replace_every = opt->replace_every;
    P.use_lossless = opt->use_lossless;
    P.lossless_any = lossless_on(opt->use_lossless, opt->demote_min_fraction, A->n_exact, A->tilenum);
    P.min_small = (float)(opt->demote_min_fraction * (double)A->tilem);
    P.min_demoted = (float)(opt->demote_min_fraction * (double)A->tilenum);
    P.relax_eta = (float)opt->relax_eta;
    P.relax_int8 = opt->relax_int8 ? 1 : 0;
    P.fp16_ok = A->n_fp16_ok == A->tilenum ? 1 : 0;
    // every tile exact in FP16: the lossless choice is the same for every tile and
    // every SpMV, so it is made here and the walk stays lookup-free (the per-slice
    // lookups with all tiles FP16 measured 37 % slower than the FP32 lean walk on
    // the 2048^2 Laplacian)
    if (opt->use_lossless && A->tilenum > 0 && A->n_exact_f16 == A->tilenum) {
        P.lean_f16 = 1;
        P.lossless_any = 0;
    }
    P.tol = opt->tol;
    P.demote16 = (float)opt->demote_fp16;
    P.demote8 = (float)opt->demote_int8;
    double to = opt->wait_timeout_s > 0 ? opt->wait_timeout_s : 10.0;
    P.timeout_ns = (unsigned long long)(to * 1e9);
    P.stall_first_barrier = opt->test_stall_barrier ? 1 : 0;
    if (opt->test_check_limit > 0) P.chk_xlen = (int)std::min<long long>(L, opt->test_check_limit & ~15LL);
    void *args[] = {&P};
    // Keep the iteration vectors in L2 while the matrix payload streams past
    // them: a persisting access-policy window over the vector block (best
    // effort; the previous stream attribute and context limit are restored).
    L2Window win;
    // (the FP64 / mixed modes never touch the narrow shadows: a smaller
    // persisting set-aside leaves more of L2 to the matrix stream -- measured
    // 3.5 % faster on the 128^3 system than a window that included p32)
    if (opt->l2_window) {
        const size_t value = mode != MODE_MIXED ? 8 : P.lean_f16 ? 2 : 4;
        const VecWindow vw = vec_window(w, mode, opt->method, (size_t)A->slice_entries * (value + 1));
        if (vw.bytes > 0) win.set(s, vw.base, vw.bytes);
    }
    const auto t_prepared = std::chrono::steady_clock::now();
    MF_CUDA_TRY(cudaEventRecord(w->e0, s));
    // One-chunk matrices (the 5- and 7-point stencils) have kernels of their own
    // in the default two-blocks-per-SM budget; everything else, parity mode and
    // the one-block variant take the general walks.
    // Systems with no more tile-rows than half-warps have kernels of theirs too.
    // (They stay out of the stalled-barrier test, which needs the grid counter.)
    const bool rows = A->one_chunk && mode != MODE_PARITY && w->lb == 2;
    const bool small = mode != MODE_PARITY && w->lb == 2 && !opt->test_stall_barrier;
    // (BiCGSTAB on more than 512 tile-rows would be summed over fewer blocks than the
    // grid's: its rounding stays as it is there.)
    const bool cluster = small && w->cluster && (opt->method == MF_METHOD_CG || w->cluster == w->G);
    const void *kfn = cluster ? mf_solve_cluster_kernel(mode, opt->method, A->one_chunk ? A->max_row : 0,
                                                          (A->tilem + w->cluster * kWarps * 2 - 1) /
                                                              (w->cluster * kWarps * 2))
                      : small && rows && opt->method == MF_METHOD_CG && A->tilem <= w->G * kWarps * 2
                          ? mf_solve_resident_kernel(mode, w->G <= w->nsm ? 1 : 2, A->max_row)
                      : rows ? mf_solve_rows_kernel(mode, opt->method, A->max_row)
                             : solve_kernel(mode, w->lb, opt->method);
    cudaError_t lerr;
    if (cluster) {
        // One cluster: its barrier and shared memory take the grid barrier's place
        // (P.cluster).  An all-reduce with the barrier takes 0.9 us on 2 - 8 blocks and
        // 1.05 on 16, through the grid counter 2.2 - 2.3 us.
        P.cluster = w->cluster;
        P.hw_begin = w->hw_begin_cl;
        cudaLaunchConfig_t cfg;
        memset(&cfg, 0, sizeof(cfg));
        cfg.gridDim = dim3(w->cluster);
        cfg.blockDim = dim3(kThreads);
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = w->cluster;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        lerr = w->cluster > 8 ? cudaFuncSetAttribute(kfn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) : cudaSuccess;
        if (lerr == cudaSuccess) lerr = cudaLaunchKernelExC(&cfg, kfn, args);
    } else {
        lerr = cudaLaunchCooperativeKernel(kfn, dim3(w->G), dim3(kThreads), args, 0, s);
    }
    if (lerr != cudaSuccess) {
        win.reset(s);
        MF_CUDA_TRY(lerr);
    }
    MF_CUDA_TRY(cudaEventRecord(w->e1, s));
    MF_CUDA_TRY(cudaMemcpyAsync(d_x, w->x, (size_t)A->n_rows * sizeof(double), cudaMemcpyDeviceToDevice, s));
    Readback rb;
    MF_CUDA_TRY(cudaMemcpyAsync(&rb, w->ctl + 128, sizeof(rb), cudaMemcpyDeviceToHost, s));
    MF_CUDA_TRY(cudaStreamSynchronize(s));
    win.reset(s);
    const double *out = rb.out;
    const unsigned long long *counts = rb.counts, *phase = rb.phase_ns;
    int err = rb.err;
    int chk = chk_take();
    if (!chk) chk = mf_rows_chk_take();
    if (!chk) chk = mf_small_chk_take();
    if (chk) err = chk;
    const auto t_done = std::chrono::steady_clock::now();
    float ms = 0.f;
    MF_CUDA_TRY(cudaEventElapsedTime(&ms, w->e0, w->e1));
    if (rep) {
        memset(rep, 0, sizeof(*rep));
        rep->host_ms[1] = std::chrono::duration<double, std::milli>(t_prepared - t_begin).count();
        rep->host_ms[2] = std::chrono::duration<double, std::milli>(t_done - t_prepared).count();
        rep->iterations = (int)out[0];
        rep->converged = (int)out[1];
        rep->relres_true = out[2];
        rep->relres_rec = out[3];
        rep->residual = out[4];
        rep->replacements = (int)out[5];
        rep->status = err ? err : (int)out[6];
        rep->time_ms = ms;
        rep->grid_blocks = cluster ? w->cluster : w->G;
        rep->threads_per_block = kThreads;
        for (int j = 0; j < 4; j++) rep->tile_uses[j] = (long long)counts[j];
        rep->tiles_skipped = (long long)counts[4];
        for (int j = 0; j < 4; j++) rep->nnz_uses[j] = (long long)counts[5 + j];
        if (mode == MODE_FP64) {
            // every tile of every SpMV phase runs in FP64: counted here, not in the kernel
            const long long nspmv = (long long)out[7];
            rep->tile_uses[0] = nspmv * A->tilenum;
            rep->nnz_uses[0] = nspmv * A->nnz;
        }
        for (int j = 0; j < 6; j++) rep->phase_ms[j] = (double)phase[j] * 1e-6;
    }
    if (err) return err;
    return (int)out[6];
}

namespace {

using SpmvFn = void (*)(SolverParams, int, double *, int);

template <int LEN>
SpmvFn spmv_kernel_len(bool f64)
{
    return f64 ? (SpmvFn)k_spmv<MODE_FP64, 2, LEN> : (SpmvFn)k_spmv<MODE_MIXED, 2, LEN>;
}

// k_spmv for a matrix and stored precision: one-chunk matrices by their longest
// row (INT8 products need the per-tile scales of the general walk).
SpmvFn spmv_kernel(const mf_matrix_s *A, int tile_prec, int *variant)
{
    const bool f64 = tile_prec == MF_P64;
    const int len = (!A->one_chunk || tile_prec == MF_P8) ? 0 : A->max_row <= 5 ? 5 : A->max_row <= 7 ? 7 : 8;
    *variant = (len == 0 ? 0 : len == 5 ? 1 : len == 7 ? 2 : 3) * 2 + (f64 ? 1 : 0);
    return len == 0 ? spmv_kernel_len<0>(f64) : len == 5 ? spmv_kernel_len<5>(f64)
           : len == 7 ? spmv_kernel_len<7>(f64) : spmv_kernel_len<8>(f64);
}

// Blocks per SM of a k_spmv variant on a device (a property of the device and
// the kernel, asked for once).
int spmv_resident(int dev, SpmvFn fn, int variant, int *occ)
{
    constexpr int kDevs = 64;
    static std::atomic<int> known[8][kDevs];
    int o = (dev >= 0 && dev < kDevs) ? known[variant][dev].load(std::memory_order_relaxed) : 0;
    if (o == 0) {
        MF_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, (const void *)fn, kThreads, 0));
        if (o < 1) o = 1;
        if (dev >= 0 && dev < kDevs) known[variant][dev].store(o, std::memory_order_relaxed);
    }
    *occ = o;
    return MF_SUCCESS;
}

// One wave: resident blocks x SMs, each half-warp a contiguous range of
// tile-rows (or every stride-th one, spmv_rows).
int spmv_launch(mf_matrix_s *A, const double *x, double *y, int tile_prec, cudaStream_t s)
{
    SolverParams P;
    fill_params(P, A, nullptr);
    P.x = const_cast<double *>(x);
    // gathers reach the columns that have entries, and column 0 of a slice's first tile (padding)
    P.chk_xlen = A->n_cols;
    int nsm = 0, dev = 0, occ = 1, variant = 0;
    MF_CUDA_TRY(cudaGetDevice(&dev));
    MF_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    SpmvFn fn = spmv_kernel(A, tile_prec, &variant);
    MF_TRY(spmv_resident(dev, fn, variant, &occ));
    const int nhw_max = nsm * occ * kWarps * 2;
    int rows_per_hw = (A->tilem + nhw_max - 1) / nhw_max;
    if (rows_per_hw < 1) rows_per_hw = 1;
    const int nhw = (A->tilem + rows_per_hw - 1) / rows_per_hw;
    int blocks = (nhw + kWarps * 2 - 1) / (kWarps * 2);
    if (blocks < 1) blocks = 1;
    fn<<<blocks, kThreads, 0, s>>>(P, tile_prec, y, rows_per_hw);
    MF_CUDA_TRY(cudaGetLastError());
    return MF_SUCCESS;
}

// Whether the product reads the caller's x where it is.  A kernel needs what a copy
// does not: x on the handle's own device (or managed), on an 8-byte boundary, and
// apart from y.  Otherwise x is copied first, which takes any alignment, another
// GPU's memory and pinned host memory (whose gathers would each cross PCIe), and
// refuses a pageable host pointer with an error where a kernel would fault.
// (Asking costs 0.06 us.)
bool spmv_in_place(const mf_matrix_s *A, const double *x, const double *y)
{
    const uintptr_t x0 = (uintptr_t)x, x1 = x0 + (size_t)A->n_cols * sizeof(double);
    const uintptr_t y0 = (uintptr_t)y, y1 = y0 + (size_t)A->n_rows * sizeof(double);
    if ((x0 < y1 && y0 < x1) || x0 % sizeof(double) != 0) return false;
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, x) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return at.type == cudaMemoryTypeManaged || (at.type == cudaMemoryTypeDevice && at.device == A->dev);
}

// x copied for a product; a refusal is this call's error, not the next launch's.
cudaError_t spmv_copy(const mf_matrix_s *A, double *to, const double *x, cudaStream_t s)
{
    const cudaError_t e = cudaMemcpyAsync(to, x, (size_t)A->n_cols * sizeof(double), cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

}  // namespace

// y = A x with every tile in one entry precision (MF_P64 .. MF_P8).  The kernel
// reads the caller's x in place: it gathers no column past n_cols, so the padded
// copy made before (33 MB moved and a 16.8 MB fill for 128^3: 20 of 75 us) is
// needed only where spmv_in_place says so.
int mf_spmv_tiles_run(mf_matrix_s *A, const double *d_x, double *d_y, int tile_prec, cudaStream_t s,
                      double *elapsed_ms)
{
    if (tile_prec < MF_P64 || tile_prec > MF_P8) return MF_ERR_INVALID;
    for (cudaEvent_t &e : A->spmv_ev)
        if (!e) MF_CUDA_TRY(cudaEventCreate(&e));
    double *copy = nullptr;
    if (!spmv_in_place(A, d_x, d_y)) {
        MF_TRY(mf_pool_array(&copy, A->n_cols, s));
        const cudaError_t e = spmv_copy(A, copy, d_x, s);
        if (e != cudaSuccess) mf_pool_free(copy, s);
        MF_CUDA_TRY(e);
        d_x = copy;
    }
    cudaError_t e0 = cudaEventRecord(A->spmv_ev[0], s);
    const int rc = e0 == cudaSuccess ? spmv_launch(A, d_x, d_y, tile_prec, s) : MF_SUCCESS;
    if (e0 == cudaSuccess) e0 = cudaEventRecord(A->spmv_ev[1], s);
    mf_pool_free(copy, s);
    MF_TRY(rc);
    MF_CUDA_TRY(e0);
    MF_CUDA_TRY(cudaStreamSynchronize(s));
    MF_TRY(chk_take());
    if (elapsed_ms) {
        float ms = 0.f;
        MF_CUDA_TRY(cudaEventElapsedTime(&ms, A->spmv_ev[0], A->spmv_ev[1]));
        *elapsed_ms = ms;
    }
    return MF_SUCCESS;
}

int mf_spmv_run(mf_matrix_s *A, const double *d_x, double *d_y, int precision, cudaStream_t s, double *elapsed_ms)
{
    return mf_spmv_tiles_run(A, d_x, d_y, precision == MF_PREC_FP64 ? MF_P64 : MF_P32, s, elapsed_ms);
}

// The parity-mode labels the last solve left in the workspace (one per column
// segment), as d_vis codes.
int mf_solver_labels_run(mf_matrix_s *A, int *vis, int nseg)
{
    Workspace *w = (Workspace *)A->ws;
    if (!w || nseg < 0 || nseg > std::max(A->tilem, A->tilen)) return MF_ERR_INVALID;
    std::vector<signed char> h((size_t)nseg + 1);
    if (nseg > 0) MF_CUDA_TRY(cudaMemcpy(h.data(), w->lab_p, (size_t)nseg, cudaMemcpyDeviceToHost));
    for (int j = 0; j < nseg; j++) vis[j] = h[j];
    return MF_SUCCESS;
}

int mf_ref_labels_run(const double *d_pold, const double *d_pnew, int nseg, int *d_vis, cudaStream_t s)
{
    if (nseg <= 0) return MF_SUCCESS;
    const int threads = 256;
    const int segs_per_block = threads / 16;
    k_ref_labels<<<(nseg + segs_per_block - 1) / segs_per_block, threads, 0, s>>>(d_pold, d_pnew, nseg, d_vis);
    MF_CUDA_TRY(cudaGetLastError());
    MF_CUDA_TRY(cudaStreamSynchronize(s));
    return MF_SUCCESS;
}

// ------------------------------------------------------------ tensor-core experiment (8 right-hand sides)
// Y = A X for 8 interleaved columns (row i's 8 values contiguous) with every
// tile's values stored in FP16, in two forms:
//  * CUDA cores (k_spmm_cc): the solver's arithmetic -- a half-warp per
//    tile-row, the FP16 value widened to FP64 against the FP64 row of X, 8
//    FP64 sums per row;
//  * tensor cores (k_spmm_tc): a warp per tile-row; each 16 x 16 tile of a
//    slice is densified in shared memory from the sparse payload (nothing
//    dense is read from HBM), X's 16 x 8 segment is rounded to FP16, and one
//    mma.sync.m16n8k16 per tile accumulates the 16 x 8 block in FP32.
// Both read the same slice payload; mf_debug_spmm times them side by side.
namespace {
constexpr int kTcWarps = 4;                          // warps per block of k_spmm_tc
constexpr int kTcSmem = kTcWarps * MF_SEG_TILES * 256 * 2;   // dense FP16 tiles of one slice per warp

__global__ void __launch_bounds__(kThreads, 2) k_spmm_cc(SolverParams P, const double *X, double *Y)
{
    const int lane = threadIdx.x & 31, i = lane & 15;
    const unsigned hmask = 0xFFFFu << (16 * (lane >> 4));
    const int R = ((blockIdx.x * blockDim.x + threadIdx.x) >> 4);
    if (R >= P.tilem) return;
    double acc[8];
#pragma unroll
    for (int q = 0; q < 8; q++) acc[q] = 0.0;
    const int sb = P.seg_ptr[R], se = P.seg_ptr[R + 1];
    if (sb < se && (!chk_in(CHK_SLICE, sb, P.nseg) || !chk_in(CHK_SLICE, se - 1, P.nseg))) return;
    for (int s = sb; s < se; s++) {
        const int4 h = P.seg_hdr[s];
        const int xb = (load_tw(P, s, i) >> 8) * MF_BS;
        const int len = load_len(P, s, i, h);
        if (!chk_in(CHK_PAYLOAD, hdr_off(h) + (long long)hdr_kp(h) * MF_BS - 1, P.n_payload)) continue;
        for (int k0 = 0; k0 < hdr_kp(h); k0 += 8) {
            const long long cb = hdr_off(h) + (long long)(k0 >> 3) * 128;
            double v64[8];
            float v[8];
            load_chunk<MF_P16>(P, cb, i, len - k0, v64, v);
            const unsigned long long m8 = __ldcs((const unsigned long long *)(P.meta + cb) + i);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const unsigned mm = (unsigned)(m8 >> (8 * j)) & 0xFFu;
                const int xi = __shfl_sync(hmask, xb, (int)(mm >> 4), 16) + (int)(mm & 15u);
                if (k0 + j < len && chk_in(CHK_X, xi, P.chk_xlen)) {
                    const double2 *xr = (const double2 *)(X + (long long)xi * 8);
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const double2 d = xr[q];
                        acc[2 * q] = fma((double)v[j], d.x, acc[2 * q]);
                        acc[2 * q + 1] = fma((double)v[j], d.y, acc[2 * q + 1]);
                    }
                }
            }
        }
    }
    const int row = R * MF_BS + i;
    if (row < P.n) {
        double2 *yr = (double2 *)(Y + (long long)row * 8);
#pragma unroll
        for (int q = 0; q < 4; q++) yr[q] = make_double2(acc[2 * q], acc[2 * q + 1]);
    }
}

__device__ __forceinline__ unsigned pack_half2(double lo, double hi)
{
    return (unsigned)__half_as_ushort(__double2half(lo)) | ((unsigned)__half_as_ushort(__double2half(hi)) << 16);
}

__global__ void __launch_bounds__(kTcWarps * 32) k_spmm_tc(SolverParams P, const double *X, double *Y)
{
    extern __shared__ __align__(16) unsigned short tc_tiles[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int R = blockIdx.x * kTcWarps + w;
    if (R >= P.tilem) return;
    unsigned short *tiles = tc_tiles + w * MF_SEG_TILES * 256;   // [slot][row][col] FP16 bits
    const int g = lane >> 2, c = lane & 3;
    float d[4] = {0.f, 0.f, 0.f, 0.f};
    const int sb = P.seg_ptr[R], se = P.seg_ptr[R + 1];
    if (sb < se && (!chk_in(CHK_SLICE, sb, P.nseg) || !chk_in(CHK_SLICE, se - 1, P.nseg))) return;
    for (int s = sb; s < se; s++) {
        const int4 h = P.seg_hdr[s];
        const int nt = hdr_nt(h);
        if (!chk_in(CHK_PAYLOAD, hdr_off(h) + (long long)hdr_kp(h) * MF_BS - 1, P.n_payload)) continue;
        for (int e = lane; e < nt * 128; e += 32) ((unsigned *)tiles)[e] = 0u;
        __syncwarp();
        // lanes 0..15 scatter their row's entries into the dense tiles
        if (lane < 16) {
            const int len = load_len(P, s, lane, h);
            for (int k0 = 0; k0 < len; k0 += 8) {
                const long long cb = hdr_off(h) + (long long)(k0 >> 3) * 128;
                const uint4 u = __ldcs((const uint4 *)(P.v16 + cb) + lane);
                const unsigned long long m8 = __ldcs((const unsigned long long *)(P.meta + cb) + lane);
                const unsigned wv[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    if (k0 + j >= len) break;
                    const unsigned mm = (unsigned)(m8 >> (8 * j)) & 0xFFu;
                    if (!chk_in(CHK_TILE, (int)(mm >> 4), nt)) continue;
                    tiles[(mm >> 4) * 256 + lane * 16 + (mm & 15u)] =
                        (unsigned short)((wv[j >> 1] >> (16 * (j & 1))) & 0xFFFFu);
                }
            }
        }
        __syncwarp();
        const int tw = (lane < nt) ? load_tw(P, s, lane) : 0;
        for (int t = 0; t < nt; t++) {
            const int xb = (__shfl_sync(0xffffffffu, tw, t) >> 8) * MF_BS;
            const unsigned *T32 = (const unsigned *)(tiles + t * 256);
            // A (16 x 16, row-major) fragment of m16n8k16
            const unsigned a0 = T32[(g * 16 + 2 * c) >> 1], a1 = T32[((g + 8) * 16 + 2 * c) >> 1];
            const unsigned a2 = T32[(g * 16 + 2 * c + 8) >> 1], a3 = T32[((g + 8) * 16 + 2 * c + 8) >> 1];
            // B (16 x 8) fragment: X rows xb + k, column g, rounded to FP16
            const double *xr = X + (long long)xb * 8 + g;
            const unsigned b0 = pack_half2(xr[(2 * c) * 8], xr[(2 * c + 1) * 8]);
            const unsigned b1 = pack_half2(xr[(2 * c + 8) * 8], xr[(2 * c + 9) * 8]);
            asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
                         "{%8, %9}, {%0, %1, %2, %3};"
                         : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                         : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
        }
        __syncwarp();
    }
    const int r0 = R * MF_BS + g, r1 = r0 + 8;
    if (r0 < P.n) *(double2 *)(Y + (long long)r0 * 8 + 2 * c) = make_double2(d[0], d[1]);
    if (r1 < P.n) *(double2 *)(Y + (long long)r1 * 8 + 2 * c) = make_double2(d[2], d[3]);
}
}  // namespace

// Y = A X for 8 right-hand sides with FP16 stored values (the columns of X
// and Y one after another, n_cols / n_rows each); tensor_cores selects
// k_spmm_tc over k_spmm_cc.  elapsed_ms: the kernel alone.
int mf_spmm_run(mf_matrix_s *A, const double *d_X, double *d_Y, int tensor_cores, cudaStream_t s,
                double *elapsed_ms)
{
    Workspace *w = nullptr;
    MF_TRY(ws_get(A, 0, &w, s));
    const long long L = A->vec_len;
    double *Xi = nullptr, *Yi = nullptr;
    MF_TRY(mf_pool_array(&Xi, L * 8, s));
    int rc = mf_pool_array(&Yi, L * 8, s);
    if (rc == MF_SUCCESS) do {
        if (cudaMemsetAsync(Xi, 0, (size_t)L * 8 * sizeof(double), s) != cudaSuccess) { rc = MF_ERR_CUDA; break; }
        k_interleave<<<592, 256, 0, s>>>(d_X, A->n_cols, (int)L, 8, 0, 8, Xi);
        SolverParams P;
        fill_params(P, A, w);
        if (cudaEventRecord(w->e0, s) != cudaSuccess) { rc = MF_ERR_CUDA; break; }
        if (tensor_cores) {
            if (cudaFuncSetAttribute(k_spmm_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem) != cudaSuccess) {
                rc = MF_ERR_CUDA;
                break;
            }
            k_spmm_tc<<<(A->tilem + kTcWarps - 1) / kTcWarps, kTcWarps * 32, kTcSmem, s>>>(P, Xi, Yi);
        } else {
            k_spmm_cc<<<(A->tilem * 16 + kThreads - 1) / kThreads, kThreads, 0, s>>>(P, Xi, Yi);
        }
        if (cudaGetLastError() != cudaSuccess || cudaEventRecord(w->e1, s) != cudaSuccess) { rc = MF_ERR_CUDA; break; }
        k_deinterleave<<<592, 256, 0, s>>>(Yi, A->n_rows, 8, 0, 8, d_Y);
        if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess) { rc = MF_ERR_CUDA; break; }
        rc = chk_take();
        float ms = 0.f;
        cudaEventElapsedTime(&ms, w->e0, w->e1);
        if (elapsed_ms) *elapsed_ms = ms;
    } while (0);
    mf_pool_free(Xi, s);
    mf_pool_free(Yi, s);
    return rc;
}

// ------------------------------------------------------------ allocation-free SpMV
// Scratch of mf_spmv_noalloc: the padded FP64 copy of x, as a file-scope device
// array (allocated with the module, one per device context), so the call
// itself allocates nothing.
static __device__ __align__(256) double g_noalloc_x[MF_SPMV_NOALLOC_MAX_LEN];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
double *g_noalloc_x_addr[kMaxDevices];

// Device address of the scratch array on the current device, looked up once
// per device (cudaGetSymbolAddress; the first lookup may load the module) and
// kept while the library stays loaded.
int noalloc_scratch(int dev, double **x)
{
    if (dev < 0 || dev >= kMaxDevices) return MF_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_x_addr[dev]) {
        void *px = nullptr;
        MF_CUDA_TRY(cudaGetSymbolAddress(&px, g_noalloc_x));
        g_noalloc_x_addr[dev] = (double *)px;
    }
    *x = g_noalloc_x_addr[dev];
    return MF_SUCCESS;
}
}  // namespace

int mf_spmv_noalloc_run(mf_matrix_s *A, const double *d_x, double *d_y, int precision, cudaStream_t s)
{
    const long long L = A->vec_len;
    if (L > MF_SPMV_NOALLOC_MAX_LEN) return MF_ERR_UNSUPPORTED;
    int dev = 0;
    MF_CUDA_TRY(cudaGetDevice(&dev));
    if (dev != A->dev) return MF_ERR_INVALID;
    double *x = nullptr;
    MF_TRY(noalloc_scratch(dev, &x));
    // the scratch is needed only where x cannot be read in place
    if (!spmv_in_place(A, d_x, d_y)) {
        MF_CUDA_TRY(spmv_copy(A, x, d_x, s));
        d_x = x;
    }
    return spmv_launch(A, d_x, d_y, precision == MF_PREC_FP64 ? MF_P64 : MF_P32, s);
}

