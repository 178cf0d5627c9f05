// adjoint.cu -- what the backward pass of a differentiable solve needs beyond
// the solver itself:
//  * mf_value_grad: dL/dA on A's stored pattern, grad[e] = -sum_k lambda_k[i] x_k[j]
//    for every stored entry e = (i, j), in the caller's CSR entry order
//    (A x = b  =>  dL/dA = -lambda x^T with lambda = A^-T dL/dx);
//  * mf_matrix_create_transposed: a handle for A^T (the adjoint system of a
//    nonsymmetric A), built from A's own CSR copy.
// No counterpart in the reference, which has no differentiation.
#include "mf_internal.cuh"

#include <type_traits>
#include <vector>

namespace {

// One warp per row; lanes stride over the row's entries, the right-hand sides
// are summed in order (deterministic).  grad is indexed from the first stored
// entry of row 0 (rowptr[0]), like the handle's nnz.
__global__ void k_value_grad(const int *__restrict__ rowptr, const int *__restrict__ colidx, int n_rows, int n_cols,
                             int nrhs, const double *__restrict__ lambda, const double *__restrict__ x,
                             double *__restrict__ grad)
{
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const int base = rowptr[0];
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n_rows; i += nw) {
        const int a = rowptr[i], b = rowptr[i + 1];
        for (int e = a + lane; e < b; e += 32) {
            const int j = colidx[e];
            double g = 0.0;
            for (int k = 0; k < nrhs; k++)
                g += lambda[(long long)k * n_rows + i] * x[(long long)k * n_cols + j];
            grad[e - base] = -g;
        }
    }
}

}  // namespace

extern "C" int mf_value_grad(mf_matrix A, int nrhs, const double *lambda, const double *x, double *grad_val,
                             int device_ptrs, void *stream)
{
    if (!A || !lambda || !x || !grad_val || nrhs < 1) return MF_ERR_INVALID;
    CallMark mark(A);
    cudaStream_t s = (cudaStream_t)stream;
    const size_t nl = (size_t)nrhs * A->n_rows, nx = (size_t)nrhs * A->n_cols, ne = (size_t)A->nnz;
    const double *dl = lambda, *dx = x;
    double *dg = grad_val, *tmp = nullptr;
    if (!device_ptrs) {
        const int rc = mf_pool_array(&tmp, (long long)(nl + nx + ne), s);
        if (rc != MF_SUCCESS) return rc;
        MF_CUDA_TRY(cudaMemcpyAsync(tmp, lambda, nl * sizeof(double), cudaMemcpyHostToDevice, s));
        MF_CUDA_TRY(cudaMemcpyAsync(tmp + nl, x, nx * sizeof(double), cudaMemcpyHostToDevice, s));
        dl = tmp;
        dx = tmp + nl;
        dg = tmp + nl + nx;
    }
    if (A->n_rows > 0 && ne > 0) {
        const int threads = 256;
        int blocks = (int)((A->n_rows + 7) / 8);
        if (blocks > 148 * 16) blocks = 148 * 16;
        k_value_grad<<<blocks, threads, 0, s>>>(A->d_rowptr, A->d_colidx, A->n_rows, A->n_cols, nrhs, dl, dx, dg);
        MF_CUDA_TRY(cudaGetLastError());
    }
    if (!device_ptrs) {
        MF_CUDA_TRY(cudaMemcpyAsync(grad_val, dg, ne * sizeof(double), cudaMemcpyDeviceToHost, s));
        mf_pool_free(tmp, s);
    }
    MF_CUDA_TRY(cudaStreamSynchronize(s));
    return mark.end(MF_SUCCESS);
}

// ------------------------------------------------------------ A^T on the GPU
// The entries of A (their positions in A's row-major order) are sorted by
// column with a stable least-significant-digit radix sort, so a row of A^T keeps
// the order of A's rows and the result does not depend on scheduling.  Columns
// take ceil(log2(n_cols) / 8) passes of 8 bits; a pass is a digit histogram per
// block, an exclusive scan over (digit, block), and a scatter in which each warp
// ranks its entries 32 at a time with __match_any_sync.  The passes move 8 bytes
// an entry each way (column, position) and are bound by the scattered stores;
// values are moved once, at the end.  A sort rather than counting columns with
// atomics and sorting each: its time does not depend on the longest column.
// 48^3 upwind system (760 K entries): 16 ms for the host's counting sort and its
// copies before, 0.2 ms for the passes now.
namespace {

constexpr int kTThreads = 256;
constexpr int kTWarps = kTThreads / 32;
constexpr int kTRounds = 16;                         // 32-entry rounds per warp
constexpr int kTTile = kTThreads * kTRounds;         // entries per block: each warp takes a contiguous run
constexpr int kDigits = 256;

// A handle has up to 2^31 - 1 entries, so counts and midpoints near that stay in range.
__host__ __device__ constexpr int sort_blocks(int n) { return (int)(((long long)n + kTTile - 1) / kTTile); }
__host__ __device__ constexpr int midpoint(int lo, int hi) { return lo + ((hi - lo) >> 1); }
static_assert(sort_blocks(2147483647) == 524288 && sort_blocks(0) == 0 && sort_blocks(kTTile + 1) == 2, "");
static_assert(midpoint(2147483640, 2147483646) == 2147483643 && midpoint(0, 1) == 0, "");

// rowptr -> the row of every entry (entries counted from row 0's first)
__global__ void k_entry_rows(const int *__restrict__ rowptr, int n_rows, int *__restrict__ row)
{
    const int lane = threadIdx.x & 7;                // 8 lanes per row
    const int base = rowptr[0];
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 3; i < n_rows; i += (gridDim.x * blockDim.x) >> 3)
        for (long long e = rowptr[i] + lane; e < rowptr[i + 1]; e += 8) row[e - base] = i;
}

__global__ void k_digit_hist(const int *__restrict__ key, int n, int shift, int nblocks, int *__restrict__ hist)
{
    __shared__ int h[kDigits];
    h[threadIdx.x] = 0;
    __syncthreads();
    const long long b0 = (long long)blockIdx.x * kTTile, b1 = b0 + kTTile < n ? b0 + kTTile : n;
    for (long long e = b0 + threadIdx.x; e < b1; e += kTThreads)
        atomicAdd(&h[(key[e] >> shift) & (kDigits - 1)], 1);
    __syncthreads();
    hist[threadIdx.x * nblocks + blockIdx.x] = h[threadIdx.x];
}

// pos_in == nullptr: the first pass (entry e is at position e)
__global__ void k_digit_scatter(const int *__restrict__ key, const int *__restrict__ pos_in, int n, int shift,
                                int nblocks, const int *__restrict__ start, int *__restrict__ key_out,
                                int *__restrict__ pos_out)
{
    __shared__ int cnt[kTWarps][kDigits];            // next output position of each digit, per warp
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int d = lane; d < kDigits; d += 32) cnt[w][d] = 0;
    __syncwarp();
    const long long w0 = (long long)blockIdx.x * kTTile + w * 32 * kTRounds;
    for (int r = 0; r < kTRounds; r++) {
        const long long e = w0 + r * 32 + lane;
        if (e < n) atomicAdd(&cnt[w][(key[e] >> shift) & (kDigits - 1)], 1);
    }
    __syncthreads();
    {
        int at = start[threadIdx.x * nblocks + blockIdx.x];
        for (int v = 0; v < kTWarps; v++) {
            const int c = cnt[v][threadIdx.x];
            cnt[v][threadIdx.x] = at;
            at += c;
        }
    }
    __syncthreads();
    for (int r = 0; r < kTRounds; r++) {
        const long long e = w0 + r * 32 + lane;
        const bool act = e < n;
        const int k = act ? key[e] : 0;
        const int d = act ? (k >> shift) & (kDigits - 1) : kDigits;
        const unsigned same = __match_any_sync(0xffffffffu, d);
        const int rank = __popc(same & ((1u << lane) - 1u));
        const int at = act ? cnt[w][d] : 0;
        __syncwarp();
        if (act && rank == 0) cnt[w][d] = at + __popc(same);
        __syncwarp();
        if (act) {
            key_out[at + rank] = k;
            pos_out[at + rank] = pos_in ? pos_in[e] : (int)e;
        }
    }
}

// row pointers of A^T from the sorted columns: row j starts at the first entry of column >= j
__global__ void k_sorted_rowptr(const int *__restrict__ key, int n, int n_cols, int *__restrict__ tp)
{
    for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j <= n_cols;
         j += (long long)gridDim.x * blockDim.x) {
        int lo = 0, hi = n;
        while (lo < hi) {
            const int mid = midpoint(lo, hi);
            if (key[mid] < j) lo = mid + 1;
            else hi = mid;
        }
        tp[j] = lo;
    }
}

__global__ void k_gather_entries(const int *__restrict__ pos, int n, const int *__restrict__ row,
                                 const double *__restrict__ val, const float *__restrict__ low,
                                 int *__restrict__ tc, double *__restrict__ tv, float *__restrict__ tl)
{
    for (long long e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
        const int p = pos[e];
        tc[e] = row[p];
        tv[e] = val[p];
        if (tl) tl[e] = low[p];
    }
}

// Pool arrays freed in stream order: by name once they are done with, the rest at the end.
struct PoolTemps {
    cudaStream_t s;
    std::vector<void *> all;
    template <typename T>
    int get(T **p, long long count)
    {
        const int rc = mf_pool_array(p, count, s);
        if (rc == MF_SUCCESS) all.push_back(*p);
        return rc;
    }
    void free_all()
    {
        for (void *p : all) mf_pool_free(p, s);
        all.clear();
    }
    ~PoolTemps() { free_all(); }
};

}  // namespace

// A handle for A^T, built from A's device CSR copy without leaving the GPU, on the
// current device as mf_matrix_create does.  Its CSR arrays become the new handle's
// and the sort's temporaries are freed before the tile build, so the call needs no
// more device memory than the handle: at most 36 bytes an entry at a time here,
// where the build goes past 46.
extern "C" int mf_matrix_create_transposed(mf_matrix *out, mf_matrix A, void *stream)
{
    if (!out || !A) return MF_ERR_INVALID;
    *out = nullptr;
    CallMark mark(A);
    cudaStream_t s = (cudaStream_t)stream;
    const int m = A->n_rows, n = A->n_cols, nnz = (int)A->nnz;
    int base = 0;                   // entries of rows [0, m) start here
    MF_CUDA_TRY(cudaMemcpyAsync(&base, A->d_rowptr, sizeof(int), cudaMemcpyDeviceToHost, s));
    MF_CUDA_TRY(cudaStreamSynchronize(s));
    PoolTemps tmp{s, {}}, csr{s, {}};
    const int *rowptr = A->d_rowptr, *colidx = A->d_colidx + base;
    const double *val = A->d_val + base;
    const float *low = A->d_val_low ? A->d_val_low + base : nullptr;
    int rc = MF_SUCCESS, dev = 0;
    MF_CUDA_TRY(cudaGetDevice(&dev));
    if (dev != A->dev) {            // kernels do not read another device's memory
        auto fetch = [&](auto **p, long long count) -> int {
            using T = std::remove_const_t<std::remove_reference_t<decltype(**p)>>;
            T *here = nullptr;
            const int e = tmp.get(&here, count);
            if (e != MF_SUCCESS) return e;
            MF_CUDA_TRY(cudaMemcpyAsync(here, *p, (size_t)count * sizeof(T), cudaMemcpyDeviceToDevice, s));
            *p = here;
            return MF_SUCCESS;
        };
        if ((rc = fetch(&rowptr, (long long)m + 1)) || (rc = fetch(&colidx, nnz)) || (rc = fetch(&val, nnz)) ||
            (low && (rc = fetch(&low, nnz))))
            return rc;
    }
    const int nblocks = sort_blocks(nnz);
    int *row, *key[2], *pos[2], *hist, *start, *tp, *tc;
    double *tv;
    float *tl = nullptr;
    if ((rc = csr.get(&tp, (long long)n + 1)) || (rc = csr.get(&tc, nnz)) || (rc = csr.get(&tv, nnz)) ||
        (low && (rc = csr.get(&tl, nnz))) || (rc = tmp.get(&row, nnz)) || (rc = tmp.get(&key[0], nnz)) ||
        (rc = tmp.get(&key[1], nnz)) || (rc = tmp.get(&pos[0], nnz)) || (rc = tmp.get(&pos[1], nnz)) ||
        (rc = tmp.get(&hist, (long long)kDigits * nblocks)) || (rc = tmp.get(&start, (long long)kDigits * nblocks + 1)))
        return rc;
    if (nnz > 0) {
        k_entry_rows<<<148 * 8, 256, 0, s>>>(rowptr, m, row);
        MF_CUDA_TRY(cudaGetLastError());
        const int *kin = colidx, *pin = nullptr;
        int at = 0;
        for (int shift = 0; shift == 0 || (shift < 31 && ((n - 1) >> shift) > 0); shift += 8, at ^= 1) {
            k_digit_hist<<<nblocks, kTThreads, 0, s>>>(kin, nnz, shift, nblocks, hist);
            MF_CUDA_TRY(cudaGetLastError());
            rc = mf_scan_i32_to_i32(hist, start, (long long)kDigits * nblocks, s);
            if (rc != MF_SUCCESS) return rc;
            k_digit_scatter<<<nblocks, kTThreads, 0, s>>>(kin, pin, nnz, shift, nblocks, start, key[at], pos[at]);
            MF_CUDA_TRY(cudaGetLastError());
            kin = key[at];
            pin = pos[at];
        }
        k_sorted_rowptr<<<(unsigned)(((long long)n + 256) / 256), 256, 0, s>>>(kin, nnz, n, tp);
        MF_CUDA_TRY(cudaGetLastError());
        k_gather_entries<<<148 * 8, 256, 0, s>>>(pin, nnz, row, val, low, tc, tv, tl);
        MF_CUDA_TRY(cudaGetLastError());
    } else {
        MF_CUDA_TRY(cudaMemsetAsync(tp, 0, ((size_t)n + 1) * sizeof(int), s));
    }
    tmp.free_all();
    csr.all.clear();                // the handle's from here on, also when the build fails
    return mark.end(mf_matrix_adopt(out, n, m, nnz, tp, tc, tv, tl, s));
}
