// scan.cu -- device exclusive prefix sums used by the GPU tiler.
// out[0..n] with out[0] = 0 and out[n] = total (the form of the reference's
// exclusive_scan over length n+1, utils.h:34-49).  Two kernels: totals per block
// of 4,096 elements, then every block adds up the totals before its own and scans
// its elements (n = 16.8 M makes 4,096 totals, 8 loads a thread).  The tiler's
// scans are short, so launches count: three levels with an add-back were 4 or 5
// kernels and two allocations each, some 30 of the 75 launches of a build.
#include "mf_internal.cuh"

namespace {

constexpr int kThreads = 512;
constexpr int kItems = 8;
constexpr int kTile = kThreads * kItems;

// what one tile-row adds to the tile, row-block and slice counts
struct Tile3 {
    int tiles, blocks, slices;
};
__device__ __forceinline__ Tile3 operator+(Tile3 x, Tile3 y)
{
    return {x.tiles + y.tiles, x.blocks + y.blocks, x.slices + y.slices};
}

__device__ __forceinline__ int shfl_up(int v, int o) { return __shfl_up_sync(0xffffffffu, v, o); }
__device__ __forceinline__ long long shfl_up(long long v, int o) { return __shfl_up_sync(0xffffffffu, v, o); }
__device__ __forceinline__ Tile3 shfl_up(Tile3 v, int o)
{
    return {shfl_up(v.tiles, o), shfl_up(v.blocks, o), shfl_up(v.slices, o)};
}

template <typename TI, typename TO>
struct PlainScan {
    using Value = TO;
    const TI *in;
    TO *out;
    __device__ Value load(long long i) const { return (TO)in[i]; }
    __device__ void store(long long i, Value v) const { out[i] = v; }
};

// Row-block split of blockspmv_cpu (blockspmv_cpu.h:35-83, PREFETCH_SMEM_TH = 4)
// and slices of up to MF_SEG_TILES tiles, from the tiles of a tile-row.
struct TileScan {
    using Value = Tile3;
    const int *ntiles;
    int *tile_ptr, *rb_ptr, *seg_ptr;
    __device__ Value load(long long i) const
    {
        const int nt = ntiles[i];
        return {nt, nt <= 4 ? 1 : (nt + 3) / 4, (nt + MF_SEG_TILES - 1) / MF_SEG_TILES};
    }
    __device__ void store(long long i, Value v) const
    {
        tile_ptr[i] = v.tiles;
        rb_ptr[i] = v.blocks;
        seg_ptr[i] = v.slices;
    }
};

// Exclusive scan of one value per thread over the block; *total: the block's sum.
template <typename T>
__device__ T block_scan(T mine, T *total)
{
    __shared__ T warp_tot[kThreads / 32], all;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    T incl = mine;
    const T zero = T();
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T t = shfl_up(incl, o);
        if (lane >= o) incl = incl + t;
    }
    if (lane == 31) warp_tot[wid] = incl;
    T before = shfl_up(incl, 1);
    if (lane == 0) before = zero;
    __syncthreads();
    if (wid == 0) {
        T wi = lane < kThreads / 32 ? warp_tot[lane] : zero;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const T t = shfl_up(wi, o);
            if (lane >= o) wi = wi + t;
        }
        T ex = shfl_up(wi, 1);
        if (lane == 0) ex = zero;
        if (lane < kThreads / 32) warp_tot[lane] = ex;
        if (lane == kThreads / 32 - 1) all = wi;
    }
    __syncthreads();
    *total = all;
    const T r = warp_tot[wid] + before;
    __syncthreads();
    return r;
}

template <typename S>
__global__ void k_block_sums(S s, typename S::Value *sums, long long n)
{
    using T = typename S::Value;
    const long long base = (long long)blockIdx.x * kTile + (long long)threadIdx.x * kItems;
    T run = T();
#pragma unroll
    for (int j = 0; j < kItems; j++)
        if (base + j < n) run = run + s.load(base + j);
    T total;
    block_scan(run, &total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

template <typename S>
__global__ void k_scan_out(S s, const typename S::Value *sums, long long n)
{
    using T = typename S::Value;
    T part = T(), offset = T();
    for (int b = threadIdx.x; b < (int)blockIdx.x; b += kThreads) part = part + sums[b];
    if (blockIdx.x > 0) block_scan(part, &offset);
    const long long base = (long long)blockIdx.x * kTile + (long long)threadIdx.x * kItems;
    T v[kItems], run = T(), total;
#pragma unroll
    for (int j = 0; j < kItems; j++) {
        v[j] = run;
        if (base + j < n) run = run + s.load(base + j);
    }
    const T off = offset + block_scan(run, &total);
#pragma unroll
    for (int j = 0; j < kItems; j++)
        if (base + j < n) s.store(base + j, off + v[j]);
    if (blockIdx.x + 1 == gridDim.x && threadIdx.x == 0) s.store(n, offset + total);
}

template <typename S>
int scan_impl(S sc, long long n, cudaStream_t s)
{
    using T = typename S::Value;
    const long long nb = n > 0 ? (n + kTile - 1) / kTile : 1;
    T *sums = nullptr;
    if (nb > 1) {
        const int rc = mf_pool_array(&sums, nb, s);
        if (rc != MF_SUCCESS) return rc;
        k_block_sums<<<(unsigned)nb, kThreads, 0, s>>>(sc, sums, n);
    }
    k_scan_out<<<(unsigned)nb, kThreads, 0, s>>>(sc, sums, n);
    mf_pool_free(sums, s);
    MF_CUDA_TRY(cudaGetLastError());
    return MF_SUCCESS;
}

}  // namespace

int mf_scan_i32_to_i32(const int *d_in, int *d_out, long long n, cudaStream_t s)
{
    return scan_impl(PlainScan<int, int>{d_in, d_out}, n, s);
}
int mf_scan_i32_to_i64(const int *d_in, long long *d_out, long long n, cudaStream_t s)
{
    return scan_impl(PlainScan<int, long long>{d_in, d_out}, n, s);
}
int mf_scan_i64_to_i64(const long long *d_in, long long *d_out, long long n, cudaStream_t s)
{
    return scan_impl(PlainScan<long long, long long>{d_in, d_out}, n, s);
}
int mf_scan_tile_counts(const int *d_ntiles, int *d_tile_ptr, int *d_rb_ptr, int *d_seg_ptr, long long n,
                        cudaStream_t s)
{
    return scan_impl(TileScan{d_ntiles, d_tile_ptr, d_rb_ptr, d_seg_ptr}, n, s);
}
