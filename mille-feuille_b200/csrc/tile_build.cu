// tile_build.cu -- GPU csr2block, precision encoder and solver-slice builder.
//
// Produces, on the device, the reference tile layout bit-exact to Tile_create
// (csr2block.h:267-422), the offsets of blockspmv_cpu (blockspmv_cpu.h:35-111),
// the nonempty-row lists of cg_solve_inc (main-cg-mixed.cu:2447-2514), the
// encoder arrays (main-cg-mixed.cu:2333-2350) and this library's solver slices.
//
// One warp per tile-row.  The distinct column tiles of a tile-row are found
// with a bitmap over the tile-row's column-tile span (in shared memory, or in
// a global scratch slice when the span is too wide), ranked with popcounts,
// so the tile order is ascending as in convert_step2 (csr2block.h:89-102).
// Entries are then ranked inside their tile in CSR order with __match_any_sync
// (the order convert_step4 appends them in, csr2block.h:204-219).
//
// The host waits four times: for the tile-rows' spans (which also check the row
// pointers), for the tile counts, for the sizes that depend on the filled tiles,
// and at the end.  With ten waits, a copy per number and up to five kernels a
// scan, a 65,280-row build took 0.44 ms for 0.15 ms of kernels.
#include "mf_internal.cuh"

#include <algorithm>
#include <chrono>
#include <vector>

namespace {

constexpr int kWarps = 8;           // warps per block in the per-tile-row kernels
constexpr int kThreads = kWarps * 32;

__device__ __forceinline__ int tile_row_end(int R, int tilem, int rowA)
{
    return (R == tilem - 1) ? rowA : (R + 1) * MF_BS;
}

// ---- K0: column-tile span per tile-row, and the maxima the host needs ----
// Also the check of the row pointers (in [0, nnz], not decreasing) and of the
// columns: a tile-row's entries are read only when its row pointers are in order.
__global__ void k_span(const int *__restrict__ rowptr, const int *__restrict__ colidx, int tilem, int rowA,
                       int colA, long long nnz, int2 *__restrict__ spans, int *__restrict__ max_words,
                       int *__restrict__ err)
{
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int R = warp; R < tilem; R += nwarps) {
        const int rows = tile_row_end(R, tilem, rowA) - R * MF_BS;
        const int rp = lane <= rows ? rowptr[R * MF_BS + lane] : 0;
        const int next = __shfl_down_sync(0xffffffffu, rp, 1);
        bool bad = lane < rows && (rp < 0 || next < rp || (long long)next > nnz);
        int jmin = INT_MAX, jmax = -1;
        if (!__any_sync(0xffffffffu, bad)) {
            const int a = __shfl_sync(0xffffffffu, rp, 0), b = __shfl_sync(0xffffffffu, rp, rows);
            for (int j = a + lane; j < b; j += 32) {
                int c = colidx[j];
                if (c < 0 || c >= colA) { bad = true; continue; }
                int jc = c >> 4;
                jmin = min(jmin, jc);
                jmax = max(jmax, jc);
            }
        }
        jmin = __reduce_min_sync(0xffffffffu, jmin);
        jmax = __reduce_max_sync(0xffffffffu, jmax);
        bad = __any_sync(0xffffffffu, bad);
        if (lane == 0) {
            if (bad) atomicExch(err, MF_ERR_INVALID);
            const int words = (jmax < 0) ? 0 : (jmax >> 5) - (jmin >> 5) + 1;
            spans[R] = make_int2((jmax < 0) ? 0 : (jmin >> 5), words);     // first word, words
            if (words > *(volatile int *)max_words) atomicMax(max_words, words);
        }
    }
}

// ---- scratch of the per-tile-row kernels ----
// k_count_tiles needs a bitmap over the tile-row's span, k_fill_tiles what
// fill_words says.  One tile-row that touches every column tile (an arrow matrix,
// a circuit's supply net) needs 17 words per tile: sized for it, the 4,736 warps
// of a launch took 20 GB at 1 M columns.  So tile-rows are sorted by what they
// need into three passes: up to kSharedWords in shared memory (the launch covers
// all tile-rows and leaves out the others), up to kMidWords in global memory with
// the full grid, and the rest with as many warps as kScratchBytes gives.
constexpr int kSharedWords = 96 * 1024 / 4 / kWarps;
constexpr int kGlobalGrid = 148 * 4;
constexpr long long kScratchBytes = 256ll << 20;
constexpr int kMidWords = (int)(kScratchBytes / 4 / kWarps / kGlobalGrid);

// bitmap, prefix (a word per span word each), next position per tile, entries per (tile, row)
__host__ __device__ constexpr int fill_words(int span, int tiles) { return 2 * span + (1 + MF_BS) * tiles; }

// What k_count_tiles finds out about the passes; rows: the mid ones from the front, the large ones from the back.
struct Passes {
    int shared_words, mid_words, large_words, n_mid, n_large;
};

// A warp's scratch, in shared memory or in global memory.
__device__ __forceinline__ unsigned int *warp_scratch(unsigned int *smem, unsigned int *gscratch, int words_per_warp,
                                                      int global_mode)
{
    const int wib = threadIdx.x >> 5;
    const long long gw = (long long)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    return global_mode ? gscratch + gw * (long long)words_per_warp : smem + (long long)wib * words_per_warp;
}

// Build the tile-row bitmap; returns the number of distinct tiles.
__device__ int build_bitmap(unsigned int *bm, const int *__restrict__ colidx, int a, int b, int base_word,
                            int words, int lane)
{
    for (int w = lane; w < words; w += 32) bm[w] = 0u;
    __syncwarp();
    for (int j = a + lane; j < b; j += 32) {
        int jc = colidx[j] >> 4;
        atomicOr(&bm[(jc >> 5) - base_word], 1u << (jc & 31));
    }
    __syncwarp();
    int cnt = 0;
    for (int w = lane; w < words; w += 32) cnt += __popc(bm[w]);
    for (int o = 16; o; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    return cnt;
}

// ---- K1: distinct tiles per tile-row, and the pass that fills it ----
__global__ void k_count_tiles(const int *__restrict__ rowptr, const int *__restrict__ colidx, int tilem, int rowA,
                              const int2 *__restrict__ spans, int words_per_warp, int global_mode,
                              unsigned int *gscratch, int *__restrict__ ntiles, int *__restrict__ rows,
                              Passes *__restrict__ passes)
{
    extern __shared__ unsigned int smem[];
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    unsigned int *bm = warp_scratch(smem, gscratch, words_per_warp, global_mode);
    for (int R = warp; R < tilem; R += nwarps) {
        const int a = rowptr[R * MF_BS], b = rowptr[tile_row_end(R, tilem, rowA)];
        const int2 sp = spans[R];
        const int c = (sp.y > 0) ? build_bitmap(bm, colidx, a, b, sp.x, sp.y, lane) : 0;
        if (lane == 0) {
            ntiles[R] = c;
            const int need = fill_words(sp.y, c);
            if (need <= kSharedWords) {
                if (need > *(volatile int *)&passes->shared_words) atomicMax(&passes->shared_words, need);
            } else if (need <= kMidWords) {
                rows[atomicAdd(&passes->n_mid, 1)] = R;
                atomicMax(&passes->mid_words, need);
            } else {
                rows[tilem - 1 - atomicAdd(&passes->n_large, 1)] = R;
                atomicMax(&passes->large_words, need);
            }
        }
        __syncwarp();
    }
}

// ---- K2: tile columns, payload offsets, scatter, uint8 row starts ----
// `rows` lists the `nrows` tile-rows of a launch; without it the launch takes all
// whose scratch fits words_per_warp.  Entries are taken 32 at a time across
// the rows of the tile-row (CSR order is row by row already): 7-point tile-rows
// are 4 steps a pass, where going row by row made 16 with two warp barriers each
// (128^3: 0.84 ms of 2 ms of kernels).  The row starts come from the (tile, row)
// counts.
__global__ void k_fill_tiles(const int *__restrict__ rowptr, const int *__restrict__ colidx,
                             const double *__restrict__ val, const float *__restrict__ val_low, int tilem,
                             int rowA, const int2 *__restrict__ spans, const int *__restrict__ rows, int nrows,
                             int words_per_warp, int global_mode, unsigned int *gscratch, const int *__restrict__ tile_ptr,
                             int *__restrict__ tile_columnidx, int *__restrict__ csr_offset,
                             int *__restrict__ csrptr_offset, double *__restrict__ tval,
                             float *__restrict__ tval_low, unsigned char *__restrict__ tcol,
                             unsigned char *__restrict__ tptr, int *__restrict__ err)
{
    extern __shared__ unsigned int smem[];
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const unsigned lt_mask = (1u << lane) - 1u;
    unsigned int *bm = warp_scratch(smem, gscratch, words_per_warp, global_mode);
    const int nz0 = rowptr[0];
    for (int q = warp; q < nrows; q += nwarps) {
        const int R = rows ? rows[q] : q;
        const int rs = R * MF_BS, re = tile_row_end(R, tilem, rowA);
        const int rowlen = re - rs;
        const int rp = lane <= rowlen ? rowptr[rs + lane] : INT_MAX;
        const int a = __shfl_sync(0xffffffffu, rp, 0), b = __shfl_sync(0xffffffffu, rp, rowlen);
        const int t0 = tile_ptr[R], nt = tile_ptr[R + 1] - t0;
        const int base_word = spans[R].x, words = spans[R].y;
        if (fill_words(words, nt) > words_per_warp) continue;      // another pass fills it
        int *pre = (int *)bm + words, *next = pre + words, *hist = next + nt;
        // csrptr_offset: exclusive scan of tile-row heights over tiles (csr2block.h:146,347)
        for (int s = lane; s < nt; s += 32) csrptr_offset[t0 + s] = t0 * MF_BS + s * rowlen;
        if (R == tilem - 1 && lane == 0) csrptr_offset[t0 + nt] = t0 * MF_BS + nt * rowlen;
        if (nt == 0) {
            if (R == tilem - 1 && lane == 0) csr_offset[t0] = b - nz0;
            continue;
        }
        for (int h = lane; h < nt * MF_BS; h += 32) hist[h] = 0;
        build_bitmap(bm, colidx, a, b, base_word, words, lane);
        // exclusive popcount prefix over the bitmap words
        int carry = 0;
        for (int w0 = 0; w0 < words; w0 += 32) {
            int w = w0 + lane;
            int c = (w < words) ? __popc(bm[w]) : 0;
            int incl = c;
            for (int o = 1; o < 32; o <<= 1) {
                int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            if (w < words) pre[w] = carry + incl - c;
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        __syncwarp();
        // tile_columnidx, ascending
        for (int w = lane; w < words; w += 32) {
            unsigned int m = bm[w];
            int r = pre[w];
            while (m) {
                int bit = __ffs(m) - 1;
                m &= m - 1u;
                tile_columnidx[t0 + r] = (base_word + w) * 32 + bit;
                r++;
            }
        }
        auto slot_of = [&](int c) -> int {
            const int jc = c >> 4, w = (jc >> 5) - base_word;
            return pre[w] + __popc(bm[w] & ((1u << (jc & 31)) - 1u));
        };
        // pass 1: entries per tile and row
        for (int j0 = a; j0 < b; j0 += 32) {
            const int j = j0 + lane;
            int ri = 0;
            for (int q = 1; q < rowlen; q++) ri += (j >= __shfl_sync(0xffffffffu, rp, q)) ? 1 : 0;
            if (j < b) atomicAdd(&hist[slot_of(colidx[j]) * MF_BS + ri], 1);
        }
        __syncwarp();
        // row starts and payload offsets: tile-row payload starts at rowptr[rs] (csr_offset scan)
        int run = a - nz0;
        for (int s0 = 0; s0 < nt; s0 += 32) {
            const int s = s0 + lane;
            int c = 0;
            if (s < nt)
                for (int ri = 0; ri < rowlen; ri++) {
                    if (c > 255) atomicExch(err, MF_ERR_UNSUPPORTED);
                    // csrptr_offset[t0 + s] = t0 * 16 + s * rowlen (only the last tile-row is short)
                    tptr[(long long)t0 * MF_BS + (long long)s * rowlen + ri] = (unsigned char)c;
                    c += hist[s * MF_BS + ri];
                }
            int incl = c;
            for (int o = 1; o < 32; o <<= 1) {
                int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            if (s < nt) {
                csr_offset[t0 + s] = run + incl - c;
                next[s] = run + incl - c;
                if (c > 256) atomicExch(err, MF_ERR_UNSUPPORTED);   // duplicate columns overflow a tile
            }
            run += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (R == tilem - 1 && lane == 0) csr_offset[t0 + nt] = run;
        __syncwarp();
        // pass 2: the payload, in CSR order within a tile
        for (int j0 = a; j0 < b; j0 += 32) {
            const int j = j0 + lane;
            const bool act = j < b;
            int slot = -1, c = 0;
            if (act) {
                c = colidx[j];
                slot = slot_of(c);
            }
            const unsigned grp = __match_any_sync(0xffffffffu, slot);
            const int rank = __popc(grp & lt_mask);
            const int o = act ? next[slot] + rank : 0;
            __syncwarp();
            if (act && rank == 0) next[slot] += __popc(grp);
            __syncwarp();
            if (act) {
                const double v = val[j];
                tval[o] = v;
                tval_low[o] = val_low ? val_low[j] : (float)v;
                tcol[o] = (unsigned char)(c & 15);
            }
        }
        __syncwarp();
    }
}

// ---- rowlists: nonempty rows per tile (main-cg-mixed.cu:2455-2514) ----
__device__ __forceinline__ int tile_row_stop(const unsigned char *ptr, int cc, int ri, int rowlen, int nnzt)
{
    return (ri == rowlen - 1) ? nnzt : (int)ptr[cc + ri + 1];
}

// Row start as the reference stores it.  exclusive_scan_char returns early for
// length 1 (utils.h:52-53), so a one-row tile-row keeps its row count as the
// "start" (csr2block.h:237,252).  The device ptr array holds the true start 0;
// the reference value is restated here and in the exported copy.
__device__ __forceinline__ int ref_row_start(const unsigned char *ptr, int cc, int ri, int rowlen, int nnzt)
{
    return (rowlen == 1) ? (int)(unsigned char)nnzt : (int)ptr[cc + ri];
}

__global__ void k_rowlist_count(const int *__restrict__ tile_ptr, const int *__restrict__ csr_offset,
                                const int *__restrict__ csrptr_offset, const unsigned char *__restrict__ tptr,
                                int tilem, int rowA, int *__restrict__ nzr, int *__restrict__ tile_rowidx,
                                int *__restrict__ block_signal)
{
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int R = warp; R < tilem; R += nwarps) {
        const int rowlen = (R == tilem - 1) ? rowA - R * MF_BS : MF_BS;
        const int t0 = tile_ptr[R], t1 = tile_ptr[R + 1];
        if (lane == 0) block_signal[R] = t1 - t0;
        for (int t = t0 + lane; t < t1; t += 32) {
            tile_rowidx[t] = R;
            const int cc = csrptr_offset[t];
            const int nnzt = csr_offset[t + 1] - csr_offset[t];
            int cnt = 0;
            for (int ri = 0; ri < rowlen; ri++)
                if (tile_row_stop(tptr, cc, ri, rowlen, nnzt) != ref_row_start(tptr, cc, ri, rowlen, nnzt)) cnt++;
            nzr[t] = cnt + 1;
        }
    }
}

__global__ void k_rowlist_fill(const int *__restrict__ tile_ptr, const int *__restrict__ csr_offset,
                               const int *__restrict__ csrptr_offset, const unsigned char *__restrict__ tptr,
                               int tilem, int rowA, const int *__restrict__ nzr_scan,
                               unsigned char *__restrict__ rowid, unsigned char *__restrict__ cptr)
{
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int R = warp; R < tilem; R += nwarps) {
        const int rowlen = (R == tilem - 1) ? rowA - R * MF_BS : MF_BS;
        for (int t = tile_ptr[R] + lane; t < tile_ptr[R + 1]; t += 32) {
            const int cc = csrptr_offset[t];
            const int nnzt = csr_offset[t + 1] - csr_offset[t];
            int base = nzr_scan[t], fl = 0;
            for (int ri = 0; ri < rowlen; ri++) {
                int stop = tile_row_stop(tptr, cc, ri, rowlen, nnzt);
                if (ri == 0) { rowid[base + fl] = 0; cptr[base + fl] = 0; fl++; }
                if (stop != ref_row_start(tptr, cc, ri, rowlen, nnzt)) {
                    rowid[base + fl] = (unsigned char)ri;
                    cptr[base + fl] = (unsigned char)stop;
                    fl++;
                }
            }
        }
    }
}

// ---- row-block split of blockspmv_cpu (blockspmv_cpu.h:35-83), PREFETCH_SMEM_TH = 4 ----
__global__ void k_rowblk_fill(const int *__restrict__ tile_ptr, int tilem, const int *__restrict__ off,
                              unsigned int *__restrict__ idx, int *__restrict__ cs, int *__restrict__ ce)
{
    int R = blockIdx.x * blockDim.x + threadIdx.x;
    if (R >= tilem) return;
    int nb = tile_ptr[R + 1] - tile_ptr[R];
    int o = off[R];
    if (nb <= 4) {
        idx[o] = (unsigned)R; cs[o] = 0; ce[o] = 0;
        return;
    }
    int num = (nb + 3) / 4;
    int len = (nb + num - 1) / num;
    for (int i = 0; i < num; i++) {
        idx[o + i] = (unsigned)R | 0x80000000u;
        cs[o + i] = tile_ptr[R] + i * len;
        ce[o + i] = (i == num - 1) ? tile_ptr[R] + nb : tile_ptr[R] + (i + 1) * len;
    }
}

// ---- encoder (main-cg-mixed.cu:2341-2346) and per-tile scaled int8 / caps ----
__device__ __forceinline__ int8_t host_trunc_i8(double v)
{
    // (int8_t)double as emitted by the x86-64 host compiler: truncate to int32
    // (0x80000000 when NaN / out of range), keep the low byte.
    int w;
    if (!(v == v) || v >= 2147483648.0 || v < -2147483648.0) w = (int)0x80000000u;
    else w = (int)v;
    return (int8_t)(unsigned char)(w & 0xFF);
}

__global__ void k_encode_ref(const double *__restrict__ tval, const float *__restrict__ tval_low, long long nnz,
                             uint16_t *__restrict__ f16, int8_t *__restrict__ i8ref)
{
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < nnz; k += (long long)gridDim.x * blockDim.x) {
        f16[k] = __half_as_ushort(__float2half_rn(tval_low[k]));
        i8ref[k] = host_trunc_i8(tval[k]);
    }
}

__global__ void k_encode_tiles(const int *__restrict__ csr_offset, int tilenum, const double *__restrict__ tval,
                               int8_t *__restrict__ q, float *__restrict__ scale, unsigned char *__restrict__ caps)
{
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < tilenum; t += gridDim.x * blockDim.x) {
        const int o = csr_offset[t], e = csr_offset[t + 1];
        double mx = 0.0, mn = INFINITY;
        bool ex32 = true, ex16 = true;
        for (int k = o; k < e; k++) {
            double a = tval[k], aa = fabs(a);
            mx = fmax(mx, aa);
            if (aa > 0.0) mn = fmin(mn, aa);
            float f = (float)a;
            if ((double)f != a) ex32 = false;
            if ((double)__half2float(__float2half_rn(f)) != a) ex16 = false;
        }
        float s = (float)(mx / 127.0);
        bool ex8 = true;
        for (int k = o; k < e; k++) {
            double a = tval[k];
            int8_t v = 0;
            if (s != 0.0f) {
                double r = rint(a / (double)s);
                r = fmin(127.0, fmax(-127.0, r));
                v = (int8_t)r;
            }
            q[k] = v;
            if ((double)((float)v * s) != a) ex8 = false;
        }
        scale[t] = s;
        unsigned char c = 0;
        if (mx <= 65504.0 && (mn == INFINITY || mn >= 6.103515625e-05)) c |= MF_CAP_FP16_OK;
        if (ex8) c |= MF_CAP_EXACT_I8;
        if (ex16) c |= MF_CAP_EXACT_F16;
        if (ex32) c |= MF_CAP_EXACT_F32;
        caps[t] = c;
    }
}

// ---- solver slices ----
// lane-per-row statistics of every segment: row lengths and padded width
__global__ void k_seg_shape(const int *__restrict__ tile_ptr, const int *__restrict__ seg_ptr,
                            const int *__restrict__ csr_offset, const int *__restrict__ csrptr_offset,
                            const unsigned char *__restrict__ tptr, int tilem, int rowA,
                            int *__restrict__ seg_tile0, int *__restrict__ seg_kp,
                            uint16_t *__restrict__ seg_rowlen, int *__restrict__ seg_entries,
                            long long *__restrict__ row_cost, int *__restrict__ shape)
{
    int longest = 0;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const int i = lane & 15;
    for (int R = warp; R < tilem; R += nwarps) {
        const int rowlen = (R == tilem - 1) ? rowA - R * MF_BS : MF_BS;
        const int t0 = tile_ptr[R], t1 = tile_ptr[R + 1];
        long long cost = 4;
        for (int s = seg_ptr[R]; s < seg_ptr[R + 1]; s++) {
            const int ta = t0 + (s - seg_ptr[R]) * MF_SEG_TILES;
            const int tb = min(t1, ta + MF_SEG_TILES);
            int len = 0;
            if (i < rowlen) {
                for (int t = ta; t < tb; t++) {
                    int cc = csrptr_offset[t], nnzt = csr_offset[t + 1] - csr_offset[t];
                    int st = tptr[cc + i];
                    int sp = (i == rowlen - 1) ? nnzt : (int)tptr[cc + i + 1];
                    len += sp - st;
                }
            }
            int K = len;
            for (int o = 8; o; o >>= 1) K = max(K, __shfl_xor_sync(0xffffffffu, K, o));
            int kp = ((K + 7) / 8) * 8;
            if (kp == 0) kp = 8;
            if (lane < 16) seg_rowlen[(long long)s * MF_BS + i] = (uint16_t)len;
            if (lane == 0) {
                seg_tile0[s] = ta;
                seg_kp[s] = kp;
                seg_entries[s] = kp * MF_BS;
            }
            cost += kp + 6;
            longest = max(longest, K);
        }
        if (lane == 0) row_cost[R] = cost;
        // not one slice of one chunk (kp + 6 = 14 past the base cost of 4)
        if (lane == 0 && cost != 18) shape[1] = 1;
    }
    // shape[0]: the longest row; shape[1]: some tile-row is not one chunk
    if (lane == 0 && longest > 0) atomicMax(&shape[0], longest);
}

// The slices' payload, a half-warp per slice: lane i collects row i's next 8 entries
// (tile by tile) and stores them as the 16-byte groups the solver loads (mf_slot),
// with zeros past the row's end.  One entry at a time, with a warp per tile-row whose
// halves took alternate slices (one of them idle on one-slice tile-rows), made 1- to
// 8-byte stores of six arrays: 91 us for 7.1 M padded entries, 59 us now for 120 MB
// written and 92 MB read.  By slice and not by tile-row: a tile-row of many slices
// would be one half-warp's serial work.
__global__ void k_seg_fill(const int4 *__restrict__ seg_hdr, const int *__restrict__ csr_offset,
                           const int *__restrict__ csrptr_offset, const unsigned char *__restrict__ tptr,
                           const unsigned char *__restrict__ tcol, const double *__restrict__ tval,
                           const float *__restrict__ tval_low, const int8_t *__restrict__ q8,
                           const int8_t *__restrict__ q8ref, int nseg, int tilem, int rowA,
                           unsigned char *__restrict__ meta, double *__restrict__ v64, float *__restrict__ v32,
                           __half *__restrict__ v16, int8_t *__restrict__ v8, int8_t *__restrict__ v8ref)
{
    const int nhw = (gridDim.x * blockDim.x) >> 4;
    const int i = threadIdx.x & 15;
    for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 4; s < nseg; s += nhw) {
        const int4 h = seg_hdr[s];
        const int R = h.y, ta = h.x, tb = ta + ((h.z >> 16) & 0xFF), kp = h.z & 0xFFFF;
        const int rowlen = (R == tilem - 1) ? rowA - R * MF_BS : MF_BS;
        const long long off = (long long)h.w << 7;
        int t = i < rowlen ? ta : tb, e = 0, end = 0;
        for (int k0 = 0; k0 < kp; k0 += 8) {
            double d[8];
            float f[8];
            unsigned short hf[8];
            unsigned long long m = 0, a8 = 0, r8 = 0;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                while (e >= end && t < tb) {          // the row's entries in the next tile
                    const int cc = csrptr_offset[t], o = csr_offset[t], nnzt = csr_offset[t + 1] - o;
                    e = o + tptr[cc + i];
                    end = o + ((i == rowlen - 1) ? nnzt : (int)tptr[cc + i + 1]);
                    t++;
                }
                d[j] = 0.0;
                f[j] = 0.0f;
                if (e < end) {
                    d[j] = tval[e];
                    f[j] = tval_low[e];
                    m |= (unsigned long long)(unsigned char)(((t - 1 - ta) << 4) | tcol[e]) << (8 * j);
                    a8 |= (unsigned long long)(unsigned char)q8[e] << (8 * j);
                    r8 |= (unsigned long long)(unsigned char)q8ref[e] << (8 * j);
                    e++;
                }
                hf[j] = __half_as_ushort(__float2half_rn(f[j]));
            }
            const long long cb = off + (long long)(k0 >> 3) * 128;
#pragma unroll
            for (int q = 0; q < 4; q++) ((double2 *)(v64 + cb + 32 * q))[i] = make_double2(d[2 * q], d[2 * q + 1]);
            ((float4 *)(v32 + cb))[i] = make_float4(f[0], f[1], f[2], f[3]);
            ((float4 *)(v32 + cb + 64))[i] = make_float4(f[4], f[5], f[6], f[7]);
            ((uint4 *)(v16 + cb))[i] = make_uint4(hf[0] | (unsigned)hf[1] << 16, hf[2] | (unsigned)hf[3] << 16,
                                                  hf[4] | (unsigned)hf[5] << 16, hf[6] | (unsigned)hf[7] << 16);
            ((unsigned long long *)(meta + cb))[i] = m;
            ((unsigned long long *)(v8 + cb))[i] = a8;
            ((unsigned long long *)(v8ref + cb))[i] = r8;
        }
    }
}

// Packed per-segment header read once per segment by the solver's pipeline:
// {first tile, tile-row, Kp | ntiles << 16 | last-slice-of-tile-row << 24,
// entry offset / 128} (offsets are multiples of 128: Kp is a multiple of 8, 16 rows).
// Also writes the slice's tile words at a fixed stride of 16 per slice
// (column-tile << 8 | capability bits, 0 past the slice's tiles), so the solver
// can fetch them by slice number without waiting for the header.
__global__ void k_seg_hdr(const int *__restrict__ seg_ptr, const int *__restrict__ seg_tile0,
                          const int *__restrict__ seg_kp, const long long *__restrict__ seg_off,
                          const int *__restrict__ tile_columnidx, const unsigned char *__restrict__ caps, int tilem,
                          int4 *__restrict__ hdr, int *__restrict__ seg_tile)
{
    int R = blockIdx.x * blockDim.x + threadIdx.x;
    if (R >= tilem) return;
    for (int s = seg_ptr[R]; s < seg_ptr[R + 1]; s++) {
        const int t0 = seg_tile0[s];
        const int nt = seg_tile0[s + 1] - t0;
        const int last = (s + 1 == seg_ptr[R + 1]) ? 1 : 0;     // last slice of its tile-row
        hdr[s] = make_int4(t0, R, seg_kp[s] | (nt << 16) | (last << 24), (int)(seg_off[s] >> 7));
        for (int i = 0; i < MF_BS; i++)
            seg_tile[(long long)s * MF_BS + i] = (i < nt) ? ((tile_columnidx[t0 + i] << 8) | caps[t0 + i]) : 0;
    }
}

int grid_for(long long work, int threads)
{
    long long b = (work + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > 148 * 32) b = 148 * 32;
    return (int)b;
}

// an array of the handle
template <typename T>
int dalloc(T **p, long long count, cudaStream_t s)
{
    return mf_pool_array(p, count, s);
}

// The build's temporaries: freed in stream order when the build ends, on every path.
struct Temps {
    cudaStream_t s;
    std::vector<void *> all;
    template <typename T>
    int get(T **p, long long count)
    {
        const int rc = mf_pool_array(p, count, s);
        if (rc == MF_SUCCESS) all.push_back(*p);
        return rc;
    }
    ~Temps()
    {
        for (void *p : all) mf_pool_free(p, s);
    }
};

}  // namespace

#define MF_TRY(expr)                        \
    do {                                    \
        int _rc = (expr);                   \
        if (_rc != MF_SUCCESS) return _rc;  \
    } while (0)

namespace {

// The numbers the host waits for, gathered on the device and read in one copy.
struct Counts {
    int err, span;                                  // written by the kernels as they go
    Passes passes;
    int longest, not_one_chunk;                     // k_seg_shape
    int tilenum, last_tile0, rowblocks, nseg, nz_lo, nz_hi;
    int nonempty;
    long long entries;
};

__global__ void k_counts_tiles(Counts *c, const int *tile_ptr, const int *rb_ptr, const int *seg_ptr,
                               const int *rowptr, int tilem, int rowA)
{
    c->tilenum = tile_ptr[tilem];
    c->last_tile0 = tilem > 0 ? tile_ptr[tilem - 1] : 0;
    c->rowblocks = rb_ptr[tilem];
    c->nseg = seg_ptr[tilem];
    c->nz_lo = rowptr[0];
    c->nz_hi = rowptr[rowA];
}

__global__ void k_counts_filled(Counts *c, const int *nonzero_row, int tilenum, const long long *seg_off, int nseg)
{
    c->nonempty = nonzero_row[tilenum];
    c->entries = seg_off[nseg];
}

int read_counts(Counts *h, const Counts *d, cudaStream_t s)
{
    MF_CUDA_TRY(cudaGetLastError());
    MF_CUDA_TRY(cudaMemcpyAsync(h, d, sizeof(*h), cudaMemcpyDeviceToHost, s));
    MF_CUDA_TRY(cudaStreamSynchronize(s));
    return h->err;
}

}  // namespace

int mf_build_tiles(mf_matrix_s *A, long long nnz_given, cudaStream_t s)
{
    auto t_start = std::chrono::steady_clock::now();
    const int rowA = A->n_rows, colA = A->n_cols;
    const int tilem = (rowA + MF_BS - 1) / MF_BS;
    const int tilen = (colA + MF_BS - 1) / MF_BS;
    A->tilem = tilem;
    A->tilen = tilen;
    A->vec_len = std::max(tilem, tilen) * MF_BS;
    Temps tmp{s, {}};
    Counts *d_c = nullptr, c;
    int2 *d_spans = nullptr;
    int *d_ntiles = nullptr, *d_rbo = nullptr, *d_rows = nullptr;
    MF_TRY(tmp.get(&d_c, 1));
    MF_TRY(tmp.get(&d_spans, tilem));
    MF_TRY(tmp.get(&d_ntiles, tilem));
    MF_TRY(tmp.get(&d_rows, tilem));
    MF_TRY(tmp.get(&d_rbo, (long long)tilem + 1));
    MF_TRY(dalloc(&A->d_tile_ptr, (long long)tilem + 1, s));
    MF_TRY(dalloc(&A->d_seg_ptr, (long long)tilem + 1, s));
    MF_CUDA_TRY(cudaMemsetAsync(d_c, 0, sizeof(Counts), s));
    const int wgrid = grid_for((long long)tilem * 32, kThreads);
    if (tilem > 0)
        k_span<<<wgrid, kThreads, 0, s>>>(A->d_rowptr, A->d_colidx, tilem, rowA, colA, nnz_given, d_spans, &d_c->span,
                                          &d_c->err);
    MF_TRY(read_counts(&c, d_c, s));

    if ((long long)tilen >= (1LL << 23)) return MF_ERR_UNSUPPORTED;   // column tile must fit 23 bits
    const int span = std::max(c.span, 1);
    // a launch's scratch: shared memory up to kSharedWords a warp, else global memory within
    // kScratchBytes (one block at least) for `rows` tile-rows, a warp each
    struct Scratch {
        int words, global_mode, grid;
        size_t smem;
        unsigned int *global;
    };
    auto scratch = [&](const void *kernel, int words, long long rows, Scratch *x) -> int {
        *x = {words, 0, grid_for(rows * 32, kThreads), (size_t)words * 4 * kWarps, nullptr};
        if (words > kSharedWords) {
            const long long fit = std::max(1LL, kScratchBytes / 4 / kWarps / words);
            x->global_mode = 1;
            x->smem = 0;
            x->grid = (int)std::min<long long>(std::min(x->grid, kGlobalGrid), fit);
            const long long total = (long long)words * x->grid * kWarps;
            MF_TRY(tmp.get(&x->global, total));
            A->build_scratch = std::max(A->build_scratch, total * 4);
        } else if (x->smem > 48 * 1024) {
            MF_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)x->smem));
        }
        return MF_SUCCESS;
    };
    if (tilem > 0) {
        Scratch x;
        MF_TRY(scratch((const void *)k_count_tiles, span, tilem, &x));
        k_count_tiles<<<x.grid, kThreads, x.smem, s>>>(A->d_rowptr, A->d_colidx, tilem, rowA, d_spans, x.words,
                                                       x.global_mode, x.global, d_ntiles, d_rows, &d_c->passes);
        MF_CUDA_TRY(cudaGetLastError());
    }
    MF_TRY(mf_scan_tile_counts(d_ntiles, A->d_tile_ptr, d_rbo, A->d_seg_ptr, tilem, s));
    k_counts_tiles<<<1, 1, 0, s>>>(d_c, A->d_tile_ptr, d_rbo, A->d_seg_ptr, A->d_rowptr, tilem, rowA);
    MF_TRY(read_counts(&c, d_c, s));

    const long long nnz = (long long)c.nz_hi - c.nz_lo;
    const int tilenum = c.tilenum, nseg = c.nseg, rb = c.rowblocks;
    A->tilenum = tilenum;
    A->csrsize = (int)nnz;
    A->nnz = nnz;
    // 16 row starts per tile, fewer in a short last tile-row
    A->csrptrlen = tilem > 0 ? c.last_tile0 * MF_BS + (tilenum - c.last_tile0) * (rowA - (tilem - 1) * MF_BS) : 0;
    A->rowblkblock = rb;
    A->nseg = nseg;
    int *d_nzr = nullptr, *d_seg_entries = nullptr;
    long long *d_cost = nullptr;
    MF_TRY(dalloc(&A->d_tile_columnidx, (long long)tilenum + 1, s));
    MF_TRY(dalloc(&A->d_csr_offset, (long long)tilenum + 1, s));
    MF_TRY(dalloc(&A->d_csrptr_offset, (long long)tilenum + 1, s));
    MF_TRY(dalloc(&A->d_tval, nnz, s));
    MF_TRY(dalloc(&A->d_tval_low, nnz, s));
    MF_TRY(dalloc(&A->d_tcol, nnz, s));
    MF_TRY(dalloc(&A->d_tptr, (long long)tilenum * MF_BS, s));
    MF_TRY(tmp.get(&d_nzr, (long long)tilenum));
    MF_TRY(dalloc(&A->d_nonzero_row_new, (long long)tilenum + 1, s));
    MF_TRY(dalloc(&A->d_tile_rowidx, (long long)tilenum + 1, s));
    MF_TRY(dalloc(&A->d_block_signal, (long long)tilem + 4, s));
    MF_TRY(dalloc(&A->d_rb_idx, (long long)rb + 1, s));
    MF_TRY(dalloc(&A->d_rb_start, (long long)rb + 1, s));
    MF_TRY(dalloc(&A->d_rb_stop, (long long)rb + 1, s));
    MF_TRY(dalloc(&A->d_val_f16, nnz, s));
    MF_TRY(dalloc(&A->d_val_i8_ref, nnz, s));
    MF_TRY(dalloc(&A->d_val_i8, nnz, s));
    MF_TRY(dalloc(&A->d_i8_scale, (long long)tilenum + 1, s));
    MF_TRY(dalloc(&A->d_tile_caps, (long long)tilenum + 1, s));
    MF_TRY(dalloc(&A->d_seg_tile0, (long long)nseg + 1, s));
    MF_TRY(dalloc(&A->d_seg_kp, (long long)nseg + 1, s));
    MF_TRY(dalloc(&A->d_seg_rowlen, (long long)nseg * MF_BS + 1, s));
    MF_TRY(tmp.get(&d_seg_entries, (long long)nseg));
    MF_TRY(dalloc(&A->d_seg_off, (long long)nseg + 1, s));
    MF_TRY(tmp.get(&d_cost, tilem));
    MF_TRY(dalloc(&A->d_row_cost, (long long)tilem + 1, s));
    MF_TRY(dalloc(&A->d_seg_hdr, (long long)nseg + 1, s));
    MF_TRY(dalloc(&A->d_seg_tile, ((long long)nseg + 1) * MF_BS, s));
    MF_CUDA_TRY(cudaMemsetAsync(A->d_block_signal, 0, ((size_t)tilem + 4) * sizeof(int), s));
    MF_CUDA_TRY(cudaMemsetAsync(A->d_seg_hdr + nseg, 0, sizeof(int4), s));
    if (tilem == 0) {
        MF_CUDA_TRY(cudaMemsetAsync(A->d_csr_offset, 0, sizeof(int), s));
        MF_CUDA_TRY(cudaMemsetAsync(A->d_csrptr_offset, 0, sizeof(int), s));
    } else {
        const Passes &ps = c.passes;
        auto fill = [&](int words, const int *rows, int nrows) -> int {
            Scratch x;
            MF_TRY(scratch((const void *)k_fill_tiles, words, nrows, &x));
            k_fill_tiles<<<x.grid, kThreads, x.smem, s>>>(A->d_rowptr, A->d_colidx, A->d_val, A->d_val_low, tilem,
                                                          rowA, d_spans, rows, nrows, x.words, x.global_mode, x.global,
                                                          A->d_tile_ptr, A->d_tile_columnidx, A->d_csr_offset,
                                                          A->d_csrptr_offset, A->d_tval, A->d_tval_low, A->d_tcol,
                                                          A->d_tptr, &d_c->err);
            MF_CUDA_TRY(cudaGetLastError());
            return MF_SUCCESS;
        };
        MF_TRY(fill(ps.shared_words, nullptr, tilem));
        if (ps.n_mid > 0) MF_TRY(fill(ps.mid_words, d_rows, ps.n_mid));
        if (ps.n_large > 0) MF_TRY(fill(ps.large_words, d_rows + tilem - ps.n_large, ps.n_large));
        // nonempty-row lists, solver-slice shapes
        k_rowlist_count<<<wgrid, kThreads, 0, s>>>(A->d_tile_ptr, A->d_csr_offset, A->d_csrptr_offset, A->d_tptr,
                                                   tilem, rowA, d_nzr, A->d_tile_rowidx, A->d_block_signal);
        MF_CUDA_TRY(cudaGetLastError());
        k_seg_shape<<<wgrid, kThreads, 0, s>>>(A->d_tile_ptr, A->d_seg_ptr, A->d_csr_offset, A->d_csrptr_offset,
                                               A->d_tptr, tilem, rowA, A->d_seg_tile0, A->d_seg_kp,
                                               A->d_seg_rowlen, d_seg_entries, d_cost, &d_c->longest);
        MF_CUDA_TRY(cudaGetLastError());
    }
    MF_TRY(mf_scan_i32_to_i32(d_nzr, A->d_nonzero_row_new, tilenum, s));
    MF_TRY(mf_scan_i32_to_i64(d_seg_entries, A->d_seg_off, nseg, s));
    MF_TRY(mf_scan_i64_to_i64(d_cost, A->d_row_cost, tilem, s));
    k_counts_filled<<<1, 1, 0, s>>>(d_c, A->d_nonzero_row_new, tilenum, A->d_seg_off, nseg);
    // encoder
    if (nnz > 0) {
        k_encode_ref<<<grid_for(nnz, 256), 256, 0, s>>>(A->d_tval, A->d_tval_low, nnz, A->d_val_f16, A->d_val_i8_ref);
        MF_CUDA_TRY(cudaGetLastError());
    }
    if (tilenum > 0) {
        k_encode_tiles<<<grid_for(tilenum, 128), 128, 0, s>>>(A->d_csr_offset, tilenum, A->d_tval, A->d_val_i8,
                                                              A->d_i8_scale, A->d_tile_caps);
        MF_CUDA_TRY(cudaGetLastError());
    }
    MF_TRY(read_counts(&c, d_c, s));

    const int cnt = c.nonempty;
    const long long ent = c.entries;
    A->cnt_non_new = cnt;
    A->slice_entries = ent;
    A->max_row = c.longest;
    A->one_chunk = tilem > 0 && c.not_one_chunk == 0 ? 1 : 0;
    if ((ent >> 7) >= (1LL << 31)) return MF_ERR_UNSUPPORTED;
    MF_TRY(dalloc(&A->d_blockrowid_new, (long long)cnt + 1, s));
    MF_TRY(dalloc(&A->d_blockcsr_ptr_new, (long long)cnt + 1, s));
    MF_TRY(dalloc(&A->d_meta, ent, s));
    MF_TRY(dalloc(&A->d_v64, ent, s));
    MF_TRY(dalloc(&A->d_v32, ent, s));
    MF_TRY(dalloc(&A->d_v16, ent, s));
    MF_TRY(dalloc(&A->d_v8, ent, s));
    MF_TRY(dalloc(&A->d_v8ref, ent, s));
    MF_CUDA_TRY(cudaMemsetAsync(A->d_blockrowid_new, 0, (size_t)cnt + 1, s));
    MF_CUDA_TRY(cudaMemsetAsync(A->d_blockcsr_ptr_new, 0, (size_t)cnt + 1, s));
    // seg_tile0[nseg] = tilenum (end sentinel)
    MF_CUDA_TRY(cudaMemcpyAsync(A->d_seg_tile0 + nseg, A->d_tile_ptr + tilem, sizeof(int), cudaMemcpyDeviceToDevice, s));
    if (tilem > 0) {
        k_rowlist_fill<<<wgrid, kThreads, 0, s>>>(A->d_tile_ptr, A->d_csr_offset, A->d_csrptr_offset, A->d_tptr,
                                                  tilem, rowA, A->d_nonzero_row_new, A->d_blockrowid_new,
                                                  A->d_blockcsr_ptr_new);
        MF_CUDA_TRY(cudaGetLastError());
        k_rowblk_fill<<<(tilem + 255) / 256, 256, 0, s>>>(A->d_tile_ptr, tilem, d_rbo, A->d_rb_idx, A->d_rb_start,
                                                         A->d_rb_stop);
        MF_CUDA_TRY(cudaGetLastError());
        k_seg_hdr<<<(tilem + 255) / 256, 256, 0, s>>>(A->d_seg_ptr, A->d_seg_tile0, A->d_seg_kp, A->d_seg_off,
                                                      A->d_tile_columnidx, A->d_tile_caps, tilem, A->d_seg_hdr,
                                                      A->d_seg_tile);
        MF_CUDA_TRY(cudaGetLastError());
    }
    if (tilem > 0 && nseg > 0) {
        k_seg_fill<<<grid_for((long long)nseg * MF_BS, kThreads), kThreads, 0, s>>>(
            A->d_seg_hdr, A->d_csr_offset, A->d_csrptr_offset, A->d_tptr, A->d_tcol, A->d_tval, A->d_tval_low,
            A->d_val_i8, A->d_val_i8_ref, nseg, tilem, rowA, A->d_meta, A->d_v64, A->d_v32, A->d_v16, A->d_v8,
            A->d_v8ref);
        MF_CUDA_TRY(cudaGetLastError());
    }
    MF_CUDA_TRY(cudaStreamSynchronize(s));
    A->build_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_start).count();
    return MF_SUCCESS;
}
