// blocked.cu -- the tensor-core (blocked) form of the Macaulay reduction.
//
// The answer is the reduced row echelon form of the Schur complement
//   D' = D - C A^-1 B
// of the A|B / C|D split (A: the known pivots restricted to the left block,
// unit upper triangular; the reference reaches the same rows by reducing one
// C|D row at a time, src/la_ff_16.c:737-835 and :601-735).  Here every step is
// a dense block operation on residue matrices, and every O(n^3) step is the
// exact modular GEMM of tc_gemm.cu (int8 tensor cores):
//
//   1. Schur complement.  W = [C | D] holds the C|D rows sorted by lead (so
//      only a prefix of rows is active for a block of A), P = [A | B] the known
//      pivots.  (a) X = C A^-1, right-looking over 128-column blocks k of A:
//        X_k = W[:, k] A_kk^-1                   (GEMM, precomputed block inverse)
//        W[:, k+1 .. e_k] -= X_k A[k, k+1 .. e_k] (GEMM; e_k = last left column the
//                                                  pivots of block k touch)
//      with X_k stored over W[:, k]; (b) D' = D - X B as one GEMM whose zero
//      tiles (staircase X, banded B) are skipped.
//   2. Echelon of D' by rounds over all pending rows: a 128-column panel whose
//      rows all have leads of their own gives them as pivots; up to 256 rows of
//      every other panel are brought to reduced echelon form inside the panel by
//      one thread-block cluster (k_panel_factor), the row transformation it
//      records is applied to the pivot rows' whole width (k_panel_apply), and
//      the round's other pending rows are eliminated against all its pivots
//      (eliminate: gathered pivot columns, block inverses, GEMMs).
//   3. Back substitution to reduced echelon form, blocks of 1024 pivots from
//      the last to the first: U_k -= U_k[:, piv(>k)] R_(>k) (GEMM against the
//      already reduced later rows), then U_k = (U_k[:, piv(k)])^-1 U_k.
//   4. Compaction into CSR rows in descending lead order (plain.cu kernels).
#include <cuda_runtime.h>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/gbgpu.h"
#include "blocked.h"
#include "common.cuh"
#include "field.cuh"
#include "internal.h"
#include "kernels.h"
#include "rounds.cuh"
#include "tc_gemm.h"
#include "tiny.cuh"

namespace gbgpu {

constexpr int KB = 128;  // pivots per elimination block, columns of an echelon panel
constexpr int PR = 256;  // candidate rows of a panel

// per-round statistics of the echelon on stderr when GBGPU_DEBUG is set
static bool trace_rounds() {
    static const bool on = getenv("GBGPU_DEBUG") != nullptr;
    return on;
}

// ---------------------------------------------------------------------------
// kernels

// Dense rows from CSR without a separate clear: row i of out (i < n) receives
// CSR row rows[i], columns [from_i, nc + pad), from_i = (i / stride) stride (0
// when stride is 0); columns left of from_i are not written.  Columns >= ncl
// move right by pad (the right block starts on a 16-byte boundary; the pad
// columns are zero).  Each CTA assembles
// DS_COLS-column segments of a row in shared memory and writes them whole
// with 16-byte stores (ld a multiple of 4, out 16-byte aligned).
constexpr int DS_COLS = 16384;
__global__ void __launch_bounds__(512)
k_densify_seg(int32_t n, const int32_t* __restrict__ rows, const int64_t* __restrict__ row_ptr,
              const int32_t* __restrict__ cols, const uint32_t* __restrict__ vals, int32_t nc,
              int32_t ncl, int32_t pad, int32_t stride, uint32_t* out, int64_t ld) {
    extern __shared__ uint4 ds_smem[];
    uint32_t* seg = (uint32_t*)ds_smem;
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        const int32_t r = rows ? rows[i] : i;
        const int64_t b = row_ptr[r], e = row_ptr[r + 1];
        const int32_t from = stride ? (i / stride) * stride : 0;
        uint32_t* o = out + (size_t)i * ld;
        for (int32_t s0 = from; s0 < nc + pad; s0 += DS_COLS) {
            const int32_t w = min(DS_COLS, nc + pad - s0);
            for (int j = threadIdx.x; j < (w + 3) / 4; j += blockDim.x)
                ds_smem[j] = make_uint4(0u, 0u, 0u, 0u);
            __syncthreads();
            for (int64_t k = b + threadIdx.x; k < e; k += blockDim.x) {
                const int32_t cc = cols[k], c = cc + (cc >= ncl ? pad : 0) - s0;
                if (c >= 0 && c < w) seg[c] = vals[k];
            }
            __syncthreads();
            uint4* o4 = (uint4*)(o + s0);
            for (int j = threadIdx.x; j < w / 4; j += blockDim.x) o4[j] = ds_smem[j];
            for (int j = (w / 4) * 4 + threadIdx.x; j < w; j += blockDim.x) o[s0 + j] = seg[j];
            __syncthreads();
        }
    }
}

// The same rows without shared memory, for the known pivots (whose written
// intervals are short): a CTA takes a row:
// it fills each interval with zeros (16-byte stores; ld a multiple of 4, out
// 16-byte aligned), waits at a barrier (the zeros are then ordered before any
// later store of the CTA) and scatters the row's entries of the interval
// straight into place.  Every entry is read once per interval.
//
// Columns >= ncl move right by pad, as in k_densify_seg.  With brange (the known
// pivots P = [A | B] of the tensor form, whose readers need less) only two
// column intervals of row i are written:
//   [from_i, e1), e1 = min(ncl, max(from_i + stride, span[i / stride] + 1)):
//       the diagonal block and the left columns the block's rows reach;
//   [ncl + pad + lo, ncl + pad + hi): the right columns of row group i / 128, from
//       brange[i / 128] = (first, last) nonzero right column of the group,
//       widened to 64-column boundaries (the limb split reads whole
//       64-column blocks); nothing when the group's right part is zero.
// Everything else in the row is left as it was: its readers (the block
// inverses, the block solves and the limb split of the Schur product's B)
// never look there.
constexpr int DS_THREADS = 256;
__global__ void __launch_bounds__(DS_THREADS)
k_densify_direct(int32_t n, const int32_t* __restrict__ rows, const int64_t* __restrict__ row_ptr,
              const int32_t* __restrict__ cols, const uint32_t* __restrict__ vals, int32_t nc,
              int32_t ncl, int32_t pad, int32_t stride, uint32_t* out, int64_t ld,
              const int32_t* __restrict__ span = nullptr,
              const int2* __restrict__ brange = nullptr) {
    const int32_t split = ncl + pad;  // first right column
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        const int32_t r = rows ? rows[i] : i;
        const int64_t b = row_ptr[r], e = row_ptr[r + 1];
        const int32_t from = stride ? (i / stride) * stride : 0;
        uint32_t* o = out + (size_t)i * ld;
        // the (one or two) intervals of this row
        int32_t iv[2][2] = {{from, nc + pad}, {0, 0}};
        int n_iv = 1;
        if (brange) {
            int32_t e1 = ncl;
            if (span && stride) e1 = min(ncl, max(from + stride, span[i / stride] + 1));
            iv[0][1] = e1;
            const int2 br = brange[i / 128];
            if (br.y >= br.x) {
                const int32_t lo = split + (br.x / 64) * 64;
                const int32_t hi = min(nc + pad, split + (br.y / 64 + 1) * 64);
                const int32_t s = lo & ~3;
                if (s <= e1) {
                    iv[0][1] = max(e1, hi);
                } else {
                    iv[1][0] = s;
                    iv[1][1] = hi;
                    n_iv = 2;
                }
            }
        }
        for (int q = 0; q < n_iv; ++q) {
            const int32_t a0 = iv[q][0], a1 = iv[q][1];  // a0 is a multiple of 4
            const int32_t w4 = (a1 - a0) / 4;
            uint4* o4 = (uint4*)(o + a0);
            for (int j = threadIdx.x; j < w4; j += blockDim.x) o4[j] = make_uint4(0u, 0u, 0u, 0u);
            for (int32_t j = a0 + 4 * w4 + threadIdx.x; j < a1; j += blockDim.x) o[j] = 0u;
            __syncthreads();
            for (int64_t k = b + threadIdx.x; k < e; k += blockDim.x) {
                const int32_t cc = cols[k], c = cc + (cc >= ncl ? pad : 0);
                if (c >= a0 && c < a1) o[c] = vals[k];
            }
        }
        __syncthreads();  // this row's stores are done before the CTA's next row
    }
}

// span[b] = largest column < limit of the known pivots of rows [bs b, bs b + bs);
// with brange, also the first and last column >= limit (as column - limit)
// of every group of 128 rows, (INT_MAX, -1) filled in before
__global__ void k_block_span(int32_t ncl, const int32_t* __restrict__ piv_row,
                             const int64_t* __restrict__ row_ptr, const int32_t* __restrict__ cols,
                             int32_t limit, int32_t bs, int32_t* span, int2* brange = nullptr) {
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int c = warp; c < ncl; c += nwarps) {
        const int32_t r = piv_row[c];
        int32_t mx = -1, blo = INT_MAX, bhi = -1;
        for (int64_t k = row_ptr[r] + lane; k < row_ptr[r + 1]; k += 32) {
            const int32_t col = cols[k];
            if (col < limit) {
                mx = max(mx, col);
            } else {
                blo = min(blo, col - limit);
                bhi = max(bhi, col - limit);
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            blo = min(blo, __shfl_xor_sync(0xffffffffu, blo, o));
            bhi = max(bhi, __shfl_xor_sync(0xffffffffu, bhi, o));
        }
        if (lane == 0 && mx >= 0) atomicMax(&span[c / bs], mx);
        if (lane == 0 && brange && bhi >= 0) {
            atomicMin(&brange[c / 128].x, blo);
            atomicMax(&brange[c / 128].y, bhi);
        }
    }
}

// every range empty: (INT_MAX, -1)
__global__ void k_clear_ranges(int32_t n, int2* r) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        r[i] = make_int2(INT_MAX, -1);
}

// lead (first column) of each listed CSR row
__global__ void k_csr_leads(int32_t n, const int32_t* __restrict__ rows,
                            const int64_t* __restrict__ row_ptr, const int32_t* __restrict__ cols,
                            int32_t* lead) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        lead[i] = cols[row_ptr[rows[i]]];
}

// number of entries of the sorted array `v` that are < bound[j], per j
__global__ void k_count_below(int32_t n, const int32_t* __restrict__ v, int32_t nb,
                              int32_t step, int32_t* out) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < nb; j += gridDim.x * blockDim.x) {
        const int32_t bound = (j + 1) * step;
        int lo = 0, hi = n;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (v[mid] < bound) lo = mid + 1;
            else hi = mid;
        }
        out[j] = lo;
    }
}

constexpr int INV_THREADS = 512;  // threads of k_neg_inverse
constexpr int INV_BYTES = (KB * (KB + 1) + KB * KB / 4) * (int)sizeof(uint32_t);

// One doubling level of k_neg_inverse: the 2 SZ x 2 SZ diagonal blocks
// [[A^-1, B], [0, C^-1]] get -A^-1 B C^-1 in place of B.  A thread owns R rows
// by CW columns of a block's product; lanes run over the columns, so the left
// factor's entries are broadcasts.
template <class F, int SZ>
__device__ __forceinline__ void inverse_level(uint32_t (*V)[KB + 1], uint32_t* T, const F& f) {
    constexpr int CW = SZ > 32 ? 2 : 1, LN = SZ / CW;       // columns of a thread, lanes of a row
    constexpr int R = SZ * KB / 2 / (INV_THREADS * CW);     // rows of a thread
    constexpr int GROUPS = SZ / R;                          // threads of a column
    const int j = threadIdx.x % LN, g = threadIdx.x / LN;
    const int pr = g / GROUPS, i0 = g % GROUPS * R, b0 = pr * 2 * SZ;
    uint64_t acc[R][CW];
    auto clear = [&]() {
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int w = 0; w < CW; ++w) acc[r][w] = 0;
    };
    // T = B C^-1 (C^-1 is upper triangular: column j needs k <= j)
    clear();
#pragma unroll
    for (int w0 = 0; w0 < CW; ++w0)
#pragma unroll 8
        for (int k = w0 * LN; k < (w0 + 1) * LN; ++k) {
            uint32_t v[CW];
#pragma unroll
            for (int w = w0; w < CW; ++w) v[w] = V[b0 + SZ + k][b0 + SZ + j + w * LN];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const uint32_t u = V[b0 + i0 + r][b0 + SZ + k];
#pragma unroll
                for (int w = w0; w < CW; ++w) acc[r][w] = f.lazy_add(acc[r][w], u, v[w]);
            }
        }
    uint32_t* Tp = T + pr * SZ * SZ;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int w = 0; w < CW; ++w) Tp[(i0 + r) * SZ + j + w * LN] = f.lazy_mod(acc[r][w]);
    __syncthreads();
    // -A^-1 T (A^-1 is upper triangular: row i needs k >= i)
    clear();
#pragma unroll 4
    for (int k = i0; k < SZ; ++k) {
        uint32_t t[CW];
#pragma unroll
        for (int w = 0; w < CW; ++w) t[w] = Tp[k * SZ + j + w * LN];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t u = V[b0 + i0 + r][b0 + k];
#pragma unroll
            for (int w = 0; w < CW; ++w) acc[r][w] = f.lazy_add(acc[r][w], u, t[w]);
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int w = 0; w < CW; ++w) {
            const uint32_t x = f.lazy_mod(acc[r][w]);
            V[b0 + i0 + r][b0 + SZ + j + w * LN] = x ? f.p - x : 0u;
        }
    __syncthreads();
}

// -U^-1 mod p for unit upper triangular blocks.  Block b is read from
// src + b * stride_b with leading dimension ld (kb x kb, kb <= KB); the result
// (KB x KB, identity-padded) goes to out + b * ostride with leading dimension
// old.  One CTA per block, V = U^-1 built in place in shared memory by
// doubling: the 8 x 8 diagonal blocks by back substitution, a thread per
// column, then for sz = 8, 16, 32, 64 every 2sz x 2sz diagonal block
// [[A, B], [0, C]] gets its top-right part -A^-1 B C^-1 as two small products.
//
// Bound by the 64-bit multiply-adds of the sz = 64 products (4 cycles a warp
// each).  A sum stays one 64-bit accumulator (below 2^39 for p < 2^16, folded
// below p^2 otherwise), a thread's products share their operands' loads, and
// 83 KB a block let two blocks share an SM: 18 us a launch of up to 296 blocks
// (36 us for p >= 2^16); with 16-bit halves in two accumulators, an entry a
// thread and 148 KB a block it was 55 us, and a second wave beyond 148 blocks.
template <class F>
__global__ void __launch_bounds__(INV_THREADS, 2)
k_neg_inverse(const uint32_t* __restrict__ src, int64_t ld, int64_t stride_b, int32_t n_blocks,
              int32_t last_kb, uint32_t* out, int64_t ostride, int64_t old, F f) {
    extern __shared__ uint32_t inv_smem[];
    uint32_t(*V)[KB + 1] = (uint32_t(*)[KB + 1])inv_smem;
    uint32_t* T = inv_smem + KB * (KB + 1);  // KB * KB / 4 entries
    const int b = blockIdx.x;
    const int kb = b == n_blocks - 1 ? last_kb : KB;
    const uint32_t* s = src + (size_t)b * stride_b;
    const int tid = threadIdx.x;
    // the block: KB * KB / blockDim.x entries per thread, 16 loads in flight
    constexpr int PER = KB * KB / INV_THREADS;
#pragma unroll 1
    for (int q0 = 0; q0 < PER; q0 += 16) {
        uint32_t v[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int t = tid + (q0 + q) * INV_THREADS;
            const int i = t / KB, j = t % KB;
            v[q] = (i < kb && j < kb && i < j) ? s[(size_t)i * ld + j] : (i == j ? 1u : 0u);
        }
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int t = tid + (q0 + q) * INV_THREADS;
            V[t / KB][t % KB] = v[q];
        }
    }
    __syncthreads();
    // 8 x 8 diagonal blocks: V[i][j] = -sum_{i<k<=j} U[i][k] V[k][j]
    uint32_t d[8];
    const int b0 = tid & (KB - 8), j = tid & 7;
    if (tid < KB) {
#pragma unroll
        for (int i = 7; i >= 0; --i) {
            uint64_t acc = 0;
#pragma unroll
            for (int k = i + 1; k < 8; ++k) acc = f.lazy_add(acc, V[b0 + i][b0 + k], d[k]);
            const uint32_t x = f.lazy_mod(acc);
            d[i] = i == j ? 1u : i < j && x ? f.p - x : 0u;
        }
    }
    __syncthreads();
    if (tid < KB) {
#pragma unroll
        for (int i = 0; i < 8; ++i) V[b0 + i][b0 + j] = d[i];
    }
    __syncthreads();
    inverse_level<F, 8>(V, T, f);
    inverse_level<F, 16>(V, T, f);
    inverse_level<F, 32>(V, T, f);
    inverse_level<F, 64>(V, T, f);
    uint32_t* o = out + (size_t)b * ostride;
    for (int t = tid; t < KB * KB; t += INV_THREADS) {
        const int i = t / KB, jj = t % KB;
        const uint32_t v = V[i][jj];
        o[(size_t)i * old + jj] = v ? f.p - v : 0u;  // -V
    }
}

// The row copies below give every piece of GB_PIECE columns of a row to one
// warp (32-bit index arithmetic, four independent loads per lane in flight);
// the loop body sees the row i and its columns [jb, je).
constexpr int GB_PIECE = 512;
#define GB_WARP_ROWS(rows, ncols)                                                    \
    const int lane = threadIdx.x & 31;                                               \
    const int warp_ = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;                  \
    const int nwarps_ = (gridDim.x * blockDim.x) >> 5;                               \
    const int npc_ = ((ncols) + GB_PIECE - 1) / GB_PIECE;                            \
    for (int it_ = warp_, i = it_ / max(npc_, 1), jb = (it_ % max(npc_, 1)) * GB_PIECE, \
             je = min((int)(ncols), jb + GB_PIECE);                                  \
         it_ < (rows) * npc_;                                                        \
         it_ += nwarps_, i = it_ / max(npc_, 1), jb = (it_ % max(npc_, 1)) * GB_PIECE, \
             je = min((int)(ncols), jb + GB_PIECE))

// dst[i][j] = src[r_i][cols[j]], r_i = rlist[i] (i without a list)
__global__ void k_gather_cols(int32_t rows, int32_t n, const uint32_t* __restrict__ src,
                              int64_t lds, const int32_t* __restrict__ cols, uint32_t* dst,
                              int64_t ldd, const int32_t* __restrict__ rlist = nullptr) {
    GB_WARP_ROWS(rows, n) {
        const int32_t r = rlist ? rlist[i] : i;
        const uint32_t* s = src + (size_t)max(r, 0) * lds;
        uint32_t* o = dst + (size_t)i * ldd;
        for (int j0 = jb + lane; j0 < je; j0 += 128) {
            uint32_t v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int jj = j0 + 32 * u;
                const int32_t col = jj < je && r >= 0 ? cols[jj] : -1;
                v[u] = col >= 0 ? s[col] : 0u;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (j0 + 32 * u < je) o[j0 + 32 * u] = v[u];
        }
    }
}

// dst row rows[i] = src row i
__global__ void k_scatter_rows_dense(int32_t nrows, const int32_t* __restrict__ rows, int32_t n,
                                     const uint32_t* __restrict__ src, int64_t lds,
                                     uint32_t* dst, int64_t ldd) {
    GB_WARP_ROWS(nrows, n) {
        const uint32_t* s = src + (size_t)i * lds;
        uint32_t* o = dst + (size_t)rows[i] * ldd;
        for (int j0 = jb + lane; j0 < je; j0 += 128) {
            uint32_t v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int jj = j0 + 32 * u;
                v[u] = jj < je ? s[jj] : 0u;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (j0 + 32 * u < je) o[j0 + 32 * u] = v[u];
        }
    }
}

// First nonzero column of every row (-1 for zero rows), one warp per row; entries of
// list below 0 stand for no row.  With from_prev the scan starts at the row's current
// lead (leads only move right under elimination).  A pass covers LEAD_U chunks of 32
// columns whose loads are in flight together.
constexpr int LEAD_U = 8;
__global__ void k_row_leads(int32_t rows, const int32_t* __restrict__ list, int32_t ncols,
                            const uint32_t* __restrict__ M, int64_t ld, int32_t* lead,
                            int32_t from_prev = 0) {
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int i = warp; i < rows; i += nwarps) {
        const int32_t r = list ? list[i] : i;
        if (r < 0) continue;
        const uint32_t* row = M + (size_t)r * ld;
        int found = -1;
        const int start = from_prev && lead[r] > 0 ? lead[r] : 0;
        for (int base = start; base < ncols && found < 0; base += 32 * LEAD_U) {
            uint32_t v[LEAD_U];
#pragma unroll
            for (int u = 0; u < LEAD_U; ++u) {
                const int c = base + 32 * u + lane;
                v[u] = c < ncols ? row[c] : 0u;
            }
#pragma unroll
            for (int u = 0; u < LEAD_U; ++u) {
                const unsigned bal = __ballot_sync(0xffffffffu, v[u] != 0u);
                if (bal && found < 0) found = base + 32 * u + __ffs(bal) - 1;
            }
        }
        if (lane == 0) lead[r] = found;
    }
}

// scale row rows[i] by the inverse of its entry at column cols[i] (one CTA
// per row; NORM_U independent loads per thread and pass)
constexpr int NORM_U = 8;
template <class F>
__global__ void k_normalize_at(const int32_t* __restrict__ n_dev, const int32_t* __restrict__ rows,
                               const int32_t* __restrict__ cols, int32_t ncols, uint32_t* M,
                               int64_t ld, F f) {
    __shared__ uint32_t s_inv;
    const int32_t n = *n_dev;
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        uint32_t* row = M + (size_t)rows[i] * ld;
        const int32_t c0 = cols[i];
        const uint32_t lv = row[c0];
        if (lv == 1u) continue;  // uniform over the CTA
        __syncthreads();  // the previous row's readers of s_inv are done
        if (threadIdx.x == 0) s_inv = f.prep(inverse_mod(lv, f.p));
        __syncthreads();
        const uint32_t inv = s_inv;
        for (int c = c0 + 1 + threadIdx.x; c < ncols; c += blockDim.x * NORM_U) {
            uint32_t v[NORM_U];
#pragma unroll
            for (int u = 0; u < NORM_U; ++u) {
                const int cc = c + u * (int)blockDim.x;
                v[u] = cc < ncols ? row[cc] : 0u;
            }
#pragma unroll
            for (int u = 0; u < NORM_U; ++u) {
                const int cc = c + u * (int)blockDim.x;
                if (v[u]) row[cc] = f.mulp(v[u], inv);
            }
        }
        if (threadIdx.x == 0) row[c0] = 1u;
    }
}

// k_panel_apply's forms by pivots of a chunk, and the lists of their chunks: cls
// holds PA_CLASSES counts, then a list of up to n_dirty chunks for each
constexpr int PA_CLASSES = 3;
__device__ __forceinline__ int pa_class(int np) { return np <= 32 ? 0 : np <= 64 ? 1 : 2; }

// Reduced row echelon form of one panel (the 128 columns of panel dpanel[d], on
// the n <= PR rows chunk_rows[d PR + i] of Dp) in the shared memory of one
// cluster (tiny.cuh).  Its pivots are registered (piv_of_col, is_piv, wflag);
// piv_rows[d KB + k]: their rows in ascending column order, n_piv[d] of them; and
// the transformation: the reduced pivot row k (unit columns at the panel's pivots)
// is sum_j F[d][k][j] (old pivot row j).  Rows of the chunk that are no pivots
// have their panel part in the span of the pivots', so the round's elimination
// clears them.
//
// What bounds it is the chain of pivots (sixteen at a time, tiny.cuh).  A step
// per pivot over all of the chunk's rows, with the transformation beside the
// panel, took 191 us for 128 rows of a full panel on one SM; here one panel takes
// 92 us with 256 candidate rows on eight SMs, and more candidates than pivots
// keep a dense panel from running short of independent rows (an 8192 x 8192
// block of rank 6144 takes 48 rounds instead of 76).

template <class F>
__global__ void __launch_bounds__(kTinyThreads, 1)
k_panel_factor(const uint32_t* __restrict__ Dp, int64_t ld, const int32_t* __restrict__ chunk_rows,
               const int32_t* __restrict__ dpanel, const int32_t* __restrict__ cursor,
               int32_t max_rows, int32_t ncr, uint32_t* F_b, int32_t* piv_rows_b, int32_t* n_piv_b,
               int32_t* piv_of_col, uint8_t* is_piv, int32_t* wflag, int32_t* cls, F f) {
    extern __shared__ __align__(16) uint32_t pf_smem[];
    const int CL = cluster_size(), rk = cluster_rank(), sh = __ffs(CL) - 1;
    const int d = blockIdx.x / CL, tid = threadIdx.x;
    const int32_t pj = dpanel[d] * KB, n = min(cursor[d], max_rows), bw = min(KB, ncr - pj);
    const int32_t* rows = chunk_rows + (size_t)d * PR;
    const TinyLayout L = tiny_layout(n, KB, CL);
    for (int t = rk; t < KB / TP; t += CL)
        for (int q = tid; q < n * TP; q += kTinyThreads) {
            const int c = t * TP + q % TP;
            pf_smem[(t >> sh) * n * TP + q] = c < bw ? Dp[(size_t)rows[q / TP] * ld + pj + c] : 0u;
        }
    const int np = tiny_echelon<true>(n, KB, pf_smem, f);
    // pivots in column order: place of column c = pivot columns left of it
    const int32_t* prow = (const int32_t*)(pf_smem + L.cols);
    __shared__ int32_t s_col[KB], s_place[KB];
    if (tid < 32) {
        int at = 0;
        for (int c = tid; c < KB; c += 32) {
            const unsigned bal = __ballot_sync(0xffffffffu, prow[c] >= 0);
            const int k = at + __popc(bal & ((1u << tid) - 1u));
            s_place[c] = prow[c] >= 0 ? k : -1;
            if (prow[c] >= 0) s_col[k] = c;
            at += __popc(bal);
        }
    }
    __syncthreads();
    if (rk == 0) {
        if (tid == 0) {
            n_piv_b[d] = np;
            if (np > 0) {
                const int q = gridDim.x == CL ? PA_CLASSES - 1 : pa_class(np);
                cls[PA_CLASSES + q * (gridDim.x / CL) + atomicAdd(&cls[q], 1)] = d;
            }
        }
        for (int k = tid; k < np; k += kTinyThreads) {
            const int32_t row = rows[prow[s_col[k]]], col = pj + s_col[k];
            piv_rows_b[d * KB + k] = row;
            piv_of_col[col] = row;
            is_piv[row] = 1;
            wflag[col] = 1;
        }
    }
    uint32_t* Fo = F_b + (size_t)d * KB * KB;
    // this CTA's columns of F
    for (int t = rk; t < KB / TP; t += CL)
        for (int q = tid; q < np * TP; q += kTinyThreads) {
            const int k = q / TP, j = s_place[t * TP + q % TP];
            if (j >= 0) Fo[k * KB + j] = pf_smem[((t >> sh) * n + prow[s_col[k]]) * TP + q % TP];
        }
}

// The panel transformation of every factorized chunk: the pivot rows of chunk d
// become F_d old over the columns from the first dirty panel on (k_panel_factor),
// np x np times np x width per chunk, in place.  A warp owns 16 columns of a chunk: it
// reads all old values there before it writes any.
//
// On CUDA cores this is bound by the 64-bit multiply-adds (four issue cycles per
// warp each: 178 us for 5000 pivot rows in chunks of 32 over 10000 columns), and
// the chunks are too small and too many for the pipeline of tc_gemm.cu.  So the
// products run on warp-level int8 matrix instructions straight from registers,
// residues in L unsigned bytes as there: the old values of four rows at a column
// are the four bytes of an operand register, and 16 columns of np rows stay in
// registers.  What is left is reading and writing the rows (and, for four bytes,
// the instructions' rate).  All rounds of a staircase matrix, CUDA cores before,
// matrix instructions now: 859 -> 475 us (20000 columns, p = 65521), 295 -> 140
// (10000, p = 251), 293 -> 264 (9001, p = 2^31 - 1); the one panel of an
// 8192-column dense block 41 -> 13 us.
//
// Forms by pivots, KC blocks of 32: registers for the old values.  A block takes
// work items (a chunk of its class, `width` columns of it) in turn: a grid over all
// chunks launched mostly blocks without work (97 us for a round of 157 chunks).
constexpr int PA_THREADS = 256;
constexpr int PA_COLS = 16;  // of a warp at a time
struct PanelApply {
    uint32_t* Dp;
    int64_t ld;
    int32_t ncr, j0, width, n_dirty;
    const int32_t *cls, *dpanel, *n_piv, *piv_rows;
    const uint32_t* F;
};

__device__ __forceinline__ void mma_u8(int32_t (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                       uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
        "{%8, %9}, {%0, %1, %2, %3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// byte l of x[0 .. 4)
template <int L>
__device__ __forceinline__ void pack_bytes(const uint32_t (&x)[4], uint32_t (&out)[L]) {
#pragma unroll
    for (int l = 0; l < L; ++l) {
        const uint32_t sel = (uint32_t)(l | ((4 + l) << 4));
        out[l] = __byte_perm(__byte_perm(x[0], x[1], sel), __byte_perm(x[2], x[3], sel), 0x5410u);
    }
}

// sum_w s[w] 2^(8 w) mod p, s[w] <= min(w + 1, 2 L - 1 - w) 128 255^2 < 2^25
template <int L, class F>
__device__ __forceinline__ uint32_t fold_weights(const int32_t (&s)[2 * L - 1], const F& f) {
    uint64_t t = (uint32_t)s[0];
#pragma unroll
    for (int w = 1; w < (L < 4 ? 2 * L - 1 : 4); ++w) t += (uint64_t)(uint32_t)s[w] << (8 * w);
    // L = 2: t < 2^41; L = 4: t < 2^50 and t <= 128 p^2, one of them below p 2^32
    uint32_t r = f.lazy_mod(t);
    if constexpr (L == 4) {
        uint64_t h = (uint32_t)s[4];
        h += (uint64_t)(uint32_t)s[5] << 8;
        h += (uint64_t)(uint32_t)s[6] << 16;
        r += f.prep(f.lazy_mod(h));  // prep: times 2^32
        r = r >= f.p ? r - f.p : r;
    }
    return r;
}

// bytes of a row of F's planes (a step of 16 beyond it: no bank conflicts)
constexpr int pa_row(int kc) { return 32 * kc + 16; }
// blocks per SM (registers)
constexpr int pa_blocks(int l, int kc) { return l == 4 ? (kc == 4 ? 1 : 2) : (kc == 1 ? 3 : 2); }
template <int L, int KC, class F>
__global__ void __launch_bounds__(PA_THREADS, pa_blocks(L, KC))
k_panel_apply(const PanelApply a, F f) {
    constexpr int ROW = pa_row(KC), PLANE = 32 * KC * ROW;
    constexpr int NT = PA_COLS / 8, NW = 2 * L - 1, CLS = KC == 1 ? 0 : KC == 2 ? 1 : 2;
    extern __shared__ __align__(16) uint8_t s_f[];  // planes of F
    __shared__ int32_t s_rows[32 * KC];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane / 4, t = lane % 4;
    const int n = a.cls[CLS];
    const int items = n * ((a.ncr - a.j0 + a.width - 1) / a.width);
    for (int i = blockIdx.x; i < items; i += gridDim.x) {
        const int d = a.cls[PA_CLASSES + CLS * a.n_dirty + i % n];
        // its rows are zero left of the chunk's panel
        const int c_lo = max(a.j0 + i / n * a.width, a.dpanel[d] * KB);
        const int c_hi = min(a.ncr, a.j0 + (i / n + 1) * a.width);
        if (c_lo >= c_hi) continue;  // uniform
        const int np = a.n_piv[d], mt = (np + 15) / 16;
        __syncthreads();  // the last item's readers are done
        for (int q = tid; q < 32 * KC; q += PA_THREADS)
            s_rows[q] = q < np ? a.piv_rows[(size_t)d * KB + q] : -1;
        const uint32_t* Fd = a.F + (size_t)d * KB * KB;
#pragma unroll 4
        for (int q = tid; q < mt * 16 * 8 * KC; q += PA_THREADS) {
            const int k = q / (8 * KC), j = 4 * (q % (8 * KC));
            uint4 e = make_uint4(0u, 0u, 0u, 0u);  // (past np: whatever is there)
            if (k < np && j < np) e = *(const uint4*)(Fd + k * KB + j);
            const uint32_t x[4] = {e.x, j + 1 < np ? e.y : 0u, j + 2 < np ? e.z : 0u,
                                   j + 3 < np ? e.w : 0u};
            uint32_t y[L];
            pack_bytes<L>(x, y);
#pragma unroll
            for (int l = 0; l < L; ++l) *(uint32_t*)&s_f[l * PLANE + k * ROW + j] = y[l];
        }
        __syncthreads();
        for (int c0 = c_lo + PA_COLS * warp; c0 < c_hi; c0 += PA_COLS * (PA_THREADS / 32)) {
            // old values: register (kc, h, nt) of a lane holds rows 32 kc + 16 h + 4 t
            // .. + 3 at column c0 + 8 nt + g
            uint32_t bv[L][KC][2][NT];
#pragma unroll
            for (int kc = 0; kc < KC; ++kc)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
                        const int col = c0 + 8 * nt + g;
                        uint32_t x[4], y[L];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int32_t r = s_rows[32 * kc + 16 * h + 4 * t + u];
                            x[u] = r >= 0 && col < c_hi ? a.Dp[(size_t)r * a.ld + col] : 0u;
                        }
                        pack_bytes<L>(x, y);
#pragma unroll
                        for (int l = 0; l < L; ++l) bv[l][kc][h][nt] = y[l];
                    }
            __syncwarp();  // every lane has read before any writes
            for (int m = 0; m < mt; ++m) {
                int32_t acc[NT][NW][4];
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int w = 0; w < NW; ++w)
#pragma unroll
                        for (int q = 0; q < 4; ++q) acc[nt][w][q] = 0;
#pragma unroll
                for (int kc = 0; kc < KC; ++kc)
#pragma unroll
                    for (int la = 0; la < L; ++la) {
                        const uint8_t* p0 = &s_f[la * PLANE + (16 * m + g) * ROW + 32 * kc + 4 * t];
                        const uint32_t af[4] = {*(const uint32_t*)p0, *(const uint32_t*)(p0 + 8 * ROW),
                                                *(const uint32_t*)(p0 + 16),
                                                *(const uint32_t*)(p0 + 8 * ROW + 16)};
#pragma unroll
                        for (int lb = 0; lb < L; ++lb)
#pragma unroll
                            for (int nt = 0; nt < NT; ++nt)
                                mma_u8(acc[nt][la + lb], af, bv[lb][kc][0][nt], bv[lb][kc][1][nt]);
                    }
                // entry q: pivot 16 m + g + 8 (q / 2), column c0 + 8 nt + 2 t + q % 2
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int32_t r = s_rows[16 * m + g + 8 * (q / 2)];
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
                        int32_t sw[NW];
#pragma unroll
                        for (int w = 0; w < NW; ++w) sw[w] = acc[nt][w][q];
                        const int col = c0 + 8 * nt + 2 * t + q % 2;
                        const uint32_t v = fold_weights<L>(sw, f);
                        if (r >= 0 && col < c_hi) a.Dp[(size_t)r * a.ld + col] = v;
                    }
                }
            }
        }
    }
}

// dst block b (NB x NB, leading dimension NB, block stride NB (NB + 1)) =
// src block b (nb_b x nb_b at src + b stride_src, leading dimension lds),
// identity-padded; nb_b = NB except for the last block
__global__ void k_copy_blocks(const uint32_t* __restrict__ src, int64_t lds, int64_t stride_src,
                              int32_t n_blocks, int32_t last_nb, int32_t NB, uint32_t* dst) {
    GB_WARP_ROWS(n_blocks * NB, NB) {
        const int32_t b = i / NB, r = i % NB;
        const int32_t nb = b == n_blocks - 1 ? last_nb : NB;
        const uint32_t* s = src + (size_t)b * stride_src + (size_t)r * lds;
        uint32_t* o = dst + (size_t)b * NB * (NB + 1) + (size_t)r * NB;
        for (int j0 = jb + lane; j0 < je; j0 += 128) {
            uint32_t v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int jj = j0 + 32 * u;
                v[u] = (r < nb && jj < nb) ? s[jj] : (r == jj ? 1u : 0u);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (j0 + 32 * u < je) o[j0 + 32 * u] = v[u];
        }
    }
}

// ---------------------------------------------------------------------------
// host helpers

struct Ctx {
    cudaStream_t s;
    uint32_t p;
    int form;
    int32_t* err;
    long long launches = 0;
    std::vector<void*> tmp;
    void* ws = nullptr;  // GEMM limb planes
    size_t ws_bytes = 0;

    template <class T>
    T* alloc(size_t n) {
        void* q = nullptr;
        if (cudaMallocAsync(&q, std::max<size_t>(n, 1) * sizeof(T), s) != cudaSuccess)
            return nullptr;
        tmp.push_back(q);
        return (T*)q;
    }
    // Buffers of one step each, for every round's step in turn: n entries of slot
    // `which`, whatever the last step left in it.  They stay until the end: freed behind
    // every step instead, each of a plan's runs waits in the pool for its largest
    // buffers, which no longer find the place of the run before (20000 x 5000 staircase:
    // 10 to 50 ms a reduction instead of 7.8).
    enum { kU, kT, kBlocks, kInverses, kGathered, kSolved, kProduct, kSlots };
    void* slot[kSlots] = {};
    size_t slot_bytes[kSlots] = {};
    uint32_t* step(int which, size_t n) {
        const size_t bytes = std::max<size_t>(n, 1) * sizeof(uint32_t);
        if (bytes > slot_bytes[which]) {
            if (slot[which]) cudaFreeAsync(slot[which], s);
            slot[which] = nullptr;
            slot_bytes[which] = 0;
            if (cudaMallocAsync(&slot[which], bytes, s) != cudaSuccess) {
                slot[which] = nullptr;
                return nullptr;
            }
            slot_bytes[which] = bytes;
        }
        return (uint32_t*)slot[which];
    }
    // all buffers, for blocked_release
    std::vector<void*>* hand_over() {
        auto* keep = new std::vector<void*>(tmp);
        if (ws) keep->push_back(ws);
        for (void* q : slot)
            if (q) keep->push_back(q);
        return keep;
    }
    void release() {
        for (void* q : tmp) cudaFreeAsync(q, s);
        tmp.clear();
        for (int k = 0; k < kSlots; ++k) {
            if (slot[k]) cudaFreeAsync(slot[k], s);
            slot[k] = nullptr;
            slot_bytes[k] = 0;
        }
        if (ws) cudaFreeAsync(ws, s);
        ws = nullptr;
        ws_bytes = 0;
    }
};

#define BL_CHECK(expr)                                                   \
    do {                                                                 \
        int rc_ = (expr);                                                \
        if (rc_) return rc_;                                             \
    } while (0)
#define BL_CUDA(expr)                                                    \
    do {                                                                 \
        cudaError_t e_ = (expr);                                         \
        if (e_ != cudaSuccess) {                                         \
            set_error(std::string(#expr) + ": " + cudaGetErrorString(e_)); \
            return GBGPU_ECUDA;                                          \
        }                                                                \
    } while (0)
#define BL_LAUNCH(...)                                                   \
    do {                                                                 \
        __VA_ARGS__;                                                     \
        ++c.launches;                                                    \
        BL_CUDA(cudaGetLastError());                                     \
    } while (0)

static int grid_of(int64_t n, int t = 256) {
    int64_t g = (n + t - 1) / t;
    return (int)std::max<int64_t>(1, std::min<int64_t>(g, 148 * 16));
}

// D (M x N) -= A (M x K) B (K x N), exact mod p, for any TcGemmArgs (batch,
// row lists); the tensor-core workspace grows on demand
static int gemm_args(Ctx& c, TcGemmArgs g) {
    if (g.M <= 0 || g.N <= 0 || g.K <= 0 || g.batch <= 0) return GBGPU_OK;
    g.p = c.p;
    if (c.form == GBGPU_FORM_PLAIN) return plain_submul(g, c.s, &c.launches);
    const size_t need = tc_workspace_bytes(c.p, g.M, g.N, g.K, g.batch);
    if (need > c.ws_bytes) {
        if (c.ws) cudaFreeAsync(c.ws, c.s);
        c.ws = nullptr;
        const size_t bytes = std::max(need, c.ws_bytes * 2);
        if (cudaMallocAsync(&c.ws, bytes, c.s) != cudaSuccess) {
            set_error("GEMM workspace allocation failed");
            return GBGPU_ENOMEM;
        }
        c.ws_bytes = bytes;
    }
    return tc_submul(g, c.ws, c.s, c.err, &c.launches);
}

static int gemm(Ctx& c, uint32_t* D, int64_t ldd, const uint32_t* A, int64_t lda,
                const uint32_t* B, int64_t ldb, int32_t M, int32_t N, int32_t K) {
    TcGemmArgs g{c.p, M, N, K, A, lda, B, ldb, D, ldd};
    return gemm_args(c, g);
}

// D <- -A B where D is A or B itself (unbatched).  The CUDA-core GEMM reads its
// operands while it writes, so there the product goes through a copy.
static int gemm_set_in_place(Ctx& c, TcGemmArgs g) {
    if (g.M <= 0 || g.N <= 0 || g.K <= 0) return GBGPU_OK;
    g.set = true;
    if (c.form != GBGPU_FORM_PLAIN) return gemm_args(c, g);
    uint32_t* D = g.D;
    const int64_t ldd = g.ldd;
    const int32_t* rows = g.d_rows;
    uint32_t* T = c.step(Ctx::kProduct, (size_t)g.M * g.N);
    if (!T) return GBGPU_ENOMEM;
    g.D = T;
    g.ldd = g.N;
    g.d_rows = nullptr;
    BL_CHECK(gemm_args(c, g));
    if (rows)
        BL_LAUNCH(k_scatter_rows_dense<<<grid_of((int64_t)g.M * g.N), 256, 0, c.s>>>(
            g.M, rows, g.N, T, g.N, D, ldd));
    else
        BL_CUDA(cudaMemcpy2DAsync(D, ldd * 4, T, (size_t)g.N * 4, (size_t)g.N * 4, g.M,
                                  cudaMemcpyDeviceToDevice, c.s));
    return GBGPU_OK;
}

// batch of `batch` products D_z <- -A_z B_z (element strides sA, sB, sD)
static int gemm_set_batched(Ctx& c, uint32_t* D, int64_t ldd, int64_t sD, const uint32_t* A,
                        int64_t lda, int64_t sA, const uint32_t* B, int64_t ldb, int64_t sB,
                        int32_t M, int32_t N, int32_t K, int32_t batch) {
    TcGemmArgs g{c.p, M, N, K, A, lda, B, ldb, D, ldd};
    g.set = true;
    g.batch = batch;
    g.sA = sA;
    g.sB = sB;
    g.sD = sD;
    return gemm_args(c, g);
}

template <int L, class F>
static int panel_apply(Ctx& c, const PanelApply& a, const F& f) {
    auto launch = [&](auto kernel, int kc) -> int {
        const int per_sm = pa_blocks(L, kc);
        const int bytes = L * 32 * kc * pa_row(kc);
        BL_CUDA(ensure_smem_limit((const void*)kernel, bytes));
        BL_LAUNCH(kernel<<<148 * per_sm, PA_THREADS, bytes, c.s>>>(a, f));
        return GBGPU_OK;
    };
    if (a.n_dirty > 1) {  // one alone is in the class of 128 (k_panel_factor)
        BL_CHECK(launch(k_panel_apply<L, 1, F>, 1));
        BL_CHECK(launch(k_panel_apply<L, 2, F>, 2));
    }
    BL_CHECK(launch(k_panel_apply<L, 4, F>, 4));
    return GBGPU_OK;
}

// elimination block size: powers of two from 128 to `cap` (1024 by default)
static int32_t nb_for(int64_t n, int32_t cap = 8 * KB) {
    int32_t nb = KB;
    while (nb < n && nb < cap) nb *= 2;
    return nb;
}

// -U^-1 for n_blocks unit upper triangular blocks of size NB (block b at
// src + b * stride_src, leading dimension lds; the last one last_nb x last_nb,
// identity-padded).  Result: out + b NB (NB + 1), leading dimension NB.  The
// 128 x 128 diagonal blocks are inverted by k_neg_inverse; blocks are then
// merged by doubling,  -[[A, B], [0, C]]^-1 = [[-A^-1, A^-1 B C^-1], [0, -C^-1]],
// with two batched GEMMs per level (the NB + 1 block stride makes the
// diagonal blocks of one level equally spaced across all big blocks).
template <class F>
static int neg_inverse_big(Ctx& c, const F& f, const uint32_t* src, int64_t lds,
                           int64_t stride_src, int32_t n_blocks, int32_t last_nb, int32_t NB,
                           uint32_t* out) {
    if (n_blocks <= 0) return GBGPU_OK;
    const int64_t bstride = (int64_t)NB * (NB + 1);
    uint32_t* U = c.step(Ctx::kU, (size_t)n_blocks * bstride);
    uint32_t* T = c.step(Ctx::kT, (size_t)n_blocks * NB * NB / 4 + 1);
    if (!U || !T) return GBGPU_ENOMEM;
    BL_LAUNCH(k_copy_blocks<<<grid_of((int64_t)n_blocks * NB * NB), 256, 0, c.s>>>(
        src, lds, stride_src, n_blocks, last_nb, NB, U));
    BL_CUDA(cudaMemsetAsync(out, 0, sizeof(uint32_t) * (size_t)n_blocks * bstride, c.s));
    BL_CUDA(ensure_smem_limit((const void*)k_neg_inverse<F>, INV_BYTES));
    const int32_t n_sub = n_blocks * (NB / KB);
    const int64_t dstep = (int64_t)KB * (NB + 1);  // between 128-blocks on the diagonal
    BL_LAUNCH(k_neg_inverse<F><<<n_sub, INV_THREADS, INV_BYTES, c.s>>>(U, NB, dstep, n_sub, KB, out,
                                                                   dstep, NB, f));
    for (int32_t sz = KB; sz < NB; sz *= 2) {
        const int32_t items = n_blocks * (NB / (2 * sz));
        const int64_t istep = (int64_t)2 * sz * (NB + 1);
        const int64_t half = (int64_t)sz * (NB + 1);
        // T = B C^-1 = -(B (-C^-1))
        BL_CHECK(gemm_set_batched(c, T, sz, (int64_t)sz * sz, U + sz, NB, istep, out + half, NB, istep,
                              sz, sz, sz, items));
        // top right of -U^-1 = A^-1 B C^-1 = -((-A^-1) T)
        BL_CHECK(gemm_set_batched(c, out + sz, NB, istep, out, NB, istep, T, sz, (int64_t)sz * sz, sz,
                              sz, sz, items));
    }
    return GBGPU_OK;
}

// out[k] = in[n - 1 - k]
__global__ void k_reverse_i32(int32_t n, const int32_t* __restrict__ in, int32_t* out) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
        out[k] = in[n - 1 - k];
}

// offs[k] = base + loc[k]
// *total = loc[n - 1], in mapped host memory: a copy would queue behind the
// answer's blocks on their way to the host (0.5 to 1 ms each), and the next block
// could not be sized before
__global__ void k_offs_write(int32_t n, const int64_t* __restrict__ loc, int64_t base,
                             int64_t* offs, int64_t* total) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        offs[k] = base + loc[k];
        if (k == n - 1) *total = loc[k];
    }
}

// Mapped host memory for one user at a time, from the pool of internal.h.
struct InfoPage {
    MappedPage p;
    cudaStream_t s;
    void *host = nullptr, *dev = nullptr;
    InfoPage(cudaStream_t s_, size_t bytes) : s(s_) {
        if (bytes <= kMappedPageBytes && mapped_page_take(&p) == cudaSuccess) {
            host = p.host;
            dev = p.dev;
        } else {
            set_error("mapped host page allocation failed");
        }
    }
    ~InfoPage() {
        cudaStreamSynchronize(s);  // an early return may leave a writer running
        mapped_page_return(p);
    }
};

// the columns of pivots 0, KB, 2 KB, ... (the last k_round_finish's)
static int first_columns(Ctx& c, const volatile RoundInfo* info, const int32_t* d_pc, int32_t n,
                         std::vector<int32_t>* out) {
    const int32_t nb = (n + KB - 1) / KB;
    out->resize((size_t)nb);
    if (nb <= kInfoFirst) {
        for (int32_t q = 0; q < nb; ++q) (*out)[q] = info->first[q];
        return GBGPU_OK;
    }
    BL_CUDA(cudaMemcpy2DAsync(out->data(), 4, d_pc, 4 * KB, 4, nb, cudaMemcpyDeviceToHost, c.s));
    BL_CUDA(cudaStreamSynchronize(c.s));
    return GBGPU_OK;
}

// Rows t_rows[0 .. rows) of M (leading dimension ld, ncols columns) are
// reduced by the pivot rows u_rows[0 .. n_p) of M (sorted by lead, monic,
// zero left of their leads, pivot columns d_pc ascending, h_first[q] = that of
// pivot q KB):
//   T <- T - T[:, pc] (U[:, pc])^-1 U,
// after which every T row is zero at every pivot column.  Blocks of NB
// pivots, left to right; the rows are read and written in place through the
// row lists (T and U rows are distinct).  With `unit`, U[:, pc] is the identity.
template <class F>
static int eliminate(Ctx& c, const F& f, uint32_t* M, int64_t ld, const int32_t* t_rows,
                     int32_t rows, int32_t ncols, const int32_t* u_rows, int32_t n_p,
                     const int32_t* d_pc, const std::vector<int32_t>& h_first, bool unit) {
    if (rows <= 0 || n_p <= 0) return GBGPU_OK;
    if (unit) {  // U[:, pc] is the identity (at most KB pivots): T -= T[:, pc] U
        uint32_t* G = c.step(Ctx::kGathered, (size_t)rows * KB);
        if (!G) return GBGPU_ENOMEM;
        const int32_t first_col = h_first[0] & ~3;
        BL_LAUNCH(k_gather_cols<<<grid_of((int64_t)rows * n_p), 256, 0, c.s>>>(rows, n_p, M, ld, d_pc,
                                                                              G, KB, t_rows));
        TcGemmArgs g{c.p, rows, ncols - first_col, n_p, G, KB, M + first_col, ld, M + first_col, ld};
        g.b_rows = u_rows;
        g.d_rows = t_rows;
        return gemm_args(c, g);
    }
    const int32_t NB = nb_for(n_p);
    const int32_t nb = (n_p + NB - 1) / NB;
    const int64_t bstride = (int64_t)NB * (NB + 1);
    uint32_t* Ublk = c.step(Ctx::kBlocks, (size_t)nb * NB * NB);  // U[:, pc] diagonal blocks
    uint32_t* Ninv = c.step(Ctx::kInverses, (size_t)nb * bstride);
    uint32_t* G = c.step(Ctx::kGathered, (size_t)rows * NB);      // T[:, pc_k]
    uint32_t* X = c.step(Ctx::kSolved, (size_t)rows * NB);
    if (!Ublk || !Ninv || !G || !X) return GBGPU_ENOMEM;
    for (int b = 0; b < nb; ++b) {
        const int kb = std::min(NB, n_p - b * NB);
        BL_LAUNCH(k_gather_cols<<<grid_of((int64_t)kb * kb), 256, 0, c.s>>>(
            kb, kb, M, ld, d_pc + b * NB, Ublk + (size_t)b * NB * NB, NB, u_rows + b * NB));
    }
    BL_CHECK(neg_inverse_big(c, f, Ublk, NB, (int64_t)NB * NB, nb, n_p - (nb - 1) * NB, NB, Ninv));
    for (int b = 0; b < nb; ++b) {
        const int kb = std::min(NB, n_p - b * NB);
        // from the block's first pivot column, or up to three left of it for the
        // GEMM's 16-byte accesses (the pivot rows are zero there)
        const int32_t first_col = h_first[b * (NB / KB)] & ~3;
        BL_LAUNCH(k_gather_cols<<<grid_of((int64_t)rows * kb), 256, 0, c.s>>>(
            rows, kb, M, ld, d_pc + b * NB, G, NB, t_rows));
        // X = G * (U_kk)^-1 = -(G * (-(U_kk)^-1))
        TcGemmArgs x{c.p, rows, kb, kb, G, NB, Ninv + (size_t)b * bstride, NB, X, NB};
        x.set = true;
        BL_CHECK(gemm_args(c, x));
        // T[:, first_col:] -= X * U_k[:, first_col:]
        TcGemmArgs g{c.p, rows, ncols - first_col, kb, X, NB, M + first_col, ld, M + first_col, ld};
        g.b_rows = u_rows + b * NB;
        g.d_rows = t_rows;
        BL_CHECK(gemm_args(c, g));
    }
    return GBGPU_OK;
}

// ---------------------------------------------------------------------------
template <class F>
static int echelon_rref(Ctx& c, const F& f, uint32_t* Dp, int64_t ld, int32_t t, int32_t ncr,
                        BlockedOutput* out);

template <class F>
static int blocked_run(const BlockedInput& in, BlockedOutput* out, Ctx& c, const F& f) {
    const int32_t ncl = in.ncl, ncr = in.ncr, nc = ncl + ncr, t = in.n_work;
    // the right block starts on a 16-byte boundary (the GEMM's wide accesses of D)
    const int32_t pad = -ncl & 3, nclp = ncl + pad;
    const int64_t ld = ((int64_t)nc + pad + 3) & ~(int64_t)3;
    cudaStream_t s = c.s;

    // ---- 1. Schur complement ---------------------------------------------------
    // C|D rows sorted by lead (stable), dense
    int32_t* lead_in = c.alloc<int32_t>(t);
    int32_t* lead_sorted = c.alloc<int32_t>(t);
    int32_t* work_sorted = c.alloc<int32_t>(t);
    uint32_t* W = c.alloc<uint32_t>((size_t)t * ld);
    if (!lead_in || !lead_sorted || !work_sorted || !W) return GBGPU_ENOMEM;
    if (t > 0) {
        BL_LAUNCH(k_csr_leads<<<grid_of(t), 256, 0, s>>>(t, in.work, in.row_ptr, in.cols, lead_in));
        size_t bytes = 0;
        cub::DeviceRadixSort::SortPairs(nullptr, bytes, lead_in, lead_sorted, in.work, work_sorted,
                                        t, 0, 32, s);
        void* tmp = c.alloc<uint8_t>(bytes);
        if (!tmp) return GBGPU_ENOMEM;
        BL_CUDA(cub::DeviceRadixSort::SortPairs(tmp, bytes, lead_in, lead_sorted, in.work,
                                                work_sorted, t, 0, 32, s));
        ++c.launches;
        BL_CUDA(ensure_smem_limit((const void*)k_densify_seg, DS_COLS * 4));
        BL_LAUNCH(k_densify_seg<<<std::min(t, 148 * 3), 512, DS_COLS * 4, s>>>(
            t, work_sorted, in.row_ptr, in.cols, in.vals, nc, ncl, pad, 0, W, ld));
    }
    if (t > 0 && ncl > 0) {
        const int32_t NB = nb_for(ncl, 16 * KB);
        const int64_t bstride = (int64_t)NB * (NB + 1);
        uint32_t* P = c.alloc<uint32_t>((size_t)ncl * ld);
        const int32_t nbk = (ncl + NB - 1) / NB;
        uint32_t* Ninv = c.alloc<uint32_t>((size_t)nbk * bstride);
        int32_t* act = c.alloc<int32_t>(nbk);
        int32_t* span = c.alloc<int32_t>(nbk);
        const int32_t ngrp = (ncl + 127) / 128;
        int2* brange = c.alloc<int2>(ngrp);
        if (!P || !Ninv || !act || !span || !brange) return GBGPU_ENOMEM;
        // active rows of each block (rows sorted by lead), the last left
        // column the known pivots of each block touch, and the right columns
        // every 128 known pivots reach
        BL_LAUNCH(k_count_below<<<grid_of(nbk), 256, 0, s>>>(t, lead_sorted, nbk, NB, act));
        BL_LAUNCH(k_fill_i32<<<grid_of(nbk), 256, 0, s>>>(span, nbk, -1));
        BL_LAUNCH(k_clear_ranges<<<grid_of(ngrp), 256, 0, s>>>(ngrp, brange));
        BL_LAUNCH(k_block_span<<<grid_of((int64_t)ncl * 32), 256, 0, s>>>(
            ncl, in.piv_row, in.row_ptr, in.cols, ncl, NB, span, brange));
        // pivot row of lead c into row c of P: on the tensor cores only the
        // parts a later step reads (its diagonal block, the left columns its
        // block reaches, the right columns its group of 128 reaches); the
        // CUDA-core GEMM reads B whole, so there P gets everything from the
        // diagonal block on
        const bool banded = c.form != GBGPU_FORM_PLAIN;
        BL_LAUNCH(k_densify_direct<<<std::min(ncl, 148 * 8), DS_THREADS, 0, s>>>(
            ncl, in.piv_row, in.row_ptr, in.cols, in.vals, nc, ncl, pad, NB, P, ld, span,
            banded ? brange : nullptr));
        // -A_kk^-1 of every NB x NB diagonal block of A (read in place from P)
        BL_CHECK(neg_inverse_big(c, f, P, ld, (int64_t)NB * ld + NB, nbk, ncl - (nbk - 1) * NB, NB,
                                 Ninv));
        std::vector<int32_t> h_act(nbk), h_span(nbk);
        BL_CUDA(cudaMemcpyAsync(h_act.data(), act, sizeof(int32_t) * nbk, cudaMemcpyDeviceToHost, s));
        BL_CUDA(cudaMemcpyAsync(h_span.data(), span, sizeof(int32_t) * nbk, cudaMemcpyDeviceToHost, s));
        BL_CUDA(cudaStreamSynchronize(s));
        // (a) X = C A^-1, in place in W[:, 0:ncl], block by block; the update of
        //     the later left columns stops at the last column block k touches
        for (int k = 0; k < nbk; ++k) {
            const int32_t c0 = k * NB, kb = std::min(NB, ncl - c0), c1 = c0 + kb;
            const int32_t rows = h_act[k];
            if (rows <= 0) continue;
            // X_k = W[:, block] A_kk^-1
            TcGemmArgs x{c.p, rows, kb, kb, W + c0, ld, Ninv + (size_t)k * bstride, NB, W + c0, ld};
            BL_CHECK(gemm_set_in_place(c, x));
            // W[:, c1:e) -= X_k A[block rows, c1:e)
            const int32_t e = std::min(ncl, h_span[k] + 1);
            if (e > c1)
                BL_CHECK(gemm(c, W + c1, ld, W + c0, ld, P + (size_t)c0 * ld + c1, ld, rows, e - c1,
                              kb));
        }
        // (b) D' = D - X B: one GEMM over the whole left block; the tile flags of
        //     the GEMM skip the zero tiles of the staircase X and of B
        {
            TcGemmArgs g{c.p, t, ncr, ncl, W, ld, P + nclp, ld, W + nclp, ld};
            if (banded) g.b_nrange = brange;  // B is zero outside these columns
            BL_CHECK(gemm_args(c, g));
        }
    }
    if (out->ms_event_schur) BL_CUDA(cudaEventRecord(out->ms_event_schur, s));
    BL_CHECK(echelon_rref(c, f, W + nclp, ld, t, ncr, out));
    out->rows = W + nclp;
    out->ld = ld;
    return GBGPU_OK;
}

// Step 3: the r echelon rows rs.prow of Dp (ascending lead, pivot columns rs.pc,
// h_first[q] = that of pivot q KB) to reduced echelon form, in place.  info: the
// host's view of rs.info.
template <class F>
static int back_substitute(Ctx& c, const F& f, uint32_t* Dp, int64_t ld, int32_t ncr, int32_t r,
                           const RoundState& rs, const volatile RoundInfo* info,
                           const std::vector<int32_t>& h_first, BlockedOutput* out) {
    cudaStream_t s = c.s;
    const int32_t *pc = rs.pc, *prow = rs.prow;
    const int32_t* piv_of_col = out->piv_of_col;
    StreamOut* so = out->stream_out;
    int32_t* pcd = nullptr;          // pivot columns, descending (the answer's order)
    int64_t* cnt = nullptr;          // [NB + 1] entries per row of a block
    int64_t* loc = nullptr;          // [NB + 1] their exclusive scan
    void* cscan = nullptr;
    size_t cscan_bytes = 0;
    cudaEvent_t blk_ev = nullptr;
    if (so) {
        pcd = c.alloc<int32_t>(r);
        cnt = c.alloc<int64_t>(nb_for(r) + 1);
        loc = c.alloc<int64_t>(nb_for(r) + 1);
        cub::DeviceScan::ExclusiveSum(nullptr, cscan_bytes, cnt, loc, nb_for(r) + 1, s);
        cscan = c.alloc<uint8_t>(cscan_bytes);
        if (!pcd || !cnt || !loc || !cscan) return GBGPU_ENOMEM;
        BL_LAUNCH(k_reverse_i32<<<grid_of(r), 256, 0, s>>>(r, pc, pcd));
        BL_CUDA(cudaEventCreateWithFlags(&blk_ev, cudaEventDisableTiming));
        so->nnz = 0;
        so->overflow = false;
    }
    // block b's answer rows [r - b NB - kb, r - b NB): compacted and sent
    auto send_block = [&](int b, int kb) -> int {
        const int64_t out0 = (int64_t)r - ((int64_t)b * nb_for(r) + kb);
        BL_LAUNCH(k_row_nnz<<<grid_of((int64_t)kb * 32), 256, 0, s>>>(
            kb, pcd + out0, piv_of_col, Dp, ld, ncr, cnt));
        BL_CUDA(cudaMemsetAsync(cnt + kb, 0, sizeof(int64_t), s));
        size_t bytes = cscan_bytes;
        BL_CUDA(cub::DeviceScan::ExclusiveSum(cscan, bytes, cnt, loc, kb + 1, s));
        ++c.launches;
        BL_LAUNCH(k_offs_write<<<grid_of(kb + 1), 256, 0, s>>>(kb + 1, loc, so->nnz,
                                                               so->offs + out0, &rs.info->entries));
        BL_CUDA(cudaStreamSynchronize(s));
        const int64_t blk = info->entries;
        if (blk > 0) {
            int32_t* bc = nullptr;
            uint8_t* bw = nullptr;
            const int vb = so->val_bytes;
            if (cudaMallocAsync((void**)&bc, sizeof(int32_t) * blk, s) != cudaSuccess ||
                cudaMallocAsync((void**)&bw, (size_t)vb * blk, s) != cudaSuccess) {
                set_error("answer block allocation failed");
                return GBGPU_ENOMEM;
            }
            BL_LAUNCH(k_row_write<<<grid_of((int64_t)kb * 32), 256, 0, s>>>(
                kb, pcd + out0, piv_of_col, Dp, ld, ncr, loc, so->col_shift, bc, bw, vb));
            cudaStream_t fs = s;
            if (!so->overflow && so->nnz + blk <= so->cap_nnz) {
                BL_CUDA(cudaEventRecord(blk_ev, s));
                BL_CUDA(cudaStreamWaitEvent(so->s_out, blk_ev, 0));
                BL_CUDA(cudaMemcpyAsync(so->h_cols + so->nnz, bc, sizeof(int32_t) * blk,
                                        cudaMemcpyDeviceToHost, so->s_out));
                BL_CUDA(cudaMemcpyAsync((uint8_t*)so->h_vals + (size_t)so->nnz * vb, bw,
                                        (size_t)vb * blk, cudaMemcpyDeviceToHost, so->s_out));
                fs = so->s_out;  // freed once copied
            } else {
                so->overflow = true;
            }
            cudaFreeAsync(bc, fs);
            cudaFreeAsync(bw, fs);
        }
        so->nnz += blk;
        return GBGPU_OK;
    };
    const int32_t NB = nb_for(r);
    const int64_t bstride = (int64_t)NB * (NB + 1);
    const int32_t nb = (r + NB - 1) / NB;
    uint32_t* Ublk = c.alloc<uint32_t>((size_t)nb * NB * NB);
    uint32_t* Ninv = c.alloc<uint32_t>((size_t)nb * bstride);
    uint32_t* G = c.alloc<uint32_t>((size_t)NB * std::max(r, 1));
    if (!Ublk || !Ninv || !G) return GBGPU_ENOMEM;
    for (int b = 0; b < nb; ++b) {
        const int kb = std::min(NB, r - b * NB);
        BL_LAUNCH(k_gather_cols<<<grid_of((int64_t)kb * kb), 256, 0, s>>>(
            kb, kb, Dp, ld, pc + b * NB, Ublk + (size_t)b * NB * NB, NB, prow + b * NB));
    }
    BL_CHECK(neg_inverse_big(c, f, Ublk, NB, (int64_t)NB * NB, nb, r - (nb - 1) * NB, NB, Ninv));
    for (int b = nb - 1; b >= 0; --b) {
        const int kb = std::min(NB, r - b * NB);
        const int32_t later = r - (b * NB + kb);
        const int32_t* rows_k = prow + b * NB;
        const int32_t c0 = h_first[b * (NB / KB)] & ~3;  // zero left of the pivot column, as below
        if (later > 0) {
            // E_k -= E_k[:, pc(>k)] R(>k)
            BL_LAUNCH(k_gather_cols<<<grid_of((int64_t)kb * later), 256, 0, s>>>(
                kb, later, Dp, ld, pc + b * NB + kb, G, later, rows_k));
            const int32_t c_later = h_first[(b + 1) * (NB / KB)] & ~3;
            TcGemmArgs g{c.p, kb, ncr - c_later, later, G, later, Dp + c_later, ld,
                         Dp + c_later, ld};
            g.b_rows = rows_k + kb;
            g.d_rows = rows_k;
            BL_CHECK(gemm_args(c, g));
        }
        // E_k = (E_k[:, pc(k)])^-1 E_k = -((-(U_kk)^-1) E_k), in place
        TcGemmArgs g{c.p, kb, ncr - c0, kb, Ninv + (size_t)b * bstride, NB, Dp + c0, ld, Dp + c0,
                     ld};
        g.b_rows = rows_k;
        g.d_rows = rows_k;
        BL_CHECK(gemm_set_in_place(c, g));
        if (so) BL_CHECK(send_block(b, kb));
    }
    if (blk_ev) cudaEventDestroy(blk_ev);
    return GBGPU_OK;
}

// Steps 2 and 3 on the dense t x ncr residue matrix Dp (leading dimension
// ld), in place: afterwards out->piv_of_col[c] is the row of Dp holding the
// reduced pivot row of column c (-1 for non-pivot columns), out->rank is the
// rank, and every other row's content is unspecified.
template <class F>
static int echelon_rref(Ctx& c, const F& f, uint32_t* Dp, int64_t ld, int32_t t, int32_t ncr,
                        BlockedOutput* out) {
    cudaStream_t s = c.s;
    // ---- 2. echelon of D' = W[:, ncl:] by rounds ----------------------------------
    // Every round looks at all pending rows (nonzero, not yet pivots) at once:
    //  * a 128-column panel in which no two pending rows share a lead is
    //    "clean": each of its rows has a lead of its own and becomes a pivot;
    //  * every other ("dirty") panel gets up to PR of its pending rows
    //    factorized in shared memory (k_panel_factor, one cluster per panel); the
    //    recorded transformation F of its pivot rows is applied to their
    //    trailing columns (k_panel_apply);
    //  * the pending rows that did not become pivots are eliminated against
    //    all pivots of the round (eliminate), which leaves them zero at every
    //    pivot column, and the next round starts from their new leads.
    const int32_t npan = (ncr + KB - 1) / KB;
    int32_t* lead = c.alloc<int32_t>(t);
    uint8_t* is_piv = c.alloc<uint8_t>(t);
    int32_t* piv_of_col = out->piv_of_col;  // [ncr], -1 if none
    int32_t* counters = c.alloc<int32_t>(8);
    // every dirty panel is factorized in the round that finds it (batch <= 4096)
    const int32_t max_dirty = std::max<int32_t>(1, std::min<int32_t>(npan, 4096));
    RoundState rs{};
    rs.t = t;
    rs.ncr = ncr;
    rs.npan = npan;
    rs.max_dirty = max_dirty;
    rs.lead = lead;
    rs.is_piv = is_piv;
    rs.piv_of_col = piv_of_col;
    rs.wflag = c.alloc<int32_t>(ncr);
    rs.hist = c.alloc<int32_t>(ncr);
    rs.pdirty = c.alloc<int32_t>(npan);
    rs.dslot = c.alloc<int32_t>(npan);
    rs.dpanel = c.alloc<int32_t>(max_dirty);
    rs.cursor = c.alloc<int32_t>(max_dirty);
    rs.chunk_rows = c.alloc<int32_t>((size_t)max_dirty * PR);
    rs.per_warp = c.alloc<int32_t>((size_t)RD_WARPS * max_dirty);
    rs.pc = c.alloc<int32_t>(ncr);    // pivot columns
    rs.prow = c.alloc<int32_t>(ncr);  // their rows
    rs.pend = c.alloc<int32_t>(t);
    rs.n_new = counters;
    rs.cls = c.alloc<int32_t>(PA_CLASSES * (1 + (size_t)max_dirty));
    int32_t *pc = rs.pc, *prow = rs.prow, *pend = rs.pend;
    uint32_t* panF = c.alloc<uint32_t>((size_t)max_dirty * KB * KB);
    int32_t* n_piv = c.alloc<int32_t>(max_dirty);
    int32_t* piv_rows = c.alloc<int32_t>((size_t)max_dirty * KB);
    if (!lead || !is_piv || !counters || !rs.wflag || !rs.hist || !rs.pdirty || !rs.dslot ||
        !rs.dpanel || !rs.cursor || !rs.chunk_rows || !rs.per_warp || !rs.cls || !pc || !prow || !pend ||
        !panF || !n_piv || !piv_rows)
        return GBGPU_ENOMEM;
    // the counts the host sizes launches from
    InfoPage page(s, sizeof(RoundInfo));
    const volatile RoundInfo* info = (const volatile RoundInfo*)page.host;
    rs.info = (RoundInfo*)page.dev;
    if (!info) return GBGPU_ENOMEM;
    BL_LAUNCH(k_fill_i32<<<grid_of(ncr), 256, 0, s>>>(piv_of_col, ncr, -1));
    if (t > 0 && ncr > 0) {
        BL_CUDA(cudaMemsetAsync(is_piv, 0, t, s));
        BL_LAUNCH(k_row_leads<<<grid_of((int64_t)t * 32), 256, 0, s>>>(t, nullptr, ncr, Dp, ld, lead));
    }
    int rounds = 0;
    bool first = true;
    while (t > 0 && ncr > 0) {
        // pending rows, clean panels claimed, the dirty panels and their chunks
        BL_LAUNCH(k_round_plan<<<1, RD_THREADS, 0, s>>>(rs, KB, PR));
        BL_CUDA(cudaStreamSynchronize(s));
        const int32_t n_pend = info->n_pend, n_dirty = info->n_dirty, n_clean = info->n_clean;
        if (first) out->dense_rows = n_pend;
        first = false;
        if (n_pend == 0) break;
        ++rounds;
        if (n_dirty > 0) {
            const int32_t j0 = info->first_panel * KB, width = ncr - j0;
            {
                // CTAs per panel: as many as leave every panel its own SMs
                int cl = kTinyMaxCluster;
                while (cl > 1 && n_dirty * cl > 148) cl /= 2;
                // many panels: the longest one sets the round's time
                int32_t nc_ = ncr, rows_ = cl == 1 ? KB : PR;
                int64_t ld_ = ld;
                F fv = f;
                void* args[] = {&Dp, &ld_, &rs.chunk_rows, &rs.dpanel, &rs.cursor, &rows_, &nc_, &panF,
                                &piv_rows, &n_piv, &piv_of_col, &is_piv, &rs.wflag, &rs.cls, &fv};
                BL_LAUNCH(BL_CUDA(launch_cluster((const void*)k_panel_factor<F>, n_dirty * cl, cl,
                                                 kTinyThreads,
                                                 (int)tiny_layout(rows_, KB, cl).words * 4, s, args)));
            }
            // pivot rows of every chunk <- F_d old, in place, columns j0..; one chunk
            // alone needs the narrow items to fill the SMs
            const PanelApply pa{Dp, ld, ncr, j0, n_dirty == 1 ? 128 : 512, n_dirty, rs.cls, rs.dpanel,
                                n_piv, piv_rows, panF};
            if constexpr (std::is_same<F, FieldSmall>::value)
                BL_CHECK(c.p < 256u ? panel_apply<1>(c, pa, f) : panel_apply<2>(c, pa, f));
            else
                BL_CHECK(panel_apply<4>(c, pa, f));
            if (trace_rounds()) {
                std::vector<int32_t> h_cur(n_dirty), h_np(n_dirty);
                BL_CUDA(cudaMemcpyAsync(h_cur.data(), rs.cursor, 4 * n_dirty, cudaMemcpyDeviceToHost, s));
                BL_CUDA(cudaMemcpyAsync(h_np.data(), n_piv, 4 * n_dirty, cudaMemcpyDeviceToHost, s));
                BL_CUDA(cudaStreamSynchronize(s));
                long long rows_in = 0, piv = 0;
                int mx = 0;
                for (int q = 0; q < n_dirty; ++q) {
                    rows_in += std::min(h_cur[q], PR);
                    piv += h_np[q];
                    mx = std::max(mx, h_cur[q]);
                }
                fprintf(stderr,
                        "gbgpu echelon round %d: pending %d, dirty panels %d (first %d), chunk rows "
                        "%lld (max %d), chunk pivots %lld\n",
                        rounds, n_pend, n_dirty, j0 / KB, rows_in, mx, piv);
            }
        }
        // all pivots of the round, ascending columns, and the rows left; the
        // panels' pivots are normalised already
        //
        // One panel alone: its pivot rows are reduced among themselves already, and
        // the elimination is one product over at most KB pivots and n_pend rows, so
        // the host does not wait for the counts (dense RREF of 48 rounds: 14.3 -> 14.1 ms).
        const bool unit = n_dirty == 1 && n_clean == 0;
        BL_LAUNCH(k_round_finish<<<1, RD_THREADS, 0, s>>>(rs, KB, 0, unit ? n_pend : 0));
        int32_t n_new = std::min(KB, ncr), n_rest = n_pend;
        std::vector<int32_t> h_first;
        if (unit) {
            h_first.assign(1, info->first_panel * KB);  // zero left of the panel
        } else {
            if (n_clean > 0)
                BL_LAUNCH(k_normalize_at<F><<<std::min(t, 148 * 8), 256, 0, s>>>(counters, prow, pc, ncr,
                                                                                 Dp, ld, f));
            BL_CUDA(cudaStreamSynchronize(s));
            n_new = info->n_new;
            n_rest = info->n_rest;
            if (trace_rounds())
                fprintf(stderr, "gbgpu echelon round %d: new pivots %d\n", rounds, n_new);
            if (n_rest == 0) break;
            // the first pivot column of every block of KB pivots
            BL_CHECK(first_columns(c, info, pc, n_new, &h_first));
        }
        BL_CHECK(eliminate(c, f, Dp, ld, pend, n_rest, ncr, prow, n_new, pc, h_first, unit));
        BL_LAUNCH(k_row_leads<<<grid_of((int64_t)n_rest * 32), 256, 0, s>>>(n_rest, pend, ncr, Dp,
                                                                             ld, lead, 1));
    }
    const int steps = rounds;
    out->echelon_rounds = steps;
    if (out->ms_event_echelon) BL_CUDA(cudaEventRecord(out->ms_event_echelon, s));

    // ---- 3. back substitution --------------------------------------------------
    // all pivots in ascending column order
    BL_LAUNCH(k_round_finish<<<1, RD_THREADS, 0, s>>>(rs, KB, 1));
    BL_CUDA(cudaStreamSynchronize(s));
    const int32_t r = info->n_new;
    out->rank = r;
    out->pivot_cols = pc;
    out->pivot_rows = prow;
    if (r > 0) {
        std::vector<int32_t> h_first;
        BL_CHECK(first_columns(c, info, pc, r, &h_first));
        BL_CHECK(back_substitute(c, f, Dp, ld, ncr, r, rs, info, h_first, out));
    } else if (out->stream_out) {
        out->stream_out->nnz = 0;
        BL_CUDA(cudaMemsetAsync(out->stream_out->offs, 0, sizeof(int64_t), s));
    }
    return GBGPU_OK;
}

// Rows with distinct leads, every one reduced by all others (dense: blocked.h).
template <class F>
static int interreduce_run(const InterreduceInput& in, Ctx& c, const F& f) {
    cudaStream_t s = c.s;
    BL_CUDA(ensure_smem_limit((const void*)k_densify_seg, DS_COLS * 4));
    BL_LAUNCH(k_densify_seg<<<std::min(in.rows, 148 * 3), 512, DS_COLS * 4, s>>>(
        in.rows, nullptr, in.row_ptr, in.cols, in.vals, in.ncols, in.ncols, 0, 0, in.D, in.ld));
    RoundState rs{};
    rs.ncr = in.ncols;
    rs.piv_of_col = in.piv_of_col;
    rs.pc = c.alloc<int32_t>(in.ncols);
    rs.prow = c.alloc<int32_t>(in.ncols);
    rs.n_new = c.alloc<int32_t>(1);
    if (!rs.pc || !rs.prow || !rs.n_new) return GBGPU_ENOMEM;
    InfoPage page(s, sizeof(RoundInfo));
    const volatile RoundInfo* info = (const volatile RoundInfo*)page.host;
    rs.info = (RoundInfo*)page.dev;
    if (!info) return GBGPU_ENOMEM;
    BL_LAUNCH(k_round_finish<<<1, RD_THREADS, 0, s>>>(rs, KB, 1));
    BL_CUDA(cudaStreamSynchronize(s));
    std::vector<int32_t> h_first;
    BL_CHECK(first_columns(c, info, rs.pc, in.rows, &h_first));
    BlockedOutput out{};
    out.piv_of_col = in.piv_of_col;
    return back_substitute(c, f, in.D, in.ld, in.ncols, in.rows, rs, info, h_first, &out);
}

int interreduce_dense(const InterreduceInput& in, BlockedOutput* out, long long* launches) {
    Ctx c;
    c.s = in.stream;
    c.p = in.p;
    c.form = in.form;
    c.err = in.err;
    int rc;
    if (in.p < 65536u)
        rc = interreduce_run(in, c, FieldSmall::make(in.p));
    else
        rc = interreduce_run(in, c, FieldMont::make(in.p));
    *launches += c.launches;
    out->keep = c.hand_over();
    return rc;
}

int blocked_reduce(const BlockedInput& in, BlockedOutput* out, long long* launches) {
    Ctx c;
    c.s = in.stream;
    c.p = in.p;
    c.form = in.form;
    c.err = in.err;
    int rc;
    if (in.p < 65536u)
        rc = blocked_run(in, out, c, FieldSmall::make(in.p));
    else
        rc = blocked_run(in, out, c, FieldMont::make(in.p));
    *launches += c.launches;
    out->keep = c.hand_over();
    return rc;
}

// dst row i = src row order[i] (all ncols), rows >= n zeroed up to `rows`
__global__ void k_order_rows(int32_t n, int32_t rows, const int32_t* __restrict__ order,
                             int32_t ncols, const uint32_t* __restrict__ src, int64_t lds,
                             uint32_t* dst, int64_t ldd) {
    const int64_t total = (int64_t)rows * ncols;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = t / ncols;
        const int j = (int)(t % ncols);
        dst[i * ldd + j] = i < n ? src[(int64_t)order[i] * lds + j] : 0u;
    }
}

template <class F>
static int dense_rref_run(const DenseRrefInput& in, int32_t* rank, Ctx& c, const F& f) {
    BlockedOutput out{};
    int32_t* piv_of_col = c.alloc<int32_t>(in.cols);
    if (!piv_of_col) return GBGPU_ENOMEM;
    out.piv_of_col = piv_of_col;
    BL_CHECK(echelon_rref(c, f, in.D, in.ld, in.rows, in.cols, &out));
    const int32_t r = (int32_t)out.rank;
    *rank = r;
    // pivot rows in ascending pivot order into the first r rows, zeros after
    uint32_t* tmp = c.alloc<uint32_t>((size_t)in.rows * in.ld);
    if (!tmp) return GBGPU_ENOMEM;
    if (r > 0)
        BL_CUDA(cudaMemcpyAsync(in.piv_cols, out.pivot_cols, sizeof(int32_t) * (size_t)r,
                                cudaMemcpyDeviceToDevice, c.s));
    BL_LAUNCH(k_order_rows<<<grid_of((int64_t)in.rows * in.cols), 256, 0, c.s>>>(
        r, in.rows, out.pivot_rows, in.cols, in.D, in.ld, tmp, in.ld));
    BL_CUDA(cudaMemcpy2DAsync(in.D, in.ld * 4, tmp, in.ld * 4, (size_t)in.cols * 4, in.rows,
                              cudaMemcpyDeviceToDevice, c.s));
    return GBGPU_OK;
}

int dense_rref(const DenseRrefInput& in, int32_t* rank, long long* launches) {
    Ctx c;
    c.s = in.stream;
    c.p = in.p;
    c.form = in.form;
    c.err = in.err;
    int rc;
    if (in.p < 65536u)
        rc = dense_rref_run(in, rank, c, FieldSmall::make(in.p));
    else
        rc = dense_rref_run(in, rank, c, FieldMont::make(in.p));
    *launches += c.launches;
    c.release();
    return rc;
}

void blocked_release(BlockedOutput* out, cudaStream_t s) {
    if (!out->keep) return;
    cudaStreamSynchronize(s);
    pool_free(out->keep->data(), out->keep->size());
    delete out->keep;
    out->keep = nullptr;
}

}  // namespace gbgpu
