// small.cu -- one-launch reduction of small Macaulay matrices (the la calls of
// the early F4 rounds, of small systems and of their prime images), built for
// latency.
//
// A general plan (api.cu) creates a stream, allocates a dozen buffers, runs
// ten or more launches and copies in and out through pageable memory; for a
// matrix of a few hundred rows that overhead is most of the call.  Here every
// host thread keeps one session per device (a stream, a device arena, pinned
// input staging and mapped pinned output memory, all grown to a high-water
// mark and reused), and a call is
//
//   rows gathered into pinned staging  ->  one host-to-device copy
//   k_small   one thread-block cluster: input checks, known pivots and the
//             C|D row list; a warp per C|D row reduces it by the known pivots
//             (src/la_ff_16.c:289-351 / :102-190) in shared memory; the reduced
//             echelon form of the right block and its compaction (tiny.cuh),
//             written straight into mapped host memory with the checks' verdict
//   one stream synchronisation.
//
// Measured on a B200, 441 x 491 matrix (141 x 191 block, p = 32003): 1425 us a
// call with one CTA for the echelon and a launch per phase, 220 us now, of it
// k_small 181 us (checks and diagonal blocks 22, rows 75, echelon 84; all three
// are chains of dependent steps on a few SMs, not throughput).  Matrices with more
// rows or a longer chain of left columns run the three phases as launches of their
// own, the rows on the whole device (kWideRows below).
//
// A batch's small matrices share one launch: the clusters take matrices from a
// work queue.  The answer is the canonical one of every other path (descending
// leads, monic, columns ascending).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/gbgpu.h"
#include "common.cuh"
#include "internal.h"
#include "kernels.h"
#include "small.h"
#include "tiny.cuh"

namespace gbgpu {

// Left columns.  The row phase adds a product per known pivot to a sum before it
// reduces it, so the field's bound on such sums is one on the left columns.
constexpr int kSmallMaxLeft = 12288;
static_assert(kSmallMaxLeft < FieldSmall::kLazyTerms, "sums of the row phase");
constexpr int LB = 32;                // left columns of a diagonal block (one per lane)

struct SmallItem {
    int32_t p, nr, ncl, ncr;
    int64_t in_off, cols_off, vals_off;  // bytes into the input buffer
    int64_t scr_off;                     // bytes into the scratch buffer
    int64_t out_off;                     // bytes into the mapped output
    FieldSmall fs;
    FieldMont fm;
};

__host__ __device__ inline int64_t rup(int64_t x, int64_t a) { return (x + a - 1) / a * a; }
// scratch of one matrix: pivot row of every left column [ncl] | its entries'
// extent [ncl] | C|D rows [nr] | checks' verdict, then the missing pivots' bit
// while the checks run | diagonal blocks [ncl][LB]
// | dense rows [n_work][ncr] of the three-launch form
struct ScrLayout {
    int64_t piv, pext, work, err, diag, D, bytes;
};
__host__ __device__ inline ScrLayout scr_layout(int32_t nr, int32_t ncl, int64_t dense = 0) {
    ScrLayout L;
    const int64_t n = ncl > 0 ? ncl : 1;
    L.piv = 0;
    L.pext = rup(4 * n, 256);
    L.work = L.pext + rup(8 * n, 256);
    L.err = L.work + rup(4 * (int64_t)nr, 256);
    L.diag = L.err + 256;
    L.D = rup(L.diag + 4 * LB * n, 256);
    L.bytes = rup(L.D + 4 * dense, 256);
    return L;
}
// mapped output of one matrix: rows, entries, verdict | offs [n_work + 1] | cols | vals
struct OutLayout {
    int64_t offs, cols, vals, bytes;
};
__host__ __device__ inline OutLayout out_layout(int32_t nr, int32_t ncl, int32_t ncr) {
    OutLayout L;
    const int64_t nw = nr - ncl > 0 ? nr - ncl : 0;
    const int64_t cap = nw * (ncr > 0 ? ncr : 0);
    L.offs = 32;
    L.cols = rup(L.offs + 8 * (nw + 1), 16);
    L.vals = rup(L.cols + 4 * (cap > 0 ? cap : 1), 16);
    L.bytes = rup(L.vals + 4 * (cap > 0 ? cap : 1), 256);
    return L;
}

// ---------------------------------------------------------------------------
// kernel phases

struct SmallMat {
    int32_t p, nr, ncl, nc;
    const int64_t* row_ptr;
    const int32_t* cols;
    const uint32_t* vals;
    int32_t* piv_row;
    int2* pext;
    int32_t* work;
    uint32_t* err;
    uint32_t* diag;
};

__host__ __device__ inline SmallMat small_mat(const SmallItem& it, const uint8_t* in,
                                               uint8_t* scr) {
    uint8_t* sb = scr + it.scr_off;
    const ScrLayout S = scr_layout(it.nr, it.ncl);
    return SmallMat{it.p,
                    it.nr,
                    it.ncl,
                    it.ncl + it.ncr,
                    (const int64_t*)(in + it.in_off),
                    (const int32_t*)(in + it.cols_off),
                    (const uint32_t*)(in + it.vals_off),
                    (int32_t*)(sb + S.piv),
                    (int2*)(sb + S.pext),
                    (int32_t*)(sb + S.work),
                    (uint32_t*)(sb + S.err),
                    (uint32_t*)(sb + S.diag)};
}

// Input checks (the contract k_check_rows enforces), the known pivot of every
// left column (first row with that lead, src/la_ff_16.c:762-772), the check
// that every left column has one, the C|D rows in row order, and, for the row
// phase, every pivot row's extent and the negated inverse of every LB x LB
// diagonal block of the known pivots (prep form).  Spread over the cluster;
// ends with the verdict.
template <class F>
__device__ uint32_t small_prep(const SmallMat& a, uint32_t* smem, int smem_words, const F f) {
    __shared__ int s_part[kTinyWarps];
    const int CL = cluster_size(), rk = cluster_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gw = rk * kTinyWarps + warp, ngw = CL * kTinyWarps;
    for (int c = rk * kTinyThreads + tid; c < a.ncl; c += CL * kTinyThreads) a.piv_row[c] = INT_MAX;
    if (rk == 0 && tid == 0) a.err[0] = a.err[1] = 0;
    cluster_sync();
    for (int i = gw; i < a.nr; i += ngw) {
        const int64_t b = a.row_ptr[i], e = a.row_ptr[i + 1];
        uint32_t bad = 0;
        if (e <= b) {
            bad |= kErrEmptyRow;
        } else {
            const int32_t lead = a.cols[b];
            if (lead < 0 || lead >= a.ncl) bad |= kErrLeadRange;
            if (a.vals[b] != 1u) bad |= kErrNotMonic;
            for (int64_t k = b + lane; k < e; k += 32) {
                const int32_t c = a.cols[k];
                const uint32_t v = a.vals[k];
                if (c < lead || c >= a.nc || (k > b && c == lead)) bad |= kErrColRange;
                if (v == 0u || v >= (uint32_t)a.p) bad |= kErrCoefRange;
            }
            if (lane == 0 && lead >= 0 && lead < a.ncl) atomicMin(&a.piv_row[lead], i);
        }
        bad = __reduce_or_sync(0xffffffffu, bad);
        if (lane == 0 && bad) atomicOr(a.err, bad);
    }
    cluster_sync();
    // the rows may be walked.  The block barriers below are inside this branch, so
    // every thread has to read the same: the loop behind it reports missing pivots
    // in a word of its own
    const bool good = __ldcg(a.err) == 0;
    for (int c = gw; c < a.ncl; c += ngw) {
        const int32_t r = __ldcg(a.piv_row + c);
        if (r == INT_MAX) {
            if (lane == 0) atomicOr(a.err + 1, kErrMissingPivot);
            continue;
        }
        if (!good) continue;
        // the applied entries (the lead excluded), as 32-bit offsets
        const int b = (int)a.row_ptr[r] + 1, e = (int)a.row_ptr[r + 1];
        if (lane == 0) a.pext[c] = make_int2(b, e);
        const int k0 = c & ~(LB - 1), k1 = min(k0 + LB, a.ncl);
        uint32_t* d = a.diag + (size_t)c * LB;
        d[lane] = 0u;
        __syncwarp();
        for (int k = b + lane; k < e; k += 32) {
            const int32_t j = a.cols[k];
            if (j >= k0 && j < k1) d[j - k0] = a.vals[k];
        }
    }
    if (rk == 0 && good) {
        // rows that are not the known pivot of their lead, in row order
        int base = 0;
        for (int r0 = 0; r0 < a.nr; r0 += kTinyThreads) {
            const int i = r0 + tid;
            const bool f = i < a.nr && __ldcg(a.piv_row + a.cols[a.row_ptr[i]]) != i;
            const unsigned bal = __ballot_sync(0xffffffffu, f);
            if (lane == 0) s_part[warp] = __popc(bal);
            __syncthreads();
            int before = 0, total = 0;
            for (int w = 0; w < kTinyWarps; ++w) {
                const int c = s_part[w];
                before += w < warp ? c : 0;
                total += c;
            }
            if (f) a.work[base + before + __popc(bal & ((1u << lane) - 1u))] = i;
            base += total;
            __syncthreads();  // s_part is rewritten by the next chunk
        }
    }
    cluster_sync();
    const uint32_t verdict = __ldcg(a.err) | __ldcg(a.err + 1);
    if (rk == 0 && tid == 0) a.err[0] = verdict;  // for the launches behind this one
    if (verdict == 0) {
        // a warp per block U (unit upper triangular), lane j column j of its
        // inverse V, from the last row up: V[i] = e_i - sum_(k > i) U[i][k] V[k]
        const int warps = min(kTinyWarps, smem_words / (2 * LB * LB));
        uint32_t* U = smem + warp * 2 * LB * LB;
        uint32_t* V = U + LB * LB;
        const int nb = (a.ncl + LB - 1) / LB;
        for (int b = rk + CL * warp; warp < warps && b < nb; b += CL * warps) {
            uint32_t* d = a.diag + (size_t)b * LB * LB;
            const int kb = min(LB, a.ncl - b * LB);
#pragma unroll 8
            for (int i = 0; i < LB; ++i) {
                U[i * LB + lane] = i < kb ? __ldcg(d + i * LB + lane) : 0u;
                V[i * LB + lane] = 0u;  // rows not there yet meet zeros of U
            }
            __syncwarp();
            for (int i = LB - 1; i >= 0; --i) {
                // terms up to the next multiple of four are zero in U
                ChainSum<F> s(f);
#pragma unroll 1
                for (int k = (i + 1) & ~3; k < LB; k += 4) {
                    const uint4 u = *(const uint4*)(U + i * LB + k);
                    s.add(f, 0, u.x, V[k * LB + lane]);
                    s.add(f, 1, u.y, V[(k + 1) * LB + lane]);
                    s.add(f, 2, u.z, V[(k + 2) * LB + lane]);
                    s.add(f, 3, u.w, V[(k + 3) * LB + lane]);
                }
                const uint32_t t = s.mod(f);  // V is kept in prep form
                const uint32_t v = lane == i ? 1u : lane > i && t ? f.p - t : 0u;
                V[i * LB + lane] = f.prep(v);
                if (i < kb) d[i * LB + lane] = v ? f.prep(f.p - v) : 0u;
                __syncwarp();
            }
        }
    }
    cluster_sync();
    return verdict;
}

// C|D rows w0, w0 + step, ... by the calling warp, whose accumulator is acc (nc
// sums of 64 bits in shared memory, reduced only when a column is read).  The
// known pivots are applied in column order, LB left columns at a time: the LB
// multipliers are the block's entries times the inverse of the pivots' diagonal
// block (independent sums, one shuffle a term), and then the pivot rows whose
// multiplier is not zero are added to the columns right of the block.  All of
// a block's multipliers are known before the first of its rows is added, so the
// rows' entries are loaded GRP rows at a time, no load waiting for an update.
// The search for the next nonzero column after every update, with a dependent
// load behind it, took 1200 cycles per pivot, and one reduction per entry.
// out(w, j, value): right column j of row w.
constexpr int GRP = 4;  // pivot rows whose first 2 x 32 entries are loaded together
template <class T>
__device__ __forceinline__ T pick(const T (&x)[GRP], int q) {
    return q == 0 ? x[0] : q == 1 ? x[1] : q == 2 ? x[2] : x[3];
}
template <class F, class Out>
__device__ void small_rows(const SmallMat& a, int n_work, int w0, int step, int out_cols,
                           uint64_t* acc, const F f, const Out out) {
    const int lane = threadIdx.x & 31;
    const int32_t ncl = a.ncl, nc = a.nc;
    for (int w = w0; w < n_work; w += step) {
        const int32_t r = __ldcg(a.work + w);
        const int rb = (int)a.row_ptr[r], re = (int)a.row_ptr[r + 1];
        const int32_t lead = a.cols[rb];
        for (int c = (lead & ~(LB - 1)) + lane; c < nc; c += 32) acc[c] = 0u;
        __syncwarp();
        for (int k = rb + lane; k < re; k += 32) acc[a.cols[k]] = a.vals[k];
        __syncwarp();
        for (int k0 = lead & ~(LB - 1); k0 < ncl; k0 += LB) {
            const int kend = min(k0 + LB, ncl);
            const bool left = k0 + lane < kend;
            const uint32_t x0 = left ? f.lazy_mod(acc[k0 + lane]) : 0u;
            if (!__any_sync(0xffffffffu, x0 != 0u)) continue;
            const int2 ext = left ? a.pext[k0 + lane] : make_int2(0, 0);
            uint32_t x;  // the negated multiplier of column k0 + lane
            {
                uint32_t d[LB];
#pragma unroll
                for (int i = 0; i < LB; ++i)
                    d[i] = k0 + i < kend ? a.diag[(size_t)(k0 + i) * LB + lane] : 0u;
                ChainSum<F> s(f);
#pragma unroll
                for (int i = 0; i < LB; ++i) s.add(f, i, d[i], __shfl_sync(0xffffffffu, x0, i));
                x = s.mod(f);
            }
            unsigned todo = __ballot_sync(0xffffffffu, x != 0u);
            // the next GRP pivot rows: extents, multipliers, first entries
            int b[GRP], e[GRP], nb[GRP], ne[GRP];
            uint32_t m[GRP], nm[GRP];
            int32_t c[GRP][2], ncol[GRP][2];
            uint32_t v[GRP][2], nv[GRP][2];
            auto fetch = [&]() {
#pragma unroll
                for (int q = 0; q < GRP; ++q) {
                    const int j = todo ? __ffs(todo) - 1 : 0;
                    nb[q] = __shfl_sync(0xffffffffu, ext.x, j);
                    ne[q] = todo ? __shfl_sync(0xffffffffu, ext.y, j) : nb[q];
                    nm[q] = __shfl_sync(0xffffffffu, x, j);
                    todo &= todo - 1u;
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int k = nb[q] + 32 * u + lane;
                        ncol[q][u] = k < ne[q] ? a.cols[k] : -1;
                        nv[q][u] = k < ne[q] ? a.vals[k] : 0u;
                    }
                }
            };
            fetch();
            for (bool more = true; more;) {
#pragma unroll
                for (int q = 0; q < GRP; ++q) {
                    b[q] = nb[q];
                    e[q] = ne[q];
                    m[q] = nm[q];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        c[q][u] = ncol[q][u];
                        v[q][u] = nv[q][u];
                    }
                }
                more = todo != 0u;
                if (more) fetch();  // in flight while these rows are added
                int longest = 0;
#pragma unroll
                for (int q = 0; q < GRP; ++q) {
                    longest = max(longest, e[q] - b[q]);
                    uint64_t y[2];
#pragma unroll
                    for (int u = 0; u < 2; ++u) y[u] = c[q][u] >= kend ? acc[c[q][u]] : 0u;
#pragma unroll
                    for (int u = 0; u < 2; ++u)
                        if (c[q][u] >= kend) acc[c[q][u]] = f.lazy_add(y[u], m[q], v[q][u]);
                    __syncwarp();  // the next row may read what this one wrote
                }
                if (longest <= 64) continue;
                // the rest of the long rows
                for (int q = 0; q < GRP; ++q) {
                    const int eq = pick(e, q);
                    const uint32_t mq = pick(m, q);
                    for (int k = pick(b, q) + 64 + lane; k < eq; k += 128) {
                        int32_t cc[4];
                        uint32_t vv[4];
                        uint64_t yy[4];  // a pivot row's columns are distinct
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            cc[u] = k + 32 * u < eq ? a.cols[k + 32 * u] : -1;
                            vv[u] = k + 32 * u < eq ? a.vals[k + 32 * u] : 0u;
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u) yy[u] = cc[u] >= kend ? acc[cc[u]] : 0u;
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (cc[u] >= kend) acc[cc[u]] = f.lazy_add(yy[u], mq, vv[u]);
                    }
                    __syncwarp();
                }
            }
        }
        for (int j = lane; j < out_cols; j += 32)
            out(w, j, ncl + j < nc ? f.lazy_mod(acc[ncl + j]) : 0u);
        __syncwarp();
    }
}

// accumulators of the row phase that fit in `words` of shared memory
__host__ __device__ inline int small_warps(int32_t nloc, int32_t nc, int64_t words) {
    const int64_t fit = words / (2 * (int64_t)(nc > 0 ? nc : 1));
    const int64_t w = fit < kTinyWarps ? fit : kTinyWarps;
    return (int)(w < nloc ? w : nloc);
}

// one matrix by the calling cluster
template <class F>
__device__ void small_matrix(const SmallMat& a, int32_t ncr, const TinyOut& to, uint32_t* smem,
                             int32_t smem_words, const F f) {
    const int CL = cluster_size(), rk = cluster_rank(), sh = __ffs(CL) - 1;
    const int n_work = a.nr - a.ncl, warp = threadIdx.x >> 5;
    const uint32_t e = small_prep(a, smem, smem_words, f);
    if (e == 0 && n_work > 0) {
        const TinyLayout L = tiny_layout(n_work, ncr, CL);
        const int warps = small_warps((n_work + CL - 1) / CL, a.nc, smem_words - L.words);
        if (warp < warps)
            // a row's right block to the CTAs that own its columns
            small_rows(a, n_work, rk + CL * warp, CL * warps, L.panels * TP,
                       (uint64_t*)(smem + L.words) + (size_t)warp * a.nc, f,
                       [&](int w, int j, uint32_t v) {
                           remote_st(remote_smem(smem + tiny_at(n_work, w, j, sh), (j / TP) & (CL - 1)),
                                     v);
                       });
        tiny_rref_body(n_work, ncr, smem, to, f);
    } else if (rk == 0 && threadIdx.x == 0) {
        to.counts[0] = 0;
        to.counts[1] = 0;
        to.offs[0] = 0;
    }
    if (rk == 0 && threadIdx.x == 0) to.counts[2] = (int64_t)e;
}

// The three phases as launches of their own, for matrices whose rows want more
// SMs than a cluster has: the row phase over the whole device, rows into D.
template <class F>
__global__ void __launch_bounds__(kTinyThreads)
k_small_prep(const SmallMat a, int32_t smem_words, F f) {
    extern __shared__ __align__(16) uint32_t sm_smem[];
    small_prep(a, sm_smem, smem_words, f);
}
template <class F>
__global__ void __launch_bounds__(kTinyThreads)
k_small_rows(const SmallMat a, int32_t n_work, uint32_t* D, int64_t ld, F f) {
    extern __shared__ __align__(16) uint32_t sm_smem[];
    if (*a.err) return;  // invalid input: nothing is read (uniform)
    const int warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    small_rows(a, n_work, blockIdx.x + gridDim.x * warp, gridDim.x * warps, a.nc - a.ncl,
               (uint64_t*)sm_smem + (size_t)warp * a.nc, f,
               [&](int w, int j, uint32_t v) { D[(size_t)w * ld + j] = v; });
}

// n matrices, items[0 .. n) from the queue, or the one in `one` (items null)
__global__ void __launch_bounds__(kTinyThreads, 1)
k_small(int32_t n, const SmallItem one, const SmallItem* items, const uint8_t* in, uint8_t* scr,
        uint8_t* out, int32_t* queue, int32_t smem_words) {
    extern __shared__ __align__(16) uint32_t sm_smem[];
    __shared__ int s_item;
    const int CL = cluster_size(), rk = cluster_rank(), tid = threadIdx.x;
    // the queue's first entry goes to the other CTAs' shared memory, which may be
    // written only once all of them have started
    if (items) cluster_sync();
    for (int pass = 0;; ++pass) {
        if (items) {
            if (rk == 0 && tid < 32) {
                int i = 0;
                if (tid == 0) i = atomicAdd(queue, 1);
                i = __shfl_sync(0xffffffffu, i, 0);
                if (tid < CL) remote_st(remote_smem(&s_item, tid), (uint32_t)i);
            }
            cluster_sync();
            if (s_item >= n) break;
        } else if (pass > 0) {
            break;
        }
        const SmallItem it = items ? items[s_item] : one;
        const int32_t nr = it.nr, ncl = it.ncl, ncr = it.ncr;
        const SmallMat a = small_mat(it, in, scr);
        const OutLayout O = out_layout(nr, ncl, ncr);
        uint8_t* ob = out + it.out_off;
        const TinyOut to{ncl, (int64_t*)(ob + O.offs), (int32_t*)(ob + O.cols),
                         (int32_t*)(ob + O.vals), nullptr, (int64_t*)ob};
        if ((uint32_t)it.p < 65536u)
            small_matrix(a, ncr, to, sm_smem, smem_words, it.fs);
        else
            small_matrix(a, ncr, to, sm_smem, smem_words, it.fm);
    }
}

// ---------------------------------------------------------------------------
// host side

namespace {

struct Session {
    DeviceInfo dev{};
    cudaStream_t s = nullptr;
    void* dmem = nullptr;  // device arena
    size_t dcap = 0;
    uint8_t* hin = nullptr;  // pinned input staging
    size_t hin_cap = 0;
    uint8_t* hout = nullptr;  // mapped pinned output
    size_t hout_cap = 0;
    ~Session() {
        // runs at thread exit; at process exit the runtime may already be
        // gone, which these calls tolerate
        if (s) cudaStreamSynchronize(s);
        if (dmem) cudaFree(dmem);
        if (hin) cudaFreeHost(hin);
        if (hout) cudaFreeHost(hout);
        if (s) cudaStreamDestroy(s);
    }
};

constexpr int kMaxDev = 64;
struct Sessions {
    Session* by_dev[kMaxDev] = {};
    ~Sessions() {
        for (auto*& x : by_dev) {
            delete x;
            x = nullptr;
        }
    }
};
thread_local Sessions t_sessions;

int grow_device(Session& S, size_t need) {
    if (need <= S.dcap) return GBGPU_OK;
    const size_t cap = std::max(need, S.dcap * 2);
    if (S.dmem) {
        cudaStreamSynchronize(S.s);
        cudaFree(S.dmem);
        S.dmem = nullptr;
        S.dcap = 0;
    }
    if (cudaMalloc(&S.dmem, cap) != cudaSuccess) {
        set_error("small-matrix arena allocation failed");
        return GBGPU_ENOMEM;
    }
    S.dcap = cap;
    return GBGPU_OK;
}

int grow_host(uint8_t** buf, size_t* capv, size_t need, unsigned flags, cudaStream_t s) {
    if (need <= *capv) return GBGPU_OK;
    const size_t cap = std::max(need, *capv * 2);
    if (*buf) {
        cudaStreamSynchronize(s);
        cudaFreeHost(*buf);
        *buf = nullptr;
        *capv = 0;
    }
    if (cudaHostAlloc((void**)buf, cap, flags) != cudaSuccess) {
        set_error("small-matrix pinned staging allocation failed");
        return GBGPU_ENOMEM;
    }
    *capv = cap;
    return GBGPU_OK;
}

// A batch leaves at most this much of each buffer in the session; what it needed
// beyond that is given back when the call ends.  (Single matrices grow the buffers to
// a high-water mark: their answer lies in them when the call returns.)
constexpr size_t kKeepHost = (size_t)64 << 20, kKeepDevice = (size_t)256 << 20;

void trim(Session& S) {
    if (S.hin_cap > kKeepHost) {
        cudaFreeHost(S.hin);
        S.hin = nullptr;
        S.hin_cap = 0;
    }
    if (S.hout_cap > kKeepHost) {
        cudaFreeHost(S.hout);
        S.hout = nullptr;
        S.hout_cap = 0;
    }
    if (S.dcap > kKeepDevice) {
        cudaFree(S.dmem);
        S.dmem = nullptr;
        S.dcap = 0;
    }
}

int session_for(int device, Session** out) {
    if (device < 0 || device >= kMaxDev) {
        set_error("device ordinal out of range");
        return GBGPU_ENODEV;
    }
    Session*& S = t_sessions.by_dev[device];
    if (!S) {
        Session* n = new Session();
        int rc = device_init(device, &n->dev);
        if (rc) {
            delete n;
            return rc;
        }
        if (cudaStreamCreateWithFlags(&n->s, cudaStreamNonBlocking) != cudaSuccess) {
            delete n;
            set_error("small-matrix session set-up failed");
            return GBGPU_ECUDA;
        }
        S = n;
    }
    *out = S;
    return GBGPU_OK;
}

// the device current on entry is made current again on return
struct DeviceGuard {
    int prev = -1;
    DeviceGuard() {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    }
    ~DeviceGuard() {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

SmallItem small_item(int32_t p, int32_t nr, int32_t ncl, int32_t ncr) {
    SmallItem it{};
    it.p = p;
    it.nr = nr;
    it.ncl = ncl;
    it.ncr = ncr;
    it.fs = FieldSmall::make((uint32_t)std::max(p, 2));
    it.fm = FieldMont::make((uint32_t)(p | 1));  // used only for odd p >= 2^16
    return it;
}

// 32-bit words of shared memory a CTA of a cluster of cl needs for a matrix of
// this shape: the echelon's, and an accumulator for every row of the CTA up to
// one per warp (at least four, or one per row), or four blocks of the prep
// phase; 0: does not fit.  A matrix of known pivots alone is only checked; it
// comes here up to the columns of two accumulators, as those of small_wide, because
// its whole input would pass through the session's pinned staging.
int64_t small_words(int32_t nr, int32_t ncl, int32_t ncr, int cl, int smem_optin) {
    const int64_t room = (smem_optin - 2048) / 4, least = 4 * 2 * LB * LB;
    if (nr <= ncl) return 4 * ((int64_t)ncl + ncr) <= room ? least : 0;
    const TinyLayout L = tiny_layout(nr - ncl, ncr, cl);
    const int32_t nc = ncl + ncr;
    const int nloc = (nr - ncl + cl - 1) / cl;
    const int w = L.words < room ? small_warps(nloc, nc, room - L.words) : 0;
    if (w < std::min(4, nloc)) return 0;
    return std::max<int64_t>(least, L.words + w * 2 * (int64_t)nc);
}

// The three-launch form takes matrices whose echelon fits a cluster (or comes to it
// in turns) and two of whose accumulators fit an SM (14400 columns).  With fewer
// than four (from 7200 columns on) a block that a plan reduces in the blocked form
// is faster there: 8000 left columns, blocks of 100 x 200, 300 x 200 and 1000 x 40,
// here / by a plan: 1777 / 5411, 1853 / 1369 and 2678 / 8239 us; 12000: 2763 / 8628,
// 2852 / 1875 and 5124 / 14713.
bool small_wide(int32_t nr, int32_t ncl, int32_t ncr, int smem_optin) {
    if (nr <= ncl || !tiny_capacity(nr - ncl, ncr, smem_optin)) return false;
    const int warps = small_warps(4, ncl + ncr, (smem_optin - 2048) / 4);
    return warps == 4 || (warps >= 2 && (nr - ncl < 128 || ncr < 128));
}

// The three-launch form is the faster one where the cluster would take its rows
// in several turns or the chain of left columns is long: measured for blocks of
// 60 x 100, 141 x 191, 200 x 300 and 250 x 450 after 200, 300, 500 and 700 left
// columns at 126 / 235 / 407 / 609 us a call against 113 / 225 / 443 / 738 us in
// one launch, and 1032 against 1645 us for 120 x 400 after 3000.
constexpr int kWideRows = 160, kWideLeft = 1024;

// Blocks of more entries are faster in the blocked form (400 x 700: 1570 us here
// against 1410 us; 300 x 600: 1100 against 1610 us).
constexpr int64_t kSmallMaxBlock = 200000;

bool small_shape(int32_t nr, int32_t ncl, int32_t ncr) {
    return nr > 0 && ncl >= 0 && ncr > 0 && nr >= ncl && ncl <= kSmallMaxLeft &&
           (int64_t)(nr - ncl) * ncr <= kSmallMaxBlock;
}

// CTAs per matrix: the most that leaves every one of n matrices its own
// cluster on the device's SMs, and at least what the matrix needs
int small_cluster(int32_t n, int sms) {
    int cl = kTinyMaxCluster;
    while (cl > 1 && (int64_t)n * cl > sms) cl /= 2;
    return cl;
}

}  // namespace

bool small_eligible(int32_t nr, int32_t ncl, int32_t ncr, int device) {
    if (!small_shape(nr, ncl, ncr)) return false;
    DeviceGuard guard;
    DeviceInfo dev{};
    if (device_init(device, &dev)) return false;
    return small_words(nr, ncl, ncr, kTinyMaxCluster, dev.smem_optin) > 0 ||
           small_wide(nr, ncl, ncr, dev.smem_optin);
}

bool small_batchable(int32_t nr, int32_t ncl, int32_t ncr, int device) {
    if (!small_shape(nr, ncl, ncr)) return false;
    DeviceGuard guard;
    DeviceInfo dev{};
    if (device_init(device, &dev)) return false;
    return small_words(nr, ncl, ncr, kTinyMaxCluster, dev.smem_optin) > 0;
}

int small_reduce(const SmallInput& in, SmallAnswer* ans) {
    DeviceGuard guard;
    Session* S = nullptr;
    int rc = session_for(in.device, &S);
    if (rc) return rc;
    const int32_t nr = in.nr, ncl = in.ncl, ncr = in.ncr;
    const int64_t nnz = in.nnz;
    // pinned staging: row_ptr | cols | vals (copied to the arena's start)
    SmallItem it = small_item(in.p, nr, ncl, ncr);
    it.cols_off = rup((int64_t)sizeof(int64_t) * (nr + 1), 16);
    it.vals_off = rup(it.cols_off + 4 * nnz, 16);
    const int64_t in_bytes = rup(it.vals_off + 4 * nnz, 16);
    if ((rc = grow_host(&S->hin, &S->hin_cap, (size_t)in_bytes, cudaHostAllocDefault, S->s)))
        return rc;
    // every call ends with a synchronisation, so the staging is free to refill
    in.fill(in.ctx, (int64_t*)S->hin, (int32_t*)(S->hin + it.cols_off),
            (uint32_t*)(S->hin + it.vals_off));
    it.scr_off = rup(in_bytes, 256);
    const int optin = S->dev.smem_optin, cl = kTinyMaxCluster, n_work = nr - ncl;
    int32_t words = (int32_t)small_words(nr, ncl, ncr, cl, optin);
    const bool wide = small_wide(nr, ncl, ncr, optin) &&
                      (words == 0 || n_work > kWideRows || ncl > kWideLeft);
    const ScrLayout L = scr_layout(nr, ncl, wide ? (int64_t)n_work * ncr : 0);
    if ((rc = grow_device(*S, (size_t)(it.scr_off + L.bytes)))) return rc;
    const OutLayout O = out_layout(nr, ncl, ncr);
    if ((rc = grow_host(&S->hout, &S->hout_cap, (size_t)O.bytes, cudaHostAllocMapped, S->s)))
        return rc;
    uint8_t* hd = nullptr;
    if (cudaHostGetDevicePointer((void**)&hd, S->hout, 0) != cudaSuccess) {
        set_error("mapped output pointer unavailable");
        return GBGPU_ECUDA;
    }
    const int64_t* counts = (const int64_t*)S->hout;
    cudaStream_t s = S->s;
    if (cudaMemcpyAsync(S->dmem, S->hin, (size_t)in_bytes, cudaMemcpyHostToDevice, s) !=
        cudaSuccess) {
        set_error("small-matrix input copy failed");
        return GBGPU_ECUDA;
    }
    uint8_t* d = (uint8_t*)S->dmem;
    cudaError_t e = cudaSuccess;
    if (wide) {
        SmallMat a = small_mat(it, d, d);
        uint32_t* D = (uint32_t*)(d + it.scr_off + L.D);
        int64_t ld = ncr;
        const int wpr = small_warps(kTinyWarps, a.nc, (optin - 2048) / 4);
        const int grid = std::min(n_work, S->dev.sms);
        const int warps = std::min(wpr, (n_work + grid - 1) / grid);
        auto run = [&](auto f) {
            using F = decltype(f);
            int32_t pw = 4 * 2 * LB * LB, nw = n_work;
            void* prep[] = {&a, &pw, &f};
            e = launch_cluster((const void*)k_small_prep<F>, cl, cl, kTinyThreads, pw * 4, s, prep);
            void* rows[] = {&a, &nw, &D, &ld, &f};
            if (e == cudaSuccess)
                e = launch_cluster((const void*)k_small_rows<F>, grid, 1, 32 * warps,
                                   warps * a.nc * 8, s, rows);
            if (e == cudaSuccess)
                e = launch_tiny_rref(n_work, ncr, D, ld, a.err, ncl, (int64_t*)(hd + O.offs),
                                     (int32_t*)(hd + O.cols), (int32_t*)(hd + O.vals), nullptr,
                                     (int64_t*)hd, tiny_capacity(n_work, ncr, optin), s, f);
        };
        if ((uint32_t)in.p < 65536u) run(it.fs);
        else run(it.fm);
        count_launch(3);
    } else {
        int32_t n = 1;
        const SmallItem* items = nullptr;
        int32_t* queue = nullptr;
        void* args[] = {&n, &it, &items, &d, &d, &hd, &queue, &words};
        e = launch_cluster((const void*)k_small, cl, cl, kTinyThreads, words * 4, s, args);
        count_launch(1);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        set_error(std::string("small-matrix run: ") + cudaGetErrorString(e));
        return GBGPU_ECUDA;
    }
    if (counts[2]) {
        std::string msg;
        rc = err_to_status((uint32_t)counts[2], &msg);
        set_error(msg);
        return rc;
    }
    ans->np = (int32_t)counts[0];
    ans->nnz = counts[1];
    ans->offs = (const int64_t*)(S->hout + O.offs);
    ans->cols = (const int32_t*)(S->hout + O.cols);
    ans->vals = (const int32_t*)(S->hout + O.vals);
    return GBGPU_OK;
}

int small_batch(int32_t n, const gbgpu_csr* const* ms, int device, gbgpu_rows* outs,
                int32_t* status) {
    if (n <= 0) return GBGPU_OK;
    DeviceGuard guard;
    Session* S = nullptr;
    int rc = session_for(device, &S);
    if (rc) return rc;
    const DeviceInfo& dev = S->dev;
    // the thread's session buffers, given back down to their bound on every
    // return: pinning and freeing the staging of one call took 4 to 20 ms
    struct Trim {
        Session* S;
        ~Trim() {
            cudaStreamSynchronize(S->s);
            trim(*S);
        }
    } trimmer{S};
    std::vector<SmallItem> items((size_t)n);
    int64_t in_bytes = 0, scr_bytes = 0, out_bytes = 0, words = 0;
    int cl = small_cluster(n, dev.sms);
    for (int32_t i = 0; i < n; ++i)
        while (cl < kTinyMaxCluster &&
               !small_words(ms[i]->nr, ms[i]->ncl, ms[i]->ncr, cl, dev.smem_optin))
            cl *= 2;
    for (int32_t i = 0; i < n; ++i) {
        const gbgpu_csr* m = ms[i];
        SmallItem& it = items[i];
        it = small_item(m->p, m->nr, m->ncl, m->ncr);
        const int64_t nnz = m->row_ptr[m->nr];
        it.in_off = in_bytes;
        it.cols_off = rup(it.in_off + 8 * (int64_t)(m->nr + 1), 16);
        it.vals_off = rup(it.cols_off + 4 * nnz, 16);
        in_bytes = rup(it.vals_off + 4 * nnz, 256);
        it.scr_off = scr_bytes;
        scr_bytes += scr_layout(m->nr, m->ncl).bytes;
        it.out_off = out_bytes;
        out_bytes += out_layout(m->nr, m->ncl, m->ncr).bytes;
        words = std::max(words, small_words(m->nr, m->ncl, m->ncr, cl, dev.smem_optin));
    }
    // device: input | items | queue | scratch (the first three in one copy)
    const int64_t o_items = rup(in_bytes, 256);
    const int64_t o_queue = o_items + rup((int64_t)sizeof(SmallItem) * n, 256);
    const int64_t o_scr = o_queue + 256;
    uint8_t* d_out = nullptr;
    if ((rc = grow_host(&S->hin, &S->hin_cap, (size_t)o_scr, cudaHostAllocDefault, S->s)) ||
        (rc = grow_host(&S->hout, &S->hout_cap, (size_t)std::max<int64_t>(out_bytes, 256),
                        cudaHostAllocMapped, S->s)) ||
        (rc = grow_device(*S, (size_t)(o_scr + scr_bytes))))
        return rc;
    if (cudaHostGetDevicePointer((void**)&d_out, S->hout, 0) != cudaSuccess) {
        set_error("mapped output pointer unavailable");
        return GBGPU_ECUDA;
    }
    uint8_t *h_in = S->hin, *h_out = S->hout, *d_in = (uint8_t*)S->dmem;
    cudaStream_t s = S->s;
    for (int32_t i = 0; i < n; ++i) {
        const gbgpu_csr* m = ms[i];
        fill_from_csr_vals((void*)m, (int64_t*)(h_in + items[i].in_off),
                           (int32_t*)(h_in + items[i].cols_off),
                           (uint32_t*)(h_in + items[i].vals_off));
    }
    memcpy(h_in + o_items, items.data(), sizeof(SmallItem) * (size_t)n);
    memset(h_in + o_queue, 0, 256);
    SmallItem* d_items = (SmallItem*)(d_in + o_items);
    int32_t* d_queue = (int32_t*)(d_in + o_queue);
    cudaError_t e = cudaMemcpyAsync(d_in, h_in, (size_t)o_scr, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        // as many clusters as the device has SMs for: the registers of k_small (128
        // for 512 threads) leave an SM one CTA
        const int grid = cl * std::max(1, std::min(n, dev.sms / cl));
        SmallItem none{};
        const SmallItem* its = d_items;
        uint8_t* scr = d_in + o_scr;
        int32_t w32 = (int32_t)words;
        void* args[] = {&n, &none, &its, &d_in, &scr, &d_out, &d_queue, &w32};
        e = launch_cluster((const void*)k_small, grid, cl, kTinyThreads, w32 * 4, s, args);
        count_launch(1);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        set_error(std::string("small-matrix batch: ") + cudaGetErrorString(e));
        for (int32_t i = 0; i < n; ++i) status[i] = GBGPU_ECUDA;
        return GBGPU_OK;
    }
    for (int32_t i = 0; i < n; ++i) {
        const uint8_t* ob = h_out + items[i].out_off;
        const OutLayout O = out_layout(items[i].nr, items[i].ncl, items[i].ncr);
        const int64_t* counts = (const int64_t*)ob;
        if (counts[2]) {
            std::string msg;
            status[i] = err_to_status((uint32_t)counts[2], &msg);
            continue;
        }
        gbgpu_rows& r = outs[i];
        r.np = (int32_t)counts[0];
        r.nnz = counts[1];
        r.row_ptr = (int64_t*)malloc(sizeof(int64_t) * (size_t)(r.np + 1));
        r.cols = (int32_t*)malloc(sizeof(int32_t) * (size_t)std::max<int64_t>(r.nnz, 1));
        r.vals = (int32_t*)malloc(sizeof(int32_t) * (size_t)std::max<int64_t>(r.nnz, 1));
        if (!r.row_ptr || !r.cols || !r.vals) {
            status[i] = GBGPU_ENOMEM;
            continue;
        }
        memcpy(r.row_ptr, ob + O.offs, sizeof(int64_t) * (size_t)(r.np + 1));
        memcpy(r.cols, ob + O.cols, sizeof(int32_t) * (size_t)r.nnz);
        memcpy(r.vals, ob + O.vals, sizeof(int32_t) * (size_t)r.nnz);
        status[i] = GBGPU_OK;
    }
    return GBGPU_OK;
}

}  // namespace gbgpu
