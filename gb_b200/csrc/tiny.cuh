// tiny.cuh -- the reduced echelon form and compaction of a small dense block in
// the shared memory of one thread-block cluster (the body of plain.cu's
// k_tiny_rref and the last phase of small.cu's k_small).
//
// What bounds it is the chain of pivots and the SMs' integer multipliers (a
// 64-bit multiply-add takes about four issue cycles per warp: one SM alone
// needs 130 us for the updates of a 141 x 191 block).  So the block is reduced
// by panels of TP columns, and the work is split by how often it has to be
// exchanged:
//   * panel k (its TP columns of all rows) belongs to CTA k % CL.  Its owner
//     copies it to every CTA, and every CTA finds the panel's pivots by itself;
//   * the columns right of the panel are updated once per panel by their
//     owners, with 64-bit sums of TP products and one reduction per entry.
// One or two cluster barriers per panel, none per pivot.
//
// The panel's pivots come from TP rows at a time (the first row of every lead,
// then any others): their TP x TP entries are brought to reduced echelon form,
// a thread per entry, and every other row r is cleared at the pivots' columns c
// at once, row_r -= sum_c row_r[c] (pivot row of c).  Rows that are still not
// zero in the panel give the next TP (a dense panel is done after one turn).
// The leads of some of the rows are leads of all of them, so every pivot found
// this way is one of the reduced echelon form.  A step per pivot over all rows
// of the panel took 1900 cycles per pivot.
//
// In the TP x TP echelon (pivot row i, column c, a = row_i[c]) every other row
// with m = row_r[c] != 0 becomes a row_r - m row_i (no inverse on the chain),
// and column c, which would be zero from here on, stores the coefficient of the
// pivot row's old value: -m s_i, s_r being the product of the factors a that
// row r took (s_i for the pivot row itself, whose own scale then is 0).  So
// the TP columns hold both the reduced rows and the transformation F, in place;
// the pivot rows are divided by their pivot entries at the end, in parallel.
#pragma once
#include <climits>
#include <stdint.h>

#include "cluster.cuh"
#include "common.cuh"

namespace gbgpu {

constexpr int kTinyThreads = 512;
constexpr int kTinyWarps = kTinyThreads / 32;
constexpr int kTinyMaxCluster = 8;          // the portable limit
constexpr int TP = 16;                      // panel columns
// Tall blocks that come in turns (k_tiny_rref): a row takes 49 words of every CTA
// however few columns it has, so 1111 rows fit.  With a launch of one CTA, whose rows
// took a word a column, blocks of up to 7130 rows had this path; all of those and the
// wider ones up to 48 columns are faster here than by the echelon rounds of a plan
// (a call, 100 left columns, p = 2^31 - 1, in turns / rounds): 1200 x 1 151 / 494 us,
// 7000 x 1 428 / 1002, 1200 x 48 236 / 2188, 4000 x 48 468 / 2423, 7000 x 20 643 /
// 1498.  Only a plan's run alone gains little with one column: 7000 x 1 862 / 854.
constexpr int kTinyTallCols = 48, kTinyTallTurns = 7;
constexpr int kRelayRows = 64;              // from here panels are passed on in two steps
// Shared memory of one CTA for an n x m block in a cluster of cl (offsets in
// 32-bit words): its panels [panels / cl][n][TP], two copies of the current
// panel [n][TP], the pivots' TP x TP blocks (F, the pivot rows in the panel, and
// eight working blocks), arrays per row and per column.
struct TinyLayout {
    int32_t panels;  // of the block
    int64_t pb, blk, rows, cols, words;
};
__host__ __device__ inline TinyLayout tiny_layout(int32_t n, int32_t m, int32_t cl) {
    TinyLayout L;
    L.panels = (m + TP - 1) / TP;
    L.pb = (int64_t)((L.panels + cl - 1) / cl) * n * TP;
    L.blk = L.pb + 2 * (int64_t)n * TP;
    L.rows = L.blk + (2 + 8) * TP * TP;
    L.cols = L.rows + (int64_t)n;
    L.words = (L.cols + 3 * (int64_t)L.panels * TP + 3) & ~(int64_t)3;
    return L;
}
// rows of a block of m columns that `words` of shared memory hold (< 0: none)
__host__ __device__ inline int64_t tiny_rows(int32_t m, int32_t cl, int64_t words) {
    const int64_t none = tiny_layout(0, m, cl).words, one = tiny_layout(64, m, cl).words;
    return 64 * (words - none - 4) / (one - none);
}
// word offset of entry (r, j) in the CTA that owns it, (j / TP) % CL
__device__ __forceinline__ int tiny_at(int n, int r, int j, int cl_shift) {
    return (((j / TP) >> cl_shift) * n + r) * TP + j % TP;
}

struct TinyOut {
    int32_t col_shift;
    int64_t* offs;      // [rank + 1]
    int32_t* cols;      // [entries]
    int32_t* vals;      // [entries]
    int32_t* piv_of_col;  // [m], or null
    int64_t* counts;    // rows, entries; [2]: the input checks' verdict
};

// in-place exclusive prefix sum of a[0..n) in shared memory; returns the total.
// Every thread sums a contiguous piece; `part` holds one int per warp.
__device__ inline int tiny_exscan(int32_t* a, int n, int* part) {
    const int per = (n + kTinyThreads - 1) / kTinyThreads;
    const int b = min(n, (int)threadIdx.x * per), e = min(n, b + per);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int s = 0;
    for (int i = b; i < e; ++i) s += a[i];
    int inc = s;
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) part[warp] = inc;
    __syncthreads();
    int before = inc - s, total = 0;
    for (int w = 0; w < kTinyWarps; ++w) {
        const int v = part[w];
        before += w < warp ? v : 0;
        total += v;
    }
    for (int i = b; i < e; ++i) {
        const int v = a[i];
        a[i] = before;
        before += v;
    }
    __syncthreads();
    return total;
}

// One turn's pivots of a panel (shared memory of the CTA).
struct TinyTurn {
    int first[TP];             // first row of every lead, INT_MAX
    int sel[TP];               // the rows of the turn
    int per_warp[kTinyWarps];
    uint32_t scl2[TP];         // scales of the turn's rows (second buffer)
    uint32_t mask;             // pivot columns found in this turn
};

// The rows of the next turn, the same in every CTA: the first row of every lead
// in the panel, then the other nonzero rows in row order.  Returns the number of
// nonzero rows that are no pivots, or TP + 1 if there are more than TP (uniform);
// the turn takes at most TP of them.
__device__ inline int tiny_select(const int n, const uint32_t* pb, const int32_t* pcol,
                                  TinyTurn& S) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto lead_of = [&](int r) {
        int ld = INT_MAX;
        if (r < n && pcol[r] < 0) {
#pragma unroll
            for (int q = TP / 4 - 1; q >= 0; --q) {
                const uint4 x = *(const uint4*)(pb + r * TP + 4 * q);
                const int f = x.x ? 0 : x.y ? 1 : x.z ? 2 : x.w ? 3 : 4;
                if (f < 4) ld = 4 * q + f;
            }
        }
        return ld;
    };
    if (tid < TP) S.first[tid] = INT_MAX;
    __syncthreads();
    const int ld0 = lead_of(tid);
    if (ld0 != INT_MAX) atomicMin(&S.first[ld0], tid);
    for (int r = tid + kTinyThreads; r < n; r += kTinyThreads) {
        const int ld = lead_of(r);
        if (ld != INT_MAX) atomicMin(&S.first[ld], r);
    }
    __syncthreads();
    const int mine = lane < TP ? S.first[lane] : INT_MAX;
    const unsigned leads = __ballot_sync(0xffffffffu, mine != INT_MAX);
    int count = __popc(leads);
    if (count == 0) {
        __syncthreads();  // S.first is rewritten by the next call
        return 0;
    }
    if (tid < TP && mine != INT_MAX) S.sel[__popc(leads & ((1u << lane) - 1u))] = mine;
    for (int r0 = 0; r0 < n && count <= TP; r0 += kTinyThreads) {
        const int r = r0 + tid, ld = r0 ? lead_of(r) : ld0;
        const bool other = ld != INT_MAX && S.first[ld] != r;
        const unsigned bal = __ballot_sync(0xffffffffu, other);
        if (lane == 0) S.per_warp[warp] = __popc(bal);
        __syncthreads();
        int slot = count + __popc(bal & ((1u << lane) - 1u));
        for (int w = 0; w < kTinyWarps; ++w) {
            const int c = S.per_warp[w];
            slot += w < warp ? c : 0;
            count += c;
        }
        if (other && slot < TP) S.sel[slot] = r;
        __syncthreads();  // per_warp is rewritten
    }
    __syncthreads();
    return min(TP + 1, count);
}

// The turn's rows: their pivots into pcol / prow / S.mask, and, by pivot column
// c, F[c] (coefficients of the old pivot rows, prep form) and PP[c] (the new
// pivot row in the panel); rows of F and PP without a pivot are 0.  One thread
// per entry (threads 0 .. TP TP - 1, which alone call this), the entries
// mirrored in two buffers of shared memory: one barrier per column, and a loop
// short enough for the instruction cache (the same steps by one warp with the
// entries in registers, unrolled, took 750 cycles per pivot).
template <class F_>
__device__ void tiny_turn(const int n_sel, const int c0, const uint32_t* pb, int32_t* pcol,
                          int32_t* prow, uint32_t* Fm, uint32_t* PP, uint32_t* buf, TinyTurn& S,
                          const F_ f) {
    const int tid = threadIdx.x, lane = tid & 31, q = tid / TP, j = tid % TP;
    const int row = q < n_sel ? S.sel[q] : -1;
    uint32_t y = row >= 0 ? pb[row * TP + j] : 0u, scl = 1u, pval = 1u;
    uint32_t pmask = 0u, done = 0u;  // pivot columns, rows that are pivots (uniform)
    int my_col = -1, cur = 0;
    uint32_t* s_scl = (uint32_t*)S.first;  // [TP], then the second buffer's
    buf[tid] = y;
    if (j == 0) s_scl[q] = 1u;
    asm volatile("bar.sync 1, 256;" ::: "memory");
#pragma unroll 1
    for (int c = 0; c < TP; ++c) {
        const uint32_t* B = buf + cur * TP * TP;
        const uint32_t col = B[(lane % TP) * TP + c];
        const unsigned cand = __ballot_sync(0xffffffffu, col != 0u) & 0xFFFFu & ~done;
        if (cand == 0u) continue;  // uniform
        const int i = __ffs(cand) - 1;
        const uint32_t a = B[i * TP + c], mr = B[q * TP + c], v = B[i * TP + j];
        const uint32_t si = cur ? S.scl2[i] : s_scl[i];
        pmask |= 1u << c;
        done |= 1u << i;
        // (selects: the pivot's warp would run both sides of a branch; a row with
        // mr = 0 is scaled by a like the others)
        const uint32_t ap = f.prep(a), mn = f.prep(f.p - mr);
        const uint32_t z = j == c ? f.mulp(si, mn) : f.ffsub(y, ap, v, mn);
        const uint32_t s2 = f.mulp(scl, ap), p2 = f.mulp(pval, ap);
        const bool pivot = q == i;
        y = pivot ? (j == c ? scl : y) : z;
        scl = pivot ? 0u : s2;
        pval = pivot ? a : p2;
        my_col = pivot ? c : my_col;
        cur ^= 1;
        buf[cur * TP * TP + tid] = y;
        if (j == 0) (cur ? S.scl2 : s_scl)[q] = scl;
        asm volatile("bar.sync 1, 256;" ::: "memory");
    }
    if (!((pmask >> q) & 1u)) Fm[tid] = PP[tid] = 0u;  // no pivot in column q
    if (my_col >= 0) {
        const uint32_t z = f.mulp(y, f.prep(f.inv(pval)));
        const bool pc = (pmask >> j) & 1u;
        Fm[my_col * TP + j] = pc ? f.prep(z) : 0u;
        PP[my_col * TP + j] = pc ? (j == my_col ? 1u : 0u) : z;
        if (j == 0) {
            pcol[row] = c0 + my_col;
            prow[c0 + my_col] = row;
        }
    }
    if (tid == 0) S.mask = pmask;
}

// G ([n][TP]) -= the turn's elimination: row r takes -= sum_c pb[r][c] P[c],
// the turn's pivot rows become P[c]; P in v by pivot column (prep form), a lane
// per column j, two rows per warp; by `parts` warps, this one the part-th.  G
// may be pb itself.  The columns of `zero` count as zero before the update.
template <class F>
__device__ __forceinline__ void tiny_update(const int n, const int c0, const uint32_t mask,
                                            const uint32_t* pb, const int32_t* pcol,
                                            const uint32_t (&v)[TP], uint32_t* G, const int part,
                                            const int parts, const F f, const uint32_t zero = 0u) {
    const int lane = threadIdx.x & 31, j = lane % TP;
    constexpr int U = 2;  // rows in flight per lane
#pragma unroll 1
    for (int r0 = 2 * U * part; r0 < n; r0 += 2 * U * parts) {
        uint4 e[U][TP / 4];
        uint32_t g[U];
        bool on[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int r = r0 + 2 * u + lane / TP;
            const int k = r < n ? pcol[r] - c0 : 0;
            on[u] = r < n && !(k >= 0 && k < TP && ((mask >> k) & 1u));
#pragma unroll
            for (int q = 0; q < TP / 4; ++q)
                e[u][q] = on[u] ? *(const uint4*)(pb + r * TP + 4 * q) : make_uint4(0u, 0u, 0u, 0u);
            g[u] = on[u] && !((zero >> j) & 1u) ? G[r * TP + j] : 0u;
        }
        __syncwarp();  // the rows are read before they are written (G = pb)
#pragma unroll
        for (int u = 0; u < U; ++u) {
            uint32_t any = 0u;
#pragma unroll
            for (int q = 0; q < TP / 4; ++q) any |= e[u][q].x | e[u][q].y | e[u][q].z | e[u][q].w;
            if (any == 0u) continue;
            ChainSum<F> acc(f);
#pragma unroll
            for (int q = 0; q < TP / 4; ++q) {
                acc.add(f, 0, e[u][q].x, v[4 * q]);
                acc.add(f, 1, e[u][q].y, v[4 * q + 1]);
                acc.add(f, 2, e[u][q].z, v[4 * q + 2]);
                acc.add(f, 3, e[u][q].w, v[4 * q + 3]);
            }
            const uint32_t t = acc.mod(f);
            G[(r0 + 2 * u + lane / TP) * TP + j] = g[u] >= t ? g[u] - t : g[u] + (f.p - t);
        }
    }
}

// One turn on this CTA's panels g in [g0, g1) (panel g at T + g n TP), none of
// them the current one (c0): the turn's pivot rows there are F times their old
// values, every other row takes their multiples (see tiny_update).  Panel `own`
// is the current one and keeps, in the turn's pivot columns, the coefficients of
// the old pivot rows.  Up to TG panels at a time, so that a few rows still fill
// the warps and the barriers are shared (a panel at a time, each turn of a
// 33-row block of 8 panels took 40000 cycles).  Reached by the whole CTA; NP:
// TG TP TP words of shared memory.
constexpr int TG = 8;
constexpr int kFewPivots = 6;
template <class F>
__device__ __forceinline__ void tiny_groups(const int n, const int c0, const uint32_t mask,
                                            const uint32_t* pb, const int32_t* pcol,
                                            const int32_t* prow, const uint32_t* Fm, uint32_t* NP,
                                            uint32_t* T, const int g0, const int g1, const int own,
                                            const F f) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int PER = TG * TP * TP / kTinyThreads;  // entries of new pivot rows per thread
    const bool few = __popc(mask) <= kFewPivots;      // the sums skip the missing terms
    for (int gb = g0; gb < g1; gb += TG) {
        const int ng = min(TG, g1 - gb);
        uint32_t np[PER];
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int e = tid + u * kTinyThreads, c = (e / TP) % TP, j = e % TP, g = e / (TP * TP);
            np[u] = 0u;
            if (g >= ng || !((mask >> c) & 1u)) continue;
            const uint32_t* G = T + (size_t)(gb + g) * n * TP;
            if (gb + g == own && ((mask >> j) & 1u)) {
                np[u] = f.mulp(1u, Fm[c * TP + j]);
                continue;
            }
            ChainSum<F> acc(f);
            if (few) {
                for (uint32_t b = mask; b; b &= b - 1u) {
                    const int q = __ffs(b) - 1;
                    acc.add(f, 0, Fm[c * TP + q], G[prow[c0 + q] * TP + j]);
                }
            } else {
                uint32_t old[TP];
#pragma unroll
                for (int q = 0; q < TP; ++q)
                    old[q] = (mask >> q) & 1u ? G[prow[c0 + q] * TP + j] : 0u;
#pragma unroll
                for (int q = 0; q < TP; ++q) acc.add(f, q, Fm[c * TP + q], old[q]);
            }
            np[u] = acc.mod(f);
        }
        __syncthreads();  // every old value is read, and the last panels' NP
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int e = tid + u * kTinyThreads, c = (e / TP) % TP, j = e % TP, g = e / (TP * TP);
            if (g >= ng) continue;
            NP[e] = f.prep(np[u]);
            if ((mask >> c) & 1u) T[(size_t)(gb + g) * n * TP + prow[c0 + c] * TP + j] = np[u];
        }
        __syncthreads();
        const int wpg = kTinyWarps / ng, g = warp / wpg;
        if (g < ng && few) {
            // few pivots: their values straight from shared memory
            uint32_t* G = T + (size_t)(gb + g) * n * TP;
            const int j = lane % TP;
            const uint32_t* P = NP + g * TP * TP + j;
            const bool zero = gb + g == own && ((mask >> j) & 1u);
            for (int r = 2 * (warp % wpg) + lane / TP; r < n; r += 2 * wpg) {
                const int k = pcol[r] - c0;
                if (k >= 0 && k < TP && ((mask >> k) & 1u)) continue;
                ChainSum<F, 2> acc(f);
                uint32_t any = 0u;
                for (uint32_t b = mask; b; b &= b - 1u) {
                    const int q = __ffs(b) - 1;
                    const uint32_t x = pb[r * TP + q];
                    any |= x;
                    acc.add(f, 0, x, P[q * TP]);
                }
                if (any == 0u) continue;
                const uint32_t t = acc.mod(f), gv = zero ? 0u : G[r * TP + j];
                G[r * TP + j] = gv >= t ? gv - t : gv + (f.p - t);
            }
        } else if (g < ng) {
            uint32_t v[TP];
#pragma unroll
            for (int q = 0; q < TP; ++q) v[q] = NP[(g * TP + q) * TP + lane % TP];
            tiny_update(n, c0, mask, pb, pcol, v, T + (size_t)(gb + g) * n * TP, warp % wpg, wpg, f,
                        gb + g == own ? mask : 0u);
        }
    }
}

// The reduced echelon form of the block in the CTAs' panels (tiny_layout, columns
// past m zero).  Reached by every thread of every CTA of the cluster,
// kTinyThreads a CTA; on return pcol[row] and prow[column] hold the pivots
// (the same in every CTA) and every CTA's panels are final and visible.  With
// COEF the pivot columns hold, instead of unit vectors, the coefficients of the
// old pivot rows: row r = sum over pivot columns c of T[r][c] old_(prow[c]).
// Returns the rank.
template <bool COEF, class F>
__device__ int tiny_echelon(const int32_t n, const int32_t m, uint32_t* smem, const F f) {
    const int CL = cluster_size(), rk = cluster_rank(), sh = __ffs(CL) - 1;
    const TinyLayout L = tiny_layout(n, m, CL);
    uint32_t* T = smem;
    uint32_t* Fm = smem + L.blk;                    // [TP][TP], see tiny_turn
    uint32_t* PP = Fm + TP * TP;
    uint32_t* NP = PP + TP * TP;  // the pivot rows in panels beside it; [TG][TP][TP]
    int32_t* pcol = (int32_t*)(smem + L.rows);      // [n] pivot column of a pivot row, -1
    int32_t* prow = (int32_t*)(smem + L.cols);      // [m] pivot row of a column, -1
    __shared__ TinyTurn S;
    const int tid = threadIdx.x, lane = tid & 31;
    // Panel k from its owner to every CTA's copy for panel k, and a cluster barrier.
    // Eight copies of 256 rows (128 KB) out of one SM take 11000 cycles with the
    // lanes of a warp storing to different CTAs, 6800 with a warp's stores to one
    // CTA, and 3600 when each CTA gets a part and passes it on, a barrier more.
    const bool relay = CL > 2 && n >= kRelayRows;
    const int quads = n * (TP / 4), part = (quads + CL - 1) >> sh;  // 16-byte groups
    auto push = [&](int k) {
        const bool mine = (k & (CL - 1)) == rk;
        const uint4* src = (const uint4*)(T + (k >> sh) * n * TP);
        const uint32_t* dst = smem + L.pb + (k & 1) * n * TP;
        if (relay) {
            if (mine)
                for (int q = tid; q < quads; q += kTinyThreads)
                    remote_st4(remote_smem(dst + 4 * q, q / part), src[q]);
            cluster_sync();
            const int q1 = min(quads, (rk + 1) * part);
            const int g = tid / 32 % CL, w = tid / 32 / CL;  // warps by destination
            if (g != rk)
                for (int q = rk * part + 32 * w + tid % 32; q < q1; q += kTinyThreads / CL)
                    remote_st4(remote_smem(dst + 4 * q, g), *(const uint4*)(dst + 4 * q));
        } else if (mine) {
            for (int q = tid; q < quads; q += kTinyThreads) {
                const uint4 x = src[q];
                for (int to = 0; to < CL; ++to) remote_st4(remote_smem(dst + 4 * q, to), x);
            }
        }
        cluster_sync();
    };
    for (int c = tid; c < L.panels * TP; c += kTinyThreads) prow[c] = -1;
    for (int r = tid; r < n; r += kTinyThreads) pcol[r] = -1;
    cluster_sync();  // every CTA has started, its panels are in place
    push(0);
    constexpr uint32_t kFull = (1u << TP) - 1u;
    int found = 0;  // pivots so far (uniform over the cluster)
    for (int k = 0; k < L.panels; ++k) {
        uint32_t* pb = smem + L.pb + (k & 1) * n * TP;
        uint32_t* own = (k & (CL - 1)) == rk ? T + (k >> sh) * n * TP : nullptr;
        const int c0 = k * TP, j = lane % TP;
        uint32_t pmask = 0u;  // the panel's pivot columns so far (uniform)
        while (pmask != kFull) {
            const int left = tiny_select(n, pb, pcol, S);
            if (left == 0) break;  // uniform over the cluster
            const bool last = left <= TP;  // every nonzero row is in this turn
            if (tid < TP * TP) tiny_turn(min(left, TP), c0, pb, pcol, prow, Fm, PP, NP, S, f);
            __syncthreads();
            const uint32_t mask = S.mask;
            pmask |= mask;
            found += __popc(mask);
            // this CTA's panels right of panel k, with COEF all of them
            tiny_groups(n, c0, mask, pb, pcol, prow, Fm, NP, T,
                        COEF ? 0 : (k + CL - rk) / CL, (L.panels - rk + CL - 1) / CL,
                        COEF && own ? k >> sh : -1, f);
            if (pmask != kFull && (!last || (!COEF && own))) {
                // the panel itself, in every CTA's copy
                __syncthreads();  // the updates above have read it
                uint32_t v[TP];
#pragma unroll
                for (int q = 0; q < TP; ++q) v[q] = f.prep(PP[q * TP + j]);
                tiny_update(n, c0, mask, pb, pcol, v, pb, tid >> 5, kTinyWarps, f);
                const int c = tid / TP;
                if (c < TP && ((mask >> c) & 1u)) pb[prow[c0 + c] * TP + j] = PP[tid];
            }
            __syncthreads();
            if (last) break;
        }
        if (!COEF && pmask != 0u && own) {
            // the owner's panel: the copy, or unit columns if all have a pivot
            for (int t = tid; t < n * TP; t += kTinyThreads)
                own[t] = pmask == kFull ? (pcol[t / TP] == c0 + t % TP ? 1u : 0u) : pb[t];
        }
        if (k + 1 == L.panels) break;
        push(k + 1);
        if (found == n) break;
    }
    cluster_sync();
    return found;
}

// The pivot rows of an n-row block to its first rows, in column order; their
// number.  Through the two copies of the current panel, which are free between
// echelons and hold 2 n rows of one panel (the callers' m is at most a panel a CTA
// and at most n).  Reached by every thread of every CTA, behind tiny_echelon.
__device__ inline int tiny_keep(const int32_t n, const int32_t m, uint32_t* smem) {
    const int CL = cluster_size(), rk = cluster_rank(), tid = threadIdx.x;
    const TinyLayout L = tiny_layout(n, m, CL);
    const int32_t* prow = (const int32_t*)(smem + L.cols);
    int32_t* place = (int32_t*)(smem + L.cols) + L.panels * TP;  // [m] pivots left of a column
    __shared__ int s_part[kTinyWarps];
    for (int c = tid; c < m; c += kTinyThreads) place[c] = prow[c] >= 0 ? 1 : 0;
    __syncthreads();
    const int np = tiny_exscan(place, m, s_part);
    const int mine = (L.panels - rk + CL - 1) / CL;  // panels of this CTA
    uint32_t* copy = smem + L.pb;
    for (int q = tid; q < mine * m * TP; q += kTinyThreads) {
        const int g = q / (m * TP), c = q / TP % m;
        if (prow[c] >= 0)
            copy[(g * np + place[c]) * TP + q % TP] = smem[((size_t)g * n + prow[c]) * TP + q % TP];
    }
    __syncthreads();
    for (int q = tid; q < mine * np * TP; q += kTinyThreads)
        smem[(size_t)(q / (np * TP)) * n * TP + q % (np * TP)] = copy[q];
    return np;
}

// tiny_echelon and the compaction of its pivot rows.
template <class F>
__device__ void tiny_rref_body(const int32_t n, const int32_t m, uint32_t* smem, const TinyOut out,
                               const F f) {
    const int CL = cluster_size(), rk = cluster_rank(), sh = __ffs(CL) - 1;
    const TinyLayout L = tiny_layout(n, m, CL);
    tiny_echelon<false>(n, m, smem, f);
    const uint32_t* T = smem;
    const int32_t* pcol = (const int32_t*)(smem + L.rows);
    const int32_t* prow = (const int32_t*)(smem + L.cols);
    int32_t* rank = (int32_t*)(smem + L.cols) + L.panels * TP;  // [m] pivots right of a column
    int32_t* cnt = rank + L.panels * TP;                        // [m] entries of the answer's rows
    __shared__ int s_part[kTinyWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // ---- compaction: pivot rows in descending pivot-column order ----
    // rank of a pivot column = pivot columns to its right
    for (int c = tid; c < m; c += kTinyThreads) rank[c] = prow[m - 1 - c] >= 0 ? 1 : 0;
    __syncthreads();
    const int np = tiny_exscan(rank, m, s_part);  // rank[m-1-c] = pivots right of c
    // four columns of a row per lane and pass, read from their owners
    constexpr int CU = 4;
    auto row_values = [&](int r, int j0, uint32_t (&v)[CU]) {
#pragma unroll
        for (int u = 0; u < CU; ++u) {
            const int j = j0 + 32 * u + lane;
            v[u] = j < m ? remote_ld(remote_smem(T + tiny_at(n, r, j, sh), (j / TP) & (CL - 1))) : 0u;
        }
    };
    for (int r = rk + CL * warp; r < n; r += CL * kTinyWarps) {
        const int p0 = pcol[r];
        if (p0 < 0) continue;
        int c = 0;
        for (int j0 = p0; j0 < m; j0 += 32 * CU) {
            uint32_t v[CU];
            row_values(r, j0, v);
#pragma unroll
            for (int u = 0; u < CU; ++u) c += v[u] != 0u;
        }
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane < CL) remote_st(remote_smem(cnt + rank[m - 1 - p0], lane), (uint32_t)c);
    }
    cluster_sync();
    const int nnz = tiny_exscan(cnt, np, s_part);
    if (rk == 0) {
        for (int q = tid; q < np; q += kTinyThreads) out.offs[q] = cnt[q];
        if (out.piv_of_col)
            for (int c = tid; c < m; c += kTinyThreads) out.piv_of_col[c] = prow[c];
        if (tid == 0) {
            out.offs[np] = nnz;
            out.counts[0] = np;
            out.counts[1] = nnz;
        }
    }
    for (int r = rk + CL * warp; r < n; r += CL * kTinyWarps) {
        const int p0 = pcol[r];
        if (p0 < 0) continue;
        int64_t pos = cnt[rank[m - 1 - p0]];
        for (int j0 = p0; j0 < m; j0 += 32 * CU) {
            uint32_t v[CU];
            row_values(r, j0, v);
#pragma unroll
            for (int u = 0; u < CU; ++u) {
                const unsigned bal = __ballot_sync(0xffffffffu, v[u] != 0u);
                if (v[u]) {
                    const int64_t q = pos + __popc(bal & ((1u << lane) - 1u));
                    out.cols[q] = j0 + 32 * u + lane + out.col_shift;
                    out.vals[q] = (int32_t)v[u];
                }
                pos += __popc(bal);
            }
        }
    }
    cluster_sync();  // the other CTAs have read this one's panels
}

}  // namespace gbgpu
