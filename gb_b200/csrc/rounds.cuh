// rounds.cuh -- the bookkeeping of one echelon round (blocked.cu) in two
// launches of one CTA.
//
// A round of the echelon needs, around its panels and products, the pending
// rows, the panels in which two of them share a lead, a chunk of rows for each
// of those, and afterwards the new pivots in column order and the rows that are
// left: about thirty small launches, clears and copies when each is a kernel of
// its own, 250 us a round while the data is a few thousand integers.  One CTA
// does either half in 8 to 15 us (8192 rows and columns; the dense RREF's 49
// rounds took 24.1 ms before, 17.9 ms now), and what the host has to know (the counts
// that size the next launches) lands in mapped host memory.
#pragma once
#include <stdint.h>

#include "common.cuh"

namespace gbgpu {

constexpr int RD_THREADS = 1024, RD_WARPS = RD_THREADS / 32;
constexpr int kInfoFirst = 16000;  // blocks of KB pivots whose first column the host can read

// mapped host memory, written by the kernels below
struct RoundInfo {
    int64_t entries;                                // of an answer block (k_offs_write)
    int32_t n_pend, n_dirty, first_panel, n_clean;  // k_round_plan
    int32_t n_new, n_rest;                          // k_round_finish
    int32_t first[kInfoFirst];                      // column of pivot 128 b
};

struct RoundState {
    int32_t t, ncr, npan, max_dirty;
    const int32_t* lead;   // [t], -1: zero row
    uint8_t* is_piv;       // [t]
    int32_t* piv_of_col;   // [ncr]
    int32_t* wflag;        // [ncr]: column got its pivot this round
    int32_t* hist;         // [ncr]
    int32_t* pdirty;       // [npan]
    int32_t* dslot;        // [npan]: chunk of a panel, -1
    int32_t* dpanel;       // [max_dirty]: panel of a chunk
    int32_t* cursor;       // [max_dirty]: rows of a chunk's panel
    int32_t* chunk_rows;   // [max_dirty][pr]
    int32_t* per_warp;     // [RD_WARPS][max_dirty]
    int32_t* cls;          // k_panel_apply's lists, their three counts first
    int32_t *pc, *prow;    // [ncr]: pivot columns ascending, their rows
    int32_t* pend;         // [t]: rows left
    int32_t* n_new;        // device copy of info->n_new
    RoundInfo* info;
};

// exclusive prefix of v over the block; *total gets the sum.  Two barriers.
__device__ __forceinline__ int block_prefix(int v, int* s_warp, int* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += x;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    const int mine = s_warp[lane];  // RD_WARPS == 32
    int sum = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += x;
    }
    *total = __shfl_sync(0xffffffffu, sum, 31);
    const int before = __shfl_sync(0xffffffffu, sum - mine, warp);
    __syncthreads();  // s_warp is rewritten by the next call
    return before + inc - v;
}

// Pending rows (nonzero, no pivots); a panel of kb columns is dirty when two of
// them share a lead in it.  The rows of the other panels become pivots; every
// dirty panel (the leftmost max_dirty) gets its pending rows, in row order, as a
// chunk of at most pr.  Every warp owns a contiguous run of rows, so the order
// does not depend on timing.
//
// Bound by the latency of its dependent loads: a warp asks for RD_GRP groups of
// 32 rows at a time (8192 rows: one batch a pass) and the counts of up to
// RD_COUNTS chunks are held in shared memory.  8192 rows in one dirty panel take
// 15 us, 37 us with one group in flight and the counts in global memory.
constexpr int RD_GRP = 8, RD_COUNTS = 256;

__global__ void __launch_bounds__(RD_THREADS) k_round_plan(const RoundState a, int32_t kb, int32_t pr) {
    __shared__ int s_pend, s_clean, s_dirty;
    __shared__ int s_cnt[RD_WARPS * RD_COUNTS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int c = tid; c < a.ncr; c += RD_THREADS) {
        a.hist[c] = 0;
        a.wflag[c] = 0;
    }
    for (int q = tid; q < a.npan; q += RD_THREADS) {
        a.pdirty[q] = 0;
        a.dslot[q] = -1;
    }
    if (tid == 0) s_pend = s_clean = s_dirty = 0;
    if (tid < 3) a.cls[tid] = 0;
    __syncthreads();
    const int run = (a.t + RD_THREADS - 1) / RD_THREADS * 32;  // rows of a warp
    const int r0 = warp * run, r1 = min(a.t, r0 + run);
    int l[RD_GRP];
    auto leads = [&](int rb) {  // of the lane's rows in the groups from rb, -1: not pending
#pragma unroll
        for (int g = 0; g < RD_GRP; ++g) {
            const int r = rb + 32 * g + lane;
            l[g] = r < r1 ? a.lead[r] : -1;
            if (r < r1 && a.is_piv[r]) l[g] = -1;
        }
    };
    int count = 0;
    for (int rb = r0; rb < r1; rb += 32 * RD_GRP) {
        leads(rb);
        bool twice[RD_GRP];
#pragma unroll
        for (int g = 0; g < RD_GRP; ++g) {
            // one atomic per lead and warp: a dense block's rows share theirs
            const unsigned same = __match_any_sync(0xffffffffu, l[g]);
            twice[g] = false;
            if (l[g] >= 0 && __ffs(same) - 1 == lane)
                twice[g] = (atomicAdd(&a.hist[l[g]], 1) > 0) | (__popc(same) > 1);
            count += l[g] >= 0;
        }
#pragma unroll
        for (int g = 0; g < RD_GRP; ++g)
            if (twice[g]) a.pdirty[l[g] / kb] = 1;
    }
    count = __reduce_add_sync(0xffffffffu, count);
    if (lane == 0 && count) atomicAdd(&s_pend, count);
    __syncthreads();
    if (warp == 0) {
        int n = 0;
        for (int q0 = 0; q0 < a.npan; q0 += 32) {
            const int q = q0 + lane;
            const bool d = q < a.npan && a.pdirty[q];
            const unsigned bal = __ballot_sync(0xffffffffu, d);
            const int slot = n + __popc(bal & ((1u << lane) - 1u));
            if (d) a.dslot[q] = slot < a.max_dirty ? slot : -2;
            if (d && slot < a.max_dirty) a.dpanel[slot] = q;
            n += __popc(bal);
        }
        if (lane == 0) s_dirty = min(n, a.max_dirty);
    }
    __syncthreads();
    const int nd = s_dirty;
    int32_t* const cnt = nd <= RD_COUNTS ? s_cnt : a.per_warp;
    int32_t* const mine = cnt + (size_t)warp * nd;
    for (int d = lane; d < nd; d += 32) mine[d] = 0;
    __syncwarp();
    int slot[RD_GRP];
    auto slots = [&]() {
#pragma unroll
        for (int g = 0; g < RD_GRP; ++g) slot[g] = l[g] >= 0 ? a.dslot[l[g] / kb] : -3;
    };
    int clean = 0;
    for (int rb = r0; rb < r1; rb += 32 * RD_GRP) {
        leads(rb);
        slots();
#pragma unroll
        for (int g = 0; g < RD_GRP; ++g) {
            if (slot[g] == -1) {  // clean
                const int r = rb + 32 * g + lane;
                a.piv_of_col[l[g]] = r;
                a.is_piv[r] = 1;
                a.wflag[l[g]] = 1;
                ++clean;
            }
            const unsigned same = __match_any_sync(0xffffffffu, slot[g]);
            if (slot[g] >= 0 && __ffs(same) - 1 == lane) mine[slot[g]] += __popc(same);
            __syncwarp();
        }
    }
    clean = __reduce_add_sync(0xffffffffu, clean);
    if (lane == 0 && clean) atomicAdd(&s_clean, clean);
    __syncthreads();
    for (int d = tid; d < nd; d += RD_THREADS) {
        int sum = 0;
        for (int w = 0; w < RD_WARPS; ++w) {
            const int x = cnt[(size_t)w * nd + d];
            cnt[(size_t)w * nd + d] = sum;
            sum += x;
        }
        a.cursor[d] = sum;
    }
    __syncthreads();
    for (int rb = r0; rb < r1; rb += 32 * RD_GRP) {
        leads(rb);  // claimed rows are pivots by now
        slots();
#pragma unroll
        for (int g = 0; g < RD_GRP; ++g) {
            const unsigned same = __match_any_sync(0xffffffffu, slot[g]);
            if (slot[g] >= 0) {
                const int at = mine[slot[g]] + __popc(same & ((1u << lane) - 1u));
                if (at < pr) a.chunk_rows[(size_t)slot[g] * pr + at] = rb + 32 * g + lane;
            }
            __syncwarp();
            if (slot[g] >= 0 && __ffs(same) - 1 == lane) mine[slot[g]] += __popc(same);
            __syncwarp();
        }
    }
    if (tid == 0) {
        a.info->n_pend = s_pend;
        a.info->n_dirty = nd;
        a.info->first_panel = nd > 0 ? a.dpanel[0] : 0;
        a.info->n_clean = s_clean;
    }
}

// The round's new pivots (`all`: every pivot) in ascending column order, and the
// rows left, in row order.  With pad_rows > 0 the lists are filled up with -1, the
// pivots to kb (they are at most as many) and the rows to pad_rows, for a
// host that does not wait for their lengths.
__global__ void __launch_bounds__(RD_THREADS)
k_round_finish(const RoundState a, int32_t kb, int32_t all, int32_t pad_rows = 0) {
    __shared__ int s_warp[RD_WARPS];
    const int tid = threadIdx.x;
    // four columns (rows) per thread and pass
    int n = 0;
    for (int c0 = 4 * tid; c0 - 4 * tid < a.ncr; c0 += 4 * RD_THREADS) {
        int row[4], k = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int c = c0 + u;
            row[u] = c < a.ncr && (all || a.wflag[c]) ? a.piv_of_col[c] : -1;
            k += row[u] >= 0;
        }
        int total;
        int at = n + block_prefix(k, s_warp, &total);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (row[u] < 0) continue;
            a.pc[at] = c0 + u;
            a.prow[at] = row[u];
            if (at % kb == 0 && at / kb < kInfoFirst) a.info->first[at / kb] = c0 + u;
            ++at;
        }
        n += total;
    }
    int rest = 0;
    for (int r0 = 4 * tid; !all && r0 - 4 * tid < a.t; r0 += 4 * RD_THREADS) {
        bool p[4];
        int k = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            p[u] = r0 + u < a.t && a.lead[r0 + u] >= 0 && !a.is_piv[r0 + u];
            k += p[u];
        }
        int total;
        int at = rest + block_prefix(k, s_warp, &total);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (p[u]) a.pend[at++] = r0 + u;
        rest += total;
    }
    if (pad_rows > 0) {
        for (int k = n + tid; k < min(kb, a.ncr); k += RD_THREADS) a.pc[k] = a.prow[k] = -1;
        for (int k = rest + tid; k < pad_rows; k += RD_THREADS) a.pend[k] = -1;
    }
    if (tid == 0) {
        *a.n_new = n;
        a.info->n_new = n;
        a.info->n_rest = rest;
    }
}

}  // namespace gbgpu
