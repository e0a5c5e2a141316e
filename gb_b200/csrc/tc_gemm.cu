// tc_gemm.cu -- exact modular GEMM  D <- (D - A B) mod p  on the int8 tensor
// cores of sm_100a (tcgen05.mma kind::i8, TMA, TMEM), and its plain CUDA-core
// twin.
//
// Residues (uint32 in [0, p), p < 2^31 odd) are split into L unsigned bytes,
// a = sum_i a_i 2^(8i) with L = 1 (p < 2^8), 2 (< 2^16), 3 (< 2^24), 4.  Then
//   A B = sum_w 2^(8w) S_w,   S_w = sum_{i+j=w} A_i B_j,   w = 0 .. 2L-2,
// and every S_w is a u8 x u8 -> s32 tensor-core product accumulated in TMEM.
// At most L limb pairs share a weight, each product is <= 255^2, so a K panel
// of at most floor((2^31-1) / (L 255^2)) columns keeps every S_w below 2^31
// (kPanelBytes below).  After each panel the epilogue folds the weights,
//   v = sum_w S_w * (2^(8w) R mod p)   (Montgomery, R = 2^32; one reduction of
//       the 64-bit sum) for two and three limbs, one Barrett step of S_0 for one,
//       three reductions for four,
// and updates D <- D - v mod p in place, so no partial sum ever leaves [0, p).
// The result is bit-identical to any exact evaluation of (D - A B) mod p.
//
// Pipeline (one CTA per 128 x BN output tile, 320 threads):
//   warp 0      TMA producer: L A-limb tiles (128 x 128 B) and L B-limb tiles
//               (BN x 128 B) per 128-byte K step into a STAGES-deep ring,
//               128-byte swizzle (the canonical K-major UMMA layout);
//   warp 1      TMEM allocation and MMA issue (one elected thread), stage
//               release through tcgen05.commit;
//   warps 2..9  epilogue: tcgen05.ld of the 2L-1 weight accumulators of its
//               32-lane TMEM quarter, fold, read-modify-write of D.
//
// What bounds it (cycle counts in the roles, B200): an MMA 128 x BN x 32 takes
// 184 / 80 / 53 cycles for BN = 256 / 128 / 64 (the rate cuBLAS's int8 product
// reaches at BN = 256), so long K is bound by the MMAs, and short K by the
// epilogue's path to D.  With the epilogue below, kernel and splits:
// 8192^3, p = 251: 879 -> 613 us; 5000 x 8000 x 1024: 359 -> 159 us (p = 251),
// 340 -> 301 us (p = 65521), 1013 -> 717 us (p = 2^31 - 1); 5000 x 20000 x 256:
// 410 -> 327, 471 -> 350, 1418 -> 679 us.  CTA pairs (cta_group::2, 256-row tiles)
// were tried before that epilogue only: 914 us against 1048 on 8192^3, p = 251, and
// equal or slower elsewhere.  They move a third less per flop, and shared memory's
// bandwidth bounds that product now (235 cycles an MMA), so this is open.
// Every mbarrier wait is bounded (clock64 budget); on expiry the CTA records
// GBGPU_ETIMEDOUT in *err, drains its in-flight copies and frees its TMEM.
// No cluster multicast is used anywhere.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <string>

#include "../../include/gbgpu.h"
#include "field.cuh"
#include "internal.h"
#include "tc_gemm.h"
#include "tc_shape.h"

namespace gbgpu {

// ---------------------------------------------------------------------------
// PTX wrappers
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Wait for the phase of parity `parity` to complete, at most `budget` cycles.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, long long budget) {
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - t0 > budget) return false;
    }
    return true;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y,
                                            uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"((uint64_t)map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     bar)
                 : "memory");
}
__device__ __forceinline__ void tc_mma_i8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                          uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// 16 consecutive TMEM columns of this warp's 32 lanes (one row per thread)
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
// the loads above have landed; `r` passes through so that no use moves before it
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                   "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                   "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])::"memory");
}

// K-major operand tile with 128-byte swizzle: rows of 128 bytes, 8-row
// groups 1024 bytes apart (SBO), LBO unused (1), descriptor version 1.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// ---------------------------------------------------------------------------
// Tile shapes (SHAPE):
//   TC_BIG   128 x BN tiles, one CTA per SM: 128 x 256 for L = 1, 128 x 128 for
//            L = 2, 128 x 64 for L = 3, 4.  One limb keeps its accumulators twice
//            (the next tile's MMAs run while the epilogue drains the last);
//            2 x NW x BN does not fit the 512 TMEM columns of the others;
//   TC_MID   one or two limbs, 128 x 64 tiles, accumulators twice.
// tc_shape.h has the rule that picks one.

template <int L, int SHAPE = TC_BIG>
struct TcCfg {
    static constexpr int BM = 128;
    static constexpr int BK = 128;  // bytes of K per stage (one swizzle row)
    static constexpr int BN = SHAPE == TC_MID ? 64 : (L == 1 ? 256 : (L == 2 ? 128 : 64));
    static constexpr int NW = 2 * L - 1;
    // accumulator sets in TMEM (see the shapes above)
    static constexpr int ACC_BUFS = 2 * (2 * L - 1) * BN <= 512 ? 2 : 1;
    static constexpr int A_BYTES = BM * BK;
    static constexpr int B_BYTES = BN * BK;
    static constexpr int STAGE_BYTES = L * (A_BYTES + B_BYTES);
    static constexpr int STAGES = L == 1 ? 4 : (L == 2 ? (BN == 128 ? 3 : 4) : 2);
    static constexpr int ACC_COLS = ACC_BUFS * NW * BN;
    static constexpr int TMEM_COLS =
        ACC_COLS <= 64 ? 64 : (ACC_COLS <= 128 ? 128 : (ACC_COLS <= 256 ? 256 : 512));
    // epilogue warps: two per TMEM lane quarter, each half of the columns
    static constexpr int EPI_WARPS = 8;
    static constexpr int THREADS = 64 + 32 * EPI_WARPS;
    static constexpr int COLS = BN / (EPI_WARPS / 4);  // columns of an epilogue warp
    // epilogue staging: a 32 x 32 block per epilogue warp (XOR-swizzled columns)
    static constexpr int STG_BYTES = EPI_WARPS * 32 * 32 * 4;
    static constexpr int BAR_OFF = STAGES * STAGE_BYTES;
    static constexpr int STG_OFF = BAR_OFF + 256;
    static constexpr int USED_BYTES = STG_OFF + STG_BYTES + 1024 /*align*/;
    static constexpr int SMEM_BYTES = USED_BYTES;
    // K bytes per panel: L * 255^2 * K < 2^31
    static constexpr int PANEL_KB = L == 1 ? 256 : (L == 2 ? 128 : (L == 3 ? 85 : 64));
    static constexpr uint32_t IDESC = (2u << 4)                      // D = s32
                                      | (0u << 7) | (0u << 10)       // A, B = u8
                                      | ((uint32_t)(BN >> 3) << 17)  // N
                                      | ((uint32_t)(BM >> 4) << 24); // M
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");
    static_assert(ACC_COLS <= 512, "TMEM columns");
};

// tiles of one batch item are visited in groups of TC_GROUP_M row tiles, all
// column tiles of a group before the next, so that the B tiles of a column are
// reused from L2 by the row tiles of the group
constexpr int TC_GROUP_M = 8;

struct TcParams {
    uint32_t* D;
    int64_t ldd, sD;
    const int32_t* d_rows;  // optional: row m of D is D + d_rows[m] ldd (< 0: not written)
    int64_t sDr;
    int32_t M, N, Mp, Np, nkb, nkbp, batch;
    // nonzero flags of the 128-row x 128-byte A tiles ([Mp/128][nkbp]) and of the
    // BN-row x 128-byte B tiles ([Np/BN][nkbp], nkbp = nkb rounded up to 64, the
    // padding zero); a K step where either tile is
    // zero contributes nothing and is skipped (NULL: no skipping)
    const uint8_t* fa;
    const uint8_t* fb;
    unsigned long long* steps;  // optional: K steps executed, summed over tiles
    uint32_t p, pneg_inv;
    uint32_t mu;     // floor(2^32 / p)
    uint32_t cw[5];    // 2^(8w) R mod p
    uint32_t r2, r3;   // R^2, R^3 mod p
    int32_t set;     // D <- -A B: D is not read
    int32_t* err;
    long long budget;
};

// VEC: D and its row and batch strides are 16-byte aligned
template <int L, int SHAPE, bool VEC>
__global__ void __launch_bounds__(TcCfg<L, SHAPE>::THREADS, 1)
k_tc_submul(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
            const TcParams prm) {
    using C = TcCfg<L, SHAPE>;
    extern __shared__ uint8_t smem_raw[];
    // 1024-byte aligned tile region (shared-window address)
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* gbase = smem_raw + (base - raw);
    uint64_t* bars = (uint64_t*)(gbase + C::BAR_OFF);
    // bars: full[STAGES], empty[STAGES], tmem_full[ACC_BUFS], tmem_empty[ACC_BUFS];
    // then tmem slot, abort flag
    const uint32_t bar0 = smem_u32(bars);
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (C::STAGES + s); };
    auto tfull_bar = [&](int b) { return bar0 + 8u * (2 * C::STAGES + b); };
    auto tempty_bar = [&](int b) { return bar0 + 8u * (2 * C::STAGES + C::ACC_BUFS + b); };
    volatile uint32_t* tmem_slot = (volatile uint32_t*)(bars + 2 * C::STAGES + 2 * C::ACC_BUFS);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nkb = prm.nkb;
    const int tiles_m = prm.Mp / C::BM, tiles_n = prm.Np / C::BN;
    const int per_z = tiles_m * tiles_n;
    const int total = per_z * prm.batch;
    // tile t -> batch item z, row tile mt, column tile nt (grouped raster)
    auto coords = [&](int t, int& z, int& mt, int& nt) {
        z = t / per_z;
        const int r = t - z * per_z;
        const int span = TC_GROUP_M * tiles_n;
        const int first_m = (r / span) * TC_GROUP_M;
        const int gm = min(TC_GROUP_M, tiles_m - first_m);
        const int rr = r - (r / span) * span;
        mt = first_m + rr % gm;
        nt = rr / gm;
    };
    // flags of the tile's A row block and B column block (NULL: all live)
    const int nkbp = prm.nkbp;
    auto flag_ptrs = [&](int z, int mt, int nt, const uint8_t*& fa, const uint8_t*& fb) {
        fa = prm.fa ? prm.fa + ((size_t)z * tiles_m + mt) * nkbp : nullptr;
        // B flags are kept per 64 rows of B's planes: the tile's BN / 64 rows
        fb = prm.fb ? prm.fb + ((size_t)z * (prm.Np / 64) + (size_t)nt * (C::BN / 64)) * nkbp
                    : nullptr;
    };
    // live K steps [64 ch, 64 ch + 64) of a tile as a bit mask, from 16-byte
    // loads of the A flag row and of the OR of the tile's B flag rows (flags
    // are 0 or 1 bytes)
    auto live_mask = [&](const uint8_t* fa, const uint8_t* fb, int ch) -> uint64_t {
        uint64_t msk = 0;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const int kb0 = ch * 64 + v * 16;
            if (kb0 >= nkb) break;  // padding only
            uint4 a = make_uint4(0x01010101u, 0x01010101u, 0x01010101u, 0x01010101u);
            uint4 b = a;
            if (fa) a = *(const uint4*)(fa + kb0);
            if (fb) {
                b = *(const uint4*)(fb + kb0);
#pragma unroll
                for (int r = 1; r < C::BN / 64; ++r) {
                    const uint4 o = *(const uint4*)(fb + (size_t)r * nkbp + kb0);
                    b.x |= o.x;
                    b.y |= o.y;
                    b.z |= o.z;
                    b.w |= o.w;
                }
            }
            const uint32_t w[4] = {a.x & b.x, a.y & b.y, a.z & b.z, a.w & b.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t x = w[j];
                const uint32_t bits = (x & 1u) | ((x >> 7) & 2u) | ((x >> 14) & 4u) | ((x >> 21) & 8u);
                msk |= (uint64_t)bits << (v * 16 + j * 4);
            }
        }
        if (!fa && !fb) {
            // no flags at all: every real K step is live
            const int rem = nkb - ch * 64;
            msk = rem >= 64 ? ~0ull : (rem > 0 ? ((1ull << rem) - 1ull) : 0ull);
        } else if (nkb - ch * 64 < 64) {
            const int rem = nkb - ch * 64;
            msk &= rem > 0 ? ((1ull << rem) - 1ull) : 0ull;
        }
        return msk;
    };
    const int nch = (nkb + 63) / 64;
    auto live_steps = [&](const uint8_t* fa, const uint8_t* fb) {
        int n_it = 0;
        for (int ch = 0; ch < nch; ++ch) n_it += __popcll(live_mask(fa, fb, ch));
        return n_it;
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int b = 0; b < C::ACC_BUFS; ++b) {
            mbar_init(tfull_bar(b), 1);
            mbar_init(tempty_bar(b), C::EPI_WARPS);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32((const void*)tmem_slot)),
                     "r"((uint32_t)C::TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    // Every role walks the same tile sequence and skips the tiles whose
    // product is zero.  The operand ring and the accumulator phases continue
    // across tiles, so the producer fetches the next tile while the epilogue
    // drains the current one.
    if (warp == 0) {
        if (lane == 0) {
            // ---- producer ----
            int it = 0;
            bool stop = false;
            for (int t = blockIdx.x; t < total && !stop; t += gridDim.x) {
                int z, mt, nt;
                coords(t, z, mt, nt);
                const uint8_t *fa, *fb;
                flag_ptrs(z, mt, nt, fa, fb);
                const int m0 = mt * C::BM, n0 = nt * C::BN;
                int n_tile = 0;
                for (int ch = 0; ch < nch && !stop; ++ch) {
                  uint64_t msk = live_mask(fa, fb, ch);
                  while (msk) {
                    const int kb = ch * 64 + __ffsll((long long)msk) - 1;
                    msk &= msk - 1;
                    const int s = it % C::STAGES;
                    const uint32_t ph = (it / C::STAGES) & 1;
                    if (*abort_flag || !mbar_wait(empty_bar(s), ph ^ 1, prm.budget)) {
                        *abort_flag = 1;
                        stop = true;
                        break;
                    }
                    mbar_expect_tx(full_bar(s), C::STAGE_BYTES);
                    const uint32_t st = base + s * C::STAGE_BYTES;
                    for (int l = 0; l < L; ++l)
                        tma_load_2d(st + l * C::A_BYTES, &mapA, kb * C::BK,
                                    (z * L + l) * prm.Mp + m0, full_bar(s));
                    for (int l = 0; l < L; ++l)
                        tma_load_2d(st + L * C::A_BYTES + l * C::B_BYTES, &mapB, kb * C::BK,
                                    (z * L + l) * prm.Np + n0, full_bar(s));
                    ++it;
                    ++n_tile;
                  }
                }
                if (prm.steps && n_tile) atomicAdd(prm.steps, (unsigned long long)n_tile);
            }
            // on abort, let the copies already issued land before the CTA exits
            for (int q = it > C::STAGES ? it - C::STAGES : 0; q < it; ++q)
                mbar_wait(full_bar(q % C::STAGES), (q / C::STAGES) & 1, prm.budget);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // ---- MMA issuer ----
            int it = 0, pc = 0;  // k steps and accumulator panels so far
            bool stop = false;
            for (int t = blockIdx.x; t < total && !stop; t += gridDim.x) {
                int z, mt, nt;
                coords(t, z, mt, nt);
                const uint8_t *fa, *fb;
                flag_ptrs(z, mt, nt, fa, fb);
                const int n_it = live_steps(fa, fb);
                int j = 0;
                for (int ch = 0; ch < nch && !stop; ++ch) {
                  uint64_t msk = live_mask(fa, fb, ch);
                  while (msk) {
                    msk &= msk - 1;
                    const int s = it % C::STAGES;
                    const uint32_t ph = (it / C::STAGES) & 1;
                    const int pk = j % C::PANEL_KB;
                    const int ab = pc % C::ACC_BUFS, au = pc / C::ACC_BUFS;
                    if (pk == 0 && au > 0) {
                        // this accumulator set is free once the epilogue read its last panel
                        if (*abort_flag || !mbar_wait(tempty_bar(ab), (au - 1) & 1, prm.budget)) {
                            *abort_flag = 1;
                            stop = true;
                            break;
                        }
                    }
                    if (*abort_flag || !mbar_wait(full_bar(s), ph, prm.budget)) {
                        *abort_flag = 1;
                        stop = true;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t st = base + s * C::STAGE_BYTES;
                    // the descriptors of the stage's operands: the start address
                    // field holds address / 16 in its low 14 bits, and every
                    // operand of the stage lies below 2^18 bytes, so an offset
                    // adds to the descriptor without a carry out of the field
                    const uint64_t dst = umma_desc_sw128(st);
#pragma unroll
                    for (int i = 0; i < L; ++i) {
#pragma unroll
                        for (int jj = 0; jj < L; ++jj) {
                            const int w = i + jj;
                            const bool first_pair = (i == (w > L - 1 ? w - (L - 1) : 0));
#pragma unroll
                            for (int kk = 0; kk < C::BK / 32; ++kk) {
                                const uint64_t ad = dst + (uint64_t)((i * C::A_BYTES + kk * 32) >> 4);
                                const uint64_t bd =
                                    dst + (uint64_t)((L * C::A_BYTES + jj * C::B_BYTES + kk * 32) >> 4);
                                const uint32_t acc = (pk == 0 && kk == 0 && first_pair) ? 0u : 1u;
                                tc_mma_i8(tmem + (uint32_t)(ab * C::NW * C::BN + w * C::BN), ad, bd,
                                          C::IDESC, acc);
                            }
                        }
                    }
                    tc_commit(empty_bar(s));
                    if (pk == C::PANEL_KB - 1 || j == n_it - 1) {
                        tc_commit(tfull_bar(ab));
                        ++pc;
                    }
                    ++it;
                    ++j;
                  }
                }
            }
        }
    } else {
        // ---- epilogue: warps 2.., TMEM lane quarter warp % 4, column half ----
        // Thread `lane` folds row q*32+lane of the tile; the 32 x 32 result
        // block goes through shared memory so that the read-modify-write of D
        // runs along rows (one 128-byte row segment per warp instruction).
        //
        // The D values of a warp's first two blocks are loaded before it waits for
        // the accumulators, and those of a later one two blocks ahead: a load of D queues behind the operand ring's copies
        // (up to 192 KB ahead of it, about 7000 cycles), so one that is only
        // issued when its block is folded costs the epilogue more than the
        // MMAs of the tile take (8192^3, p = 251: 25000 cycles per 32 x 32
        // block, and the MMA warp waited 43% of its time for a free set of
        // accumulators).
        const int e = warp - 2;
        const int q = warp & 3;
        constexpr int NB = C::COLS / 32;  // blocks of this warp
        const int cbeg = (e / 4) * C::COLS;
        const int row = q * 32 + lane;
        const uint32_t p = prm.p;
        uint32_t* stg = (uint32_t*)(gbase + C::STG_OFF + (size_t)e * 32 * 32 * 4);
        int pc = 0;
        bool stop = false;
        for (int t = blockIdx.x; t < total && !stop; t += gridDim.x) {
            int z, mt, nt;
            coords(t, z, mt, nt);
            const uint8_t *fa, *fb;
            flag_ptrs(z, mt, nt, fa, fb);
            const int n_it = live_steps(fa, fb);
            if (n_it == 0 && !prm.set) continue;  // A B is zero here: D stays as it is
            const int npanels = (n_it + C::PANEL_KB - 1) / C::PANEL_KB;
            const int m0 = mt * C::BM, n0 = nt * C::BN;
            const int gm = m0 + row;
            uint32_t* Dz = prm.D + (size_t)z * prm.sD;
            // row `lane` of the warp's 32 rows in D (< 0: not written)
            int32_t ri = -1;
            if (gm < prm.M) ri = prm.d_rows ? prm.d_rows[(size_t)z * prm.sDr + gm] : gm;
            const bool rows_here = __any_sync(0xffffffffu, ri >= 0);
            const int rows_q = prm.M - (m0 + q * 32);  // rows of the warp in the matrix
            uint32_t* Dq = Dz + (size_t)(m0 + q * 32) * prm.ldd;
            // A 32 x 32 block of D in registers.  VEC: entry 4 i + u of a lane is
            // row 4 i + lane / 8, column 4 (lane % 8) + u (one 16-byte access per
            // four entries); otherwise entry r is row r, column `lane`.
            const int vr = lane / 8, vc = 4 * (lane % 8);
            auto load_d = [&](int c0, uint32_t (&dv)[32]) {
                if constexpr (VEC) {
                    const int gn = n0 + c0 + vc;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int r = 4 * i + vr;
                        const int32_t rr = prm.d_rows ? __shfl_sync(0xffffffffu, ri, r)
                                                      : (r < rows_q ? m0 + q * 32 + r : -1);
                        const uint32_t* o = Dz + (size_t)(rr < 0 ? 0 : rr) * prm.ldd + gn;
                        uint4 x = make_uint4(0u, 0u, 0u, 0u);
                        if (rr >= 0 && gn + 4 <= prm.N) {
                            x = *(const uint4*)o;
                        } else if (rr >= 0) {
                            if (gn < prm.N) x.x = o[0];
                            if (gn + 1 < prm.N) x.y = o[1];
                            if (gn + 2 < prm.N) x.z = o[2];
                        }
                        dv[4 * i] = x.x;
                        dv[4 * i + 1] = x.y;
                        dv[4 * i + 2] = x.z;
                        dv[4 * i + 3] = x.w;
                    }
                } else {
                    const int gn = n0 + c0 + lane;
                    const bool col_ok = gn < prm.N;
                    if (prm.d_rows) {
#pragma unroll
                        for (int r = 0; r < 32; ++r) {
                            const int32_t rr = __shfl_sync(0xffffffffu, ri, r);
                            dv[r] = (rr >= 0 && col_ok) ? Dz[(size_t)rr * prm.ldd + gn] : 0u;
                        }
                    } else {
                        const uint32_t* o = Dq + gn;
#pragma unroll
                        for (int r = 0; r < 32; ++r, o += prm.ldd)
                            dv[r] = (r < rows_q && col_ok) ? *o : 0u;
                    }
                }
            };
            if (n_it == 0) {  // D <- 0
                for (int r = 0; r < 32; ++r) {
                    const int32_t rr = __shfl_sync(0xffffffffu, ri, r);
                    for (int j = lane; j < C::COLS; j += 32)
                        if (rr >= 0 && n0 + cbeg + j < prm.N)
                            Dz[(size_t)rr * prm.ldd + n0 + cbeg + j] = 0u;
                }
                continue;
            }
            for (int panel = 0; panel < npanels; ++panel, ++pc) {
                const int ab = pc % C::ACC_BUFS, au = pc / C::ACC_BUFS;
                const uint32_t acc_base = (uint32_t)(ab * C::NW * C::BN);
                // (this lane wrote the same addresses in the previous panel, if any)
                // blocks in flight (unaligned one-limb tiles: two spill, 259 us
                // against 225 for 8192 x 8001 x 128)
                constexpr int PRE = NB > 1 && (VEC || L > 1) ? 2 : 1;
                const bool fresh = prm.set && panel == 0;  // nothing to read
                uint32_t dv[PRE][32];
#pragma unroll
                for (int b = 0; b < PRE; ++b) {
                    if (rows_here && !fresh) {
                        load_d(cbeg + 32 * b, dv[b]);
                    } else {
#pragma unroll
                        for (int r = 0; r < 32; ++r) dv[b][r] = 0u;
                    }
                }
                bool ok = true;
                if (lane == 0) ok = !*abort_flag && mbar_wait(tfull_bar(ab), au & 1, prm.budget);
                ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                if (!ok) {
                    if (lane == 0) *abort_flag = 1;
                    stop = true;
                    break;
                }
                tc_fence_after();
                // a warp with no row to write keeps only its place in the
                // accumulator handshake
                if (!rows_here) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(tempty_bar(ab));
                    continue;
                }
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    const int c0 = cbeg + 32 * b;
                    uint32_t(&d)[32] = dv[b % PRE];
                    uint32_t v[32];
                    const uint32_t acc_q = tmem + ((uint32_t)(q * 32) << 16) + acc_base + (uint32_t)c0;
                    if constexpr (L == 1) {
                        // S_0 < 2^31: one Barrett step (through the weights' sum
                        // 8192 x 8192 x 128 took 190 us, 181 now)
                        uint32_t a[2][16];
                        tmem_ld16(acc_q, a[0]);
                        tmem_ld16(acc_q + 16, a[1]);
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            tmem_wait(a[h]);
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                const uint32_t r = a[h][j] - __umulhi(a[h][j], prm.mu) * p;
                                v[16 * h + j] = r >= p ? r - p : r;
                            }
                        }
                    } else if constexpr (L <= 3) {
                        // one Montgomery reduction of the weighted sum:
                        // T = sum_w S_w (2^(8w) R mod p) < (2L - 1) 2^31 p, so
                        // (T + q p) / 2^32 < 2^32, then one Barrett step; 16
                        // columns at a time (registers)
#pragma unroll
                        for (int h = 0; h < 32; h += 16) {
                            uint32_t a[C::NW][16];
#pragma unroll
                            for (int w = 0; w < C::NW; ++w)
                                tmem_ld16(acc_q + (uint32_t)(w * C::BN + h), a[w]);
                            uint64_t T[16];
#pragma unroll
                            for (int w = 0; w < C::NW; ++w) {
                                tmem_wait(a[w]);
                                const uint32_t cw = prm.cw[w];
#pragma unroll
                                for (int j = 0; j < 16; ++j)
                                    T[j] = (w == 0 ? 0ull : T[j]) + (uint64_t)a[w][j] * cw;
                            }
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                const uint32_t qq = (uint32_t)T[j] * prm.pneg_inv;
                                const uint32_t t = (uint32_t)((T[j] + (uint64_t)qq * p) >> 32);
                                const uint32_t r = t - __umulhi(t, prm.mu) * p;
                                v[h + j] = r >= p ? r - p : r;
                            }
                        }
                    } else {
                        // t0 = S_0 + .. + S_3 2^24 and t1 = S_4 + .. + S_6 2^16, both
                        // below 2^56 <= p 2^32: redc(t0) R^2 + redc(t1) R^3 < 2 p^2,
                        // and its redc is t0 + t1 2^32 (a reduction per two weights
                        // took 388 us for 8192 x 8192 x 128, 349 now).  The same
                        // by shifts for two limbs needs registers in flight that the
                        // D values have: 225 -> 233 to 296 us
                        auto redc = [&](uint64_t T) {
                            const uint32_t qq = (uint32_t)T * prm.pneg_inv;
                            const uint32_t r = (uint32_t)((T + (uint64_t)qq * p) >> 32);
                            return r >= p ? r - p : r;
                        };
#pragma unroll
                        for (int h = 0; h < 32; h += 16) {
                            uint32_t a[4][16], u[16];
#pragma unroll
                            for (int w = 0; w < 4; ++w)
                                tmem_ld16(acc_q + (uint32_t)(w * C::BN + h), a[w]);
#pragma unroll
                            for (int w = 0; w < 4; ++w) tmem_wait(a[w]);
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                u[j] = redc(a[0][j] + ((uint64_t)a[1][j] << 8) +
                                            ((uint64_t)a[2][j] << 16) + ((uint64_t)a[3][j] << 24));
#pragma unroll
                            for (int w = 4; w < 7; ++w)
                                tmem_ld16(acc_q + (uint32_t)(w * C::BN + h), a[w - 4]);
#pragma unroll
                            for (int w = 0; w < 3; ++w) tmem_wait(a[w]);
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                const uint32_t y = redc(a[0][j] + ((uint64_t)a[1][j] << 8) +
                                                        ((uint64_t)a[2][j] << 16));
                                v[h + j] = redc((uint64_t)u[j] * prm.r2 + (uint64_t)y * prm.r3);
                            }
                        }
                    }
                    if (b == NB - 1) {  // the accumulators are read: free for the next tile
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(tempty_bar(ab));
                    }
                    if constexpr (VEC) {
                        // 16-byte group g of row `lane` at group g ^ (lane % 8)
#pragma unroll
                        for (int g = 0; g < 8; ++g)
                            *(uint4*)&stg[lane * 32 + ((g ^ (lane & 7)) << 2)] =
                                make_uint4(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
                        __syncwarp();
                        const int gv = n0 + c0 + vc;
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const int r = 4 * i + vr;
                            uint4 x = *(const uint4*)&stg[r * 32 + (((lane & 7) ^ (r & 7)) << 2)];
                            x.x = d[4 * i] >= x.x ? d[4 * i] - x.x : d[4 * i] + (p - x.x);
                            x.y = d[4 * i + 1] >= x.y ? d[4 * i + 1] - x.y : d[4 * i + 1] + (p - x.y);
                            x.z = d[4 * i + 2] >= x.z ? d[4 * i + 2] - x.z : d[4 * i + 2] + (p - x.z);
                            x.w = d[4 * i + 3] >= x.w ? d[4 * i + 3] - x.w : d[4 * i + 3] + (p - x.w);
                            const int32_t rr = prm.d_rows ? __shfl_sync(0xffffffffu, ri, r)
                                                          : (r < rows_q ? m0 + q * 32 + r : -1);
                            uint32_t* o = Dz + (size_t)(rr < 0 ? 0 : rr) * prm.ldd + gv;
                            if (rr >= 0 && gv + 4 <= prm.N) {
                                *(uint4*)o = x;
                            } else if (rr >= 0) {
                                if (gv < prm.N) o[0] = x.x;
                                if (gv + 1 < prm.N) o[1] = x.y;
                                if (gv + 2 < prm.N) o[2] = x.z;
                            }
                        }
                    } else {
                        // (row lane, column j) at [lane][j ^ lane]
                        const int gn = n0 + c0 + lane;
                        const bool col_ok = gn < prm.N;
#pragma unroll
                        for (int j = 0; j < 32; ++j) stg[lane * 32 + (j ^ lane)] = v[j];
                        __syncwarp();
#pragma unroll
                        for (int r = 0; r < 32; ++r) {
                            const uint32_t x = stg[r * 32 + (lane ^ r)];
                            v[r] = d[r] >= x ? d[r] - x : d[r] + (p - x);
                        }
                        if (prm.d_rows) {
#pragma unroll
                            for (int r = 0; r < 32; ++r) {
                                const int32_t rr = __shfl_sync(0xffffffffu, ri, r);
                                if (rr >= 0 && col_ok) Dz[(size_t)rr * prm.ldd + gn] = v[r];
                            }
                        } else {
                            uint32_t* o = Dq + gn;
#pragma unroll
                            for (int r = 0; r < 32; ++r, o += prm.ldd)
                                if (r < rows_q && col_ok) *o = v[r];
                        }
                    }
                    if (b + PRE < NB && !fresh) load_d(cbeg + 32 * (b + PRE), d);
                    __syncwarp();
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag) atomicExch(prm.err, GBGPU_ETIMEDOUT);
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"((uint32_t)C::TMEM_COLS)
                     : "memory");
    }
}

// ---------------------------------------------------------------------------
// Limb planes of both operands and their tile flags, one launch per GEMM.
//
// A part (blocks [0, a_blocks)): one 128-row x 128-column tile of A per
// block; out[l][m][k] = byte l of A[m][k], zero padded; row m of A is
// A + a_rows[m] lda when a_rows is given (negative: a zero row).  Every item
// is 16 consecutive k of one row (one 16-byte store per limb); with `vec` (A
// and its row and batch strides 16-byte aligned) a full item is read as four
// 16-byte loads.  The block writes its tile flag fa[mt][kb] (0 or 1).
//
// B part (the other blocks): transposing split, out[l][n][k] = byte l of
// B[k][n]; row k of B is B + b_rows[k] ldb when b_rows is given (negative: a
// zero row).  One 128 (k) x 64 (n) tile per block: rows of B are read 256
// bytes per pair of warps; the bytes go to shared memory as [l][n][k] (rows
// padded to 132 bytes: conflict-free in both phases) and leave as whole
// 128-byte k-rows of every n, four threads per row.  The block writes its flag
// fb[n / 64][kb]; the GEMM ORs the flags of the 64-row groups of its tile.
// With nrange (see TcGemmArgs::b_nrange) a tile outside its rows' column range
// is not read: it is written as zeros when another part of its bn-wide GEMM
// tile is live, and not at all otherwise (the GEMM never loads it).
//
// Every flag of the GEMM is written here, so nothing clears them first.
constexpr int SPLIT_ROW = 132;
struct SplitArgs {
    const uint32_t* A;
    int64_t lda, sA;
    const int32_t* a_rows;
    int64_t sAr;
    int32_t M, K, Mp, Kp, L;
    uint8_t* Ap;
    uint8_t* fa;
    int32_t nkbp, vec;
    const uint32_t* B;
    int64_t ldb, sB;
    const int32_t* b_rows;
    int64_t sBr;
    int32_t N, Np, bn;
    uint8_t* Bp;
    uint8_t* fb;
    const int2* nrange;
    int32_t a_blocks;  // (Mp / 128) (Kp / 128)
};

__global__ void __launch_bounds__(256) k_split_ab(const SplitArgs a) {
    extern __shared__ uint8_t split_smem[];  // [L][64][SPLIT_ROW] bytes (B part)
    __shared__ const uint32_t* rowp[128];
    const int z = blockIdx.z;  // batch item
    const int nkb = a.Kp / 128;
    const int L = a.L;
    if ((int)blockIdx.x < a.a_blocks) {
        // ---- A part ----
        const int mt = blockIdx.x / nkb, kbi = blockIdx.x % nkb;
        const uint32_t* A = a.A + (size_t)z * a.sA;
        const int32_t* a_rows = a.a_rows ? a.a_rows + (size_t)z * a.sAr : nullptr;
        uint8_t* out = a.Ap + (size_t)z * L * a.Mp * a.Kp;
        uint32_t any = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int item = threadIdx.x + 256 * q;
            const int m = mt * 128 + (item >> 3);
            const int k = kbi * 128 + (item & 7) * 16;
            int64_t src = -1;
            if (m < a.M) src = a_rows ? (int64_t)a_rows[m] : (int64_t)m;
            const uint32_t* row = src >= 0 ? A + (size_t)src * a.lda : nullptr;
            uint32_t v[16];
            if (a.vec && row && k + 16 <= a.K) {
                const uint4* r4 = (const uint4*)(row + k);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint4 w = r4[u];
                    v[4 * u] = w.x;
                    v[4 * u + 1] = w.y;
                    v[4 * u + 2] = w.z;
                    v[4 * u + 3] = w.w;
                }
            } else {
#pragma unroll
                for (int e = 0; e < 16; ++e) v[e] = (row && k + e < a.K) ? row[k + e] : 0u;
            }
#pragma unroll
            for (int e = 0; e < 16; ++e) any |= v[e];
            for (int l = 0; l < L; ++l) {
                uint32_t w[4];
#pragma unroll
                for (int jj = 0; jj < 4; ++jj)
                    w[jj] = ((v[4 * jj] >> (8 * l)) & 255u) |
                            (((v[4 * jj + 1] >> (8 * l)) & 255u) << 8) |
                            (((v[4 * jj + 2] >> (8 * l)) & 255u) << 16) |
                            (((v[4 * jj + 3] >> (8 * l)) & 255u) << 24);
                *(uint4*)(out + ((size_t)l * a.Mp + m) * a.Kp + k) =
                    make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
        any = __syncthreads_or(any != 0);
        if (threadIdx.x == 0)
            a.fa[((size_t)z * (a.Mp / 128) + mt) * a.nkbp + kbi] = any ? 1 : 0;
        return;
    }
    // ---- B part ----
    const int bq = blockIdx.x - a.a_blocks;
    const int nx = bq % (a.Np / 64), kbi = bq / (a.Np / 64);
    const int k0 = kbi * 128, n0 = nx * 64;
    const uint32_t* B = a.B + (size_t)z * a.sB;
    const int32_t* b_rows = a.b_rows ? a.b_rows + (size_t)z * a.sBr : nullptr;
    uint8_t* out = a.Bp + (size_t)z * L * a.Np * a.Kp;
    uint8_t* flag = a.fb + ((size_t)z * (a.Np / 64) + nx) * a.nkbp + kbi;
    if (a.nrange) {  // uniform over the block
        const int2 rg = k0 < a.K ? a.nrange[kbi] : make_int2(1, 0);
        const int t0 = (n0 / a.bn) * a.bn;
        const bool tile_live = !(rg.y < rg.x || t0 + a.bn <= rg.x || t0 > rg.y);
        if (!tile_live || n0 + 64 <= rg.x || n0 > rg.y) {
            if (threadIdx.x == 0) *flag = 0;
            if (!tile_live) return;
            // zeros: 64 k-rows of 128 bytes per limb, four threads per row
            const int nn = threadIdx.x >> 2, part = threadIdx.x & 3;
            for (int l = 0; l < L; ++l) {
                uint4* dst = (uint4*)(out + ((size_t)l * a.Np + n0 + nn) * a.Kp + k0 + 32 * part);
                dst[0] = make_uint4(0u, 0u, 0u, 0u);
                dst[1] = make_uint4(0u, 0u, 0u, 0u);
            }
            return;
        }
    }
    if (threadIdx.x < 128) {
        const int k = k0 + threadIdx.x;
        int64_t src = -1;
        if (k < a.K) src = b_rows ? (int64_t)b_rows[k] : (int64_t)k;
        rowp[threadIdx.x] = src >= 0 ? B + (size_t)src * a.ldb : nullptr;
    }
    __syncthreads();
    uint32_t any = 0;
    {
        const int c = threadIdx.x & 63, r0 = threadIdx.x >> 6;  // 4 k rows per pass
        const int n = n0 + c;
        // all 32 loads first (no shared-memory store between them)
        uint32_t v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            const uint32_t* rp = rowp[r0 + 4 * i];
            v[i] = (rp && n < a.N) ? rp[n] : 0u;
        }
        for (int l = 0; l < L; ++l) {
            uint8_t* dst = split_smem + ((size_t)l * 64 + c) * SPLIT_ROW + r0;
#pragma unroll
            for (int i = 0; i < 32; ++i) dst[4 * i] = (uint8_t)(v[i] >> (8 * l));
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) any |= v[i];
    }
    any = __syncthreads_or(any != 0);
    // thread: n = tid / 4, bytes [32 part, 32 part + 32) of the 128-byte k row
    const int nn = threadIdx.x >> 2, part = threadIdx.x & 3;
    const int n = n0 + nn;  // n < Np and k0 + 128 <= Kp by the grid
    for (int l = 0; l < L; ++l) {
        const uint32_t* src =
            (const uint32_t*)(split_smem + ((size_t)l * 64 + nn) * SPLIT_ROW + 32 * part);
        uint32_t w[8];
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) w[jj] = src[jj];
        uint4* dst = (uint4*)(out + ((size_t)l * a.Np + n) * a.Kp + k0 + 32 * part);
        dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
        dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
    if (threadIdx.x == 0) *flag = any ? 1 : 0;
}

// row index lists of the plain GEMM (see TcGemmArgs)
struct RowLists {
    const int32_t *a, *b, *d;
    int64_t sa, sb, sd;
    int32_t set;  // D is not read
};

// ---------------------------------------------------------------------------
// plain CUDA-core modular GEMM: 64 x 64 tile per 256 threads, 4 x 4 per thread;
// b is split into 16-bit halves so 2^16 products fit the u64 partial sums.
__global__ void __launch_bounds__(256)
k_plain_submul(const uint32_t* __restrict__ A, int64_t lda, const uint32_t* __restrict__ B,
               int64_t ldb, uint32_t* D, int64_t ldd, int32_t M, int32_t N, int32_t K,
               int64_t strideA, int64_t strideB, int64_t strideD, RowLists rl, FieldMont f) {
    A += (size_t)blockIdx.z * strideA;
    B += (size_t)blockIdx.z * strideB;
    D += (size_t)blockIdx.z * strideD;
    const int32_t* a_rows = rl.a ? rl.a + (size_t)blockIdx.z * rl.sa : nullptr;
    const int32_t* b_rows = rl.b ? rl.b + (size_t)blockIdx.z * rl.sb : nullptr;
    const int32_t* d_rows = rl.d ? rl.d + (size_t)blockIdx.z * rl.sd : nullptr;
    __shared__ uint32_t sA[16][64 + 1];
    __shared__ uint32_t sB[16][64 + 1];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int m0 = blockIdx.y * 64, n0 = blockIdx.x * 64;
    // row index of A row m / B row k (negative: zero row)
    auto arow = [&](int m) -> int64_t { return a_rows ? (int64_t)a_rows[m] : (int64_t)m; };
    auto brow = [&](int k) -> int64_t { return b_rows ? (int64_t)b_rows[k] : (int64_t)k; };
    uint64_t lo[4][4], hi[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) lo[i][j] = hi[i][j] = 0;
    int since = 0;
    for (int k0 = 0; k0 < K; k0 += 16) {
        for (int t = threadIdx.x; t < 16 * 64; t += 256) {
            const int kk = t & 15, mm = t >> 4;
            const int m = m0 + mm, k = k0 + kk;
            const int64_t ra = (m < M && k < K) ? arow(m) : -1;
            sA[kk][mm] = ra >= 0 ? A[(size_t)ra * lda + k] : 0u;
            const int nn = t & 63, kr = t >> 6;
            const int n = n0 + nn, k2 = k0 + kr;
            const int64_t rb = (n < N && k2 < K) ? brow(k2) : -1;
            sB[kr][nn] = rb >= 0 ? B[(size_t)rb * ldb + n] : 0u;
        }
        __syncthreads();
#pragma unroll 4
        for (int kk = 0; kk < 16; ++kk) {
            uint32_t a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = sA[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = sB[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    lo[i][j] += (uint64_t)a[i] * (b[j] & 0xFFFFu);
                    hi[i][j] += (uint64_t)a[i] * (b[j] >> 16);
                }
        }
        __syncthreads();
        since += 16;
        if (since >= 32768) {  // keep the partial sums far from 2^64
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    lo[i][j] %= f.p;
                    hi[i][j] %= f.p;
                }
            since = 0;
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
        const int64_t rd = d_rows ? (int64_t)d_rows[m] : (int64_t)m;
        if (rd < 0) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n >= N) continue;
            const uint64_t h = (hi[i][j] % f.p) << 16;
            const uint32_t v = (uint32_t)((lo[i][j] % f.p + h % f.p) % f.p);
            const uint32_t d = rl.set ? 0u : D[(size_t)rd * ldd + n];
            D[(size_t)rd * ldd + n] = d >= v ? d - v : d + (f.p - v);
        }
    }
}

// ---------------------------------------------------------------------------
// host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

static int make_map(CUtensorMap* map, const void* base, int64_t inner, int64_t rows,
                    int box_inner, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) {
        set_error("cuTensorMapEncodeTiled unavailable");
        return GBGPU_ENODEV;
    }
    cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)inner};
    cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides,
                    box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed");
        return GBGPU_ECUDA;
    }
    return GBGPU_OK;
}

static thread_local GemmProfile* g_profile = nullptr;
GemmProfile* gemm_profile() { return g_profile; }
void set_gemm_profile(GemmProfile* p) { g_profile = p; }

int limbs_for(uint32_t p) {
    if (p < (1u << 8)) return 1;
    if (p < (1u << 16)) return 2;
    if (p < (1u << 24)) return 3;
    return 4;
}

// SMs of the current device (persistent GEMM grid)
static int num_sms() {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
        return 148;
    return n;
}

template <int L, int SHAPE>
static int tc_run(const TcGemmArgs& g, uint8_t* planes, cudaStream_t s, int32_t* err,
                  long long* launches) {
    using Cfg = TcCfg<L, SHAPE>;
    const int32_t Mp = (g.M + Cfg::BM - 1) / Cfg::BM * Cfg::BM;
    const int32_t Np = (g.N + Cfg::BN - 1) / Cfg::BN * Cfg::BN;
    const int32_t Kp = (g.K + Cfg::BK - 1) / Cfg::BK * Cfg::BK;
    const int32_t nb = g.batch;
    uint8_t* Ap = planes;                                    // [nb][L][Mp][Kp]
    uint8_t* Bp = planes + (size_t)nb * L * Mp * Kp;         // [nb][L][Np][Kp]
    const int32_t nkb = Kp / Cfg::BK;
    const int32_t nkbp = (nkb + 63) / 64 * 64;
    uint8_t* fa = Bp + (size_t)nb * L * Np * Kp;             // [nb][Mp/128][nkbp]
    uint8_t* fb = fa + (size_t)nb * (Mp / Cfg::BM) * nkbp;   // [nb][Np/64][nkbp]
    GemmProfile* prof = gemm_profile();
    if (prof) {
        cudaEvent_t es = nullptr;
        cudaEventCreate(&es);
        cudaEventRecord(es, s);
        prof->split_events.push_back(es);
    }
    {
        SplitArgs sa{};
        sa.A = g.A;
        sa.lda = g.lda;
        sa.sA = g.sA;
        sa.a_rows = g.a_rows;
        sa.sAr = g.sAr;
        sa.M = g.M;
        sa.K = g.K;
        sa.Mp = Mp;
        sa.Kp = Kp;
        sa.L = L;
        sa.Ap = Ap;
        sa.fa = fa;
        sa.nkbp = nkbp;
        sa.vec = ((uintptr_t)g.A % 16 == 0) && g.lda % 4 == 0 && g.sA % 4 == 0;
        sa.B = g.B;
        sa.ldb = g.ldb;
        sa.sB = g.sB;
        sa.b_rows = g.b_rows;
        sa.sBr = g.sBr;
        sa.N = g.N;
        sa.Np = Np;
        sa.bn = Cfg::BN;
        sa.Bp = Bp;
        sa.fb = fb;
        sa.nrange = nb == 1 && !g.b_rows ? g.b_nrange : nullptr;
        sa.a_blocks = (Mp / 128) * (Kp / 128);
        const int64_t blocks = (int64_t)sa.a_blocks + (int64_t)(Np / 64) * (Kp / 128);
        k_split_ab<<<dim3((unsigned)blocks, 1, nb), 256, L * 64 * SPLIT_ROW, s>>>(sa);
        *launches += 1;
    }
    CUtensorMap ma, mb;
    int rc = make_map(&ma, Ap, Kp, (int64_t)nb * L * Mp, Cfg::BK, Cfg::BM);
    if (rc) return rc;
    rc = make_map(&mb, Bp, Kp, (int64_t)nb * L * Np, Cfg::BK, Cfg::BN);
    if (rc) return rc;
    TcParams prm{};
    prm.D = g.D;
    prm.ldd = g.ldd;
    prm.sD = g.sD;
    prm.d_rows = g.d_rows;
    prm.sDr = g.sDr;
    prm.M = g.M;
    prm.N = g.N;
    prm.Mp = Mp;
    prm.Np = Np;
    prm.nkb = nkb;
    prm.nkbp = nkbp;
    prm.fa = fa;
    prm.fb = fb;
    const FieldMont f = FieldMont::make(g.p);
    prm.p = g.p;
    prm.pneg_inv = f.pneg_inv;
    prm.mu = (uint32_t)((((uint64_t)1) << 32) / g.p);
    const uint64_t R = ((uint64_t)1 << 32) % g.p;
    prm.r2 = (uint32_t)(R * R % g.p);
    prm.r3 = (uint32_t)((uint64_t)prm.r2 * R % g.p);
    uint64_t pw = 1;
    for (int w = 0; w < 5; ++w) {
        prm.cw[w] = (uint32_t)((pw % g.p) * R % g.p);
        pw = (pw << 8) % g.p;
    }
    prm.err = err;
    prm.budget = 4000000000LL;  // about 2 s at 2 GHz per wait
    const bool vec = (uintptr_t)g.D % 16 == 0 && g.ldd % 4 == 0 && g.sD % 4 == 0;
    const void* kernel = vec ? (const void*)k_tc_submul<L, SHAPE, true>
                             : (const void*)k_tc_submul<L, SHAPE, false>;
    cudaError_t e = ensure_smem_limit(kernel, Cfg::SMEM_BYTES);
    if (e != cudaSuccess) {
        set_error(std::string("tc smem attribute: ") + cudaGetErrorString(e));
        return GBGPU_ECUDA;
    }
    prm.batch = nb;
    prm.set = g.set;
    const int64_t tiles = (int64_t)(Np / Cfg::BN) * (Mp / Cfg::BM) * nb;
    const dim3 grid((unsigned)std::max<int64_t>(
        1, std::min<int64_t>(tiles, (int64_t)num_sms())));
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (prof) {
        const int slot = (int)prof->events.size();
        prm.steps = slot < prof->capacity ? prof->d_steps + slot : nullptr;
        prof->shape.insert(prof->shape.end(), {g.M, g.N, g.K, nb});
        cudaEventCreate(&e0);
        cudaEventCreate(&e1);
        cudaEventRecord(e0, s);
    }
    void* args[] = {&ma, &mb, &prm};
    e = cudaLaunchKernel(kernel, grid, dim3(Cfg::THREADS), args, Cfg::SMEM_BYTES, s);
    ++*launches;
    if (prof) {
        cudaEventRecord(e1, s);
        prof->events.push_back({e0, e1});
        // int8 MACs of one executed K step of one tile
        prof->macs_per_step.push_back((double)Cfg::BM * Cfg::BN * Cfg::BK * L * L);
    }
    if (e != cudaSuccess) {
        set_error(std::string("tc launch: ") + cudaGetErrorString(e));
        return GBGPU_ECUDA;
    }
    return GBGPU_OK;
}

size_t tc_workspace_bytes(uint32_t p, int32_t M, int32_t N, int32_t K, int32_t batch) {
    const int L = limbs_for(p);
    // planes padded for the widest tile (256 columns), flags counted for the
    // narrowest (64) with flag rows padded to 64 K steps: enough for either
    // tile shape
    const size_t Mp = (size_t)(M + 127) / 128 * 128, Np = (size_t)(N + 255) / 256 * 256;
    const size_t Kp = (size_t)(K + 127) / 128 * 128;
    const size_t nkbp = (Kp / 128 + 63) / 64 * 64;
    const size_t nb = (size_t)(batch > 0 ? batch : 1);
    const size_t flags = nb * (Mp / 128 + Np / 64) * nkbp;
    return nb * L * (Mp + Np) * Kp + ((flags + 255) & ~(size_t)255);
}

int tc_submul(const TcGemmArgs& g, void* workspace, cudaStream_t s, int32_t* err,
              long long* launches) {
    if (g.M <= 0 || g.N <= 0 || g.K <= 0 || g.batch <= 0) return GBGPU_OK;
    if (g.batch > 65535) {
        set_error("tensor-core GEMM: batch too large");
        return GBGPU_ERANGE;
    }
    if ((g.p & 1u) == 0 || g.p < 3) {
        set_error("tensor-core path needs an odd prime");
        return GBGPU_EINVAL;
    }
    const int L = limbs_for(g.p);
    const int shape = tc_shape(L, g.M, g.N, g.K, g.batch, num_sms(), tc_shape_for(L, g.K));
    return tc_submul_shape(g, workspace, s, err, launches, shape);
}

// the shapes: 0 big, 2 mid (L <= 2); any other request falls back to big
int tc_submul_shape(const TcGemmArgs& g, void* workspace, cudaStream_t s, int32_t* err,
                    long long* launches, int shape) {
    if (g.M <= 0 || g.N <= 0 || g.K <= 0 || g.batch <= 0) return GBGPU_OK;
    uint8_t* planes = (uint8_t*)workspace;
    const bool mid = shape == TC_MID;
    switch (limbs_for(g.p)) {
        case 1:
            return mid ? tc_run<1, TC_MID>(g, planes, s, err, launches)
                       : tc_run<1, TC_BIG>(g, planes, s, err, launches);
        case 2:
            return mid ? tc_run<2, TC_MID>(g, planes, s, err, launches)
                       : tc_run<2, TC_BIG>(g, planes, s, err, launches);
        case 3: return tc_run<3, TC_BIG>(g, planes, s, err, launches);
        default: return tc_run<4, TC_BIG>(g, planes, s, err, launches);
    }
}

int plain_submul(const TcGemmArgs& g, cudaStream_t s, long long* launches) {
    if (g.M <= 0 || g.N <= 0 || g.K <= 0 || g.batch <= 0) return GBGPU_OK;
    dim3 grid((g.N + 63) / 64, (g.M + 63) / 64, g.batch);
    FieldMont f{};
    f.p = g.p;
    const RowLists rl{g.a_rows, g.b_rows, g.d_rows, g.sAr, g.sBr, g.sDr, g.set};
    k_plain_submul<<<grid, 256, 0, s>>>(g.A, g.lda, g.B, g.ldb, g.D, g.ldd, g.M, g.N, g.K, g.sA,
                                        g.sB, g.sD, rl, f);
    ++*launches;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error(std::string("plain gemm launch: ") + cudaGetErrorString(e));
        return GBGPU_ECUDA;
    }
    return GBGPU_OK;
}

}  // namespace gbgpu
