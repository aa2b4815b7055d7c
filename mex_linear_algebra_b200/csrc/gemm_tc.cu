// gemm_tc.cu -- GF(2) product on the sm_100a tensor cores (tcgen05, kind::i8).
//
// Both operands are 0/1 bytes (expanded from the packed bits by
// expand_kernel), K-major: A8 is m x k, Bt8 is n x k (B transposed).  The
// tensor cores accumulate the integer dot products in 32-bit TMEM cells;
// bit (i,j) of the GF(2) product is the low bit of the sum.  The sum is at
// most k < 2^31, and the low bit of a 32-bit two's-complement sum is exact
// even past that, so the result is bit-exact for every k.
//
// Kernel structure (one 128 x 256 output tile per CTA, 192 threads):
//   warp 0  lane 0 : TMA producer, 4-stage ring of (A 128x128 B, B 256x128 B)
//   warp 1         : allocates 256 TMEM columns; lane 0 issues 4 UMMAs of
//                    K=32 per stage and commits each stage back to its
//                    producer barrier
//   warps 2..5     : epilogue; each reads its 32 TMEM lanes (= 32 output
//                    rows) x 256 columns, keeps the parity bit and writes 4
//                    packed words per row.
// Where the tiles leave most of the chip idle, K is split over gridDim.y: each
// CTA multiplies its slice of the stages and XORs its parity bits into C, which
// starts as zero.
// Tiles are rasterised in bands of 16 tile-rows so that the CTAs resident
// at one time share A and B tiles in L2.
//
// FP4 form (F4 = true): the operands are packed E2M1 values (0x2 = 1.0,
// 0x0 = 0; two per byte), the instruction is tcgen05 kind::mxf4 with one
// UE8M0 scale factor per 32 values of K, at twice the INT8 rate.  Every scale
// factor is 1.0, so the scale-factor columns of TMEM are one constant block
// (bytes 0x7F) written once per CTA and addressed by every instruction.  The
// f32 accumulator holds the integer dot product exactly; K < 2^23 is
// required so that adding 2^23 puts the integer in the low mantissa bits,
// whose bit 0 is the parity (one float add per value instead of a
// float-to-int conversion).
#include <cstdlib>

#include "mela_common.cuh"
#include "mela_internal.h"
#include "tc_ptx.cuh"

namespace mela {

namespace {

constexpr int BM = 128, BN = 256, BK = 128;  // BK in bytes (= K elements)
constexpr int STAGES = 4;
constexpr int A_BYTES = BM * BK;
constexpr int B_BYTES = BN * BK;
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
constexpr u32 SF_COL = 256;   // first TMEM column of the 32 constant scale-factor columns (FP4 form)
constexpr int GROUP_M = 16;

struct Ctl {
    u64 full[STAGES];
    u64 empty[STAGES];
    u64 acc;
    u64 drain;
    u32 tmem;
    int abort;
};

}  // namespace

template <bool F4>
__global__ void __launch_bounds__(192, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               u64 *__restrict__ C, i64 ldc, i64 m, i64 n, int tiles_m, int tiles_n, int all_stages,
               int split_stages, u32 *err)
{
    constexpr u32 TMEM_COLS = F4 ? 512 : 256;
    // this CTA's stages of K: ks0 .. ks0 + kstages - 1
    const int ks0 = (int)blockIdx.y * split_stages;
    const int kstages = all_stages - ks0 < split_stages ? all_stages - ks0 : split_stages;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem =
        reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    Ctl *ctl = reinterpret_cast<Ctl *>(smem + STAGES * STAGE_BYTES);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // grouped rasterisation
    const int t = blockIdx.x;
    const int per_group = GROUP_M * tiles_n;
    const int group = t / per_group;
    const int first_m = group * GROUP_M;
    const int gsize = (tiles_m - first_m) < GROUP_M ? (tiles_m - first_m) : GROUP_M;
    const int tm = first_m + (t % per_group) % gsize;
    const int tn = (t % per_group) / gsize;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            ptx::mbar_init(&ctl->full[s], 1);
            ptx::mbar_init(&ctl->empty[s], 1);
        }
        ptx::mbar_init(&ctl->acc, 1);
        ptx::mbar_init(&ctl->drain, 1);
        ctl->abort = 0;
        ptx::fence_barrier_init();
    }
    if (warp == 0 && lane == 0) {
        ptx::prefetch_tmap(&tmA);
        ptx::prefetch_tmap(&tmB);
    }
    if (warp == 1) {
        ptx::tmem_alloc(&ctl->tmem, TMEM_COLS);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const u32 tmem = ctl->tmem;
    volatile int *abort_flag = &ctl->abort;
    if constexpr (F4) {
        // constant scale factors: every byte of columns SF_COL.. = 0x7F (2^0)
        if (warp >= 2) {
            const u32 lane_base = (u32)((warp & 3) * 32) << 16;
            ptx::tmem_st_32x32b_x16(tmem + lane_base + SF_COL, 0x7F7F7F7Fu);
            ptx::tmem_st_32x32b_x16(tmem + lane_base + SF_COL + 16, 0x7F7F7F7Fu);
            ptx::tmem_st_wait();
        }
        ptx::tc_fence_before();
        __syncthreads();
        ptx::tc_fence_after();
    }

    if (warp == 0) {
        if (lane == 0) {
            int last_round[STAGES];
#pragma unroll
            for (int s = 0; s < STAGES; ++s) last_round[s] = -1;
            for (int ks = 0; ks < kstages; ++ks) {
                const int s = ks % STAGES, round = ks / STAGES;
                if (round > 0 && !ptx::mbar_wait(&ctl->empty[s], (round - 1) & 1, err)) {
                    *abort_flag = 1;
                    break;
                }
                if (*abort_flag) break;
                unsigned char *sa = smem + s * STAGE_BYTES;
                ptx::mbar_arrive_expect_tx(&ctl->full[s], STAGE_BYTES);
                ptx::tma_load_2d(sa, &tmA, &ctl->full[s], (ks0 + ks) * BK, tm * BM);
                ptx::tma_load_2d(sa + A_BYTES, &tmB, &ctl->full[s], (ks0 + ks) * BK, tn * BN);
                last_round[s] = round;
            }
            if (*abort_flag) {
                // let every issued copy land before the CTA's shared memory goes away
                for (int s = 0; s < STAGES; ++s)
                    if (last_round[s] >= 0) ptx::mbar_wait(&ctl->full[s], last_round[s] & 1, nullptr);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr u32 idesc = F4 ? ptx::idesc_mxf4(BM, BN) : ptx::idesc_i8(BM, BN);
            bool ok = true;
            for (int ks = 0; ks < kstages; ++ks) {
                const int s = ks % STAGES, round = ks / STAGES;
                if (!ptx::mbar_wait(&ctl->full[s], round & 1, err) || *abort_flag) {
                    *abort_flag = 1;
                    ok = false;
                    break;
                }
                ptx::tc_fence_after();
                const u32 a0 = ptx::smem_u32(smem + s * STAGE_BYTES);
                const u32 b0 = a0 + A_BYTES;
#pragma unroll
                for (int kk = 0; kk < BK / 32; ++kk) {
                    // 32 bytes of K per instruction: 32 int8 values or 64 packed e2m1 values
                    if constexpr (F4)
                        ptx::umma_mxf4(tmem, ptx::desc_k_sw128(a0 + kk * 32), ptx::desc_k_sw128(b0 + kk * 32),
                                       idesc, tmem + SF_COL, tmem + SF_COL + 8, (ks | kk) != 0);
                    else
                        ptx::umma_i8(tmem, ptx::desc_k_sw128(a0 + kk * 32), ptx::desc_k_sw128(b0 + kk * 32),
                                     idesc, (ks | kk) != 0);
                }
                ptx::umma_commit(&ctl->empty[s]);
            }
            if (ok) {
                ptx::umma_commit(&ctl->acc);
            } else {
                // drain UMMAs still reading shared memory, then release the epilogue
                ptx::umma_commit(&ctl->drain);
                ptx::mbar_wait(&ctl->drain, 0, nullptr);
                ptx::mbar_arrive(&ctl->acc);
            }
        }
        __syncwarp();
    } else {
        const bool ok = ptx::mbar_wait(&ctl->acc, 0, err);
        ptx::tc_fence_after();
        if (ok && !*abort_flag) {
            const int ew = warp & 3;  // TMEM lane quarter this warp may access
            const i64 row = (i64)tm * BM + ew * 32 + lane;
            u32 bits[BN / 32];
#pragma unroll
            for (int c = 0; c < BN / 32; ++c) {
                u32 r[32];
                ptx::tmem_ld_32x32b_x32(tmem + ((u32)(ew * 32) << 16) + (u32)(c * 32), r);
                ptx::tmem_ld_wait();
                u32 b = 0;
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    const u32 v = F4 ? __float_as_uint(__uint_as_float(r[j]) + 8388608.0f) : r[j];
                    b |= (v & 1u) << j;
                }
                bits[c] = b;
            }
            const i64 nw = words_of(n);
            if (row < m) {
#pragma unroll
                for (int q = 0; q < BN / 64; ++q) {
                    const i64 w = (i64)tn * (BN / 64) + q;
                    const u64 v = (u64)bits[2 * q] | ((u64)bits[2 * q + 1] << 32);
                    if (w >= nw) continue;
                    if (gridDim.y == 1)
                        C[row * ldc + w] = v;
                    else
                        atomicXor(&C[row * ldc + w], v);
                }
            }
        }
    }

    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem, TMEM_COLS);
    }
}

// ---------------------------------------------------------------- CTA pairs
// The same product with 256 x 256 output tiles computed by a cluster of two
// CTAs (tcgen05 cta_group::2).  CTA r of the pair loads rows r*128..+127 of
// the tile's A rows and of its B rows (B transposed) into its own shared
// memory; the TMA completions of both CTAs are counted on the even CTA's
// stage barrier, and the even CTA's MMA thread issues M = 256 instructions
// that read both CTAs' halves and accumulate, in each CTA's TMEM, that CTA's
// 128 rows x 256 columns.  Each SM thereby fills half as many B bytes into
// shared memory per instruction as with one CTA per tile.  The MMA commits
// arrive on the barrier of the same offset in both CTAs, so each CTA's
// producer learns when a stage is free and each CTA's epilogue when its
// accumulator is ready.  No TMA load uses cluster multicast.
namespace {
constexpr int P_STAGES = 7;
constexpr int P_A_BYTES = 128 * BK;                    // this CTA's 128 rows of A
constexpr int P_B_BYTES = 128 * BK;                    // this CTA's 128 rows of B
constexpr int P_STAGE_BYTES = P_A_BYTES + P_B_BYTES;
constexpr int P_SMEM_BYTES = P_STAGES * P_STAGE_BYTES + 1024 + 256;

struct PairCtl {
    u64 full[P_STAGES];   // even CTA: both CTAs' bytes of a stage have landed
    u64 empty[P_STAGES];  // both CTAs: the pair's MMAs have read a stage
    u64 acc_full;         // both CTAs: the accumulator holds a finished tile
    u64 acc_empty;        // even CTA: both CTAs' epilogues have read the accumulator
    u64 drain;
    u32 tmem;
    int abort;
};
constexpr int P_EPI_WARPS = 8;                         // two per TMEM lane quarter, 128 columns each
constexpr int P_THREADS = 64 + 32 * P_EPI_WARPS;

// Up to two blocks of C (pitch ldc) that one product goes to.
struct PairSum {
    u64 *c[2];
    i64 rows[2], words[2];  // 0: none
    int add[2];             // XOR into the block instead of writing it
};

// Pins registers that an asynchronous TMEM load fills behind the wait for it.
__device__ __forceinline__ void tie(u32 (&r)[32])
{
#pragma unroll
    for (int j = 0; j < 32; ++j) asm volatile("" : "+r"(r[j]));
}
// The parities of 32 accumulators as one word, value j in bit j: four chains
// of 8 funnel shifts, each of which moves a value's low bit in from the top.
template <bool F4>
__device__ __forceinline__ u32 low_bits(const u32 (&r)[32])
{
    u32 b[4] = {};
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const u32 x = r[8 * q + j];
            b[q] = __funnelshift_r(b[q], F4 ? __float_as_uint(__uint_as_float(x) + 8388608.0f) : x, 1);
        }
    return __byte_perm(__byte_perm(b[0], b[1], 0x0073), __byte_perm(b[2], b[3], 0x0073), 0x5410);
}
}  // namespace

// Persistent: cluster c computes tiles c, c + clusters, ... (grouped
// rasterisation over 256 x 256 tiles).  The stage ring runs on across tiles,
// so the producer fills the next tile's stages while the current tile's last
// MMAs and its epilogue run; the MMA thread starts a tile once both CTAs'
// epilogues have read the previous one out of TMEM.
// SUM: the product is written or added (XOR) to the blocks of `out` instead.
template <bool F4, bool SUM>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(P_THREADS, 1)
gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    u64 *__restrict__ C, i64 ldc, i64 m, i64 n, int tiles_m, int tiles_n, int kstages, u32 *err,
                    const __grid_constant__ PairSum out)
{
    constexpr u32 TMEM_COLS = F4 ? 512 : 256;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem =
        reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    PairCtl *ctl = reinterpret_cast<PairCtl *>(smem + P_STAGES * P_STAGE_BYTES);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const u32 rank = ptx::cluster_ctarank();
    const bool leader = rank == 0;
    const int cid = blockIdx.x >> 1, clusters = gridDim.x >> 1;
    const int ntiles = tiles_m * tiles_n;
    auto coords = [&](int t, int &tm, int &tn) {
        const int per_group = GROUP_M * tiles_n;
        const int group = t / per_group;
        const int first_m = group * GROUP_M;
        const int gsize = (tiles_m - first_m) < GROUP_M ? (tiles_m - first_m) : GROUP_M;
        tm = first_m + (t % per_group) % gsize;
        tn = (t % per_group) / gsize;
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < P_STAGES; ++s) {
            ptx::mbar_init(&ctl->full[s], 1);
            ptx::mbar_init(&ctl->empty[s], 1);
        }
        ptx::mbar_init(&ctl->acc_full, 1);
        ptx::mbar_init(&ctl->acc_empty, 2 * P_EPI_WARPS);
        ptx::mbar_init(&ctl->drain, 1);
        ctl->abort = 0;
        ptx::fence_barrier_init();
    }
    if (warp == 0 && lane == 0) {
        ptx::prefetch_tmap(&tmA);
        ptx::prefetch_tmap(&tmB);
    }
    if (warp == 1) {
        ptx::tmem_alloc_pair(&ctl->tmem, TMEM_COLS);
        ptx::tmem_relinquish_pair();
    }
    ptx::tc_fence_before();
    ptx::cluster_sync();  // both CTAs' barriers and TMEM exist before any copy or MMA
    ptx::tc_fence_after();
    const u32 tmem = ctl->tmem;
    volatile int *abort_flag = &ctl->abort;
    if constexpr (F4) {
        if (warp >= 2 && warp < 6) {
            const u32 lane_base = (u32)((warp & 3) * 32) << 16;
            ptx::tmem_st_32x32b_x16(tmem + lane_base + SF_COL, 0x7F7F7F7Fu);
            ptx::tmem_st_32x32b_x16(tmem + lane_base + SF_COL + 16, 0x7F7F7F7Fu);
            ptx::tmem_st_wait();
        }
        ptx::tc_fence_before();
        ptx::cluster_sync();  // the scale factors of both CTAs are in place
        ptx::tc_fence_after();
    }

    if (warp == 0) {
        if (lane == 0) {
            const u32 full0 = ptx::mapa_shared(ptx::smem_u32(&ctl->full[0]), 0);
            int g = 0;  // stage counter over all tiles of this cluster
            bool ok = true;
            for (int t = cid; t < ntiles && ok; t += clusters) {
                int tm, tn;
                coords(t, tm, tn);
                for (int ks = 0; ks < kstages; ++ks, ++g) {
                    const int s = g % P_STAGES, round = g / P_STAGES;
                    if ((round > 0 && !ptx::mbar_wait(&ctl->empty[s], (round - 1) & 1, err)) || *abort_flag) {
                        *abort_flag = 1;
                        ok = false;
                        break;
                    }
                    unsigned char *sa = smem + s * P_STAGE_BYTES;
                    if (leader) ptx::mbar_arrive_expect_tx(&ctl->full[s], 2 * P_STAGE_BYTES);
                    const u32 bar = full0 + (u32)(s * sizeof(u64));
                    ptx::tma_load_2d_pair(sa, &tmA, bar, ks * BK, tm * 256 + (int)rank * 128);
                    ptx::tma_load_2d_pair(sa + P_A_BYTES, &tmB, bar, ks * BK, tn * 256 + (int)rank * 128);
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && leader) {
            constexpr u32 idesc = F4 ? ptx::idesc_mxf4(256, BN) : ptx::idesc_i8(256, BN);
            bool ok = true;
            int g = 0, i = 0;
            for (int t = cid; t < ntiles && ok; t += clusters, ++i) {
                // the previous tile has left TMEM (both CTAs)
                if (i > 0 && (!ptx::mbar_wait_cluster(&ctl->acc_empty, (i - 1) & 1, err) || *abort_flag)) {
                    ok = false;
                    break;
                }
                ptx::tc_fence_after();
                for (int ks = 0; ks < kstages; ++ks, ++g) {
                    const int s = g % P_STAGES, round = g / P_STAGES;
                    if (!ptx::mbar_wait(&ctl->full[s], round & 1, err) || *abort_flag) {
                        ok = false;
                        break;
                    }
                    ptx::tc_fence_after();
                    const u32 a0 = ptx::smem_u32(smem + s * P_STAGE_BYTES);
                    const u32 b0 = a0 + P_A_BYTES;
#pragma unroll
                    for (int kk = 0; kk < BK / 32; ++kk) {
                        if constexpr (F4)
                            ptx::umma_mxf4_pair(tmem, ptx::desc_k_sw128(a0 + kk * 32),
                                                ptx::desc_k_sw128(b0 + kk * 32), idesc, tmem + SF_COL,
                                                tmem + SF_COL + 8, (ks | kk) != 0);
                        else
                            ptx::umma_i8_pair(tmem, ptx::desc_k_sw128(a0 + kk * 32), ptx::desc_k_sw128(b0 + kk * 32),
                                              idesc, (ks | kk) != 0);
                    }
                    ptx::umma_commit_pair(&ctl->empty[s], 0x3);
                }
                if (ok) ptx::umma_commit_pair(&ctl->acc_full, 0x3);
            }
            if (!ok) {
                *abort_flag = 1;
                // drain the MMAs still reading either CTA's shared memory
                ptx::umma_commit_pair(&ctl->drain, 0x1);
                ptx::mbar_wait(&ctl->drain, 0, nullptr);
            }
        }
        __syncwarp();
    } else {
        const int ew = warp & 3;  // TMEM lane quarter this warp may access
        const u32 acc_empty0 = ptx::mapa_shared(ptx::smem_u32(&ctl->acc_empty), 0);
        const int side = (warp - 2) >> 2;  // its half of the tile's columns
        const i64 nw = words_of(n);
        int i = 0;
        for (int t = cid; t < ntiles; t += clusters, ++i) {
            const bool ok = ptx::mbar_wait(&ctl->acc_full, i & 1, err);
            ptx::tc_fence_after();
            if (!ok || *abort_flag) {
                *abort_flag = 1;
                break;
            }
            int tm, tn;
            coords(t, tm, tn);
            const i64 row = (i64)tm * 256 + (i64)rank * 128 + ew * 32 + lane;
            // two chunks of 32 columns in registers: one on its way from TMEM
            // while the other's bits are gathered (the tile's MMAs wait for
            // this: 3.3K cycles a tile, 3.6K with four warps one chunk at a
            // time; 16384 x 1024 x 16384 in 323K cycles against 338K)
            u32 bits[4], r[2][32];
            const u32 tcol = tmem + ((u32)(ew * 32) << 16) + (u32)(128 * side);
            ptx::tmem_ld_32x32b_x32(tcol, r[0]);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                ptx::tmem_ld_wait();
                tie(r[c & 1]);
                if (c < 3) ptx::tmem_ld_32x32b_x32(tcol + (u32)(32 * (c + 1)), r[(c + 1) & 1]);
                bits[c] = low_bits<F4>(r[c & 1]);
            }
            // this warp's TMEM reads are done: the next tile may overwrite them
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive_cluster(acc_empty0);
            const i64 w0 = (i64)tn * (BN / 64) + 2 * side;
            const u64 v[2] = {(u64)bits[0] | ((u64)bits[1] << 32), (u64)bits[2] | ((u64)bits[3] << 32)};
            if constexpr (SUM) {
#pragma unroll
                for (int d = 0; d < 2; ++d) {
                    u64 *c = out.c[d] + row * ldc + w0;
                    const i64 left = row < out.rows[d] ? out.words[d] - w0 : 0;
                    u64 old[2] = {};
                    if (out.add[d]) {
#pragma unroll
                        for (int q = 0; q < 2; ++q)
                            if (q < left) old[q] = c[q];
                    }
#pragma unroll
                    for (int q = 0; q < 2; ++q)
                        if (q < left) c[q] = old[q] ^ v[q];
                }
            } else if (row < m) {
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    if (w0 + q < nw) C[row * ldc + w0 + q] = v[q];
            }
        }
    }

    ptx::tc_fence_before();
    __syncthreads();
    ptx::cluster_sync();  // neither CTA leaves while the pair's MMAs may still read its shared memory
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc_pair(tmem, TMEM_COLS);
    }
}

// ---------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn()
{
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

// K-major byte matrix rows x kp, box (128 bytes, box_rows rows), 128-byte swizzle.
static mela_status make_map(CUtensorMap *map, const unsigned char *base, i64 rows, i64 kp,
                            int box_rows)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) {
        set_error("cuTensorMapEncodeTiled unavailable");
        return MELA_ERR_CUDA;
    }
    cuuint64_t dims[2] = {(cuuint64_t)kp, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)kp};
    cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void *)base, dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed (%d)", (int)r);
        return MELA_ERR_CUDA;
    }
    return MELA_OK;
}

mela_status make_u8_kmajor_map(CUtensorMap *map, const unsigned char *base, i64 rows, i64 kp, int box_rows)
{
    return make_map(map, base, rows, kp, box_rows);
}

mela_status make_u64_rows_map(CUtensorMap *map, const u64 *base, i64 rows, i64 words, i64 ld, int box_words,
                              int box_rows)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) {
        set_error("cuTensorMapEncodeTiled unavailable");
        return MELA_ERR_CUDA;
    }
    cuuint64_t dims[2] = {(cuuint64_t)words, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 8};
    cuuint32_t box[2] = {(cuuint32_t)box_words, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, (void *)base, dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled (packed rows) failed (%d)", (int)r);
        return MELA_ERR_CUDA;
    }
    return MELA_OK;
}

// CTA pairs are used whenever the padded row count allows (mp % 256 == 0),
// unless the tile choice asks for single CTAs (tile 1) or, for the default
// choice, MELA_TC_PAIR=0 is set in the environment.
static bool use_pairs(i64 mp, int tile)
{
    if (mp % 256 || tile == 1) return false;
    if (tile == 2) return true;
    const char *e = getenv("MELA_TC_PAIR");
    return !(e && e[0] == '0');
}

// The pair kernel over mp x np x kp expanded operands.
template <bool SUM>
static mela_status launch_pairs(const unsigned char *A8, const unsigned char *Bt8, i64 mp, i64 np, i64 kp, u64 *C,
                                i64 ldc, i64 m, i64 n, bool fp4, const PairSum &out, cudaStream_t s)
{
    CUtensorMap ma, mb;
    mela_status st = make_map(&ma, A8, mp, kp, 128);
    if (st != MELA_OK) return st;
    st = make_map(&mb, Bt8, np, kp, 128);
    if (st != MELA_OK) return st;
    const i64 tiles_m = mp / 256, tiles_n = np / BN, ntiles = tiles_m * tiles_n, clusters_max = sm_count() / 2;
    const unsigned grid = (unsigned)(2 * (ntiles < clusters_max ? ntiles : clusters_max));
    const auto kernel = fp4 ? gemm_tc_pair_kernel<true, SUM> : gemm_tc_pair_kernel<false, SUM>;
    MELA_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, P_SMEM_BYTES));
    kernel<<<grid, P_THREADS, P_SMEM_BYTES, s>>>(ma, mb, C, ldc, m, n, (int)tiles_m, (int)tiles_n, (int)(kp / BK),
                                           device_error_word(), out);
    MELA_LAUNCH_CHECK("gemm_tc_pair_kernel");
    return MELA_OK;
}

mela_status launch_gemm_tc(const unsigned char *A8, const unsigned char *Bt8, i64 mp, i64 np,
                           i64 kp, u64 *C, i64 ldc, i64 m, i64 n, cudaStream_t s, bool fp4, int tile)
{
    if (m <= 0 || n <= 0) return MELA_OK;
    if (mp % BM || np % BN || kp % BK || kp <= 0) {
        set_error("gemm_tc: padded shape %lld x %lld x %lld not tile-aligned", mp, np, kp);
        return MELA_ERR_INVALID;
    }
    if (((uintptr_t)A8 | (uintptr_t)Bt8) & 15) {
        set_error("gemm_tc: operands must be 16-byte aligned");
        return MELA_ERR_INVALID;
    }
    const i64 tiles_m = mp / BM, tiles_n = np / BN, kst = kp / BK;
    if (tiles_m * tiles_n > 0x7fffffffLL || kst > 0x7fffffffLL || kp > (1LL << 31)) {
        set_error("gemm_tc: problem too large for one launch");
        return MELA_ERR_UNSUPPORTED;
    }
    if (use_pairs(mp, tile)) {
        return launch_pairs<false>(A8, Bt8, mp, np, kp, C, ldc, m, n, fp4, PairSum{}, s);
    }
    CUtensorMap ma, mb;
    mela_status st = make_map(&ma, A8, mp, kp, BM);
    if (st != MELA_OK) return st;
    st = make_map(&mb, Bt8, np, kp, BN);
    if (st != MELA_OK) return st;
    // Slices of K: as many as fill one wave (a CTA takes an SM), each of at least
    // 4 stages, and only past 16 stages, where the time saved (0.2 us a stage)
    // passes the clearing of C (200 x 20000 x 300 in FP4: 12.4 us in 19 slices,
    // 34.3 us in one).
    i64 splits = kst >= 16 ? sm_count() / (tiles_m * tiles_n) : 1, per = kst;
    if (splits > kst / 4) splits = kst / 4;
    if (splits > 1) {
        per = (kst + splits - 1) / splits;
        splits = (kst + per - 1) / per;
        MELA_CUDA_TRY(cudaMemset2DAsync(C, (size_t)ldc * 8, 0, (size_t)words_of(n) * 8, (size_t)m, s));
    } else {
        splits = 1;
    }
    const dim3 grid((unsigned)(tiles_m * tiles_n), (unsigned)splits);
    const auto kernel = fp4 ? gemm_tc_kernel<true> : gemm_tc_kernel<false>;
    MELA_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
    kernel<<<grid, 192, SMEM_BYTES, s>>>(ma, mb, C, ldc, m, n, (int)tiles_m, (int)tiles_n, (int)kst, (int)per,
                                         device_error_word());
    MELA_LAUNCH_CHECK("gemm_tc_kernel");
    return MELA_OK;
}

// ---------------------------------------------------------------- Strassen
// Seven products of half-size blocks instead of eight (Strassen 1969; over
// GF(2) every sign is +).  The sums of blocks cost no pass of their own: the
// expansion reads both blocks of an operand and XORs them, and the epilogue
// adds a product to each block of C that it belongs to.  Blocks are halves of
// whole 256-bit tiles; the second ones are as short as the matrix leaves them
// and count as zero past that.
// Where it pays (device time, whole -> seven products): the seventh of the MMA
// work saved has to cover 7/4 of the expansion and the worse efficiency of
// products of half the K.  FP4: 32768^3 11.33 -> 9.97 ms (under the power cap
// either way), 30001 x 27003 x 29999 7.85 -> 7.22, 27200^3 6.53 -> 6.24, 24576^3
// 4.58 -> 4.59, 16384^3 1.39 -> 1.54; with K = 16384, 40000 x 16384 x 32768
// 6.50 -> 6.59.  INT8, half the rate: 32768^3 20.9 -> 17.7 ms, 20480^3 4.87 ->
// 4.66, 22000 x 16384 x 22300 4.56 -> 4.40, 16384^3 2.49 -> 2.50.
constexpr i64 ST_MIN = 16384, ST_K_F4 = 20480;
constexpr double ST_CELLS_F4 = 2e13, ST_CELLS_I8 = 8e12;

bool gemm_strassen_fits(const u64 *A, i64 lda, const u64 *B, i64 ldb, const u64 *C, i64 ldc, i64 m, i64 k, i64 n,
                        bool fp4, int tile)
{
    if (m < ST_MIN || k < (fp4 ? ST_K_F4 : ST_MIN) || n < ST_MIN || !use_pairs(256, tile)) return false;
    if ((double)m * (double)k * (double)n < (fp4 ? ST_CELLS_F4 : ST_CELLS_I8)) return false;
    // blocks of A and B are read after blocks of C are written
    return packed_apart(A, lda, m, k, C, ldc, m, n) && packed_apart(B, ldb, k, n, C, ldc, m, n);
}

mela_status launch_gemm_strassen(const u64 *A, i64 lda, const u64 *B, i64 ldb, u64 *C, i64 ldc, i64 m, i64 k, i64 n,
                                 void *ws, size_t ws_bytes, bool fp4, cudaStream_t s)
{
    auto half = [](i64 x) { return ((x + 1) / 2 + 255) / 256 * 256; };
    const i64 mh = half(m), kh = half(k), nh = half(n), kp = fp4 ? kh / 2 : kh;
    unsigned char *A8 = (unsigned char *)ws, *B8 = A8 + (size_t)mh * kp;
    if ((uintptr_t)ws & 15) {
        set_error("gemm_tc: operands must be 16-byte aligned");
        return MELA_ERR_INVALID;
    }
    if ((size_t)(mh + nh) * kp > ws_bytes) {
        set_error("gemm_strassen: workspace of %zu bytes needed, %zu given", (size_t)(mh + nh) * kp, ws_bytes);
        return MELA_ERR_INVALID;
    }
    auto a = [&](int i, int j) {
        return ExpandBlock{A + i * mh * lda + j * (kh / 64), i ? m - mh : mh, j ? k - kh : kh};
    };
    auto b = [&](int i, int j) {
        return ExpandBlock{B + i * kh * ldb + j * (nh / 64), i ? k - kh : kh, j ? n - nh : nh};
    };
    const ExpandBlock none;
    const struct {
        ExpandBlock a[2], b[2];
        int c[2], first[2];  // blocks of C (2 i + j, -1: none), and whether this product is the first there
    } step[7] = {
        {{a(0, 0), a(1, 1)}, {b(0, 0), b(1, 1)}, {0, 3}, {1, 1}},
        {{a(1, 0), a(1, 1)}, {b(0, 0), none}, {2, 3}, {1, 0}},
        {{a(0, 0), none}, {b(0, 1), b(1, 1)}, {1, 3}, {1, 0}},
        {{a(1, 1), none}, {b(1, 0), b(0, 0)}, {0, 2}, {0, 0}},
        {{a(0, 0), a(0, 1)}, {b(1, 1), none}, {0, 1}, {0, 0}},
        {{a(1, 0), a(0, 0)}, {b(0, 0), b(0, 1)}, {3, -1}, {0, 0}},
        {{a(0, 1), a(1, 1)}, {b(1, 0), b(1, 1)}, {0, -1}, {0, 0}},
    };
    for (const auto &p : step) {
        mela_status st = launch_expand_sum(p.a, lda, mh, A8, p.b, ldb, nh, B8, kp, fp4, s);
        if (st != MELA_OK) return st;
        PairSum out{};
        for (int d = 0; d < 2; ++d) {
            if (p.c[d] < 0) continue;
            const int i = p.c[d] >> 1, j = p.c[d] & 1;
            out.c[d] = C + i * mh * ldc + j * (nh / 64);
            out.rows[d] = i ? m - mh : mh;
            out.words[d] = words_of(j ? n - nh : nh);
            out.add[d] = !p.first[d];
        }
        if ((st = launch_pairs<true>(A8, B8, mh, nh, kp, nullptr, ldc, mh, nh, fp4, out, s)) != MELA_OK) return st;
    }
    return MELA_OK;
}

}  // namespace mela
