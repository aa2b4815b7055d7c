// elim_small.cu -- reduced row echelon form of one small matrix by one CTA in
// one launch, the matrix in shared memory throughout.
//
// Same results as the other forms (elim.cu): greedy pivot columns and the
// unique RREF rows of gf2_rref_standard (src/mela_null_gf2.c:88-131).  The
// columns go 32 at a time: up to 64 unused rows with bits left there are
// eliminated among themselves by one warp (half_word_select, basis.cuh), and
// every row then takes the combination of the round's original pivot rows
// that clears its bits at the round's pivot columns, through 4-bit tables of
// those rows.  Rounds repeat until no unused row has a bit left in the 32
// columns.
//
// Bound by the serial chain of a round (about 2600 cycles of half_word_select,
// five barriers and the table reads), not by throughput: 100 x 200 takes 13 us
// and 256 x 512 36 us, against 112 and about 300 us one pivot and one barrier
// at a time, and 27 and 43 us in tensor-core windows (which pass it at about
// 300 rows: 400 x 800 92 us here, 80 there).
#include "mela_common.cuh"
#include "mela_internal.h"
#include "mela_host.h"
#include "elim.h"
#include "basis.cuh"

namespace mela {

namespace {

constexpr int SM_THREADS = 512;
constexpr int SM_MAX_ROWS = SM_THREADS;  // a thread per row lists the candidates
constexpr int SM_MAX_BYTES = 192 * 1024;  // the matrix and the tables

struct SmallHead {
    HalfRound r;
    int crow[kHalfCand];    // row of a candidate
    int colrow[32];         // pivot row of column b of the current half word
    int wcnt[2][32];        // candidates per warp, alternating
    int pcol_of[SM_MAX_ROWS];  // column of the row's pivot in this round (-1: none)
};

struct SmallLayout {
    int wc, pitch;  // words per row; per row in shared memory (odd: rows fall on different banks)
    size_t a, vt, total;
};
__host__ __device__ inline SmallLayout small_layout(int m, int n)
{
    SmallLayout L;
    L.wc = (n + 63) >> 6;
    L.pitch = L.wc | 1;
    L.a = (sizeof(SmallHead) + 15) & ~(size_t)15;
    L.vt = L.a + (size_t)m * L.pitch * 8;
    L.total = L.vt + (size_t)128 * L.wc * 8;
    return L;
}

static_assert(sizeof(SmallHead) <= 8 * 1024, "shared memory head");

__global__ void __launch_bounds__(SM_THREADS, 1)
elim_small_kernel(u64 *__restrict__ M, i64 ld, int m, int n, int lanes_log2, long long *rank, long long *piv,
                  long long *prow)
{
    extern __shared__ __align__(16) unsigned char sm_raw[];
    SmallHead &S = *reinterpret_cast<SmallHead *>(sm_raw);
    const SmallLayout L = small_layout(m, n);
    const int wc = L.wc, pitch = L.pitch;
    u64 *A = reinterpret_cast<u64 *>(sm_raw + L.a);
    u64 *vt = reinterpret_cast<u64 *>(sm_raw + L.vt);  // entry (g, e), word x: vt[(16 g + e) wc + x]
    const u32 *A32 = reinterpret_cast<const u32 *>(A);
    constexpr int NW = SM_THREADS / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // P = 2^lanes_log2 lanes take a row's words together
    const int P = 1 << lanes_log2, part = tid & (P - 1), rows_per_pass = SM_THREADS >> lanes_log2;

    for (int e = tid; e < m * wc; e += SM_THREADS) {
        const int j = e / wc, x = e - j * wc;
        A[j * pitch + x] = M[(i64)j * ld + x];
    }
    bool used = tid >= m;  // row tid is a pivot row (or no row)
    int r = 0, par = 0;
    __syncthreads();
    for (int h = 0; h < 2 * wc && r < m; ++h) {
        const int x0 = h >> 1;
        u32 H = 0;  // pivot columns of this half word
        while (r + __popc(H) < m) {
            const u32 d = used ? 0u : A32[2 * tid * pitch + h];
            const unsigned bal = __ballot_sync(0xffffffffu, d != 0);
            par ^= 1;
            if (lane == 0) S.wcnt[par][warp] = __popc(bal);
            S.pcol_of[tid] = -1;
            __syncthreads();
            const int wv = lane < NW ? S.wcnt[par][lane] : 0;
            const int total = __reduce_add_sync(0xffffffffu, wv);
            if (total == 0) break;
            int idx = __reduce_add_sync(0xffffffffu, lane < warp ? wv : 0) + __popc(bal & ((1u << lane) - 1));
            if (d == 0 || idx >= kHalfCand) idx = -1;
            if (idx >= 0) {
                S.r.cand[idx] = d;
                S.r.pcol[idx] = -1;
                S.crow[idx] = tid;
            }
            __syncthreads();
            if (warp == 0) half_word_select(S.r, total < kHalfCand ? total : kHalfCand);
            __syncthreads();
            const u32 C = S.r.C;
            const int pc = idx >= 0 ? S.r.pcol[idx] : -1;
            if (pc >= 0) {
                used = true;
                S.colrow[pc] = tid;
                S.pcol_of[tid] = pc;
            }
            // tables over the round's original pivot rows (words x0 ..) and T
            for (int e = tid; e < 128 * (wc - x0); e += SM_THREADS) {
                const int ge = e / (wc - x0), x = x0 + e - ge * (wc - x0), g = ge >> 4, v = ge & 15;
                u64 a = 0;
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const int ci = S.r.ci[4 * g + b];
                    if (((v >> b) & 1) && ci >= 0) a ^= A[S.crow[ci] * pitch + x];
                }
                vt[ge * wc + x] = a;
            }
            if (tid >= SM_THREADS - 128) half_word_tt(S.r, tid - (SM_THREADS - 128));
            __syncthreads();
            for (int j0 = 0; j0 < m; j0 += rows_per_pass) {
                const int j = j0 + (tid >> lanes_log2);
                u32 z = 0;
                u64 keep = ~0ull;
                if (j < m) {
                    const int own = S.pcol_of[j];
                    const u32 y = A32[2 * j * pitch + h] & C;
                    z = own >= 0 ? S.r.T[own] : y ? half_word_times_T(S.r, y) : 0u;
                    keep = own >= 0 ? 0ull : ~0ull;
                }
                __syncwarp();  // the row's lanes have read its half word
                if (z) {
                    for (int x = x0 + part; x < wc; x += P) {
                        u64 a = A[j * pitch + x] & keep;
#pragma unroll
                        for (int g = 0; g < 8; ++g) a ^= vt[(16 * g + ((z >> (4 * g)) & 15)) * wc + x];
                        A[j * pitch + x] = a;
                    }
                }
            }
            H |= C;
            __syncthreads();
        }
        if (tid < 32 && ((H >> tid) & 1)) {
            const int t = r + __popc(H & ((1u << tid) - 1));
            piv[t] = 32 * h + tid;
            prow[t] = S.colrow[tid];
        }
        r += __popc(H);
        __syncwarp();
    }
    __syncthreads();
    for (int e = tid; e < m * wc; e += SM_THREADS) {
        const int j = e / wc, x = e - j * wc;
        M[(i64)j * ld + x] = A[j * pitch + x];
    }
    if (tid == 0) *rank = r;
}

}  // namespace

bool small_elim_fits(i64 m, i64 n)
{
    if (m > SM_MAX_ROWS || n > 64 * 256) return false;
    const SmallLayout L = small_layout((int)m, (int)n);
    return L.total - L.a <= SM_MAX_BYTES;
}

mela_status launch_small_elim(u64 *M, i64 ld, i64 m, i64 n, long long *d_rank, long long *d_piv, long long *d_prow,
                              cudaStream_t s)
{
    const SmallLayout L = small_layout((int)m, (int)n);
    int lg = 0;
    while (lg < 4 && (2 << lg) <= L.wc) ++lg;
    MELA_CUDA_TRY(cudaFuncSetAttribute(elim_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       SM_MAX_BYTES + 8 * 1024));
    elim_small_kernel<<<1, SM_THREADS, L.total, s>>>(M, ld, (int)m, (int)n, lg, d_rank, d_piv, d_prow);
    MELA_LAUNCH_CHECK("elim_small_kernel");
    return MELA_OK;
}

}  // namespace mela
