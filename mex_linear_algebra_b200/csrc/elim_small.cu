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
constexpr int SM_NULL_COLS = 512;         // columns of a null space written by the same launch

struct SmallHead {
    HalfRound r;
    int crow[kHalfCand];    // row of a candidate
    int colrow[32];         // pivot row of column b of the current half word
    int wcnt[2][32];        // candidates per warp, alternating
    int pcol_of[SM_MAX_ROWS];  // column of the row's pivot in this round (-1: none)
    short prow_of[SM_NULL_COLS];  // null space: row of the column's pivot (-1: free column)
    short fcol[SM_NULL_COLS];     // the free columns
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

// POST: for the gateways' calls.  Nothing is written back but what the caller
// waits for, straight into its page-locked words: the rank, the device error
// word and, where Z is given, the null-space basis as n x (n - rank) logical
// bytes, column by column: the unit bit of a free column, and at the pivot
// columns the RREF rows' bits there.  One launch and one wait instead of five
// launches, three copies and two waits: 72 x 149 null space 86 -> 42 us a call,
// rank 58 -> 40; 256 x 512 null space 146 -> 111.  The basis is gathered as bits
// first (a byte at a time from the rows: 39 us for 158 KB, 28 this way, which
// is what one SM's writes to host memory take).
template <bool POST>
__global__ void __launch_bounds__(SM_THREADS, 1)
elim_small_kernel(u64 *__restrict__ M, i64 ld, int m, int n, int lanes_log2, long long *rank, long long *piv,
                  long long *prow, unsigned char *Z, const u32 *err, u32 *err_out)
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

    const u64 last = n & 63 ? (1ull << (n & 63)) - 1 : ~0ull;  // bits past the last column are no columns
    for (int e = tid; e < m * wc; e += SM_THREADS) {
        const int j = e / wc, x = e - j * wc;
        A[j * pitch + x] = M[(i64)j * ld + x] & (x == wc - 1 ? last : ~0ull);
    }
    if (POST) S.prow_of[tid] = -1;
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
            if (POST) {
                if (Z) S.prow_of[32 * h + tid] = (short)S.colrow[tid];
            } else {
                piv[t] = 32 * h + tid;
                prow[t] = S.colrow[tid];
            }
        }
        r += __popc(H);
        __syncwarp();
    }
    __syncthreads();
    if (tid == 0) *rank = r;
    if constexpr (POST) {
        if (tid == 0) *err_out = *err;
        if (!Z) return;
        const int f = n - r;
        if (warp == 0) {
            for (int c0 = 0, at = 0; c0 < n; c0 += 32) {
                const bool free_col = c0 + lane < n && S.prow_of[c0 + lane] < 0;
                const unsigned bal = __ballot_sync(0xffffffffu, free_col);
                if (free_col) S.fcol[at + __popc(bal & ((1u << lane) - 1))] = (short)(c0 + lane);
                at += __popc(bal);
            }
        }
        __syncthreads();
        // the basis as bits, column c's rows 32 k .. in word k: a warp holds 32
        // rows' places and takes every column's word of them by a ballot
        const int kw = (n + 31) >> 5;
        u32 *zb = reinterpret_cast<u32 *>(sm_raw + L.total);
        {
            static_assert(SM_NULL_COLS <= 32 * NW, "a warp per word of a column");
            const int k = warp % kw, step = NW / kw;
            const int i = 32 * k + lane, p = i < n ? S.prow_of[i] : -1;
            for (int c = warp / kw; c < f; c += step) {
                const int q = S.fcol[c];
                const bool bit = p >= 0 ? (A32[2 * p * pitch + (q >> 5)] >> (q & 31)) & 1u : i == q;
                const unsigned bal = __ballot_sync(0xffffffffu, bit);
                if (lane == 0) zb[c * (kw + 1) + k] = bal;
            }
        }
        for (int c = tid; c < f; c += SM_THREADS) zb[c * (kw + 1) + kw] = 0;
        __syncthreads();
        // 16 bytes a thread: 16 bits from place i on, past row n those of the next column
        for (int e = 16 * tid; e < f * n; e += 16 * SM_THREADS) {
            int c = e / n, i = e - c * n;
            u32 bits = 0;
            for (int got = 0; got < 16 && c < f; ++c, i = 0) {
                const u32 *w = zb + c * (kw + 1) + (i >> 5);
                bits |= (__funnelshift_r(w[0], w[1], i & 31) & 0xFFFFu) << got;
                got += n - i;
            }
            const uint4 v = make_uint4(((bits & 15u) * 0x00204081u) & 0x01010101u,
                                       (((bits >> 4) & 15u) * 0x00204081u) & 0x01010101u,
                                       (((bits >> 8) & 15u) * 0x00204081u) & 0x01010101u,
                                       (((bits >> 12) & 15u) * 0x00204081u) & 0x01010101u);
            *reinterpret_cast<uint4 *>(Z + e) = v;
        }
    } else {
        for (int e = tid; e < m * wc; e += SM_THREADS) {
            const int j = e / wc, x = e - j * wc;
            M[(i64)j * ld + x] = A[j * pitch + x];
        }
    }
}

}  // namespace

bool small_elim_fits(i64 m, i64 n)
{
    if (m > SM_MAX_ROWS || n > 64 * 256) return false;
    const SmallLayout L = small_layout((int)m, (int)n);
    return L.total - L.a <= SM_MAX_BYTES;
}

static int small_lanes(const SmallLayout &L)
{
    int lg = 0;
    while (lg < 4 && (2 << lg) <= L.wc) ++lg;
    return lg;
}

mela_status launch_small_elim(u64 *M, i64 ld, i64 m, i64 n, long long *d_rank, long long *d_piv, long long *d_prow,
                              cudaStream_t s)
{
    const SmallLayout L = small_layout((int)m, (int)n);
    MELA_CUDA_TRY(cudaFuncSetAttribute(elim_small_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       SM_MAX_BYTES + 8 * 1024));
    elim_small_kernel<false><<<1, SM_THREADS, L.total, s>>>(M, ld, (int)m, (int)n, small_lanes(L), d_rank, d_piv,
                                                            d_prow, nullptr, nullptr, nullptr);
    MELA_LAUNCH_CHECK("elim_small_kernel");
    return MELA_OK;
}

bool small_null_fits(i64 m, i64 n) { return n <= SM_NULL_COLS && small_elim_fits(m, n); }

mela_status launch_small_post(const u64 *M, i64 ld, i64 m, i64 n, const Posted &to, bool null_space, cudaStream_t s)
{
    const SmallLayout L = small_layout((int)m, (int)n);
    if (null_space && (!small_null_fits(m, n) || to.bytes_size < (size_t)n * (size_t)n)) {
        set_error("small null space: result buffer too small");
        return MELA_ERR_INVALID;
    }
    MELA_CUDA_TRY(cudaFuncSetAttribute(elim_small_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       SM_MAX_BYTES + 8 * 1024));
    const size_t smem = L.total + (null_space ? (size_t)n * ((n + 31) / 32 + 1) * 4 : 0);
    elim_small_kernel<true><<<1, SM_THREADS, smem, s>>>(const_cast<u64 *>(M), ld, (int)m, (int)n, small_lanes(L),
                                                           to.value, nullptr, nullptr,
                                                           null_space ? to.bytes : nullptr, to.err_word, to.err);
    MELA_LAUNCH_CHECK("elim_small_kernel");
    return MELA_OK;
}

}  // namespace mela
