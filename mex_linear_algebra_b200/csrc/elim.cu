// elim.cu -- Gaussian elimination over GF(2) on packed device matrices:
// rank (forward elimination) and reduced row echelon form, in two forms.
//
// Results are those of the reference's algorithms: the rank of
// bitrank_packed / rank_m4ri (src/mela_rank_gf2.c:27-121,
// src/mela_rank_m4ri.c:94-279), and the pivot columns and RREF rows of
// gf2_rref_standard (src/mela_null_gf2.c:88-131).  Both are properties of
// the row space (greedy pivot columns, unique RREF), so any elimination
// order that keeps the pivots greedy reproduces them bit for bit.
//
// Rows never move in memory.  Each row is "active" (not yet a pivot) or a
// pivot; pivot t of the result lives in physical row prow[t] and has its
// leading one in column piv[t].  RREF row t is therefore M[prow[t]].
//
// Blocked form (the Four-Russians / PLE form), one 64-column panel (one
// word column w) at a time:
//   panel_select  one CTA.  Brings the active rows' panel words to reduced row
//                   echelon form (lowest set bit leading) in chunks of a row
//                   per thread, 32 columns at a time (basis.cuh); the walk ends
//                   once the basis spans the panel.  Gives the panel's greedy
//                   pivot columns b, the row S_b that entered the basis at
//                   each, and the combination coef[b] of the S rows whose panel
//                   part is the unit vector of column b.
//   panel_rows    R_b = XOR of the S rows in coef[b] (full width from word
//                   w on), written to a panel buffer and over row S_b.
//   panel_update  every other row j (active rows for rank; all rows for
//                 RREF) XORs sum_k bit(c_k of row j) * R_k, looked up 8 pivot
//                 bits at a time in shared-memory tables of the 256
//                 combinations of 8 R rows.
// Plain form: one cooperative persistent kernel, one grid barrier per
// column: every CTA searches its rows for the first active row holding the
// column's bit (atomicMin over the grid), then every CTA XORs that pivot row
// into its rows holding the bit.
#include <climits>
#include <cstring>

#include "mela_common.cuh"
#include "mela_internal.h"
#include "mela_host.h"
#include "elim.h"
#include "basis.cuh"

namespace mela {

// ---------------------------------------------------------------- helpers
// Panel bookkeeping shared by the blocked kernels (device memory); everything
// of a pivot is indexed by its column in the panel.
struct PanelState {
    long long rank;  // pivots found so far
    int p;           // pivots in the current panel
    int pad;
    u64 pivmask;     // pivot columns of the current panel
    int srow[64];    // physical row S_b of pivot column b (-1: none), which receives R_b
    u64 coef[64];    // R_b = XOR_{j in coef[b]} row S_j
};

// ---------------------------------------------------------------- panel_select
// The state before the first panel: every row active, no pivots, word 0 of every
// row (the first panel's words).  One launch instead of three fills and one.
__global__ void panel_init_kernel(const u64 *__restrict__ M, i64 ld, i64 m, unsigned char *state, int *stamp,
                                  PanelState *ps, u64 *__restrict__ y)
{
    for (i64 j = blockIdx.x * (i64)blockDim.x + threadIdx.x; j < m; j += (i64)gridDim.x * blockDim.x) {
        y[j] = M[j * ld];
        state[j] = 1;
        stamp[j] = -1;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) ps->rank = 0;
}

namespace {
constexpr int SEL_THREADS = 512;
struct SelSmem {
    u64 basis[64];     // in-place vector of pivot column b
    u64 tab[16][16];   // 4-bit tables of the basis
    u64 vt[8][16];     // 4-bit tables of a round's pivot rows
    u64 cv[kHalfCand]; // the candidates' vectors
    int prow[64];
    int wcnt[2][32];
    HalfRound r;
};

// A row's vector after a round with pivot columns C of half word h and the
// combination z of the round's pivot rows.
__device__ __forceinline__ u64 sel_apply(const SelSmem &S, u64 v, int h, u32 C, u32 z)
{
    v &= ~((u64)C << (32 * h));
#pragma unroll
    for (int g = 0; g < 8; ++g) v ^= S.vt[g][(z >> (4 * g)) & 15];
    return v | ((u64)z << (32 * h));
}
}  // namespace

// The panel words y come packed (the update of the panel before writes them),
// so a chunk is one coalesced read; on dense matrices the first chunk fills
// the basis.  Bound by its serial chain (one CTA): half_word_select and four
// barriers a round of up to 32 pivots, 7.8 us for a full panel of 64 against
// 44 us with warp-local XOR bases merged pairwise.  Whole calls with the rows
// and update kernels below: rank of 1501 x 2900 760 us, of 16384 x 32768 (rank
// 12000) 28.0 ms, before 3.0 and 56.7 ms.
__global__ void __launch_bounds__(SEL_THREADS, 1)
panel_select_kernel(const u64 *__restrict__ y, i64 m, i64 n, i64 w, unsigned char *state, int *stamp, int panel,
                    PanelState *ps, long long *piv, long long *prow)
{
    __shared__ SelSmem S;
    constexpr int NW = SEL_THREADS / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int valid = n - 64 * w < 64 ? (int)(n - 64 * w) : 64;
    const long long r0 = ps->rank;
    u64 H = 0;  // pivot columns so far
    int nb = 0, par = 0;
    for (i64 base = 0; base < m && nb < valid; base += SEL_THREADS) {
        const u64 H0 = H;  // basis vectors of earlier chunks
        if (H0) {
            for (int e = tid; e < 256; e += SEL_THREADS) {
                const int g = e >> 4, v = e & 15;
                u64 a = 0;
#pragma unroll
                for (int b = 0; b < 4; ++b)
                    if (((v >> b) & 1) && ((H0 >> (4 * g + b)) & 1)) a ^= S.basis[4 * g + b];
                S.tab[g][v] = a;
            }
            __syncthreads();
        }
        const i64 j = base + tid;
        u64 v = (j < m && state[j]) ? y[j] : 0ull;
        const u64 yb = v & H0;
        if (yb) {
            v ^= yb;
#pragma unroll
            for (int g = 0; g < 16; ++g) v ^= S.tab[g][(yb >> (4 * g)) & 15];
        }
        if (r0 >= m) break;  // every row is a pivot row
        int mycol = -1;
        for (int h = 0; h < 2 && nb < valid; ++h) {
            u32 Hh = (u32)(H >> (32 * h));
            while (Hh != 0xffffffffu && nb < valid) {
                const u32 d = mycol < 0 ? (u32)(v >> (32 * h)) & ~Hh : 0u;
                const unsigned bal = __ballot_sync(0xffffffffu, d != 0);
                par ^= 1;
                if (lane == 0) S.wcnt[par][warp] = __popc(bal);
                __syncthreads();
                const int wv = lane < NW ? S.wcnt[par][lane] : 0;
                const int total = __reduce_add_sync(0xffffffffu, wv);
                if (total == 0) break;
                int idx = __reduce_add_sync(0xffffffffu, lane < warp ? wv : 0) + __popc(bal & ((1u << lane) - 1));
                if (d == 0 || idx >= kHalfCand) idx = -1;
                if (idx >= 0) {
                    S.r.cand[idx] = d;
                    S.cv[idx] = v;
                    S.r.pcol[idx] = -1;
                }
                __syncthreads();
                if (warp == 0) half_word_select(S.r, total < kHalfCand ? total : kHalfCand);
                __syncthreads();
                const u32 C = S.r.C;
                if (tid < 128) {
                    const int g = tid >> 4, e = tid & 15;
                    u64 a = 0;
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        const int ci = S.r.ci[4 * g + b];
                        if (((e >> b) & 1) && ci >= 0) a ^= S.cv[ci];
                    }
                    S.vt[g][e] = a & ~((u64)C << (32 * h));
                } else if (tid < 256) {
                    half_word_tt(S.r, tid - 128);
                }
                const int pc = idx >= 0 ? S.r.pcol[idx] : -1;
                __syncthreads();
                if (pc >= 0) {
                    mycol = 32 * h + pc;
                    S.prow[mycol] = (int)j;
                    v = sel_apply(S, 0, h, C, S.r.T[pc]);
                } else {
                    const u32 yr = (u32)(v >> (32 * h)) & C;
                    if (yr) v = sel_apply(S, v, h, C, half_word_times_T(S.r, yr));
                }
                if (tid < 64 && ((H0 >> tid) & 1)) {
                    const u64 o = S.basis[tid];
                    const u32 yr = (u32)(o >> (32 * h)) & C;
                    if (yr) S.basis[tid] = sel_apply(S, o, h, C, half_word_times_T(S.r, yr));
                }
                nb += __popc(C);
                Hh |= C;
                H |= (u64)C << (32 * h);
            }
        }
        if (mycol >= 0) S.basis[mycol] = v;
        __syncthreads();
    }
    __syncthreads();  // every thread has read the rank before it is advanced
    if (tid < 64) {
        int r = -1;
        if ((H >> tid) & 1) {
            const int t = __popcll(H & ((1ull << tid) - 1));
            r = S.prow[tid];
            ps->coef[tid] = S.basis[tid] & H;
            piv[r0 + t] = 64 * w + tid;
            prow[r0 + t] = r;
            state[r] = 0;
            stamp[r] = panel;
        }
        ps->srow[tid] = r;
    }
    if (tid == 0) {
        ps->p = nb;
        ps->pivmask = H;
        ps->rank = r0 + nb;
    }
}

// ---------------------------------------------------------------- panel_rows
// Block: 4 words x every pivot, a thread per (column, word).  R_b is looked
// up four columns at a time in 16 tables of the 16 combinations of the S rows
// of columns 4g..4g+3; every S row is read before any is overwritten.
__global__ void __launch_bounds__(256)
panel_rows_kernel(u64 *__restrict__ M, i64 ld, i64 wc, i64 w, const PanelState *ps,
                  u64 *__restrict__ Rbuf)
{
    __shared__ u64 rows[64][4];
    __shared__ u64 tab[16][16][4];
    if (ps->p == 0) return;
    const int tid = threadIdx.x, b = tid >> 2, q = tid & 3;
    const i64 word = w + (i64)blockIdx.x * 4 + q;
    const int sr = ps->srow[b];
    const u64 coef = sr >= 0 ? ps->coef[b] : 0ull;
    const bool ok = sr >= 0 && word < wc;
    rows[b][q] = ok ? M[(i64)sr * ld + word] : 0ull;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int e = (tid >> 2) + 64 * i, g = e >> 4, v = e & 15;
        u64 a = 0;
#pragma unroll
        for (int h = 0; h < 4; ++h) a ^= ((v >> h) & 1) ? rows[4 * g + h][q] : 0ull;
        tab[g][v][q] = a;
    }
    __syncthreads();
    u64 acc = 0;
#pragma unroll
    for (int g = 0; g < 16; ++g) acc ^= tab[g][(coef >> (4 * g)) & 15][q];
    if (ok) {
        M[(i64)sr * ld + word] = acc;
        Rbuf[(i64)b * wc + word] = acc;
    }
}

// ---------------------------------------------------------------- panel_update
// Four-Russians update with tables of K pivot bits (M4RI k = K).  The panel's
// 64 bit positions are cut into G = ceil(64/K) groups of consecutive
// positions (the last one shorter when K does not divide 64); group g's table
// holds the 2^bits(g) XOR combinations of the reduced rows R of its positions
// (zero rows where a position holds no pivot), built in two steps: the
// combinations of the low and of the high half of the group's bits from the
// rows, then every other entry from one of each.  Every other row j
// (active rows for the rank; all rows for the RREF) then XORs, per word,
// one entry per group, indexed by its panel bits at the pivot positions.
// Each CTA covers TW words (columns) and `rt` rows; the table build is paid
// once per CTA, so a larger K (fewer lookups per row) pays off with more
// rows per CTA.  Shared memory: (G-1)*2^K + 2^bits(G-1) entries of TW words.
template <int K>
struct M4riGroups {
    static constexpr int G = (64 + K - 1) / K;
    static constexpr int last_bits = 64 - (G - 1) * K;
    static constexpr int entries = (G - 1) * (1 << K) + (1 << last_bits);
    __host__ __device__ static constexpr int bits(int g) { return g == G - 1 ? last_bits : K; }
};

template <int K, int TW>
__global__ void __launch_bounds__(256)
panel_update_kernel(u64 *__restrict__ M, i64 ld, i64 m, i64 wc, i64 w, const PanelState *ps,
                    const u64 *__restrict__ Rbuf, const unsigned char *state, const int *stamp,
                    int panel, int rref, const u64 *__restrict__ y, u64 *__restrict__ ynext, int rt)
{
    using Gr = M4riGroups<K>;
    extern __shared__ __align__(16) unsigned char upd_raw[];
    u64 *T = reinterpret_cast<u64 *>(upd_raw);  // entry e of group g: T[((g << K) + e) * TW + t]
    const int p = ps->p;
    const int tid = threadIdx.x;
    const i64 row0 = (i64)blockIdx.y * rt;
    // the next panel's words (word w + 1, in the first column tile) also go,
    // packed, to ynext, unless every row is a pivot row and none is looked at
    // any more (55 x 5400, 84 panels behind the last pivot: 958 -> 780 us)
    if (p == 0) {
        if (blockIdx.x == 0 && w + 1 < wc && ps->rank < m)
            for (i64 j = row0 + tid; j < row0 + rt && j < m; j += 256) ynext[j] = M[j * ld + w + 1];
        return;
    }
    const u64 pm = ps->pivmask;
    const i64 w0 = w + (i64)blockIdx.x * TW;

    // entry 0 of every group is zero, entry 2^h of group g is R_(gK + h)
    for (int e = tid; e < Gr::G * TW; e += 256) T[(((e / TW) << K)) * TW + e % TW] = 0;
    for (int e = tid; e < 64 * TW; e += 256) {
        const int t = e % TW, b = e / TW, g = b / K, h = b - g * K;
        const i64 word = w0 + t;
        T[((g << K) + (1 << h)) * TW + t] = (((pm >> b) & 1) && word < wc) ? Rbuf[(i64)b * wc + word] : 0ull;
    }
    __syncthreads();
    // combinations of the low LB bits (entries x) and of the others (x << LB)
    constexpr int LB = K / 2, HB = K - LB, NX = (1 << LB) + (1 << HB);
    for (int e = tid; e < Gr::G * NX * TW; e += 256) {
        const int t = e % TW, rest = e / TW, g = rest / NX, i = rest % NX;
        const int x = i < (1 << LB) ? i : (i - (1 << LB)) << LB;
        if (x >= (1 << Gr::bits(g)) || (x & (x - 1)) == 0) continue;
        const u64 *Tg = T + ((size_t)g << K) * TW;
        u64 a = 0;
#pragma unroll
        for (int h = 0; h < K; ++h) a ^= ((x >> h) & 1) ? Tg[(1 << h) * TW + t] : 0ull;
        T[(((size_t)g << K) + x) * TW + t] = a;
    }
    __syncthreads();
    for (int e = tid; e < Gr::entries * TW; e += 256) {
        const int t = e % TW, ge = e / TW, g = ge >> K, x = ge & ((1 << K) - 1);
        const int lo = x & ((1 << LB) - 1), hi = x ^ lo;
        if (!lo || !hi) continue;
        const u64 *Tg = T + ((size_t)g << K) * TW;
        T[(size_t)e] = Tg[lo * TW + t] ^ Tg[hi * TW + t];
    }
    __syncthreads();

    const int t = tid % TW;
    const i64 word = w0 + t;
    const bool next = word == w + 1;
    if (word >= wc) return;
    for (int rr = tid / TW; rr < rt; rr += 256 / TW) {
        const i64 j = row0 + rr;
        if (j >= m) break;
        const u64 yj = (rref ? (stamp[j] == panel) : (state[j] == 0)) ? 0ull : y[j] & pm;
        if (!yj) {
            if (next) ynext[j] = M[j * ld + word];
            continue;
        }
        u64 acc = M[j * ld + word];
#pragma unroll
        for (int g = 0; g < Gr::G; ++g)
            acc ^= T[((g << K) + (int)((yj >> (g * K)) & ((1ull << Gr::bits(g)) - 1))) * TW + t];
        M[j * ld + word] = acc;
        if (next) ynext[j] = acc;
    }
}

// The (K, TW) pairs the blocked form runs with: TW (words per CTA) shrinks as
// the tables grow, keeping them within 100 KB of shared memory.
template <int K>
struct M4riTile;
template <> struct M4riTile<4> { static constexpr int TW = 8; };
template <> struct M4riTile<6> { static constexpr int TW = 8; };
template <> struct M4riTile<7> { static constexpr int TW = 4; };
template <> struct M4riTile<8> { static constexpr int TW = 4; };
template <> struct M4riTile<9> { static constexpr int TW = 2; };
template <> struct M4riTile<10> { static constexpr int TW = 2; };

template <int K>
static mela_status launch_panel_update(u64 *M, i64 ld, i64 m, i64 wc, i64 w, const PanelState *ps,
                                       const u64 *Rbuf, const unsigned char *state, const int *stamp,
                                       int panel, int rref, const u64 *y, u64 *ynext, int rt,
                                       cudaStream_t s, bool configure)
{
    constexpr int TW = M4riTile<K>::TW;
    constexpr size_t smem = (size_t)M4riGroups<K>::entries * TW * 8;
    if (configure) {
        MELA_CUDA_TRY(cudaFuncSetAttribute(panel_update_kernel<K, TW>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        return MELA_OK;
    }
    const i64 rem = wc - w;
    const i64 rtiles = (m + rt - 1) / rt;
    panel_update_kernel<K, TW><<<dim3((unsigned)((rem + TW - 1) / TW), (unsigned)rtiles), 256, smem, s>>>(
        M, ld, m, wc, w, ps, Rbuf, state, stamp, panel, rref, y, ynext, rt);
    return MELA_OK;
}

using PanelUpdateFn = mela_status (*)(u64 *, i64, i64, i64, i64, const PanelState *, const u64 *,
                                      const unsigned char *, const int *, int, int, const u64 *, u64 *,
                                      int, cudaStream_t, bool);

static PanelUpdateFn panel_update_for(int k)
{
    switch (k) {
    case 4: return launch_panel_update<4>;
    case 6: return launch_panel_update<6>;
    case 7: return launch_panel_update<7>;
    case 8: return launch_panel_update<8>;
    case 9: return launch_panel_update<9>;
    case 10: return launch_panel_update<10>;
    default: return nullptr;
    }
}

// ---------------------------------------------------------------- plain form
struct GridBar {
    unsigned count;
    unsigned gen;
    int abort;
};

__device__ bool grid_sync(GridBar *gb, unsigned nblocks, u32 *err)
{
    __syncthreads();
    __shared__ int s_abort;
    if (threadIdx.x == 0) {
        volatile unsigned *vgen = &gb->gen;
        const unsigned g = *vgen;
        __threadfence();
        if (atomicAdd(&gb->count, 1u) == nblocks - 1) {
            gb->count = 0;
            __threadfence();
            atomicAdd(&gb->gen, 1u);
        } else {
            const unsigned long long t0 = global_ns();
            int spins = 0;
            while (*vgen == g) {
                if (((++spins) & 255) == 0) {
                    if (*((volatile int *)&gb->abort)) break;
                    if (global_ns() - t0 > kWaitLimitNs) {
                        atomicOr(err, kErrWaitTimeout);
                        atomicExch(&gb->abort, 1);
                        break;
                    }
                }
            }
        }
        __threadfence();
        s_abort = *((volatile int *)&gb->abort);
    }
    __syncthreads();
    return s_abort == 0;
}

__global__ void __launch_bounds__(512)
ge_plain_kernel(u64 *__restrict__ M, i64 ld, i64 m, i64 n, int rref, unsigned char *state,
                long long *piv, long long *prow, long long *rank_out, int *cand, GridBar *gb,
                u32 *err)
{
    extern __shared__ u64 prow_buf[];
    __shared__ int s_min;
    const i64 wc = words_of(n);
    const i64 per = (m + gridDim.x - 1) / gridDim.x;
    const i64 r0 = (i64)blockIdx.x * per;
    const i64 r1 = (r0 + per < m) ? r0 + per : m;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;

    auto search = [&](i64 c) {
        // first active row of this CTA holding bit c -> atomicMin(cand[c % 3])
        if (tid == 0) s_min = INT_MAX;
        __syncthreads();
        if (c < n) {
            const i64 cw = c >> 6;
            const u64 bit = 1ull << (c & 63);
            for (i64 j = r0 + tid; j < r1; j += blockDim.x) {
                if (state[j] && (M[j * ld + cw] & bit)) {
                    atomicMin(&s_min, (int)j);
                    break;
                }
            }
        }
        __syncthreads();
        if (tid == 0 && s_min != INT_MAX) atomicMin(&cand[c % 3], s_min);
    };

    long long r = 0;
    search(0);
    for (i64 c = 0; c < n; ++c) {
        if (!grid_sync(gb, gridDim.x, err)) break;
        const int p = *((volatile int *)&cand[c % 3]);
        if (blockIdx.x == 0 && tid == 0) cand[(c + 2) % 3] = INT_MAX;
        if (p == INT_MAX) {
            search(c + 1);
            continue;
        }
        if (blockIdx.x == 0 && tid == 0) {
            piv[r] = c;
            prow[r] = p;
        }
        ++r;
        if (p >= r0 && p < r1 && tid == 0) state[p] = 0;
        const i64 cw = c >> 6;
        const u64 bit = 1ull << (c & 63);
        for (i64 t = cw + tid; t < wc; t += blockDim.x) prow_buf[t] = M[(i64)p * ld + t];
        __syncthreads();
        // warp per row, lanes over words
        for (i64 j = r0 + warp; j < r1; j += nwarps) {
            if (j == p) continue;
            if (!rref && !state[j]) continue;
            if (!(M[j * ld + cw] & bit)) continue;
            for (i64 t = cw + lane; t < wc; t += 32) M[j * ld + t] ^= prow_buf[t];
        }
        __syncthreads();
        search(c + 1);
        if (r >= m) break;  // every row is a pivot: no later column can hold one
    }
    if (blockIdx.x == 0 && tid == 0 && rank_out) *rank_out = r;
}

// ---------------------------------------------------------------- null basis
// Z^T row i = e_{f_i} + sum_p R_p[f_i] e_{piv[p]}: the r bits of column f_i of
// the RREF rows, deposited at the pivot columns.  Three launches:
//   null_words     per column word W: the pivots before it, its pivot mask
//                  and the six move masks of the deposit
//   null_columns   the free columns of the RREF rows as rows of r bits
//   null_rows      the deposit, and the unit bits
// Bound by memory traffic: the RREF rows are read once, their free part is
// written and read once as rows and the basis written once (rank 12000 of
// 16384 x 32768: 49 + 31 + 31 + 85 MB; 100 us in all against 387 us with all
// columns transposed and a bit-by-bit deposit).
struct NullMeta {       // wc entries each
    u64 *mask;          // pivot columns of the word
    long long *before;  // pivots before the word
    u64 *mv;            // [6][wc] move masks
};

// A warp per word (piv is ascending).
__global__ void __launch_bounds__(256) null_words_kernel(const long long *__restrict__ piv, long long r, i64 wc,
                                                         NullMeta N)
{
    const int lane = threadIdx.x & 31;
    const i64 W = (i64)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (W >= wc) return;
    long long lo = 0, hi = r;  // first pivot >= 64 W, by 32 probes at a time
    while (lo < hi) {
        const long long step = (hi - lo + 31) / 32, at = lo + lane * step;
        const int below = __popc(__ballot_sync(0xffffffffu, at < hi && piv[at < hi ? at : lo] < 64 * W));
        if (below == 0) break;
        const long long up = lo + below * step;
        lo += (below - 1) * step + 1;
        hi = up < hi ? up : hi;
    }
    u32 m0 = 0, m1 = 0;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const long long t = lo + 32 * q + lane;
        const long long c = t < r ? piv[t] - 64 * W : 64;
        if (c < 32)
            m0 |= 1u << c;
        else if (c < 64)
            m1 |= 1u << (c - 32);
    }
    m0 = __reduce_or_sync(0xffffffffu, m0);
    m1 = __reduce_or_sync(0xffffffffu, m1);
    if (lane) return;
    const u64 mask = (u64)m0 | ((u64)m1 << 32);
    N.mask[W] = mask;
    N.before[W] = lo;
    // the bits to move by 1, 2, 4, ... when compressing under the mask (H. S.
    // Warren, Hacker's Delight, "Compress, or Generalized Extract"); the
    // deposit applies them in reverse
    u64 m = mask, mk = ~mask << 1;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        u64 mp = mk;
#pragma unroll
        for (int sh = 1; sh < 64; sh <<= 1) mp ^= mp << sh;
        const u64 mv = mp & m;
        N.mv[(i64)i * wc + W] = mv;
        m = (m ^ mv) | (mv >> (1 << i));
        mk &= ~mp;
    }
}

// Block: 256 RREF rows x 4 words.  A lane reads 32 bytes of its row, eight
// 32 x 32 warp transposes turn the warp's rows into 32-bit column slices, and
// a thread per column writes the block's 256 bits of a free column as one 32-byte
// piece of row (its rank among the free columns) of X.
__global__ void __launch_bounds__(256) null_columns_kernel(const u64 *__restrict__ M, i64 ld,
                                                           const long long *__restrict__ prow, long long r, i64 n,
                                                           i64 wc, NullMeta N, u64 *__restrict__ X, i64 ldx)
{
    __shared__ u32 U[256][9];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const i64 w0 = (i64)blockIdx.x * 4, t0 = (i64)blockIdx.y * 256;
    const i64 t = t0 + 32 * warp + lane;
    u32 a[8] = {};
    if (t < r) {
        const u64 *src = M + prow[t] * ld + w0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const u64 v = w0 + q < wc ? src[q] : 0ull;
            a[2 * q] = (u32)v;
            a[2 * q + 1] = (u32)(v >> 32);
        }
    }
#pragma unroll
    for (int g = 0; g < 8; ++g) U[32 * g + lane][warp] = transpose32_warp(a[g]);
    __syncthreads();
    const i64 W = w0 + (tid >> 6), c = 64 * W + (tid & 63);
    if (c >= n) return;
    const u64 mask = N.mask[W];
    if ((mask >> (tid & 63)) & 1) return;
    const i64 f = 64 * W - N.before[W] + __popcll(~mask & ((1ull << (tid & 63)) - 1));
    const i64 words = words_of(r), ow = (i64)blockIdx.y * 4;
    u64 *dst = X + f * ldx + ow;
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (ow + q < words) dst[q] = (u64)U[tid][2 * q] | ((u64)U[tid][2 * q + 1] << 32);
}

// Block: 32 words x NULL_ROWS basis rows, a lane per word, eight rows at a time.
constexpr int NULL_ROWS = 64;
__global__ void __launch_bounds__(256) null_rows_kernel(const u64 *__restrict__ X, i64 ldx, NullMeta N, long long f,
                                                        i64 n, i64 wc, u64 *__restrict__ Zt, i64 ldz)
{
    const i64 wtiles = (wc + 31) / 32;
    const i64 W = (i64)blockIdx.x % wtiles * 32 + threadIdx.x;
    if (W >= wc) return;
    const u64 mask = N.mask[W];
    const long long s = N.before[W];
    u64 mv[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) mv[i] = N.mv[(i64)i * wc + W];
    const int len = __popcll(mask), sb = (int)(s & 63);
    const u64 keep = len == 64 ? ~0ull : (1ull << len) - 1;
    const u64 vm = n - 64 * W >= 64 ? ~0ull : (1ull << (n - 64 * W)) - 1;
    const u64 fm = ~mask & vm;               // the word's free columns
    const long long f0 = 64 * W - s;         // free columns before it
    const int fn = __popcll(fm);
    const i64 i0 = (i64)blockIdx.x / wtiles * NULL_ROWS;
#pragma unroll 2
    for (int k = threadIdx.y; k < NULL_ROWS; k += 8) {
        const i64 i = i0 + k;
        if (i >= f) break;
        u64 x = 0;
        if (len) {
            const u64 *src = X + i * ldx + (s >> 6);
            x = src[0] >> sb;
            if (sb + len > 64) x |= src[1] << (64 - sb);
            x &= keep;
#pragma unroll
            for (int b = 5; b >= 0; --b) x = (x & ~mv[b]) | ((x << (1 << b)) & mv[b]);
            x &= mask;
        }
        const long long e = i - f0;  // this row's own free column, if in the word
        if (e >= 0 && e < fn) {
            // position of the e-th free column
            u64 t = fm;
            int left = (int)e, pos = 0;
#pragma unroll
            for (int sh = 32; sh; sh >>= 1) {
                const int c = __popcll(t & ((1ull << sh) - 1));
                if (left >= c) {
                    left -= c;
                    t >>= sh;
                    pos += sh;
                }
            }
            x |= 1ull << pos;
        }
        Zt[i * ldz + W] = x;
    }
}

// Packed rows -> row-major bytes (row i of Zt = column i of the n x f logical
// Z).  A thread writes 16 consecutive bytes of the result, from 16 bits of
// one row or the end of one and the start of the next (8192 x 8192: 16.2 us
// against 131 us with a division per byte).
__device__ __forceinline__ u32 spread4_01(u32 v) { return ((v & 15u) * 0x00204081u) & 0x01010101u; }
__global__ void __launch_bounds__(256) unpack_rows_kernel(const u64 *__restrict__ P, i64 ld, i64 rows, i64 n,
                                                          unsigned char *__restrict__ out)
{
    const i64 total = rows * n;
    const bool aligned = ((uintptr_t)out & 15) == 0;
    for (i64 e = (blockIdx.x * (i64)blockDim.x + threadIdx.x) * 16; e < total;
         e += (i64)gridDim.x * blockDim.x * 16) {
        const i64 i = total <= 0xffffffffll ? (i64)((u32)e / (u32)n) : e / n;
        const i64 j = e - i * n;
        if (aligned && n >= 16 && e + 16 <= total) {
            const u64 *src = P + i * ld + (j >> 6);
            const int sb = (int)(j & 63);
            u32 v = (u32)(src[0] >> sb);
            const i64 rem = n - j;  // columns left in row i
            if (sb + (rem < 16 ? (int)rem : 16) > 64) v |= (u32)(src[1] << (64 - sb));
            if (rem < 16) v = (v & ((1u << rem) - 1)) | ((u32)P[(i + 1) * ld] << rem);
            *reinterpret_cast<uint4 *>(out + e) =
                make_uint4(spread4_01(v), spread4_01(v >> 4), spread4_01(v >> 8), spread4_01(v >> 12));
        } else {
            i64 ii = i, jj = j;
            for (int q = 0; q < 16 && e + q < total; ++q) {
                out[e + q] = (unsigned char)((P[ii * ld + (jj >> 6)] >> (jj & 63)) & 1);
                if (++jj == n) {
                    jj = 0;
                    ++ii;
                }
            }
        }
    }
}

// ---------------------------------------------------------------- host side
static int grid_cap(i64 total, int threads)
{
    i64 g = (total + threads - 1) / threads;
    const i64 cap = (i64)sm_count() * 16;
    if (g > cap) g = cap;
    return (int)(g < 1 ? 1 : g);
}

static size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

ElimLayout elim_layout(i64 m, i64 n)
{
    ElimLayout L{};
    const i64 wc = words_of(n);
    size_t off = 0;
    L.state = off;  off += al256((size_t)m);
    L.stamp = off;  off += al256((size_t)m * 4);
    L.ps = off;     off += al256(sizeof(PanelState));
    L.rbuf = off;   off += al256((size_t)64 * (size_t)(wc ? wc : 1) * 8);
    L.cand = off;   off += al256(3 * sizeof(int));
    L.gb = off;     off += al256(sizeof(GridBar));
    L.ysnap = off;  off += 2 * al256((size_t)m * 8);  // this and the next panel's words
    L.total = off;
    return L;
}

size_t elim_workspace(i64 m, i64 n)
{
    const size_t a = elim_layout(m, n).total, b = fused_workspace(m, n), c = elim_tc_workspace(m, n);
    const size_t ab = a > b ? a : b;
    return ab > c ? ab : c;
}

mela_status elim_device(int variant_arg, u64 *M, i64 ld, i64 m, i64 n, int rref, long long *d_rank,
                        long long *d_piv, long long *d_prow, void *ws, size_t ws_bytes,
                        cudaStream_t s, bool resolved)
{
    Tuning tune{};
    const bool chosen = resolved || MELA_VARIANT_BASE(variant_arg) == MELA_ELIM_AUTO;
    if (m > 0 && n > 0) variant_arg = resolve_elim_variant(variant_arg, M, ld, m, n, rref, s);
    if (!decode_elim_variant(variant_arg, &tune)) {
        set_error("elimination: bad variant argument 0x%x", variant_arg);
        return MELA_ERR_INVALID;
    }
    int variant = tune.base;
    if (m == 0 || n == 0) {
        MELA_CUDA_TRY(cudaMemsetAsync(d_rank, 0, sizeof(long long), s));
        return MELA_OK;
    }
    if (m > INT_MAX - 1) {
        set_error("elimination: more than 2^31-2 rows");
        return MELA_ERR_UNSUPPORTED;
    }
    if (variant == MELA_ELIM_FUSED)
        return launch_fused_elim(M, ld, m, n, d_rank, d_piv, d_prow, ws, ws_bytes, s);
    // The Four-Russians form without tuning fields also goes by windows.  Where
    // AUTO picks the windows it leaves the update to the tables up to 40M cells:
    // there the update hides behind the factorization either way, and the
    // tables take fewer and shorter launches (rank 3000 x 5000 372 us, 409 on
    // the tensor cores; RREF 4096 x 8192 603 / 656, 8192 x 8192 1230 / 1183).
    // The windows want a 16-byte aligned workspace, and more of it than the
    // panels: a Four-Russians call that brings less takes panels, and so does
    // AUTO on another alignment.
    const bool aligned = ((uintptr_t)ws & 15) == 0, room = ws_bytes >= elim_tc_workspace(m, n);
    // An RREF of one panel goes by it in either form: a window's launches and
    // fork cost more (Four-Russians form 20 x 20 27 against 37 us a call, 5000 x
    // 64 32 against 38, 50000 x 64 32 against 56; tensor-core form, ones at 0.5
    // and 0.01: 100000 x 64 35 and 41 against 79 and 432, 3000000 x 16 152 and
    // 145 against 1152 and 768; a rank ends with the factorization, 16 us).
    // More rows than the panels take stay with the windows in the tensor-core
    // form.
    const bool one = rref && n <= 64;
    const bool tables = (variant_arg == MELA_ELIM_M4RI && aligned && room && !one) ||
                        (chosen && variant == MELA_ELIM_TC && aligned && (double)m * (double)n <= 4e7);
    if (variant == MELA_ELIM_TC && (aligned ? one && room && m <= 1024ll * 65535 : chosen)) {
        variant = MELA_ELIM_M4RI;
        decode_elim_variant(variant, &tune);
    } else if (variant == MELA_ELIM_TC || tables)
        return elim_windows_device(M, ld, m, n, rref, tables, variant_arg == MELA_ELIM_M4RI, d_rank, d_piv, d_prow, ws,
                                   ws_bytes, s);
    ElimLayout L = elim_layout(m, n);
    if (ws_bytes < L.total || !ws) {
        set_error("elimination workspace of %zu bytes needed, %zu given", elim_workspace(m, n), ws_bytes);
        return MELA_ERR_INVALID;
    }
    unsigned char *w = (unsigned char *)ws;
    unsigned char *state = w + L.state;
    int *stamp = (int *)(w + L.stamp);
    PanelState *ps = (PanelState *)(w + L.ps);
    u64 *rbuf = (u64 *)(w + L.rbuf);
    int *cand = (int *)(w + L.cand);
    GridBar *gb = (GridBar *)(w + L.gb);
    u64 *ysnap[2] = {(u64 *)(w + L.ysnap), (u64 *)(w + L.ysnap + al256((size_t)m * 8))};
    const i64 wc = words_of(n);

    if (variant == MELA_ELIM_PLAIN) {
        MELA_CUDA_TRY(cudaMemsetAsync(state, 1, (size_t)m, s));
        int init[3] = {INT_MAX, INT_MAX, INT_MAX};
        MELA_CUDA_TRY(cudaMemcpyAsync(cand, init, sizeof init, cudaMemcpyHostToDevice, s));
        MELA_CUDA_TRY(cudaMemsetAsync(gb, 0, sizeof(GridBar), s));
        int dev = 0, per_sm = 0;
        MELA_CUDA_TRY(cudaGetDevice(&dev));
        const size_t smem = (size_t)wc * 8;
        if (smem > 200 * 1024) {
            set_error("plain elimination: rows of %lld words exceed the shared-memory pivot buffer", wc);
            return MELA_ERR_UNSUPPORTED;
        }
        MELA_CUDA_TRY(cudaFuncSetAttribute(ge_plain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem));
        MELA_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ge_plain_kernel, 512, smem));
        if (per_sm < 1) {
            set_error("plain elimination kernel cannot be resident");
            return MELA_ERR_UNSUPPORTED;
        }
        i64 blocks = (i64)sm_count();  // one CTA per SM keeps barriers cheap
        const i64 by_rows = (m + 31) / 32;
        if (blocks > by_rows) blocks = by_rows;
        if (blocks < 1) blocks = 1;
        u32 *err = device_error_word();
        long long *rank_out = d_rank;
        void *args[] = {&M, &ld, &m, &n, &rref, &state, &d_piv, &d_prow, &rank_out, &cand, &gb, &err};
        MELA_CUDA_TRY(cudaLaunchCooperativeKernel((void *)ge_plain_kernel, dim3((unsigned)blocks),
                                                  dim3(512), args, smem, s));
        MELA_LAUNCH_CHECK("ge_plain_kernel");
        return MELA_OK;
    }
    if (variant != MELA_ELIM_M4RI && variant != MELA_ELIM_M4RI_K4) {
        set_error("unknown elimination variant %d", variant);
        return MELA_ERR_INVALID;
    }
    const PanelUpdateFn update = panel_update_for(tune.k);
    if (!update) {
        set_error("blocked elimination: M4RI k = %d (4 or 6..10 supported)", tune.k);
        return MELA_ERR_INVALID;
    }
    // Rows per update CTA, unless the variant names them: 256 while those CTAs
    // make at most two waves of three per SM, else 1024.  A CTA's table build
    // is a fixed cost that 256 rows pay back worse, but smaller matrices need
    // the CTAs (rank, k = 8: 2048 x 4096 1150 us with 256 rows, 1385 with 1024;
    // 4096 x 8192 2853 / 3226; 16384 x 32768 35.7 / 28.0 ms).
    const int col_tile = tune.k <= 6 ? 8 : tune.k <= 8 ? 4 : 2;
    auto rows_per_cta = [&](i64 rem) -> int {
        if (tune.row_tile) return tune.row_tile;
        return (rem + col_tile - 1) / col_tile * ((m + 255) / 256) <= 6ll * sm_count() ? 256 : 1024;
    };
    const int rt_min = rows_per_cta(1);
    if (mela_status st = check_grid_yz((m + rt_min - 1) / rt_min, 1, "blocked elimination update"); st != MELA_OK)
        return st;
    if (mela_status st = update(M, ld, m, wc, 0, ps, rbuf, state, stamp, 0, rref, nullptr, nullptr, 0, s, true);
        st != MELA_OK)
        return st;
    panel_init_kernel<<<grid_cap(m, 256), 256, 0, s>>>(M, ld, m, state, stamp, ps, ysnap[0]);
    for (i64 pw = 0; pw < wc; ++pw) {  // every word column is one panel
        const u64 *y = ysnap[pw & 1];
        panel_select_kernel<<<1, SEL_THREADS, 0, s>>>(y, m, n, pw, state, stamp, (int)pw, ps, d_piv, d_prow);
        panel_rows_kernel<<<(unsigned)((wc - pw + 3) / 4), 256, 0, s>>>(M, ld, wc, pw, ps, rbuf);
        update(M, ld, m, wc, pw, ps, rbuf, state, stamp, (int)pw, rref, y, ysnap[(pw + 1) & 1], rows_per_cta(wc - pw), s,
               false);
    }
    MELA_LAUNCH_CHECK("panel elimination");
    MELA_CUDA_TRY(cudaMemcpyAsync(d_rank, &ps->rank, sizeof(long long), cudaMemcpyDeviceToDevice, s));
    return MELA_OK;
}

NullLayout null_layout(i64 n, i64 rank)
{
    NullLayout L{};
    const i64 wc = words_of(n);
    const i64 ldx = even_words(rank > 0 ? rank : 1);
    size_t off = 0;
    L.mask = off;    off += al256((size_t)wc * 8);
    L.before = off;  off += al256((size_t)wc * 8);
    L.mv = off;      off += al256((size_t)wc * 6 * 8);
    // n - rank rows are used; room for n, so that a workspace for some rank
    // also serves every smaller one
    L.x = off;       off += al256((size_t)(n ? n : 1) * (size_t)ldx * 8);
    L.ldx = ldx;
    L.total = off;
    return L;
}

mela_status null_basis_device(const u64 *M, i64 ld, i64 m, i64 n, i64 rank, const long long *d_piv,
                              const long long *d_prow, u64 *Zt, i64 ldz, void *ws, size_t ws_bytes,
                              cudaStream_t s)
{
    (void)m;
    const i64 f = n - rank;
    if (f <= 0) return MELA_OK;
    NullLayout L = null_layout(n, rank);
    if (ws_bytes < L.total || !ws) {
        set_error("null-space workspace of %zu bytes needed, %zu given", L.total, ws_bytes);
        return MELA_ERR_INVALID;
    }
    unsigned char *w = (unsigned char *)ws;
    const NullMeta N{(u64 *)(w + L.mask), (long long *)(w + L.before), (u64 *)(w + L.mv)};
    u64 *X = (u64 *)(w + L.x);
    const i64 wc = words_of(n);
    if (mela_status st = check_grid_yz((rank + 255) / 256, 1, "null basis"); st != MELA_OK) return st;
    null_words_kernel<<<(unsigned)((wc + 7) / 8), 256, 0, s>>>(d_piv, rank, wc, N);
    if (rank > 0)
        null_columns_kernel<<<dim3((unsigned)((wc + 3) / 4), (unsigned)((rank + 255) / 256)), 256, 0, s>>>(
            M, ld, d_prow, rank, n, wc, N, X, L.ldx);
    null_rows_kernel<<<(unsigned)((f + NULL_ROWS - 1) / NULL_ROWS * ((wc + 31) / 32)), dim3(32, 8), 0, s>>>(
        X, L.ldx, N, f, n, wc, Zt, ldz);
    MELA_LAUNCH_CHECK("null basis");
    return MELA_OK;
}

mela_status launch_unpack_rows(const u64 *P, i64 ld, i64 rows, i64 n, unsigned char *out, cudaStream_t s)
{
    if (rows <= 0 || n <= 0) return MELA_OK;
    unpack_rows_kernel<<<grid_cap((rows * n + 15) / 16, 256), 256, 0, s>>>(P, ld, rows, n, out);
    MELA_LAUNCH_CHECK("unpack_rows_kernel");
    return MELA_OK;
}

}  // namespace mela
