// elim_tc.cu -- blocked GF(2) elimination by 256-column windows, the trailing
// (Schur) update on the sm_100a tensor cores or, in the Four-Russians form, by
// tables on the CUDA cores.
//
// Results are those of the other forms (elim.cu): the rank of
// bitrank_packed / rank_m4ri (src/mela_rank_gf2.c:27-121,
// src/mela_rank_m4ri.c:94-279), the greedy pivot columns and the unique RREF
// rows of gf2_rref_standard (src/mela_null_gf2.c:88-131).  Rows never move:
// pivot t lives in physical row prow[t].
//
// One window of 256 columns (4 words) at a time:
//   window_factor   one CTA.  Walks the list of active rows in chunks of up to
//                   320 nonzero ones and brings the window part to reduced row echelon form
//                   (lowest set bit leading), 32 columns at a time.  Every
//                   basis vector carries its combination ("tag") over the rows
//                   P_b that entered the basis, so R_window = tag * A[P, window].
//                   The walk stops as soon as the basis spans every column of
//                   the window.  The walked part of the list is then compacted
//                   in place (pivot rows and rows found zero from the window on
//                   are dropped, order kept).
//   window_near     the next window's words of every other row to update (rank:
//                   the active rows; RREF: all rows), all that the next
//                   factorization reads, by tables over the tags and the P
//                   rows; a row whose bits at the window's pivot columns are
//                   not all zero gets a slot, those bits as a row of 0/1 bytes.
//   window_combine  R_b = sum_j tag[b][j] A[P_j] over the words from the window
//                   on, into the panel buffer (a block per 4 words, 4-bit
//                   tables over the P rows).
//   window_rt       R transposed as 0/1 bytes, Rt8[j][b] = bit j of R_b (the
//                   columns of each 32 in the order the update's epilogue
//                   gathers them), and R_b written over row P_b.
//   tc_update       the other words: A[row(slot)] ^= parity(X8[slot] . Rt8^T): tcgen05
//                   kind::i8 128 x 256 tiles with K = 256.  A persistent CTA
//                   keeps a 256-column strip of Rt8 in shared memory and
//                   streams 128-row tiles of X8 through a 4-stage ring into two
//                   TMEM accumulators; four groups of four epilogue warps XOR
//                   the parity bits into the packed rows while the next tiles
//                   are multiplied, and flag the rows that are still nonzero.
// Since the basis is reduced, a row's coefficient for R_b is its own bit at
// pivot column b, and XORing sum_b x_b R_b clears every pivot column of the
// window; a row whose window part lies in the basis' span (every active row,
// once the scan has ended) is then zero across the window.
#include <algorithm>
#include <climits>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

#include "mela_common.cuh"
#include "mela_internal.h"
#include "mela_host.h"
#include "elim.h"
#include "basis.cuh"
#include "tc_ptx.cuh"

namespace mela {

namespace {

constexpr int WW = 4;         // words per window
constexpr int WBITS = 256;    // columns per window
constexpr int WF_ROWS = 320;     // a chunk of rows; 320 random rows span 256 columns but with probability 2^-64
// Warps 3, 7, 11 share one scheduler: warp 3 selects, the other two only help
// with the tables; the rest hold the rows, a thread each.
constexpr int WF_WARPS = WF_ROWS / 32 + 3;
constexpr int WF_THREADS = 32 * WF_WARPS;
constexpr int WF_SELECTOR = 3;
constexpr int WF_SPARSE = 32;  // set bits up to which a row is reduced bit by bit
static_assert(WF_ROWS == 320, "ten row warps on three schedulers");

// Everything that belongs to a pivot of a window is indexed by its column in
// the window (0..255), so the coefficient of a row is its window part masked
// by `have`.
struct WinState {
    long long rank;         // pivots so far (every window)
    int rt;                 // pivots of the current window
    int nu;                 // rows to update in the current window
    int na;                 // rows in the active-row list
    int lbase;              // the list is list[lbase .. lbase + na)
    u64 have[WW];           // pivot columns of the window
    int prow[WBITS];        // physical row P_b of pivot column b (-1: none)
    alignas(16) u64 tag[WBITS][WW];  // R_b = sum_j bit j * A[P_j]
};

struct WfSmem {
    uint4 basis[WBITS][2];    // vector of pivot column b (in-place form)
    uint4 tab[2][64][16];     // 4-bit tables of the basis, a plane per 16-byte half
    uint4 vt[2][8][16];       // 4-bit tables of a round's pivot rows
    uint4 cv[kHalfCand][2];   // the candidates' vectors
    HalfRound r;
    uint4 vrow[WF_ROWS][2];   // the chunk being gathered: vectors
    int grow[WF_ROWS];        //   and rows
    int cut;                  // first row of the block that did not fit
    int prow[WBITS];          // physical row of pivot column b
    int cnt;
    int wcnt[2][32];          // candidates per warp, alternating
    int wsum[32];
};

// Half word h of an 8-word vector held in registers (selects, no local memory).
__device__ __forceinline__ u32 sel8(const u32 (&v)[8], int h)
{
    const u32 a = (h & 1) ? v[1] : v[0], b = (h & 1) ? v[3] : v[2];
    const u32 c = (h & 1) ? v[5] : v[4], d = (h & 1) ? v[7] : v[6];
    const u32 e = (h & 2) ? b : a, f = (h & 2) ? d : c;
    return (h & 4) ? f : e;
}
__device__ __forceinline__ void xor8(u32 (&v)[8], const uint4 &a, const uint4 &b)
{
    v[0] ^= a.x;
    v[1] ^= a.y;
    v[2] ^= a.z;
    v[3] ^= a.w;
    v[4] ^= b.x;
    v[5] ^= b.y;
    v[6] ^= b.z;
    v[7] ^= b.w;
}
__device__ __forceinline__ uint4 xor4u(const uint4 &a, const uint4 &b)
{
    return make_uint4(a.x ^ b.x, a.y ^ b.y, a.z ^ b.z, a.w ^ b.w);
}


// Exclusive position of this thread's flag among the block's flags (thread
// order) and the block total; every thread of the block must call it.
__device__ __forceinline__ int block_slot(bool flag, int *wsum, int &total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned bal = __ballot_sync(0xffffffffu, flag);
    if (lane == 0) wsum[warp] = __popc(bal);
    __syncthreads();
    if (warp == 0) {
        int v = lane < (int)(blockDim.x >> 5) ? wsum[lane] : 0;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, off);
            if (lane >= off) v += u;
        }
        wsum[lane] = v;
    }
    __syncthreads();
    total = wsum[31];
    const int slot = (warp ? wsum[warp - 1] : 0) + __popc(bal & ((1u << lane) - 1));
    __syncthreads();  // wsum may be rewritten by the next call
    return slot;
}

}  // namespace

// ---------------------------------------------------------------- window_factor
namespace {

// A row's vector v after a round with pivot columns C of half word h: its
// bits y at C select sum_k y_k T_k = z, the combination of the round's
// original pivot rows to add; z itself takes the place of the bits at C.
__device__ __forceinline__ void wf_apply(const WfSmem &S, u32 (&v)[8], int h, u32 C, u32 z)
{
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] &= q == h ? ~C : ~0u;
#pragma unroll
    for (int g = 0; g < 8; ++g) {
        const int e = (int)((z >> (4 * g)) & 15);
        xor8(v, S.vt[0][g][e], S.vt[1][g][e]);
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] |= q == h ? z : 0u;
}
// Half word ht of what wf_apply makes of v.
__device__ __forceinline__ u32 wf_half(const WfSmem &S, const u32 (&v)[8], int h, int ht, u32 C, u32 z)
{
    u32 x = sel8(v, ht);
    if (z) {
        if (ht == h) x &= ~C;
        const u32 *t = reinterpret_cast<const u32 *>(&S.vt[ht >> 2][0][0]) + (ht & 3);
#pragma unroll
        for (int g = 0; g < 8; ++g) x ^= t[4 * (16 * g + ((z >> (4 * g)) & 15))];
        if (ht == h) x |= z;
    }
    return x;
}

}  // namespace

// Blocked Gauss-Jordan of the window, in place: a row is 256 bits, which at
// the pivot columns found so far hold its combination over the pivot rows P_b
// and elsewhere its data (a row with bit c set gets v ^= v_p without bit c, so
// its bit c stays set and becomes the coefficient of P_c).  One CTA walks the
// active rows in chunks of a row per thread, leaving out the rows that are zero
// modulo the basis so far (most rows of a sparse matrix; few-bit rows are reduced
// bit by bit, others through tables); the columns go 32 at a time (half words): up to 64 rows with data left there are eliminated by one warp
// (half_word_select), and every row of the chunk then takes the round's pivots
// in through 4-bit tables; rounds repeat until no unused row has data left in
// the half word.  Where a round fills its half word, the rows first bring only
// the next half word up to date, so that the next round's selection runs in a
// warp of its own beside the rest of the row updates.
// Bound by the serial chain, not by throughput (one CTA): a round of up to 32
// pivots costs about 2600 cycles in half_word_select, four barriers, the
// tables and one half word of every row: about 29 us for a full window, against
// 133 us when the rows are eliminated one pivot and one barrier at a time
// (rank of a 2000 x 4100 parity-check matrix 637 us, 976 with the zero rows in
// the chunks).
__global__ void __launch_bounds__(WF_THREADS, 1)
window_factor_kernel(const u64 *__restrict__ M, i64 ld, i64 m, i64 n, i64 w, int *list, const unsigned char *live,
                     unsigned char *state, int *stamp, int wid, const WinState *prev, WinState *ws, long long *piv,
                     long long *prow, long long *rank)
{
    extern __shared__ __align__(16) unsigned char wf_raw[];
    WfSmem &S = *reinterpret_cast<WfSmem *>(wf_raw);
    constexpr int NW = WF_ROWS / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool holds = (warp & 3) != 3;            // this warp holds rows:
    const int rw = holds ? warp - (warp >> 2) : NW;  // 32 rw .. of the chunk
    const int ri = 32 * rw + lane;
    const i64 wc = words_of(n);
    const int wn = (wc - w) < WW ? (int)(wc - w) : WW;
    const i64 vb = n - 64 * w;
    const int valid = vb < WBITS ? (int)vb : WBITS;  // columns of this window inside the matrix
    const int na = prev->na;
    if (na == 0) {  // every row is a pivot or zero: nothing in any later window
        if (tid == 0) {
            ws->rt = 0;
            ws->na = 0;
            ws->rank = prev->rank;
        }
        return;
    }
    int *L0 = list + prev->lbase;

    u32 H[8] = {};  // pivot columns so far (the same in every thread)
    int nb = 0;     // their number
    int walked = 0, par = 0, chunks = 0;
    while (walked < na && nb < valid) {
        const bool older = nb > 0;  // basis vectors of earlier chunks
        u32 H0[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) H0[q] = H[q];
        const bool obasis = older && holds && ri < WBITS && ((sel8(H0, (ri >> 5) & 7) >> (ri & 31)) & 1);
        if (older) {
            // tables of the 16 combinations of basis vectors 4g..4g+3
            for (int e = tid; e < 2 * 64 * 16; e += WF_THREADS) {
                const int half = e >> 10, g = (e >> 4) & 63, v = e & 15;
                uint4 a = make_uint4(0, 0, 0, 0);
#pragma unroll
                for (int b = 0; b < 4; ++b)
                    if (((v >> b) & 1) && ((sel8(H0, g >> 3) >> ((4 * g + b) & 31)) & 1))
                        a = xor4u(a, S.basis[4 * g + b][half]);
                S.tab[half][g][v] = a;
            }
            __syncthreads();
        }
        // the next rows that are not zero modulo the basis, from blocks of
        // WF_ROWS list entries, until there are enough of them to span the
        // columns that are left: more with each chunk of the window, as the rows
        // of a sparse matrix depend on one another.  (Always WF_ROWS of them
        // walked all of a tall sparse matrix for its last columns: rank of
        // 1000000 x 64 of density 0.001 3.46 ms, 0.17 this way, 100000 x 200 of
        // 0.01 216 and 70 us; fewer from the start cost sparse square matrices
        // chunks: 8192 x 1024 of 0.003 480 us with half of this, 376.)
        const int goal = min(WF_ROWS, (4 << min(chunks, 6)) * (valid - nb) + 8);
        ++chunks;
        int row = -1, filled = 0;
        u32 v[8] = {};
        auto words_of_row = [&](int r, u32 (&x)[8]) {
#pragma unroll
            for (int q = 0; q < WW; ++q) {
                const u64 t = r >= 0 && q < wn ? M[(i64)r * ld + w + q] : 0ull;
                x[2 * q] = (u32)t;
                x[2 * q + 1] = (u32)(t >> 32);
            }
        };
        int kr = holds && walked + ri < na ? L0[walked + ri] : -1;
        u32 x[8];
        words_of_row(kr, x);
        for (;;) {
            const int next = walked + WF_ROWS + ri, kn = holds && next < na ? L0[next] : -1;
            if (older) {
                u32 y[8];
                int bits = 0;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    y[q] = x[q] & H0[q];
                    x[q] &= ~H0[q];
                    bits += __popc(y[q]);
                }
                if (__reduce_max_sync(0xffffffffu, bits) <= WF_SPARSE) {  // (sparse rows: 64 table steps for a few bits)
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        for (u32 c = y[q]; c; c &= c - 1) {
                            const uint4 *u = S.basis[32 * q + __ffs((int)c) - 1];
                            xor8(x, u[0], u[1]);
                        }
                } else {
#pragma unroll
                    for (int g = 0; g < 64; ++g) {
                        const int e = (int)((y[g >> 3] >> (4 * (g & 7))) & 15);
                        if (e) xor8(x, S.tab[0][g][e], S.tab[1][g][e]);
                    }
                }
            }
            u32 any = 0;
#pragma unroll
            for (int q = 0; q < 8; ++q) any |= x[q] & ~H0[q];
            const unsigned bal = __ballot_sync(0xffffffffu, any != 0);
            par ^= 1;
            if (holds && lane == 0) S.wcnt[par][rw] = __popc(bal);
            const int total = __syncthreads_count(any != 0);
            const bool last = walked + WF_ROWS >= na;
            if (filled == 0 && (last || total >= goal || 4 * total >= 3 * WF_ROWS)) {
                // the block as it is: filling it up would not save a chunk
                row = kr;
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] = x[q];
                walked = last ? na : walked + WF_ROWS;
                filled = total;
                break;
            }
            u32 xn[8];  // on their way while this block is written out
            words_of_row(kn, xn);
            const int wv = lane < rw && lane < NW ? S.wcnt[par][lane] : 0;
            const int idx = filled + __reduce_add_sync(0xffffffffu, wv) + __popc(bal & ((1u << lane) - 1));
            if (any && idx < WF_ROWS) {
                S.vrow[idx][0] = make_uint4(x[0], x[1], x[2], x[3]);
                S.vrow[idx][1] = make_uint4(x[4], x[5], x[6], x[7]);
                S.grow[idx] = kr;
            }
            if (any && idx == WF_ROWS) S.cut = ri;
            __syncthreads();
            const bool over = filled + total > WF_ROWS;
            walked = over ? walked + S.cut : last ? na : walked + WF_ROWS;
            filled = over ? WF_ROWS : filled + total;
            if (filled >= goal || walked >= na) {
                if (ri < filled) {
                    const uint4 a = S.vrow[ri][0], b = S.vrow[ri][1];
                    v[0] = a.x;
                    v[1] = a.y;
                    v[2] = a.z;
                    v[3] = a.w;
                    v[4] = b.x;
                    v[5] = b.y;
                    v[6] = b.z;
                    v[7] = b.w;
                    row = S.grow[ri];
                }
                break;
            }
            kr = kn;
#pragma unroll
            for (int q = 0; q < 8; ++q) x[q] = xn[q];
        }
        if (filled == 0) break;  // only rows inside the span were left
        int mycol = -1;  // this row's pivot column
        // the last round, while its pivots are not in v yet: half word h,
        // columns C, combination z of this row
        bool pend = false;
        int h = 0;
        u32 C = 0, z = 0;
        auto take_in = [&]() {
            if (z) wf_apply(S, v, h, C, z);
            if (obasis) {
                const uint4 a = S.basis[ri][0], b = S.basis[ri][1];
                u32 o[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
                const u32 y = sel8(o, h) & C;
                if (y) {
                    wf_apply(S, o, h, C, half_word_times_T(S.r, y));
                    S.basis[ri][0] = make_uint4(o[0], o[1], o[2], o[3]);
                    S.basis[ri][1] = make_uint4(o[4], o[5], o[6], o[7]);
                }
            }
        };
        while (h < 8 && nb < valid) {
            int ht = h;  // the half word of the next round
            if (pend && sel8(H, h) == 0xffffffffu && ++ht == 8) break;
            const u32 Ht = sel8(H, ht);
            u32 d = 0;
            unsigned bal = 0;
            par ^= 1;
            if (holds) {
                if (mycol < 0) d = (pend ? wf_half(S, v, h, ht, C, z) : sel8(v, ht)) & ~Ht;
                bal = __ballot_sync(0xffffffffu, d != 0);
                if (lane == 0) S.wcnt[par][rw] = __popc(bal);
            }
            __syncthreads();
            const int wv = lane < NW ? S.wcnt[par][lane] : 0;
            const int total = __reduce_add_sync(0xffffffffu, wv);
            if (total == 0) {  // no unused row has data left in half word ht
                if (pend && holds) take_in();
                pend = false;
                h = ht + 1;
                continue;
            }
            int idx = __reduce_add_sync(0xffffffffu, lane < rw ? wv : 0) + __popc(bal & ((1u << lane) - 1));
            if (d == 0 || idx >= kHalfCand) idx = -1;
            if (idx >= 0) {
                S.r.cand[idx] = d;
                S.r.pcol[idx] = -1;
            }
            __syncthreads();
            if (warp == WF_SELECTOR) {
                half_word_select(S.r, total < kHalfCand ? total : kHalfCand);
            } else if (holds) {
                if (pend) take_in();
                if (idx >= 0) {
                    S.cv[idx][0] = make_uint4(v[0], v[1], v[2], v[3]);
                    S.cv[idx][1] = make_uint4(v[4], v[5], v[6], v[7]);
                }
            }
            __syncthreads();
            C = S.r.C;
            // tables over the round's pivots: their original rows (without
            // the bits at C) and the rows of T
            if (holds && ri < 256) {
                const int half = ri >> 7, g = (ri >> 4) & 7, e = ri & 15;
                uint4 a = make_uint4(0, 0, 0, 0);
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const int ci = S.r.ci[4 * g + b];
                    if (((e >> b) & 1) && ci >= 0) a = xor4u(a, S.cv[ci][half]);
                }
                if (half == (ht >> 2)) {
                    const int q = ht & 3;
                    a.x &= q == 0 ? ~C : ~0u;
                    a.y &= q == 1 ? ~C : ~0u;
                    a.z &= q == 2 ? ~C : ~0u;
                    a.w &= q == 3 ? ~C : ~0u;
                }
                S.vt[half][g][e] = a;
            }
            if (!holds)
                for (int e = 32 * (warp >> 2) + lane; e < 128; e += 96) half_word_tt(S.r, e);
            const int pc = idx >= 0 ? S.r.pcol[idx] : -1;
            __syncthreads();
            if (pc >= 0) {
                mycol = 32 * ht + pc;
                S.prow[mycol] = row;
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] = 0;
                z = S.r.T[pc];
            } else {
                const u32 y = sel8(v, ht) & C;
                z = y ? half_word_times_T(S.r, y) : 0u;
            }
            pend = true;
            h = ht;
            nb += __popc(C);
#pragma unroll
            for (int q = 0; q < 8; ++q) H[q] |= q == ht ? C : 0u;
        }
        if (pend && holds) take_in();
        if (mycol >= 0) {
            S.basis[mycol][0] = make_uint4(v[0], v[1], v[2], v[3]);
            S.basis[mycol][1] = make_uint4(v[4], v[5], v[6], v[7]);
        }
        __syncthreads();
    }

    // results, by column; pivot t of the window is its t-th pivot column
    const long long r0 = prev->rank;
    if (tid < WBITS) {
        const u32 hq = sel8(H, tid >> 5);
        int r = -1;
        if ((hq >> (tid & 31)) & 1) {
            int t = __popc(hq & ((1u << (tid & 31)) - 1));
#pragma unroll
            for (int q = 0; q < 8; ++q) t += q < (tid >> 5) ? __popc(H[q]) : 0;
            const uint4 a = S.basis[tid][0], b = S.basis[tid][1];
            ws->tag[tid][0] = (u64)(a.x & H[0]) | ((u64)(a.y & H[1]) << 32);
            ws->tag[tid][1] = (u64)(a.z & H[2]) | ((u64)(a.w & H[3]) << 32);
            ws->tag[tid][2] = (u64)(b.x & H[4]) | ((u64)(b.y & H[5]) << 32);
            ws->tag[tid][3] = (u64)(b.z & H[6]) | ((u64)(b.w & H[7]) << 32);
            r = S.prow[tid];
            piv[r0 + t] = 64 * w + tid;
            prow[r0 + t] = r;
            state[r] = 0;
            stamp[r] = wid;
        }
        ws->prow[tid] = r;
    }
    if (tid < WW) {
        const u32 a = tid == 0 ? H[0] : tid == 1 ? H[2] : tid == 2 ? H[4] : H[6];
        const u32 b = tid == 0 ? H[1] : tid == 1 ? H[3] : tid == 2 ? H[5] : H[7];
        ws->have[tid] = (u64)a | ((u64)b << 32);
    }
    if (tid == 0) S.cnt = walked;
    __syncthreads();
    // compact the walked part [0, walked) of the list to its right end, in
    // order, dropping this window's pivot rows and rows known to be zero from
    // the window on; chunks go from the last to the first, so every write lands
    // at or after the chunk being read
    for (int c0 = ((walked - 1) / WF_ROWS) * WF_ROWS; walked > 0 && c0 >= 0; c0 -= WF_ROWS) {
        const int k = c0 + tid;
        int row = -1;
        if (tid < WF_ROWS && k < walked) row = L0[k];
        const bool keep = row >= 0 && state[row] && live[row];
        int total;
        const int slot = block_slot(keep, S.wsum, total);
        const int wpos = S.cnt - total;
        if (keep) L0[wpos + slot] = row;
        __syncthreads();
        if (tid == 0) S.cnt = wpos;
        __syncthreads();
    }
    if (tid == 0) {
        ws->rt = nb;
        ws->nu = 0;
        ws->lbase = prev->lbase + S.cnt;  // S.cnt = entries dropped
        ws->na = na - S.cnt;
        ws->rank = r0 + nb;
        *rank = r0 + nb;
    }
}

// ---------------------------------------------------------------- window_combine
// Block: CB_W words x every pivot.  R_b = XOR_j tag[b][j] A[P_j] is evaluated
// four columns j at a time from 64 tables of the 16 combinations of the pivot
// rows of columns 4g..4g+3 (restricted to the block's words).
namespace {
constexpr int CB_W = 4;
struct CbSmem {
    u64 tab[64][16][CB_W];  // 32 KB
    u64 rows[WBITS][CB_W];  // the P rows' words
    u64 tag[WBITS][WW];
};
}

__global__ void __launch_bounds__(256)
window_combine_kernel(const u64 *__restrict__ M, i64 ld, i64 wc, i64 w, const WinState *ws,
                      u64 *__restrict__ Rbuf, i64 ldr)
{
    extern __shared__ __align__(16) unsigned char cb_raw[];
    CbSmem &S = *reinterpret_cast<CbSmem *>(cb_raw);
    if (ws->rt == 0) return;
    const int tid = threadIdx.x;
    const i64 w0 = w + (i64)blockIdx.x * CB_W;
    {
        const int j = tid;  // 256 threads: a column each
        const int pr = ws->prow[j];
        u64 v[CB_W];
        if (pr >= 0) {
            const u64 *src = M + (i64)pr * ld + w0;
#pragma unroll
            for (int q = 0; q < CB_W; ++q) v[q] = (w0 + q < wc) ? src[q] : 0ull;
        } else {
#pragma unroll
            for (int q = 0; q < CB_W; ++q) v[q] = 0;
        }
#pragma unroll
        for (int q = 0; q < CB_W; ++q) S.rows[j][q] = v[q];
#pragma unroll
        for (int q = 0; q < WW; ++q) S.tag[j][q] = pr >= 0 ? ws->tag[j][q] : 0ull;
    }
    __syncthreads();
    for (int e = tid; e < 64 * 16; e += 256) {
        const int g = e >> 4, v = e & 15;
        u64 a[CB_W] = {};
#pragma unroll
        for (int h = 0; h < 4; ++h)
            if ((v >> h) & 1) {
#pragma unroll
                for (int q = 0; q < CB_W; ++q) a[q] ^= S.rows[4 * g + h][q];
            }
#pragma unroll
        for (int q = 0; q < CB_W; ++q) S.tab[g][v][q] = a[q];
    }
    __syncthreads();
    // thread: word q = tid % CB_W, columns b = tid / CB_W + 64 i (zero where
    // there is no pivot)
    const int q = tid % CB_W;
    for (int b = tid / CB_W; b < WBITS; b += 256 / CB_W) {
        u64 acc = 0;
#pragma unroll
        for (int qq = 0; qq < WW; ++qq) {
            const u64 tg = S.tag[b][qq];
#pragma unroll
            for (int g = 0; g < 16; ++g) acc ^= S.tab[16 * qq + g][(tg >> (4 * g)) & 15][q];
        }
        if (w0 + q < wc) Rbuf[(i64)b * ldr + (w0 + q - w)] = acc;
    }
}

// 4 bits -> 4 bytes of 0/1.
__device__ __forceinline__ u32 nib_bytes(u32 v) { return ((v & 15u) * 0x00204081u) & 0x01010101u; }

// ---------------------------------------------------------------- window_near
namespace {
struct NrSmem {
    uint4 tag[2][16][64];   // 4-bit tables of the tags, entry-major: [16-byte half][entry][group]
    uint4 prow[2][16][64];  // the same of the pivot rows' words of the next window
    int cnt[8];
    int base;
};

// Half words 0..7 in a group of 8 lanes, one a lane -> nibble s of half word k
// in bits 4k .. 4k + 3 (s: the lane's place in its group).
__device__ __forceinline__ u32 gather_nibbles(u32 v, int lane)
{
    const int s = lane & 7;
    u32 r = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k)
        r |= ((__shfl_sync(0xffffffffu, v, (lane & 24) + k) >> (4 * s)) & 15u) << (4 * k);
    return r;
}
// XOR over a group of 8 lanes of an 8-word vector, word s left in lane s.
__device__ __forceinline__ u32 xor_scatter(const u32 (&a)[8], int lane)
{
    u32 b[4], c[2];
    const bool h4 = lane & 4, h2 = lane & 2, h1 = lane & 1;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const u32 send = h4 ? a[i] : a[4 + i], keep = h4 ? a[4 + i] : a[i];
        b[i] = keep ^ __shfl_xor_sync(0xffffffffu, send, 4);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const u32 send = h2 ? b[i] : b[2 + i], keep = h2 ? b[2 + i] : b[i];
        c[i] = keep ^ __shfl_xor_sync(0xffffffffu, send, 2);
    }
    return (h1 ? c[1] : c[0]) ^ __shfl_xor_sync(0xffffffffu, h1 ? c[0] : c[1], 1);
}
// sum over the lane's groups s, s + 8, .. of table entries, XORed over the 8
// lanes: the lanes of a row read 8 different 16-byte bank groups.
__device__ __forceinline__ u32 near_lookup(const uint4 (&t)[2][16][64], u32 nib, int lane)
{
    u32 a[8] = {};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int e = (int)((nib >> (4 * k)) & 15), g = (lane & 7) + 8 * k;
        xor8(a, t[0][e][g], t[1][e][g]);
    }
    return xor_scatter(a, lane);
}
}  // namespace

// The next window's words of every row to update (rank: the active rows;
// RREF: every row but this window's pivots), which is all that the next
// factorization reads, and the coefficients of the tensor-core update.  A
// group of 8 lanes per row, a half word each: the row's bits y at the window's
// pivot columns give z = sum_b y_b tag[b], the combination of the original
// pivot rows, and the words change by sum_j z_j A[P_j] -- 64 table reads each,
// without waiting for the reduced rows R.  Rows with y != 0 get a slot of
// ulist and their coefficients in X8 (256 0/1 bytes, or the 32 bytes of y as
// they are, for table_update); live says whether the
// row's words of the next window are nonzero (the update adds the others).
// Latency-bound: about 2 us of table building and dependent loads, then
// 1000 cycles per 32 rows.  It takes the place, on the critical path, of the
// combine, transpose and one-strip tensor-core launches (15 us a window):
// rank of 3000 x 5000 (rank 2200) 422 against 516 us, 8192 x 8192 1.22 ms.
__global__ void __launch_bounds__(256)
window_near_kernel(u64 *__restrict__ M, i64 ld, i64 m, i64 wc, i64 w, const int *__restrict__ list, const int *stamp,
                   int wid, int rref, WinState *ws, int *ulist, unsigned char *X8, int bytes, unsigned char *live)
{
    extern __shared__ __align__(16) unsigned char nr_raw[];
    NrSmem &S = *reinterpret_cast<NrSmem *>(nr_raw);
    if (ws->rt == 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, s = lane & 7;
    {
        // a thread per (table, 16-byte half, group): its 16 entries in Gray-code order
        const int half = (tid >> 6) & 1, g = tid & 63;
        const i64 pw = w + WW + 2 * half;
        uint4 v[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int pr = ws->prow[4 * g + b];
            v[b] = make_uint4(0, 0, 0, 0);
            if (pr >= 0 && tid < 128) v[b] = reinterpret_cast<const uint4 *>(ws->tag[4 * g + b])[half];
            if (pr >= 0 && tid >= 128) {
                const u64 *src = M + (i64)pr * ld + pw;
                const u64 x0 = pw < wc ? src[0] : 0ull, x1 = pw + 1 < wc ? src[1] : 0ull;
                v[b] = make_uint4((u32)x0, (u32)(x0 >> 32), (u32)x1, (u32)(x1 >> 32));
            }
        }
        uint4 *T = tid < 128 ? &S.tag[half][0][g] : &S.prow[half][0][g];
        uint4 a = make_uint4(0, 0, 0, 0);
        T[0] = a;
#pragma unroll
        for (int i = 1; i < 16; ++i) {
            a = xor4u(a, v[(i & 1) ? 0 : (i & 2) ? 1 : (i & 4) ? 2 : 3]);
            T[(i ^ (i >> 1)) * 64] = a;
        }
    }
    const u32 have = reinterpret_cast<const u32 *>(ws->have)[s];
    const i64 cnt = rref ? m : (i64)ws->na;
    list += ws->lbase;
    __syncthreads();
    for (i64 i0 = (i64)blockIdx.x * 32; i0 < cnt; i0 += (i64)gridDim.x * 32) {
        const i64 idx = i0 + (tid >> 3);
        i64 row = -1;
        if (idx < cnt) {
            row = rref ? idx : (i64)list[idx];
            if (rref && stamp[row] == wid) row = -1;
        }
        u32 *p = reinterpret_cast<u32 *>(M + row * ld + w) + s;
        const bool in_y = row >= 0 && w + (s >> 1) < wc, in_v = row >= 0 && w + WW + (s >> 1) < wc;
        const u32 y = in_y ? p[0] & have : 0u;
        u32 v = in_v ? p[2 * WW] : 0u;
        const unsigned nzl = __ballot_sync(0xffffffffu, y != 0);
        const unsigned nz4 = ((nzl & 0xffu) != 0) | ((nzl & 0xff00u) != 0) << 1 | ((nzl & 0xff0000u) != 0) << 2 |
                             ((nzl & 0xff000000u) != 0) << 3;  // the warp's four rows
        if (lane == 0) S.cnt[warp] = __popc(nz4);
        __syncthreads();
        if (tid == 0) {
            int t = 0;
#pragma unroll
            for (int q = 0; q < 8; ++q) t += S.cnt[q];
            S.base = t ? atomicAdd(&ws->nu, t) : 0;
        }
        const bool nz = (nz4 >> (lane >> 3)) & 1;
        if (nz4) {
            const u32 z = near_lookup(S.tag, gather_nibbles(y, lane), lane);
            v ^= near_lookup(S.prow, gather_nibbles(z, lane), lane);
            if (nz && in_v) p[2 * WW] = v;
            const unsigned vl = __ballot_sync(0xffffffffu, in_v && v != 0);
            if (nz && s == 0) live[row] = ((vl >> (lane & 24)) & 0xffu) != 0;
        }
        __syncthreads();
        if (nz) {
            int slot = S.base + __popc(nz4 & ((1u << (lane >> 3)) - 1));
#pragma unroll
            for (int q = 0; q < 8; ++q) slot += q < warp ? S.cnt[q] : 0;
            if (s == 0) ulist[slot] = (int)row;
            if (bytes) {
                uint4 *dst = reinterpret_cast<uint4 *>(X8 + (size_t)slot * WBITS + 32 * s);
                dst[0] = make_uint4(nib_bytes(y), nib_bytes(y >> 4), nib_bytes(y >> 8), nib_bytes(y >> 12));
                dst[1] = make_uint4(nib_bytes(y >> 16), nib_bytes(y >> 20), nib_bytes(y >> 24), nib_bytes(y >> 28));
            } else {
                reinterpret_cast<u32 *>(X8)[(size_t)slot * 8 + s] = y;
            }
        }
        __syncthreads();  // cnt and base are read before the next rows write them
    }
}

// The parity bits of 32 columns from 16 registers of column pairs (low 16 bits
// of columns 2i and 2i + 1): columns 2i in bits 0..15, 2i + 1 in bits 16..31.
__device__ __forceinline__ u32 parity_pairs(const u32 *r)
{
    u32 b = r[0] & 0x00010001u;
#pragma unroll
    for (int i = 1; i < 16; ++i) b |= (r[i] << i) & (0x00010001u << i);
    return b;
}
// Place of column bit b of a 32-column group in the strip, so that
// parity_pairs leaves it in bit b.
__device__ __forceinline__ int pair_place(int b) { return b < 16 ? 2 * b : 2 * (b - 16) + 1; }

// ---------------------------------------------------------------- window_rt
// Block W (word w + W): Rt8 rows 64W..64W+63 (in pair_place order) and word
// w + W of every row P_b.
__global__ void __launch_bounds__(256)
window_rt_kernel(u64 *__restrict__ M, i64 ld, i64 w, const u64 *__restrict__ Rbuf, i64 ldr, const WinState *ws,
                 unsigned char *Rt8)
{
    __shared__ u64 col[WBITS];
    if (ws->rt == 0) return;
    const int tid = threadIdx.x;
    const i64 W = blockIdx.x;
    const u64 v = Rbuf[(i64)tid * ldr + W];  // zero where the column has no pivot
    col[tid] = v;
    const int pr = ws->prow[tid];
    if (pr >= 0) M[(i64)pr * ld + w + W] = v;
    __syncthreads();
    for (int e = tid; e < 64 * 16; e += 256) {
        const int jl = e >> 4, c = e & 15;
        u32 o[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            u32 x = 0;
#pragma unroll
            for (int b = 0; b < 4; ++b) x |= (u32)((col[16 * c + 4 * r + b] >> jl) & 1) << (8 * b);
            o[r] = x;
        }
        const int place = (jl & 32) + pair_place(jl & 31);
        *reinterpret_cast<uint4 *>(Rt8 + ((size_t)(W * 64 + place)) * WBITS + 16 * c) =
            make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// ---------------------------------------------------------------- tc_update
namespace {
constexpr int UM = 128, UN = 256;             // output tile
constexpr int UBOX = 128;                     // K bytes per TMA box (128-byte swizzle)
constexpr int UA_BOX = UM * UBOX;             // 16 KB
constexpr int UB_BOX = UN * UBOX;             // 32 KB
constexpr int UA_BYTES = 2 * UA_BOX;          // K = 256
constexpr int UB_BYTES = 2 * UB_BOX;
constexpr int U_STAGES = 4;                   // X8 tiles in flight
constexpr int U_BSTAGES = 1;                  // Rt8 strips in shared memory
constexpr int U_GROUPS = 4;                   // epilogue groups, tile t to group t % 4
constexpr int U_STAGE_BYTES = U_GROUPS * UM * 4 * 8;  // per group, 128 rows x 4 words
constexpr int U_SMEM = U_BSTAGES * UB_BYTES + U_STAGES * UA_BYTES + U_STAGE_BYTES + 1024 + 256;
constexpr int U_MCH = 8;                      // row tiles per work unit (far part)
constexpr int U_EPI_THREADS = 128;           // a group: one warp per TMEM lane quarter
constexpr int U_THREADS = 64 + U_GROUPS * U_EPI_THREADS;

struct UCtl {
    u64 bfull[U_BSTAGES], bempty[U_BSTAGES];
    u64 afull[U_STAGES], aempty[U_STAGES];
    u64 accfull[U_GROUPS], accempty[2];
    u64 drain;
    u32 tmem;
    int abort;
};

}  // namespace

// Bound by the matrix instructions (M = 128 kind::i8 reads 12 KB of shared
// memory an instruction: 87 us of the 100 us that a launch over 16384 rows x
// 32256 columns takes without any epilogue work).  Before, 134 us: the parity
// bits one by one (two logical operations an element against one for a pair
// of columns read together), and each epilogue warp waiting for the row
// numbers of its own tile.
__global__ void __launch_bounds__(U_THREADS, 1)
tc_update_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmR,
                 u64 *__restrict__ M, i64 ld, i64 wc, i64 w, const WinState *ws, const int *__restrict__ ulist,
                 unsigned char *live, int strip_lo, int strip_hi, int skip, int mch, u32 *err)
{
    // strips strip_lo .. strip_hi-1 (256 columns each, from the window's first
    // column) except strip `skip` (-1: none); work units of mch row tiles
    const int rt = ws->rt, nu = ws->nu;
    if (rt == 0 || nu == 0) return;
    const i64 lw = wc - w;
    const int s_end = (int)((lw + 3) / 4) < strip_hi ? (int)((lw + 3) / 4) : strip_hi;
    const int strips = s_end - strip_lo - (skip >= strip_lo && skip < s_end ? 1 : 0);
    if (strips <= 0) return;
    auto strip_of = [&](long long vs) -> int {
        const int st = strip_lo + (int)vs;
        return (skip >= 0 && st >= skip) ? st + 1 : st;
    };
    const int mt = (nu + UM - 1) / UM;
    const int chunks = (mt + mch - 1) / mch;
    const long long units = (long long)strips * chunks;
    const long long ub = units * blockIdx.x / gridDim.x, ue = units * (blockIdx.x + 1) / gridDim.x;
    if (ub >= ue) return;

    extern __shared__ unsigned char u_raw[];
    unsigned char *smem =
        reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(u_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char *sB = smem;
    unsigned char *sA = smem + U_BSTAGES * UB_BYTES;
    u64 *stage = reinterpret_cast<u64 *>(sA + U_STAGES * UA_BYTES);  // [group][UM][4]
    UCtl *ctl = reinterpret_cast<UCtl *>(sA + U_STAGES * UA_BYTES + U_STAGE_BYTES);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < U_BSTAGES; ++s) {
            ptx::mbar_init(&ctl->bfull[s], 1);
            ptx::mbar_init(&ctl->bempty[s], 1);
        }
        for (int s = 0; s < U_STAGES; ++s) {
            ptx::mbar_init(&ctl->afull[s], 1);
            ptx::mbar_init(&ctl->aempty[s], 1);
        }
        for (int q = 0; q < U_GROUPS; ++q) ptx::mbar_init(&ctl->accfull[q], 1);
        for (int a = 0; a < 2; ++a) ptx::mbar_init(&ctl->accempty[a], U_EPI_THREADS);
        ptx::mbar_init(&ctl->drain, 1);
        ctl->abort = 0;
        ptx::fence_barrier_init();
    }
    if (warp == 0 && lane == 0) {
        ptx::prefetch_tmap(&tmX);
        ptx::prefetch_tmap(&tmR);
    }
    if (warp == 1) {
        ptx::tmem_alloc(&ctl->tmem, 512);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const u32 tmem = ctl->tmem;
    volatile int *abort_flag = &ctl->abort;

    if (warp == 0) {
        if (lane == 0) {
            // strip loads (nbl) and tile loads (it) in the order the MMA warp consumes them
            int nbl = 0, it = 0, prev_strip = -1;
            int last_a[U_STAGES], last_b[U_BSTAGES];
#pragma unroll
            for (int q = 0; q < U_STAGES; ++q) last_a[q] = -1;
#pragma unroll
            for (int q = 0; q < U_BSTAGES; ++q) last_b[q] = -1;
            bool ok = true;
            for (long long u = ub; u < ue && ok; ++u) {
                const int strip = strip_of(u / chunks), chunk = (int)(u % chunks);
                if (strip != prev_strip) {
                    const int bs = nbl % U_BSTAGES;
                    if (nbl >= U_BSTAGES && !ptx::mbar_wait(&ctl->bempty[bs], ((nbl / U_BSTAGES) - 1) & 1, err)) {
                        ok = false;
                        break;
                    }
                    if (*abort_flag) {
                        ok = false;
                        break;
                    }
                    unsigned char *b = sB + bs * UB_BYTES;
                    ptx::mbar_arrive_expect_tx(&ctl->bfull[bs], UB_BYTES);
                    ptx::tma_load_2d(b, &tmR, &ctl->bfull[bs], 0, strip * UN);
                    ptx::tma_load_2d(b + UB_BOX, &tmR, &ctl->bfull[bs], UBOX, strip * UN);
                    last_b[bs] = nbl / U_BSTAGES;
                    ++nbl;
                    prev_strip = strip;
                }
                const int t1 = (chunk + 1) * mch < mt ? (chunk + 1) * mch : mt;
                for (int tile = chunk * mch; tile < t1; ++tile, ++it) {
                    const int s = it % U_STAGES;
                    if (it >= U_STAGES && !ptx::mbar_wait(&ctl->aempty[s], ((it / U_STAGES) - 1) & 1, err)) {
                        ok = false;
                        break;
                    }
                    if (*abort_flag) {
                        ok = false;
                        break;
                    }
                    unsigned char *a = sA + s * UA_BYTES;
                    ptx::mbar_arrive_expect_tx(&ctl->afull[s], UA_BYTES);
                    ptx::tma_load_2d(a, &tmX, &ctl->afull[s], 0, tile * UM);
                    ptx::tma_load_2d(a + UA_BOX, &tmX, &ctl->afull[s], UBOX, tile * UM);
                    last_a[s] = it / U_STAGES;
                }
            }
            if (!ok) {
                *abort_flag = 1;
                // let every issued copy land before the CTA's shared memory goes away
                for (int s = 0; s < U_BSTAGES; ++s)
                    if (last_b[s] >= 0) ptx::mbar_wait(&ctl->bfull[s], last_b[s] & 1, nullptr);
                for (int s = 0; s < U_STAGES; ++s)
                    if (last_a[s] >= 0) ptx::mbar_wait(&ctl->afull[s], last_a[s] & 1, nullptr);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr u32 idesc = ptx::idesc_i8(UM, UN);
            int nbl = 0, it = 0, prev_strip = -1, bs = 0;
            bool ok = true;
            for (long long u = ub; u < ue && ok; ++u) {
                const int strip = strip_of(u / chunks), chunk = (int)(u % chunks);
                if (strip != prev_strip) {
                    bs = nbl % U_BSTAGES;
                    if (!ptx::mbar_wait(&ctl->bfull[bs], (nbl / U_BSTAGES) & 1, err) || *abort_flag) {
                        ok = false;
                        break;
                    }
                    ++nbl;
                    prev_strip = strip;
                }
                const u32 b0 = ptx::smem_u32(sB + bs * UB_BYTES);
                const int t1 = (chunk + 1) * mch < mt ? (chunk + 1) * mch : mt;
                for (int tile = chunk * mch; tile < t1; ++tile, ++it) {
                    const int s = it % U_STAGES, acc = it & 1;
                    if (!ptx::mbar_wait(&ctl->afull[s], (it / U_STAGES) & 1, err) ||
                        (it >= 2 && !ptx::mbar_wait(&ctl->accempty[acc], ((it >> 1) - 1) & 1, err)) ||
                        *abort_flag) {
                        ok = false;
                        break;
                    }
                    ptx::tc_fence_after();
                    const u32 a0 = ptx::smem_u32(sA + s * UA_BYTES);
                    const u32 d = tmem + (u32)(acc * UN);
#pragma unroll
                    for (int kb = 0; kb < 2; ++kb)
#pragma unroll
                        for (int kk = 0; kk < UBOX / 32; ++kk)
                            ptx::umma_i8(d, ptx::desc_k_sw128(a0 + kb * UA_BOX + kk * 32),
                                         ptx::desc_k_sw128(b0 + kb * UB_BOX + kk * 32), idesc, (kb | kk) != 0);
                    ptx::umma_commit(&ctl->aempty[s]);
                    ptx::umma_commit(&ctl->accfull[it % U_GROUPS]);
                }
                if (!ok) break;
                // the strip's buffer is free once this unit's products are done
                const bool next_same = (u + 1 < ue) && (strip_of((u + 1) / chunks) == strip);
                if (!next_same) ptx::umma_commit(&ctl->bempty[bs]);
            }
            if (!ok) {
                *abort_flag = 1;
                ptx::umma_commit(&ctl->drain);
                ptx::mbar_wait(&ctl->drain, 0, nullptr);
            }
        }
        __syncwarp();
    } else {
        // Four groups of four warps take the tiles in turn, a warp per TMEM
        // lane quarter (32 rows): a group has four tiles' time for the memory
        // latencies of its own.  A tile's packed parity words go through
        // shared memory, within the warp, so that the read-modify-write of the
        // rows is done with 32 contiguous bytes per row (4 lanes a row, 8 rows a
        // warp instruction).  The rows' numbers are fetched a tile ahead of
        // their words, and the words before the previous tile is drained.
        const int ew = warp & 3;          // TMEM lane quarter of this warp
        const int g = (warp - 2) >> 2;    // group: tiles 4k + g of the CTA
        const int r8 = lane >> 2, q = lane & 3;  // item c: row r8 + 8c of the quarter, word q
        u64 *wstage = stage + (size_t)(g * UM + ew * 32) * 4;
        int k = 0;  // own tiles so far
        bool ok = true;
        // previous own tile
        i64 p_w = 0;
        int p_row[4] = {-1, -1, -1, -1};
        u64 p_old[4] = {0, 0, 0, 0};
        bool p_in = false;
        auto drain_and_write = [&]() -> bool {
            const bool good = !*abort_flag && ptx::mbar_wait(&ctl->accfull[g], (k - 1) & 1, err);
            if (!good) {
                *abort_flag = 1;
                return false;
            }
            ptx::tc_fence_after();
            const u32 tbase = tmem + ((u32)(ew * 32) << 16) + (u32)((g & 1) * UN);
            u32 pb[8];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                u32 r[32];
                ptx::tmem_ld_32x32b_x32_pack16(tbase + 64 * h, r);
                ptx::tmem_ld_wait();
                pb[2 * h] = parity_pairs(r);
                pb[2 * h + 1] = parity_pairs(r + 16);
            }
            ptx::tc_fence_before();
            ptx::mbar_arrive(&ctl->accempty[g & 1]);
            __syncwarp();  // the previous tile's words have been read
            uint4 *st = reinterpret_cast<uint4 *>(wstage + 4 * lane);
            st[0] = make_uint4(pb[0], pb[1], pb[2], pb[3]);
            st[1] = make_uint4(pb[4], pb[5], pb[6], pb[7]);
            __syncwarp();
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                u64 v = 0;
                if (p_row[c] >= 0 && p_in) {
                    v = p_old[c] ^ wstage[lane + 32 * c];
                    M[(i64)p_row[c] * ld + p_w] = v;
                }
                // one flag per row: the four lanes of a row combine their words
                const unsigned nz = __ballot_sync(0xffffffffu, v != 0);
                if (q == 0 && p_row[c] >= 0 && ((nz >> (4 * r8)) & 15u)) live[p_row[c]] = 1;
            }
            return true;
        };
        // the CTA's tiles in order
        long long at = ub;
        int vs = (int)(ub / chunks), chunk = (int)(ub % chunks), tile = chunk * mch;
        auto step = [&]() {
            if (++tile < mt && tile < (chunk + 1) * mch) return;
            ++at;
            if (++chunk == chunks) {
                chunk = 0;
                ++vs;
            }
            tile = chunk * mch;
        };
        auto rows_of = [&](int (&row)[4]) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int slot = tile * UM + 32 * ew + r8 + 8 * c;
                row[c] = at < ue && slot < nu ? ulist[slot] : -1;
            }
        };
        int n_row[4];  // rows of the next own tile
        for (int i = 0; i < g && at < ue; ++i) step();
        rows_of(n_row);
        while (at < ue && ok) {
            const i64 pw = w + (i64)strip_of(vs) * 4 + q;
            const bool in = pw < wc;
            const int row[4] = {n_row[0], n_row[1], n_row[2], n_row[3]};
            u64 old[4] = {0, 0, 0, 0};
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (row[c] >= 0 && in) old[c] = M[(i64)row[c] * ld + pw];
            for (int i = 0; i < U_GROUPS && at < ue; ++i) step();
            rows_of(n_row);
            if (k > 0 && !drain_and_write()) ok = false;
            ++k;
            p_w = pw;
            p_in = in;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                p_row[c] = row[c];
                p_old[c] = old[c];
            }
        }
        if (ok && k > 0 && !drain_and_write()) ok = false;
        if (!ok) *abort_flag = 1;
    }

    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem, 512);
    }
}

// ---------------------------------------------------------------- table_update
// The update of the words that window_near leaves, on the CUDA cores (the
// Four-Russians form): strip q is words w + 4q .. w + 4q + 3.  A CTA builds the
// 4-bit tables of the reduced rows' words of its strip (32 KB) and takes every
// gridDim.y-th group of 32 listed rows, 8 lanes a row and a half word each as
// in window_near: 64 conflict-free table reads a row.  For the RREF the CTAs of
// the first row group also write the reduced rows over the pivot rows, in
// strip `skip` (whose listed rows window_near has done) nothing else.
// Bound by the shared-memory reads, 4 cycles a row word and SM, where the
// matrix is large; up to 4096 x 8192 it hides behind the next factorization
// and costs the window fewer launches than the tensor cores (rank of 2048 x
// 4096, rank 1800: 308 us, 331 on the tensor cores, 1074 in 64-column panels;
// 16384 x 32768, rank 12000: 7.8, 5.5 and 27.9 ms).
namespace {
struct TuSmem {
    uint4 t[2][16][64];
};
}  // namespace

__global__ void __launch_bounds__(256)
table_update_kernel(u64 *__restrict__ M, i64 ld, i64 wc, i64 w, const WinState *ws, const u64 *__restrict__ Rbuf,
                    i64 ldr, const int *__restrict__ ulist, const u32 *__restrict__ Y, unsigned char *live,
                    int strip_lo, int skip, int rref)
{
    extern __shared__ __align__(16) unsigned char tu_raw[];
    TuSmem &S = *reinterpret_cast<TuSmem *>(tu_raw);
    if (ws->rt == 0) return;
    const int nu = ws->nu;
    const int strip = strip_lo + (int)blockIdx.x;
    if (strip == skip && blockIdx.y > 0) return;
    const i64 w0 = 4 * (i64)strip;            // from the window's first word
    const int tid = threadIdx.x, lane = tid & 31, s = lane & 7;
    const int nwords = wc - w - w0 < 4 ? (int)(wc - w - w0) : 4;
    if (tid < 128) {
        const int half = tid >> 6, g = tid & 63;
        uint4 v[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const u64 *src = Rbuf + (i64)(4 * g + b) * ldr + w0 + 2 * half;
            const u64 x0 = 2 * half < nwords ? src[0] : 0ull, x1 = 2 * half + 1 < nwords ? src[1] : 0ull;
            v[b] = make_uint4((u32)x0, (u32)(x0 >> 32), (u32)x1, (u32)(x1 >> 32));
        }
        uint4 a = make_uint4(0, 0, 0, 0);
        S.t[half][0][g] = a;
#pragma unroll
        for (int i = 1; i < 16; ++i) {
            a = xor4u(a, v[(i & 1) ? 0 : (i & 2) ? 1 : (i & 4) ? 2 : 3]);
            S.t[half][i ^ (i >> 1)][g] = a;
        }
    }
    __syncthreads();
    const bool in = (s >> 1) < nwords;
    if (rref && blockIdx.y == 0) {
        for (int b = tid >> 3; b < WBITS; b += 32) {
            const int pr = ws->prow[b];
            if (pr >= 0 && in)
                reinterpret_cast<u32 *>(M + (i64)pr * ld + w + w0)[s] =
                    reinterpret_cast<const u32 *>(Rbuf + (i64)b * ldr + w0)[s];
        }
    }
    if (strip == skip) return;  // its listed rows are up to date (window_near)
    for (int i0 = 32 * (int)blockIdx.y; i0 < nu; i0 += 32 * (int)gridDim.y) {
        const int slot = i0 + (tid >> 3);
        const bool ok = slot < nu;
        const int row = ok ? ulist[slot] : 0;
        const u32 y = ok ? Y[(size_t)slot * 8 + s] : 0u;
        u32 *p = reinterpret_cast<u32 *>(M + (i64)row * ld + w + w0) + s;
        u32 v = ok && in ? *p : 0u;
        v ^= near_lookup(S.t, gather_nibbles(y, lane), lane);
        if (ok && in) *p = v;
        const unsigned vl = __ballot_sync(0xffffffffu, ok && in && v != 0);
        if (ok && s == 0 && ((vl >> (lane & 24)) & 0xffu)) live[row] = 1;
    }
}

// ---------------------------------------------------------------- host side
static size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

// The state before the first window: every row active, possibly nonzero and
// in the list, in order; no pivots.
__global__ void window_init_kernel(i64 m, int *list, unsigned char *state, int *stamp, unsigned char *live0,
                                   unsigned char *live1, WinState *prev, long long *rank)
{
    for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < m; i += (i64)gridDim.x * blockDim.x) {
        list[i] = (int)i;
        state[i] = 1;
        stamp[i] = -1;
        live0[i] = 1;
        live1[i] = 1;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        prev->rank = 0;
        prev->rt = 0;
        prev->nu = 0;
        prev->na = (int)m;
        prev->lbase = 0;
        *rank = 0;
    }
}

static int grid_for(i64 total)
{
    i64 g = (total + 255) / 256;
    const i64 cap = (i64)sm_count() * 8;
    return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

namespace {
struct TcLayout {
    size_t state, stamp, live, ws, ulist, list, x8, rt8, rbuf, total;
    i64 mpad, npad;
};

TcLayout tc_layout(i64 m, i64 n)
{
    TcLayout L{};
    const i64 wc = words_of(n);
    L.mpad = (m + UM - 1) / UM * UM;
    L.npad = (64 * wc + UN - 1) / UN * UN;
    size_t off = 0;
    L.state = off;  off += al256((size_t)m);
    L.stamp = off;  off += al256((size_t)m * 4);
    L.live = off;   off += 2 * al256((size_t)m);          // one flag array per window parity
    L.ws = off;     off += 2 * al256(sizeof(WinState));   // one state per window parity
    L.ulist = off;  off += al256((size_t)m * 4);
    L.list = off;   off += al256((size_t)m * 4);
    L.x8 = off;     off += al256((size_t)L.mpad * WBITS);
    L.rt8 = off;    off += al256((size_t)L.npad * WBITS);
    L.rbuf = off;   off += al256((size_t)WBITS * (size_t)wc * 8);
    L.total = off;
    return L;
}
}  // namespace

size_t elim_tc_workspace(i64 m, i64 n) { return tc_layout(m, n).total; }

namespace {
// Captured eliminations, kept for the life of the process (at most
// kMaxElimGraphs of calls that name the Four-Russians form and as many of the
// others, so that neither keeps the other from being captured; further shapes
// or buffers run without a graph).
struct ElimGraphKey {
    int dev;
    const void *p[5];
    long long v[4];
};
struct ElimGraph {
    ElimGraphKey k;
    cudaGraphExec_t exec;
};
constexpr long long kElimTables = 2, kElimNamed = 4;  // bits of v[3]: update by tables, form named by the caller
constexpr size_t kMaxElimGraphs = 16;
constexpr size_t kMaxElimSeen = 64;
std::mutex g_elim_graph_mu;
struct ElimGraphs {
    std::vector<ElimGraph> kept;
    std::vector<ElimGraphKey> seen;  // calls made once, without a graph
    size_t seen_next = 0;            // the oldest entry, replaced once the list is full
};
ElimGraphs *g_elim_graphs[2] = {};
// of a call's kind (under g_elim_graph_mu)
ElimGraphs &elim_graphs(const ElimGraphKey &k)
{
    ElimGraphs *&g = g_elim_graphs[(k.v[3] & kElimNamed) != 0];
    if (!g) g = new ElimGraphs();
    return *g;
}

bool elim_graphs_enabled()
{
    const char *e = std::getenv("MELA_ELIM_GRAPH");
    return !(e && e[0] == '0');
}
cudaGraphExec_t elim_graph_lookup(const ElimGraphKey &k)
{
    if (!elim_graphs_enabled()) return nullptr;
    std::lock_guard<std::mutex> lk(g_elim_graph_mu);
    for (const ElimGraph &g : elim_graphs(k).kept)
        if (std::memcmp(&g.k, &k, sizeof k) == 0) return g.exec;
    return nullptr;
}
// Capture now: the same call (device, buffers, shape, form) was made before
// -- a one-off call does not pay for instantiating a graph --, the stream is
// not being captured by the caller and there is room to keep one more graph.
bool elim_graph_capturable(const ElimGraphKey &k, cudaStream_t s)
{
    if (!elim_graphs_enabled()) return false;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return false;
    }
    std::lock_guard<std::mutex> lk(g_elim_graph_mu);
    ElimGraphs &G = elim_graphs(k);
    if (G.kept.size() >= kMaxElimGraphs) return false;
    for (const ElimGraphKey &q : G.seen)
        if (std::memcmp(&q, &k, sizeof k) == 0) return true;
    // remember the call; a full list forgets its oldest entry, so a stream of
    // one-off shapes never keeps a repeated call from being captured
    if (G.seen.size() < kMaxElimSeen) {
        G.seen.push_back(k);
    } else {
        G.seen[G.seen_next] = k;
        G.seen_next = (G.seen_next + 1) % kMaxElimSeen;
    }
    return false;
}
void elim_graph_store(const ElimGraphKey &k, cudaGraphExec_t exec)
{
    std::lock_guard<std::mutex> lk(g_elim_graph_mu);
    elim_graphs(k).kept.push_back(ElimGraph{k, exec});
}
}  // namespace

mela_status elim_windows_device(u64 *M, i64 ld, i64 m, i64 n, int rref, bool tables, bool named, long long *d_rank,
                                long long *d_piv, long long *d_prow, void *wsp, size_t ws_bytes, cudaStream_t s)
{
    const TcLayout L = tc_layout(m, n);
    if (!wsp || ws_bytes < L.total) {
        set_error("elimination workspace of %zu bytes needed, %zu given", L.total, ws_bytes);
        return MELA_ERR_INVALID;
    }
    if (L.mpad / UM > INT_MAX / 2 || L.npad > ((i64)1 << 31)) {
        set_error("tensor-core elimination: matrix too large");
        return MELA_ERR_UNSUPPORTED;
    }
    unsigned char *b = (unsigned char *)wsp;
    unsigned char *state = b + L.state;
    int *stamp = (int *)(b + L.stamp);
    WinState *wsv[2] = {(WinState *)(b + L.ws), (WinState *)(b + L.ws + al256(sizeof(WinState)))};
    int *ulist = (int *)(b + L.ulist);
    unsigned char *X8 = b + L.x8;
    unsigned char *Rt8 = b + L.rt8;
    u64 *Rbuf = (u64 *)(b + L.rbuf);
    int *list = (int *)(b + L.list);
    unsigned char *livev[2] = {b + L.live, b + L.live + al256((size_t)m)};
    const i64 wc = words_of(n);

    CUtensorMap mx, mr;
    mela_status st = make_u8_kmajor_map(&mx, X8, L.mpad, WBITS, UM);
    if (st != MELA_OK) return st;
    st = make_u8_kmajor_map(&mr, Rt8, L.npad, WBITS, UN);
    if (st != MELA_OK) return st;
    cudaStream_t s2;
    if ((st = side_stream(&s2)) != MELA_OK) return st;

    const size_t wf_smem = sizeof(WfSmem);
    MELA_CUDA_TRY(cudaFuncSetAttribute(window_factor_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)wf_smem));
    MELA_CUDA_TRY(cudaFuncSetAttribute(tc_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, U_SMEM));
    const int cb_smem = (int)sizeof(CbSmem);
    MELA_CUDA_TRY(cudaFuncSetAttribute(window_combine_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, cb_smem));
    const int sms = sm_count();
    const int tu_smem = (int)sizeof(TuSmem);
    MELA_CUDA_TRY(cudaFuncSetAttribute(table_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, tu_smem));
    const int nr_smem = (int)sizeof(NrSmem);
    MELA_CUDA_TRY(cudaFuncSetAttribute(window_near_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, nr_smem));
    const int near_blocks = (int)std::min<i64>((m + 31) / 32, 2 * sms);
    const i64 tiles_max = L.mpad / UM, chunks_max = (tiles_max + U_MCH - 1) / U_MCH;
    u32 *err = device_error_word();

    // Look-ahead: window_near brings window w + 1's columns of every row up to
    // date, so the next factorization follows it at once; the reduced rows and
    // the update of the other columns are forked to the side stream and run
    // beside it (on SMs the fork leaves free).  window_near of window w + 1
    // waits for them: it reads the pivot rows' later words, and the coefficient
    // and R buffers are the ones the update still reads.  Window states and row
    // flags alternate by window parity so that the factorization of w + 1 never
    // writes what the update of w reads.
    cudaEvent_t evs[2] = {};
    for (int i = 0; i < 2; ++i) {
        if (cudaEventCreateWithFlags(&evs[i], cudaEventDisableTiming) != cudaSuccess) {
            for (int j = 0; j < i; ++j) cudaEventDestroy(evs[j]);
            set_error("cudaEventCreate failed");
            return MELA_ERR_CUDA;
        }
    }
    cudaEvent_t ev_fork = evs[0], ev_join = evs[1];
    cudaStream_t sx = s;  // the stream the launches go to (a capture stream while capturing)
    auto run = [&]() -> mela_status {
        window_init_kernel<<<grid_for(m), 256, 0, sx>>>(m, list, state, stamp, livev[0], livev[1], wsv[1], d_rank);
        bool forked = false;
        int wid = 0;
        for (i64 w = 0; w < wc; w += WW, ++wid) {
            const i64 lw = wc - w;
            WinState *cur = wsv[wid & 1], *prev = wsv[(wid + 1) & 1];
            unsigned char *live = livev[wid & 1];  // flags of window wid-2 (complete); then this window's
            window_factor_kernel<<<1, WF_THREADS, wf_smem, sx>>>(M, ld, m, n, w, list, live, state, stamp, wid, prev,
                                                                cur, d_piv, d_prow, d_rank);
            if (forked) {
                MELA_CUDA_TRY(cudaStreamWaitEvent(sx, ev_join, 0));
                forked = false;
            }
            if (!rref && w + WW >= wc) break;  // a rank: no column is left to update
            window_near_kernel<<<near_blocks, 256, nr_smem, sx>>>(M, ld, m, wc, w, list, stamp, wid, rref, cur, ulist,
                                                                 X8, tables ? 0 : 1, live);
            MELA_CUDA_TRY(cudaEventRecord(ev_fork, sx));
            MELA_CUDA_TRY(cudaStreamWaitEvent(s2, ev_fork, 0));
            window_combine_kernel<<<(unsigned)((lw + CB_W - 1) / CB_W), 256, cb_smem, s2>>>(M, ld, wc, w, cur, Rbuf,
                                                                                           wc);
            if (!tables) window_rt_kernel<<<(unsigned)lw, 256, 0, s2>>>(M, ld, w, Rbuf, wc, cur, Rt8);
            // strips 2.. and, for the RREF, strip 0 (the window's own columns;
            // for the rank every updated row is in the window basis' span and
            // its window part becomes zero)
            const i64 strips = (lw + 3) / 4;
            const int far_lo = rref ? 0 : 2, far_skip = (rref && strips >= 2) ? 1 : -1;
            const i64 far_strips = (strips > far_lo ? strips - far_lo : 0) - (far_skip >= 0 ? 1 : 0);
            if (tables) {
                const i64 all = strips > far_lo ? strips - far_lo : 0;
                if (all > 0) {
                    const i64 groups = (m + 31) / 32, want = (4 * sms + all - 1) / all;
                    table_update_kernel<<<dim3((unsigned)all, (unsigned)(groups < want ? groups : want)), 256, tu_smem,
                                          s2>>>(M, ld, wc, w, cur, Rbuf, wc, ulist, (const u32 *)X8, live, far_lo,
                                                far_skip, rref);
                }
            } else if (far_strips > 0) {
                const i64 units = far_strips * chunks_max;
                const int cap = sms > 4 ? sms - 2 : sms;  // SMs left for the next factorization
                const int grid_far = (int)(units < cap ? units : cap);
                tc_update_kernel<<<grid_far, U_THREADS, U_SMEM, s2>>>(mx, mr, M, ld, wc, w, cur, ulist, live, far_lo,
                                                                     (int)strips, far_skip, U_MCH, err);
            }
            MELA_CUDA_TRY(cudaEventRecord(ev_join, s2));
            forked = true;
        }
        if (forked) MELA_CUDA_TRY(cudaStreamWaitEvent(sx, ev_join, 0));
        MELA_LAUNCH_CHECK("tensor-core elimination");
        return MELA_OK;
    };
    // The launch sequence depends only on the shape and the buffers, so from
    // the second call on it is captured once into a CUDA graph per (device,
    // buffers, shape, form), on the thread's capture stream, and replayed on
    // the caller's stream: about
    // 1.4 ms less per 16384 x 32768 call than launching the 770 kernels and
    // events one by one.  A caller that is itself capturing gets the launches
    // in its own graph.
    ElimGraphKey key;
    std::memset(&key, 0, sizeof key);
    cudaGetDevice(&key.dev);
    key.p[0] = M;
    key.p[1] = d_rank;
    key.p[2] = d_piv;
    key.p[3] = d_prow;
    key.p[4] = wsp;
    key.v[0] = ld;
    key.v[1] = m;
    key.v[2] = n;
    key.v[3] = rref + (tables ? kElimTables : 0) + (named ? kElimNamed : 0);
    cudaGraphExec_t exec = elim_graph_lookup(key);
    cudaStream_t cap = nullptr;
    if (exec) {
        st = cudaGraphLaunch(exec, s) == cudaSuccess ? MELA_OK : MELA_ERR_CUDA;
        if (st != MELA_OK) set_error("cudaGraphLaunch (tensor-core elimination) failed");
    } else if (elim_graph_capturable(key, s) && capture_stream(&cap) == MELA_OK) {
        st = MELA_OK;
        if (cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
            cudaGetLastError();
            st = run();
        } else {
            sx = cap;
            const mela_status bst = run();
            sx = s;
            cudaGraph_t g = nullptr;
            const cudaError_t ee = cudaStreamEndCapture(cap, &g);
            cudaGraphExec_t ex = nullptr;
            if (bst == MELA_OK && ee == cudaSuccess && g && cudaGraphInstantiate(&ex, g, 0) == cudaSuccess) {
                elim_graph_store(key, ex);
                st = cudaGraphLaunch(ex, s) == cudaSuccess ? MELA_OK : MELA_ERR_CUDA;
                if (st != MELA_OK) set_error("cudaGraphLaunch (tensor-core elimination) failed");
            } else {
                cudaGetLastError();
                st = bst != MELA_OK ? bst : run();  // not capturable here: launch directly
            }
            if (g) cudaGraphDestroy(g);
        }
    } else {
        st = run();
    }
    for (cudaEvent_t e : evs) cudaEventDestroy(e);
    return st;
}

}  // namespace mela
