// basis.cuh -- Gauss-Jordan elimination of a few rows over a 32-column half
// word by one warp: the pivot search of the blocked eliminations (elim.cu,
// elim_tc.cu) and of small matrices (elim_small.cu), and the tables of a round's
// pivots, which the batch engine's selection (batch.cu) also uses.
//
// Rows are kept in in-place form: at the pivot columns found so far a row
// holds its combination over the pivot rows (bit c: contains the original row
// of pivot column c), elsewhere its data.  Eliminating with pivot row p of
// column c is v ^= v_p without bit c for every other row with bit c set, whose
// bit c thereby turns from data into the coefficient of that pivot row.
#pragma once

#include "mela_common.cuh"

namespace mela {

__device__ __forceinline__ int ctz64_(u64 x) { return __ffsll((long long)x) - 1; }

constexpr int kHalfCand = 64;  // rows one selection round eliminates among themselves

// One round's shared state.
struct HalfRound {
    u32 tt[8][16];         // 4-bit tables of T
    u32 cand[kHalfCand];   // the candidates' data bits in the half word
    u32 T[32];             // row of T of the pivot in column c of the half word
    int ci[32];            // its candidate (-1: no pivot)
    int pcol[kHalfCand];   // column of a candidate's pivot (-1: none)
    u32 C;                 // the round's pivot columns
};

// Gauss-Jordan of the first ncand candidates by one warp, columns in lanes:
// lane c's mask (bit r = row r, two registers) holds column c.  A step
// broadcasts column c, takes its lowest unused row p as the pivot and, in
// every other lane whose column has bit p, XORs in the rows that hold bit c.
// Lane c's own mask is left alone: it becomes column c of the combinations.
// Column c + 1 is fetched while the step before it runs and brought up to
// date in registers, so a step's chain has no shuffle latency; selects, no
// branches (64 cycles a step against 115 with a branch on the own column).
__device__ __forceinline__ void half_word_select(HalfRound &S, int ncand)
{
    const int lane = threadIdx.x & 31;
    u32 lo = transpose32_warp(lane < ncand ? S.cand[lane] : 0u);
    u32 hi = transpose32_warp(lane + 32 < ncand ? S.cand[lane + 32] : 0u);
    u32 ulo = ~0u, uhi = ~0u;    // unused rows
    u32 mlo = 0, mhi = 0;        // this column's pivot row
    u32 xlo, xhi;                // the step's column
    auto step = [&](int c, int next) {
        const u32 nlo = __shfl_sync(0xffffffffu, lo, next);
        const u32 nhi = __shfl_sync(0xffffffffu, hi, next);
        const u32 alo = xlo & ulo, ahi = xhi & uhi;
        const u32 plo = alo & (0u - alo), phi = alo ? 0u : ahi & (0u - ahi);
        const u32 rlo = xlo ^ plo, rhi = xhi ^ phi;
        ulo ^= plo;
        uhi ^= phi;
        const bool own = lane == c;
        mlo = own ? plo : mlo;
        mhi = own ? phi : mhi;
        const bool hit = ((lo & plo) | (hi & phi)) != 0 && !own;
        lo ^= hit ? rlo : 0u;
        hi ^= hit ? rhi : 0u;
        const bool nhit = ((nlo & plo) | (nhi & phi)) != 0;
        xlo = nhit ? nlo ^ rlo : nlo;
        xhi = nhit ? nhi ^ rhi : nhi;
    };
    xlo = __shfl_sync(0xffffffffu, lo, 0);
    xhi = __shfl_sync(0xffffffffu, hi, 0);
#pragma unroll
    for (int c = 0; c < 32; ++c) step(c, (c + 1) & 31);
    const u32 C = __ballot_sync(0xffffffffu, (mlo | mhi) != 0);
    const u32 wlo = transpose32_warp(lo), whi = transpose32_warp(hi);
    const int ci = mlo ? __ffs(mlo) - 1 : mhi ? 31 + __ffs(mhi) : -1;
    const u32 t0 = __shfl_sync(0xffffffffu, wlo, ci & 31), t1 = __shfl_sync(0xffffffffu, whi, ci & 31);
    S.T[lane] = ci < 0 ? 0u : ((ci < 32 ? t0 : t1) & C);
    S.ci[lane] = ci;
    if (ci >= 0) S.pcol[ci] = lane;
    if (lane == 0) S.C = C;
}

// Entry x = 16 g + e of the tables of T.
__device__ __forceinline__ void half_word_tt(HalfRound &S, int x)
{
    const int g = x >> 4, e = x & 15;
    u32 a = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b) a ^= ((e >> b) & 1) ? S.T[4 * g + b] : 0u;
    S.tt[g][e] = a;
}
// sum_k y_k T_k: the combination of the round's original pivot rows that
// clears the bits y at its pivot columns.
__device__ __forceinline__ u32 half_word_times_T(const HalfRound &S, u32 y)
{
    u32 z = 0;
#pragma unroll
    for (int g = 0; g < 8; ++g) z ^= S.tt[g][(y >> (4 * g)) & 15];
    return z;
}

}  // namespace mela
