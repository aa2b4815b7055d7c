// pack.cu -- data-format kernels on the path into and out of the GF(2) kernels.
//
//  * rand_dense   seeded Bernoulli(1/2) packed matrices (counter-based
//                 splitmix64, identical bits to the CPU generator)
//  * pack         MATLAB column-major logical / double -> packed rows
//                 (reference: pack_rows_logical / pack_rows_double,
//                 src/mela_matmul_gf2.c:42-69; inline packs in
//                 src/mela_rank_gf2.c:154-176, src/mela_null_gf2.c:169-187)
//  * unpack       packed rows -> column-major logical bytes
//                 (reference: src/mela_matmul_gf2.c:193-205)
//  * transpose    64x64 bit-block transpose with warp ballots
//  * expand       packed bits -> 0/1 bytes or e2m1 pairs (operands of the
//                 tensor-core GEMM, B transposed on the way)
//
// All of these are HBM-bound byte/word moves: each thread reads and writes
// whole words or bytes with warp-contiguous addresses; no GEMM reshaping.
#include "mela_common.cuh"
#include "mela_internal.h"

namespace mela {

// ---------------------------------------------------------------- generator
__host__ __device__ __forceinline__ u64 mix64(u64 z)
{
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}

u64 stream_key(u64 seed, u64 stream)
{
    return mix64(seed * 0x9E3779B97F4A7C15ULL + 0x632BE59BD9B4E019ULL) ^
           mix64(stream + 0xD1B54A32D192ED03ULL);
}

__global__ void rand_dense_kernel(u64 key, i64 m, i64 n, i64 wc, u64 *out, i64 ld)
{
    const u64 tail = (n & 63) ? ((1ULL << (n & 63)) - 1) : ~0ULL;
    i64 total = m * ld;
    for (i64 t = blockIdx.x * (i64)blockDim.x + threadIdx.x; t < total;
         t += (i64)gridDim.x * blockDim.x) {
        i64 i = t / ld, w = t - i * ld;
        u64 v = 0;
        if (w < wc) {
            v = mix64(key + (u64)(i * wc + w + 1) * 0x9E3779B97F4A7C15ULL);
            if (w == wc - 1) v &= tail;
        }
        out[t] = v;
    }
}

// Bernoulli(density) bits: entry e = i*n + j takes 16-bit slice e%4 of word
// e/4 of the stream and is 1 when the slice is below `thresh` (density*65536).
__global__ void rand_bernoulli_kernel(u64 key, i64 m, i64 n, unsigned thresh, u64 *out, i64 ld)
{
    const i64 wc = words_of(n);
    const i64 total = m * ld;
    for (i64 t = blockIdx.x * (i64)blockDim.x + threadIdx.x; t < total; t += (i64)gridDim.x * blockDim.x) {
        const i64 i = t / ld, w = t - i * ld;
        u64 v = 0;
        if (w < wc) {
            const int cols = (n - 64 * w) < 64 ? (int)(n - 64 * w) : 64;
            for (int b = 0; b < cols; ++b) {
                const i64 e = i * n + 64 * w + b;
                const u64 word = mix64(key + (u64)(e / 4 + 1) * 0x9E3779B97F4A7C15ULL);
                const unsigned sl = (unsigned)(word >> (16 * (e & 3))) & 0xFFFFu;
                if (sl < thresh) v |= 1ull << b;
            }
        }
        out[t] = v;
    }
}

// ---------------------------------------------------------------- pack
// Parity of a double as the reference reads it, ((int)x) & 1, with the
// x86-64 result for NaN and out-of-range values (INT_MIN, even) spelled out.
__device__ __forceinline__ u32 parity_of(double x)
{
    if (!(x >= -2147483648.0 && x < 2147483648.0)) return 0;
    return (u32)__double2int_rz(x) & 1u;
}
__device__ __forceinline__ u32 parity_of(unsigned char x) { return x != 0; }

// Doubles.  Block: 32 rows x 4 output words, a warp per word, a lane per row:
// each load instruction reads 32 consecutive rows of one column.  The 64
// columns of a word are fetched 16 at a time, all in flight together: the
// kernel is bound by the latency of its loads until the array passes a few tens
// of MB (a 2048 x 512 block, 8.4 MB: 3.1 us against 7.9 us with the loads one
// after the other; 8192 x 8192 80.9 us = 6.6 TB/s).
__global__ void __launch_bounds__(128) pack_double_kernel(const double *__restrict__ in, i64 m, i64 n,
                                                          u64 *__restrict__ out, i64 ld, i64 out_words)
{
    __shared__ u64 tile[32][5];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const i64 row0 = (i64)blockIdx.x * 32;
    const i64 w = (i64)blockIdx.y * 4 + warp;
    const i64 row = row0 + lane;
    u64 word = 0;
    if (row < m && w * 64 < n) {
        const i64 c0 = w * 64;
        const int cols = (int)((n - c0) < 64 ? (n - c0) : 64);
        const double *p = in + row + c0 * m;
#pragma unroll 1
        for (int j0 = 0; j0 < cols; j0 += 16) {
            double x[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) x[j] = j0 + j < cols ? p[(i64)(j0 + j) * m] : 0.0;
            u32 bits = 0;
#pragma unroll
            for (int j = 0; j < 16; ++j) bits |= parity_of(x[j]) << j;
            word |= (u64)bits << j0;
        }
    }
    tile[lane][warp] = word;
    __syncthreads();
    const int r = threadIdx.x >> 2, q = threadIdx.x & 3;
    const i64 orow = row0 + r, ow = (i64)blockIdx.y * 4 + q;
    if (orow < m && ow < out_words) out[orow * ld + ow] = tile[r][q];
}

// Bytes 0x01 / 0x00 of the nonzero bytes of x, in the top bit of each byte.
__device__ __forceinline__ u32 nonzero_hi(u32 x) { return (((x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x) & 0x80808080u; }

// Logical bytes (nonzero = 1).  Block: 128 rows x 4 output words, a warp per
// word, a lane per 4 rows.  A lane reads its 4 bytes of a column as one word
// -- the aligned words of its first and last row and a funnel shift, as the
// column may start anywhere in a word (odd m) -- so a warp's load is 128
// consecutive bytes, and each word read holds a byte of the array, so it never
// leaves the array's allocation.  Five logical operations
// per word shift its nonzero bits into one byte per row, 16 columns into 16
// bits of each row's packed word.  Latency-bound like the doubles, with 16
// columns in flight; the loop is kept short because a call runs it once and
// would fetch an unrolled body from L2.  (3001 x 2500: 5.3 us against 6.5 us
// with a byte a load; 8192 x 8192 18.6 against 43.8 us.)
constexpr int kTilePitch = 9;  // u32 per row of 4 words: rows 4 apart fall on different banks
__global__ void __launch_bounds__(128) pack_logical_kernel(const unsigned char *__restrict__ in, i64 m, i64 n,
                                                           u64 *__restrict__ out, i64 ld, i64 out_words)
{
    __shared__ u32 tile[128 * kTilePitch];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const i64 row0 = (i64)blockIdx.x * 128;
    const i64 w = (i64)blockIdx.y * 4 + warp;
    const i64 row = row0 + 4 * lane;
    const i64 c0 = w * 64;
    const int cols = row >= m || c0 >= n ? 0 : (int)((n - c0) < 64 ? (n - c0) : 64);
    const int left = m - row < 4 ? (int)(m - row) : 4;
    const uintptr_t p = (uintptr_t)(in + row + c0 * m);
    unsigned short *t16 = reinterpret_cast<unsigned short *>(tile) + 4 * lane * (2 * kTilePitch) + 4 * warp;
#pragma unroll 1
    for (int o2 = 0; o2 < 4; ++o2) {
        u32 oct[2] = {0, 0};  // byte r: bits of 8 columns of row r
        if (16 * o2 < cols) {
            u32 x[16];
            u32 v0[16], v1[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const int c = 16 * o2 + j < cols ? 16 * o2 + j : cols - 1;
                const uintptr_t q = p + (uintptr_t)(c * m);
                v0[j] = __ldg(reinterpret_cast<const u32 *>(q & ~(uintptr_t)3));
                v1[j] = __ldg(reinterpret_cast<const u32 *>((q + left - 1) & ~(uintptr_t)3));
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const u32 q = (u32)p + (u32)(16 * o2 + j) * (u32)m;
                x[j] = 16 * o2 + j < cols ? __funnelshift_r(v0[j], v1[j], 8 * (q & 3)) : 0u;
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                u32 &a = oct[j >> 3];
                a = ((a >> 1) & 0x7F7F7F7Fu) | nonzero_hi(x[j]);
            }
        }
        const u32 r01 = __byte_perm(oct[0], oct[1], 0x5140), r23 = __byte_perm(oct[0], oct[1], 0x7362);
        t16[0 * 2 * kTilePitch + o2] = (unsigned short)r01;
        t16[1 * 2 * kTilePitch + o2] = (unsigned short)(r01 >> 16);
        t16[2 * 2 * kTilePitch + o2] = (unsigned short)r23;
        t16[3 * 2 * kTilePitch + o2] = (unsigned short)(r23 >> 16);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = (threadIdx.x >> 2) + 32 * i, q = threadIdx.x & 3;
        const i64 orow = row0 + r, ow = (i64)blockIdx.y * 4 + q;
        const u32 *t = tile + r * kTilePitch + 2 * q;
        if (orow < m && ow < out_words) out[orow * ld + ow] = (u64)t[0] | ((u64)t[1] << 32);
    }
}

// ---------------------------------------------------------------- unpack
// One warp: 32 rows x 64 columns; each store instruction writes 32
// consecutive rows of one column (column-major output).
__global__ void __launch_bounds__(256) unpack_kernel(const u64 *__restrict__ in, i64 ld, i64 m,
                                                     i64 n, unsigned char *__restrict__ out)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const i64 row = (i64)blockIdx.x * 32 + lane;
    const i64 w = (i64)blockIdx.y * 8 + warp;
    if (w * 64 >= n) return;
    const i64 c0 = w * 64;
    const int cols = (int)((n - c0) < 64 ? (n - c0) : 64);
    if (row >= m) return;
    u64 word = in[row * ld + w];
    unsigned char *p = out + row + c0 * m;
    for (int j = 0; j < cols; ++j) p[(i64)j * m] = (unsigned char)((word >> j) & 1);
}

// ---------------------------------------------------------------- transpose
// Block: 256 input rows x 64 input columns.  Warp w loads rows
// 32w..32w+31 (one word each); two 32x32 warp transposes give, per input
// column b, the 32 bits of rows 32w..32w+31.  Output row (column b) receives
// 4 words.
__global__ void __launch_bounds__(256) transpose_kernel(const u64 *__restrict__ in, i64 ld_in,
                                                        i64 rows, i64 cols,
                                                        u64 *__restrict__ out, i64 ld_out)
{
    __shared__ u32 part[8][65];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const i64 wcol = blockIdx.x;           // input word column
    const i64 r0 = (i64)blockIdx.y * 256;  // input row group
    const i64 row = r0 + warp * 32 + lane;
    u64 x = (row < rows) ? in[row * ld_in + wcol] : 0ull;
    const u32 keep0 = transpose32_warp((u32)x), keep1 = transpose32_warp((u32)(x >> 32));
    part[warp][lane] = keep0;
    part[warp][lane + 32] = keep1;
    __syncthreads();
    const int b = threadIdx.x >> 2, q = threadIdx.x & 3;
    const i64 ocol_row = wcol * 64 + b;  // output row index
    const i64 ow = (i64)blockIdx.y * 4 + q;
    const i64 owc = words_of(rows);
    if (ocol_row < cols && ow < owc)
        out[ocol_row * ld_out + ow] = (u64)part[2 * q][b] | ((u64)part[2 * q + 1][b] << 32);
}

// ---------------------------------------------------------------- expand to bytes
__device__ __forceinline__ u32 spread4(u32 nib) { return (nib * 0x00204081u) & 0x01010101u; }
// 16 bits -> 16 bytes of 0/1.
__device__ __forceinline__ uint4 bytes_16(u32 v)
{
    return make_uint4(spread4(v & 15), spread4((v >> 4) & 15), spread4((v >> 8) & 15), spread4((v >> 12) & 15));
}
// 8 bits at 1..8 of v -> bit 1 of 8 nibbles (e2m1 values 0x2 = 1.0, 0).
__device__ __forceinline__ u32 e2m1_8(u32 v)
{
    v = (v | (v << 12)) & 0x001E001Eu;
    v = (v | (v << 6)) & 0x06060606u;
    return (v | (v << 3)) & 0x22222222u;
}
// 32 bits -> 32 e2m1 values, value j in nibble j & 1 of byte j / 2.
__device__ __forceinline__ uint4 e2m1_32(u32 v)
{
    return make_uint4(e2m1_8((v << 1) & 0x1FEu), e2m1_8((v >> 7) & 0x1FEu), e2m1_8((v >> 15) & 0x1FEu),
                      e2m1_8((v >> 23) & 0x1FEu));
}

// Rows of A: out (rows_pad x kpad bytes) = the values of bits 0 .. kpad's of
// each packed row, zero outside rows x kbits (whole words; the matrix's bits
// past its columns are zero).  A thread per 16 bytes, the lanes' pieces side by
// side: bound by the writes (both operands of 32768^3: FP4 260 us, 5.2 TB/s,
// against 368 with a word and a 64-bit division a thread; INT8 427 against 567;
// of 2048 x 2048 x 1024 in FP4 3.1 against 4.5).  Row and piece advance by the
// grid's step in both, so that only the step is divided out.
template <bool F4, bool SUM>
__device__ __forceinline__ void expand_rows(const u64 *__restrict__ in, i64 ld, i64 rows, i64 kbits,
                                            const ExpandBlock &in2, i64 rows_pad, i64 kpad,
                                            unsigned char *__restrict__ out, i64 block, i64 blocks)
{
    constexpr int PPW = F4 ? 2 : 4;  // pieces per packed word
    const i64 ppr = kpad >> 4, total = rows_pad * ppr, step = blocks * 256;
    const i64 pc = words_of(kbits) * PPW, pc2 = words_of(in2.cols) * PPW;
    auto piece = [&](const u64 *p, i64 r, i64 q) -> u32 {
        if (F4) return reinterpret_cast<const u32 *>(p)[r * 2 * ld + q];
        return reinterpret_cast<const unsigned short *>(p)[r * 4 * ld + q];
    };
    i64 t = block * 256 + threadIdx.x, r, dr = 0;
    if (total + step <= 0x7fffffff) {
        r = (u32)t / (u32)ppr;
        if (step < total) dr = (u32)step / (u32)ppr;
    } else {
        r = t / ppr;
        dr = step / ppr;
    }
    i64 q = t - r * ppr;
    const i64 dq = step - dr * ppr;
    for (; t < total; t += step) {
        u32 v = r < rows && q < pc ? piece(in, r, q) : 0u;
        if (SUM && r < in2.rows && q < pc2) v ^= piece(in2.p, r, q);
        *reinterpret_cast<uint4 *>(out + r * kpad + 16 * q) = F4 ? e2m1_32(v) : bytes_16(v);
        r += dr;
        q += dq;
        if (q >= ppr) {
            q -= ppr;
            ++r;
        }
    }
}

// 256 bits of row k from column j0 (a multiple of 256), zero past rows and
// cols: two 16-byte loads where the row's words are so aligned and all inside.
__device__ __forceinline__ void load_256(const u64 *__restrict__ in, i64 ld, i64 k, i64 rows, i64 j0, i64 cols,
                                         u32 (&a)[8])
{
    if (k < rows && j0 + 256 <= cols && !((ld & 1) | ((uintptr_t)in & 15))) {
        const uint4 *src = reinterpret_cast<const uint4 *>(in + k * ld + (j0 >> 6));
        const uint4 x = src[0], y = src[1];
        a[0] = x.x;
        a[1] = x.y;
        a[2] = x.z;
        a[3] = x.w;
        a[4] = y.x;
        a[5] = y.y;
        a[6] = y.z;
        a[7] = y.w;
        return;
    }
    const u32 *in32 = reinterpret_cast<const u32 *>(in);
#pragma unroll
    for (int g = 0; g < 8; ++g) {
        const i64 c = j0 + 32 * g;  // first column of word g
        u32 v = 0;
        if (k < rows && c < cols) {
            v = in32[k * 2 * ld + (c >> 5)];
            if (cols - c < 32) v &= (1u << (cols - c)) - 1u;
        }
        a[g] = v;
    }
}

// Transposing expansion: out row j (j < cols_pad) holds column j of the packed
// kbits x cols matrix `in` as K-major tensor-core values -- 0/1 bytes (F4 =
// false, kpad bytes per row) or e2m1 pairs (F4 = true, kpad bytes per row =
// two values each) -- zero past kbits and past cols.  It replaces a bit
// transpose followed by an expansion.  Block: 256 k x 256 columns.  Each
// warp reads 32 rows of 256 bits (a lane per row) and turns them into
// 32-bit column slices by five rounds of shuffle butterflies; the output rows
// are written in 16-byte pieces, contiguous along k.
template <bool F4, bool SUM>
__device__ __forceinline__ void expand_t(const u64 *__restrict__ in, i64 ld, i64 kbits, i64 cols,
                                         const ExpandBlock &in2, i64 kpad,
                                         unsigned char *__restrict__ out, i64 jb, i64 kb0, u32 (&U)[256][9])
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const i64 j0 = jb * 256, k0 = kb0 * 256;
    // lane = row k0 + 32 warp + lane; a[g] = its 32 bits of columns j0 + 32 g ...
    const i64 k = k0 + 32 * warp + lane;
    u32 a[8];
    load_256(in, ld, k, kbits, j0, cols, a);
    if (SUM) {
        u32 b[8];
        load_256(in2.p, ld, k, in2.rows, j0, in2.cols, b);
#pragma unroll
        for (int g = 0; g < 8; ++g) a[g] ^= b[g];
    }
    // 32 x 32 bit transposes across the warp: afterwards lane l's a[g] holds,
    // at bit r, row k0 + 32 warp + r of column j0 + 32 g + l
#pragma unroll
    for (int g = 0; g < 8; ++g) a[g] = transpose32_warp(a[g]);
#pragma unroll
    for (int g = 0; g < 8; ++g) U[32 * g + lane][warp] = a[g];
    __syncthreads();
    if (F4) {
        // column j, k slice q (32 values): 16 bytes, value k in nibble k & 1 of byte k / 2
        for (int e = tid; e < 256 * 8; e += 256) {
            const int j = e >> 3, q = e & 7;
            const i64 kb = (k0 + 32 * q) / 2;  // byte offset in the output row
            if (kb >= kpad) continue;
            *reinterpret_cast<uint4 *>(out + (j0 + j) * kpad + kb) = e2m1_32(U[j][q]);
        }
    } else {
        // column j, k slice q (16 values): 16 bytes of 0/1
        for (int e = tid; e < 256 * 16; e += 256) {
            const int j = e >> 4, q = e & 15;
            const i64 kb = k0 + 16 * q;
            if (kb >= kpad) continue;
            *reinterpret_cast<uint4 *>(out + (j0 + j) * kpad + kb) = bytes_16(U[j][q >> 1] >> (16 * (q & 1)));
        }
    }
}

// Both operands of a tensor-core product in one launch: blocks 0 .. tb-1 take
// B's 256 x 256 tiles (tj tiles a row), the others A's rows.  Either part may
// be empty.  One launch instead of two: 2 us less per product of a few
// thousand rows, where the expansion is launch-bound (2048 x 2048 x 1024: 11.3
// us for the product against 13.4).
// SUM: each operand is the sum of two blocks, A + A2 and B + B2 (A2, B2 may be
// empty), of k rows or columns and zero past their own sizes.
template <bool F4, bool SUM>
__global__ void __launch_bounds__(256) expand_kernel(const u64 *__restrict__ A, i64 lda, i64 m, i64 mp,
                                                     unsigned char *__restrict__ A8, const u64 *__restrict__ B,
                                                     i64 ldb, i64 n, unsigned char *__restrict__ B8, i64 ka, i64 kb,
                                                     i64 kp, i64 tb, i64 tj, ExpandBlock A2, ExpandBlock B2)
{
    __shared__ u32 U[256][9];
    if ((i64)blockIdx.x < tb)
        expand_t<F4, SUM>(B, ldb, kb, n, B2, kp, B8, (i64)blockIdx.x % tj, (i64)blockIdx.x / tj, U);
    else
        expand_rows<F4, SUM>(A, lda, m, ka, A2, mp, kp, A8, (i64)blockIdx.x - tb, (i64)gridDim.x - tb);
}

// ---------------------------------------------------------------- launchers
static int grid_for(i64 total, int threads)
{
    i64 g = (total + threads - 1) / threads;
    i64 cap = (i64)sm_count() * 16;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    return (int)g;
}

mela_status launch_expand(const u64 *A, i64 lda, i64 m, i64 mp, unsigned char *A8, const u64 *B, i64 ldb, i64 n,
                          i64 np, unsigned char *B8, i64 k, i64 kp, bool fp4, cudaStream_t s)
{
    if (kp <= 0) return MELA_OK;
    if (np % 256) {
        set_error("expand: padded column count %lld is not a multiple of 256", np);
        return MELA_ERR_INVALID;
    }
    const i64 kvals = fp4 ? 2 * kp : kp, tj = np > 0 ? np / 256 : 1, tk = (kvals + 255) / 256;
    if (np > 0)
        if (mela_status st = check_grid_yz(tk, 1, "expand_t"); st != MELA_OK) return st;
    const i64 tb = np > 0 ? tj * tk : 0;
    const i64 ta = mp > 0 ? grid_for(mp * (kp >> 4), 256) : 0;
    if (ta + tb == 0) return MELA_OK;
    const auto kernel = fp4 ? expand_kernel<true, false> : expand_kernel<false, false>;
    kernel<<<(unsigned)(ta + tb), 256, 0, s>>>(A, lda, m, mp, A8, B, ldb, n, B8, k, k, kp, tb, tj, ExpandBlock{},
                                               ExpandBlock{});
    MELA_LAUNCH_CHECK("expand_kernel");
    return MELA_OK;
}

mela_status launch_expand_sum(const ExpandBlock (&A)[2], i64 lda, i64 mp, unsigned char *A8, const ExpandBlock (&B)[2],
                              i64 ldb, i64 np, unsigned char *B8, i64 kp, bool fp4, cudaStream_t s)
{
    const i64 kvals = fp4 ? 2 * kp : kp, tj = np / 256, tk = (kvals + 255) / 256;
    if (mela_status st = check_grid_yz(tk, 1, "expand_t"); st != MELA_OK) return st;
    const i64 tb = tj * tk, ta = grid_for(mp * (kp >> 4), 256);
    const auto kernel = fp4 ? expand_kernel<true, true> : expand_kernel<false, true>;
    kernel<<<(unsigned)(ta + tb), 256, 0, s>>>(A[0].p, lda, A[0].rows, mp, A8, B[0].p, ldb, B[0].cols, B8, A[0].cols,
                                               B[0].rows, kp, tb, tj, A[1], B[1]);
    MELA_LAUNCH_CHECK("expand_kernel");
    return MELA_OK;
}

mela_status launch_transpose(const u64 *in, i64 ld_in, i64 rows, i64 cols, u64 *out, i64 ld_out,
                             cudaStream_t s)
{
    if (rows <= 0 || cols <= 0) return MELA_OK;
    if (mela_status st = check_grid_yz((rows + 255) / 256, 1, "transpose"); st != MELA_OK) return st;
    dim3 grid((unsigned)words_of(cols), (unsigned)((rows + 255) / 256));
    transpose_kernel<<<grid, 256, 0, s>>>(in, ld_in, rows, cols, out, ld_out);
    MELA_LAUNCH_CHECK("transpose_kernel");
    return MELA_OK;
}

mela_status launch_pack(int kind, i64 m, i64 n, const void *in, u64 *out, i64 ld, cudaStream_t s)
{
    return launch_pack_words(kind, m, n, in, out, ld, ld, s);
}

mela_status launch_pack_words(int kind, i64 m, i64 n, const void *in, u64 *out, i64 ld, i64 out_words,
                              cudaStream_t s)
{
    if (m <= 0) return MELA_OK;
    i64 wgroups = (out_words + 3) / 4;
    if (wgroups == 0) return MELA_OK;
    if (mela_status st = check_grid_yz((out_words + 7) / 8, 1, "pack"); st != MELA_OK) return st;
    if (wgroups > 65535) {  // more columns than one launch takes: in parts of whole words
        const i64 part = 65535 * 4;
        const size_t esz = kind == MELA_KIND_DOUBLE ? 8 : 1;
        for (i64 w0 = 0; w0 < out_words; w0 += part) {
            const i64 ow = out_words - w0 < part ? out_words - w0 : part;
            const i64 nc = n - 64 * w0 < 0 ? 0 : n - 64 * w0 < 64 * ow ? n - 64 * w0 : 64 * ow;
            mela_status st = launch_pack_words(kind, m, nc, (const char *)in + (size_t)(64 * w0) * (size_t)m * esz,
                                               out + w0, ld, ow, s);
            if (st != MELA_OK) return st;
        }
        return MELA_OK;
    }
    if (kind == MELA_KIND_DOUBLE)
        pack_double_kernel<<<dim3((unsigned)((m + 31) / 32), (unsigned)wgroups), 128, 0, s>>>((const double *)in, m, n,
                                                                                             out, ld, out_words);
    else
        pack_logical_kernel<<<dim3((unsigned)((m + 127) / 128), (unsigned)wgroups), 128, 0, s>>>(
            (const unsigned char *)in, m, n, out, ld, out_words);
    MELA_LAUNCH_CHECK("pack_kernel");
    return MELA_OK;
}

mela_status launch_unpack(const u64 *in, i64 ld, i64 m, i64 n, unsigned char *out, cudaStream_t s)
{
    if (m <= 0 || n <= 0) return MELA_OK;
    if (mela_status st = check_grid_yz((words_of(n) + 7) / 8, 1, "unpack"); st != MELA_OK) return st;
    dim3 grid((unsigned)((m + 31) / 32), (unsigned)((words_of(n) + 7) / 8));
    unpack_kernel<<<grid, 256, 0, s>>>(in, ld, m, n, out);
    MELA_LAUNCH_CHECK("unpack_kernel");
    return MELA_OK;
}

mela_status launch_rand_bernoulli(u64 seed, u64 stream_id, i64 m, i64 n, double density, u64 *out,
                                  i64 ld, cudaStream_t s)
{
    if (m <= 0 || ld <= 0) return MELA_OK;
    double t = density * 65536.0;
    unsigned thresh = t <= 0 ? 0u : (t >= 65536.0 ? 65536u : (unsigned)t);
    rand_bernoulli_kernel<<<grid_for(m * ld, 256), 256, 0, s>>>(stream_key(seed, stream_id), m, n, thresh,
                                                                 out, ld);
    MELA_LAUNCH_CHECK("rand_bernoulli_kernel");
    return MELA_OK;
}

mela_status launch_rand_dense(u64 seed, u64 stream_id, i64 m, i64 n, u64 *out, i64 ld,
                              cudaStream_t s)
{
    if (m <= 0 || ld <= 0) return MELA_OK;
    rand_dense_kernel<<<grid_for(m * ld, 256), 256, 0, s>>>(stream_key(seed, stream_id), m, n,
                                                            words_of(n), out, ld);
    MELA_LAUNCH_CHECK("rand_dense_kernel");
    return MELA_OK;
}

}  // namespace mela

// ---------------------------------------------------------------- C ABI
using namespace mela;

extern "C" mela_status mela_dev_rand_dense(uint64_t seed, uint64_t stream_id, int64_t m,
                                           int64_t n, uint64_t *d_out, int64_t ld, void *stream)
{
    if (m < 0 || n < 0 || ld < words_of(n) || (m > 0 && ld > 0 && !d_out)) {
        set_error("mela_dev_rand_dense: bad shape or pointer");
        return MELA_ERR_INVALID;
    }
    return launch_rand_dense(seed, stream_id, m, n, (u64 *)d_out, ld, (cudaStream_t)stream);
}

extern "C" mela_status mela_dev_rand_bernoulli(uint64_t seed, uint64_t stream_id, int64_t m,
                                               int64_t n, double density, uint64_t *d_out, int64_t ld,
                                               void *stream)
{
    if (m < 0 || n < 0 || ld < words_of(n) || (m > 0 && ld > 0 && !d_out) || !(density >= 0.0)) {
        set_error("mela_dev_rand_bernoulli: bad shape, pointer or density");
        return MELA_ERR_INVALID;
    }
    return launch_rand_bernoulli(seed, stream_id, m, n, density, (u64 *)d_out, ld, (cudaStream_t)stream);
}

extern "C" mela_status mela_dev_pack(int32_t kind, int64_t m, int64_t n, const void *d_in,
                                     uint64_t *d_out, int64_t ld, void *stream)
{
    if (m < 0 || n < 0 || ld < words_of(n) || (kind != MELA_KIND_LOGICAL && kind != MELA_KIND_DOUBLE)) {
        set_error("mela_dev_pack: bad shape or kind");
        return MELA_ERR_INVALID;
    }
    if (m > 0 && ld > 0 && (!d_out || (n > 0 && !d_in))) {
        set_error("mela_dev_pack: null pointer");
        return MELA_ERR_INVALID;
    }
    return launch_pack(kind, m, n, d_in, (u64 *)d_out, ld, (cudaStream_t)stream);
}

extern "C" mela_status mela_dev_unpack(const uint64_t *d_in, int64_t ld, int64_t m, int64_t n,
                                       uint8_t *d_out, void *stream)
{
    if (m < 0 || n < 0 || ld < words_of(n) || (m > 0 && n > 0 && (!d_in || !d_out))) {
        set_error("mela_dev_unpack: bad shape or pointer");
        return MELA_ERR_INVALID;
    }
    return launch_unpack((const u64 *)d_in, ld, m, n, d_out, (cudaStream_t)stream);
}

extern "C" mela_status mela_dev_transpose(const uint64_t *d_in, int64_t ld_in, int64_t rows,
                                          int64_t cols, uint64_t *d_out, int64_t ld_out,
                                          void *stream)
{
    if (rows < 0 || cols < 0 || ld_in < words_of(cols) || ld_out < words_of(rows) ||
        (rows > 0 && cols > 0 && (!d_in || !d_out))) {
        set_error("mela_dev_transpose: bad shape or pointer");
        return MELA_ERR_INVALID;
    }
    return launch_transpose((const u64 *)d_in, ld_in, rows, cols, (u64 *)d_out, ld_out,
                            (cudaStream_t)stream);
}
