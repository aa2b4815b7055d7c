// mela_internal.h -- launchers shared between the library's translation units.
#pragma once

#include <cuda.h>

#include "mela_common.cuh"

namespace mela {

u64 stream_key(u64 seed, u64 stream);

mela_status launch_rand_dense(u64 seed, u64 stream_id, i64 m, i64 n, u64 *out, i64 ld,
                              cudaStream_t s);
mela_status launch_rand_bernoulli(u64 seed, u64 stream_id, i64 m, i64 n, double density, u64 *out,
                                  i64 ld, cudaStream_t s);
mela_status launch_pack(int kind, i64 m, i64 n, const void *in, u64 *out, i64 ld, cudaStream_t s);
// The same, writing only the first out_words words of each packed row (the
// words of a column block, for packing a matrix block by block).
mela_status launch_pack_words(int kind, i64 m, i64 n, const void *in, u64 *out, i64 ld, i64 out_words,
                              cudaStream_t s);
mela_status launch_unpack(const u64 *in, i64 ld, i64 m, i64 n, unsigned char *out, cudaStream_t s);
mela_status launch_transpose(const u64 *in, i64 ld_in, i64 rows, i64 cols, u64 *out, i64 ld_out,
                             cudaStream_t s);
// A block of a packed matrix (its pitch given beside it); rows = 0: empty.
struct ExpandBlock {
    const u64 *p = nullptr;
    i64 rows = 0, cols = 0;
};
// Both operands as sums of two blocks, A[0] + A[1] (K in columns) and B[0] +
// B[1] (K in rows), expanded to mp x kp and np x kp.
mela_status launch_expand_sum(const ExpandBlock (&A)[2], i64 lda, i64 mp, unsigned char *A8, const ExpandBlock (&B)[2],
                              i64 ldb, i64 np, unsigned char *B8, i64 kp, bool fp4, cudaStream_t s);
// Tensor-core operands, both K-major with kp bytes per row (0/1 bytes, or e2m1
// pairs when fp4), zero past the matrices' edges: A8 (mp rows) from the packed
// m x k matrix A, B8 (np rows, a multiple of 256) from the columns of the packed
// k x n matrix B.  mp or np 0: that operand is left out.
mela_status launch_expand(const u64 *A, i64 lda, i64 m, i64 mp, unsigned char *A8, const u64 *B, i64 ldb, i64 n,
                          i64 np, unsigned char *B8, i64 k, i64 kp, bool fp4, cudaStream_t s);

// ---- products (packed, device)
// The words of two packed matrices (pitch, rows, columns) lie apart, one after
// the other or as column blocks of one buffer: a product that writes its result
// before it has read all of an operand needs that.
inline bool packed_apart(const u64 *x, i64 ldx, i64 rx, i64 cx, const u64 *y, i64 ldy, i64 ry, i64 cy)
{
    const i64 wx = words_of(cx), wy = words_of(cy);
    if (x + (rx - 1) * ldx + wx <= y || y + (ry - 1) * ldy + wy <= x) return true;
    if (ldx != ldy) return false;
    const i64 at = (y >= x ? y - x : ldx - 1 - (x - y - 1) % ldx) % ldx;  // y's first word in a row from x's
    return at >= wx && at + wy <= ldx;
}
// Plain AND+popcount product: C (m x n) = A (m x k) * B (k x n), with the
// transposed right operand Bt (n x k) already formed.
mela_status launch_gemm_plain(const u64 *A, i64 lda, const u64 *Bt, i64 ldbt, u64 *C, i64 ldc,
                              i64 m, i64 k, i64 n, cudaStream_t s);
// Tensor-core product on 0/1 byte operands A8 (mp x kp) and Bt8 (np x kp),
// both K-major; mp % 128 == 0, np % 256 == 0, kp % 128 == 0.  Writes the
// valid m x n block of packed C.
// fp4 = true: packed e2m1 operands (kp counts bytes, two values each), kind::mxf4.
// tile: 0 = CTA pairs (256 x 256 tiles) when mp % 256 == 0, else one CTA per
// 128 x 256 tile; 1 = always one CTA per tile; 2 = pairs where mp allows.
mela_status launch_gemm_tc(const unsigned char *A8, const unsigned char *Bt8, i64 mp, i64 np,
                           i64 kp, u64 *C, i64 ldc, i64 m, i64 n, cudaStream_t s, bool fp4, int tile = 0);
// One level of Strassen's algorithm over packed operands, the workspace (two
// expanded quarter operands) at ws; fits: where it beats one product of the
// whole, and C overlaps neither operand.
bool gemm_strassen_fits(const u64 *A, i64 lda, const u64 *B, i64 ldb, const u64 *C, i64 ldc, i64 m, i64 k, i64 n,
                        bool fp4, int tile);
mela_status launch_gemm_strassen(const u64 *A, i64 lda, const u64 *B, i64 ldb, u64 *C, i64 ldc, i64 m, i64 k, i64 n,
                                 void *ws, size_t ws_bytes, bool fp4, cudaStream_t s);
// TMA map of a K-major byte matrix rows x kp (row pitch kp bytes): boxes of
// 128 bytes x box_rows rows with 128-byte swizzle, as the tcgen05 kernels read them.
mela_status make_u8_kmajor_map(CUtensorMap *map, const unsigned char *base, i64 rows, i64 kp, int box_rows);
// TMA map of packed rows (rows x words uint64, row pitch ld words; ld * 8 must
// be a multiple of 16 and base 16-byte aligned): boxes of box_words x box_rows,
// no swizzle, zeros read past the edges.
mela_status make_u64_rows_map(CUtensorMap *map, const u64 *base, i64 rows, i64 words, i64 ld, int box_words,
                              int box_rows);
// tile: 0 / 2 = 16 warps of 32 rows per 512-row CTA, 1 = 8 warps of 64 rows.
mela_status launch_gemm_m4ri(const u64 *A, i64 lda, const u64 *B, i64 ldb, u64 *C, i64 ldc,
                             i64 m, i64 k, i64 n, cudaStream_t s, int tile = 0);

// Product of small arrays in MATLAB layout (column-major, element kinds and
// sizes as given) in one launch: C (m x n logical), and the device error word
// copied to err_out where that is given.  fits: where it beats packing
// (gemm_small.cu).
bool gemm_small_fits(i64 m, i64 k, i64 n, size_t a_size, size_t b_size);
mela_status launch_gemm_small(int kind_a, const void *A, int kind_b, const void *B, unsigned char *C, i64 m, i64 k,
                              i64 n, const u32 *err, u32 *err_out, cudaStream_t s);

// Whole RREF of one matrix by one CTA in one launch: in shared memory where it
// fits (elim_small.cu: up to 512 rows, 192 KB with its tables), else by the
// batch engine for big matrices over the workspace (batch.cu).
bool small_elim_fits(i64 m, i64 n);
mela_status launch_small_elim(u64 *M, i64 ld, i64 m, i64 n, long long *d_rank, long long *d_piv,
                              long long *d_prow, cudaStream_t s);
// The calling thread's page-locked words (api.cu: posted), which a kernel may
// write itself: a value, the device error word (read at err_word) and bytes.
struct Posted {
    long long *value;
    u32 *err;
    const u32 *err_word;
    unsigned char *bytes, *in;  // results; inputs on their way up (24 KB)
    size_t bytes_size;          // of the results
};
// The same elimination for a call that waits for the result: the rank and, for
// a null space (of at most small_null_fits columns), the basis as logical
// bytes, written to the caller's page-locked words.  M is left as it was.
bool small_null_fits(i64 m, i64 n);
mela_status launch_small_post(const u64 *M, i64 ld, i64 m, i64 n, const Posted &to, bool null_space, cudaStream_t s);
size_t fused_workspace(i64 m, i64 n);
mela_status launch_fused_elim(u64 *M, i64 ld, i64 m, i64 n, long long *d_rank, long long *d_piv,
                              long long *d_prow, void *ws, size_t ws_bytes, cudaStream_t s);

}  // namespace mela
