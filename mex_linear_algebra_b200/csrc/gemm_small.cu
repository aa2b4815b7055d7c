// gemm_small.cu -- small product on arrays in MATLAB layout, in one launch.
//
// C (m x n logical, column-major) = A (m x k) * B (k x n) over GF(2), A and B
// column-major logical or double, nothing packed in memory.  For the gateways'
// small calls, which otherwise spend most of their time on six launches and
// their buffers (pack A, pack B, transpose, product, unpack).
//
// Block: 32 x 32 of C, 256 threads, all of K (up to 256 bits).  A warp packs
// 32 rows x 32 columns of A as one word per lane (32 loads of 32 neighbouring
// rows in flight), a column of B by ballots of 32 neighbouring rows; then each
// thread ANDs and XORs a row of A with four columns of B, the parity of the
// final word giving the bit.
// Bound by launch and load latency.  Whole gateway call, packed path -> this:
// 16^3 52 -> 28 us, 64^3 62 -> 30, 100 x 120 x 80 logical 59 -> 33, double
// 79 -> 55.
#include "mela_common.cuh"
#include "mela_internal.h"

namespace mela {

namespace {

constexpr int SP_T = 32;  // rows and columns of C per block
constexpr int SP_KW = 8;  // 32-bit words of K

__device__ __forceinline__ u32 bit_of(double x)
{
    // ((int)x) & 1 as the reference reads it; NaN and out-of-range values are even
    if (!(x >= -2147483648.0 && x < 2147483648.0)) return 0;
    return (u32)__double2int_rz(x) & 1u;
}
__device__ __forceinline__ u32 bit_of(unsigned char x) { return x != 0; }

template <typename TA, typename TB>
__global__ void __launch_bounds__(256)
gemm_small_kernel(const TA *__restrict__ A, const TB *__restrict__ B, unsigned char *__restrict__ C, int m, int k, int n,
                  const u32 *err, u32 *err_out)
{
    __shared__ u32 As[SP_T][SP_KW + 1], Bs[SP_T][SP_KW + 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int i0 = (int)blockIdx.x * SP_T, j0 = (int)blockIdx.y * SP_T;
    const int i = i0 + lane;
    u32 acc[4] = {0, 0, 0, 0};
    if (err_out && tid == 0 && blockIdx.x == 0 && blockIdx.y == 0) *err_out = *err;
    const int kw = (k + 31) >> 5;
    for (int q = warp; q < kw; q += 8) {
        const int c0 = 32 * q;
        u32 v = 0;
#pragma unroll 16
        for (int b = 0; b < 32; ++b)
            if (i < m && c0 + b < k) v |= bit_of(A[(size_t)(c0 + b) * m + i]) << b;
        As[lane][q] = v;
    }
    for (int e = warp; e < SP_T * kw; e += 8) {
        const int c = e / kw, q = e - c * kw, j = j0 + c, r = 32 * q + lane;
        const u32 bit = j < n && r < k ? bit_of(B[(size_t)j * k + r]) : 0u;
        const u32 v = __ballot_sync(0xffffffffu, bit);
        if (lane == 0) Bs[c][q] = v;
    }
    __syncthreads();
    for (int q = 0; q < kw; ++q) {
        const u32 a = As[lane][q];
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[c] ^= a & Bs[4 * warp + c][q];
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int j = j0 + 4 * warp + c;
        if (i < m && j < n) C[(size_t)j * m + i] = (unsigned char)(__popc(acc[c]) & 1);
    }
}

}  // namespace

bool gemm_small_fits(i64 m, i64 k, i64 n, size_t a_size, size_t b_size)
{
    if (m <= 0 || k <= 0 || n <= 0 || m > 4096 || n > 4096 || k > 32 * SP_KW) return false;
    // Every block reads its rows of A and columns of B in full.  Up to 8 MiB of
    // that and 256 bits of K it beats packing (200^3 logical 48 against 73 us,
    // double 88 against 93; 256^3 double 110 against 115; 1000 x 64 x 1000
    // logical 250 against 276); near 8 MiB the two draw level (1000 x 200 x 500
    // logical 188 and 199).  A longer K is a serial chain of loads in each
    // block: 128 x 512 x 128 double 121 against 110, 64 x 2000 x 64 156
    // against 95.
    const i64 bi = (m + SP_T - 1) / SP_T, bj = (n + SP_T - 1) / SP_T;
    return bi * bj * SP_T * k * (i64)(a_size + b_size) <= (i64)8 << 20;
}

mela_status launch_gemm_small(int kind_a, const void *A, int kind_b, const void *B, unsigned char *C, i64 m, i64 k,
                              i64 n, const u32 *err, u32 *err_out, cudaStream_t s)
{
    const dim3 grid((unsigned)((m + SP_T - 1) / SP_T), (unsigned)((n + SP_T - 1) / SP_T));
    const int mi = (int)m, ki = (int)k, ni = (int)n;
    const bool da = kind_a == MELA_KIND_DOUBLE, db = kind_b == MELA_KIND_DOUBLE;
    if (da && db)
        gemm_small_kernel<<<grid, 256, 0, s>>>((const double *)A, (const double *)B, C, mi, ki, ni, err, err_out);
    else if (da)
        gemm_small_kernel<<<grid, 256, 0, s>>>((const double *)A, (const unsigned char *)B, C, mi, ki, ni, err, err_out);
    else if (db)
        gemm_small_kernel<<<grid, 256, 0, s>>>((const unsigned char *)A, (const double *)B, C, mi, ki, ni, err, err_out);
    else
        gemm_small_kernel<<<grid, 256, 0, s>>>((const unsigned char *)A, (const unsigned char *)B, C, mi, ki, ni, err, err_out);
    MELA_LAUNCH_CHECK("gemm_small_kernel");
    return MELA_OK;
}

}  // namespace mela
