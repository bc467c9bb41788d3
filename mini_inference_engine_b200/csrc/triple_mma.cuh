// Products of float32 operands on the warps' tensor-core instruction (mma.sync), for kernels whose tiles are too small, or depend too much on one another, for tcgen05.
//
// A float32 number is the sum of three bfloat16 numbers: the nearest one, the nearest to what is left, and the rest.  Of the nine products of parts six are
// formed; the three left out are at most 2^-24 of the product together and of either sign.  The instruction's sum is cut off towards zero, so the product of
// the high parts (16 digits: 16 of them add up with next to nothing cut off) and the small ones, 2^-8 of it, have sums of their own, and both are added up in float32
// registers rounded to nearest every 16 products: a sum of 128 products with random signs is 6e-8 off (2-norm) where a chain of fused multiply-adds is 1.9e-7 off.
//
// Numbers beyond 2^127 may not have three parts (the nearest bfloat16 is infinite): callers look for them.  Of a number below 2^-110 the last part loses digits.
#pragma once
#include "common.cuh"

__device__ __forceinline__ uint32_t magnitude(float v) { return __float_as_uint(v) & 0x7fffffffu; }
__device__ __forceinline__ uint32_t magnitude(float4 v) { return max(max(magnitude(v.x), magnitude(v.y)), max(magnitude(v.z), magnitude(v.w))); }
__device__ __forceinline__ bool has_no_parts(uint32_t magnitude_bits) { return magnitude_bits >= 0x7f000000u; }

// Two numbers as [high, middle, low] parts, the first in the lower half.
__device__ __forceinline__ uint32_t nearest2(float a, float b) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
}
__device__ __forceinline__ void split3(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    h = nearest2(a, b);
    a -= __uint_as_float(h << 16);
    b -= __uint_as_float(h & 0xffff0000u);
    m = nearest2(a, b);
    a -= __uint_as_float(m << 16);
    b -= __uint_as_float(m & 0xffff0000u);
    l = nearest2(a, b);
}
// A left operand of 16 x 16 from a lane's eight numbers: (row, column) + (0, 0 .. 1), (8, 0 .. 1), (0, 8 .. 9), (8, 8 .. 9) from (lane / 4, 2 (lane % 4)) on.
__device__ __forceinline__ void split_left(uint32_t (&a)[3][4], const float4& v, const float4& w) {
    split3(v.x, v.y, a[0][0], a[1][0], a[2][0]);
    split3(v.z, v.w, a[0][1], a[1][1], a[2][1]);
    split3(w.x, w.y, a[0][2], a[1][2], a[2][2]);
    split3(w.z, w.w, a[0][3], a[1][3], a[2][3]);
}

__device__ __forceinline__ void mma_zero(float (&d)[4], const uint32_t* a, const uint32_t* b) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}
__device__ __forceinline__ void mma_more(float (&d)[4], const uint32_t* a, const uint32_t* b) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// sum[n] += A B_n over 16 of the contraction, for N tiles of 8 columns; a, b: parts.
template <int N>
__device__ __forceinline__ void triple_step(float (*sum)[4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][N][2]) {
    float t[N][4], h[N][4];
#pragma unroll
    for (int n = 0; n < N; ++n) mma_zero(t[n], a[2], b[0][n]);
#pragma unroll
    for (int n = 0; n < N; ++n) mma_zero(h[n], a[0], b[0][n]);
#pragma unroll
    for (int n = 0; n < N; ++n) mma_more(t[n], a[0], b[2][n]);
#pragma unroll
    for (int n = 0; n < N; ++n) mma_more(t[n], a[1], b[1][n]);
#pragma unroll
    for (int n = 0; n < N; ++n) mma_more(t[n], a[1], b[0][n]);
#pragma unroll
    for (int n = 0; n < N; ++n) mma_more(t[n], a[0], b[1][n]);
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) sum[n][i] = h[n][i] + (sum[n][i] + t[n][i]);
}
// Tiles of bfloat16 numbers in shared memory: rows of COLS numbers in pieces of 16 bytes, a row's pieces permuted so that eight neighbouring rows
// lie in different banks (rows of 128 bytes and more by the row, rows of 32 bytes by a quarter of the row).
template <int COLS>
__device__ __forceinline__ uint32_t tile_at(int row, int piece) {
    return (uint32_t)(row * (COLS * 2) + ((piece ^ (COLS >= 64 ? row & 7 : (row >> 2) & 1)) << 4));
}
__device__ __forceinline__ void ldm4(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(at) : "memory");
}
__device__ __forceinline__ void ldm4t(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(at) : "memory");
}
// Left operand (16 x 16) from three tiles, `plane` bytes apart, whose rows are its rows.
template <int COLS>
__device__ __forceinline__ void left_rows(uint32_t (&a)[3][4], uint32_t tile, int plane, int m, int k, int lane) {
    const uint32_t at = tile + tile_at<COLS>(m * 16 + (lane & 15), k * 2 + (lane >> 4));
#pragma unroll
    for (int p = 0; p < 3; ++p) ldm4(a[p][0], a[p][1], a[p][2], a[p][3], at + p * plane);
}
// Right operand, two tiles of 8 columns (n, n + 1) into b[..][first] and the next, from tiles whose rows run along the contraction ...
template <int COLS, int N>
__device__ __forceinline__ void right_rows(uint32_t (&b)[3][N][2], int first, uint32_t tile, int plane, int k, int n, int lane) {
    const uint32_t at = tile + tile_at<COLS>(k * 16 + (lane & 15), n + (lane >> 4));
#pragma unroll
    for (int p = 0; p < 3; ++p) ldm4t(b[p][first][0], b[p][first][1], b[p][first + 1][0], b[p][first + 1][1], at + p * plane);
}
// ... or along its columns.
template <int COLS, int N>
__device__ __forceinline__ void right_columns(uint32_t (&b)[3][N][2], int first, uint32_t tile, int plane, int k, int n, int lane) {
    const uint32_t at = tile + tile_at<COLS>(n * 8 + (lane & 7) + ((lane >> 4) << 3), k * 2 + ((lane >> 3) & 1));
#pragma unroll
    for (int p = 0; p < 3; ++p) ldm4(b[p][first][0], b[p][first][1], b[p][first + 1][0], b[p][first + 1][1], at + p * plane);
}
