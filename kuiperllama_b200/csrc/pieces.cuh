// Products of 32-bit operands on the tensor cores, and what the walks over chunks of a prompt share (outer_chunked.cu, delta_chunked.cu): a number
// as the sum of three bfloat16 ones, the six products of two such operands, tiles in shared memory whose rows are read by ldmatrix, bulk
// copies.
#pragma once
#include "tcgen05.cuh"

namespace kl {

// `bytes` (a multiple of 16) that lie together, counted by a barrier
__device__ __forceinline__ void pc_bulk(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void pc_ldm4(uint32_t a, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void pc_ldm4t(uint32_t a, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void pc_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// the same from zero
__device__ __forceinline__ void pc_mma0(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// two numbers as three packed pairs of bfloat16 that add up to them
__device__ __forceinline__ void pc_split(float x, float y, uint32_t& a, uint32_t& b, uint32_t& c) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    float2 f = __bfloat1622float2(h);
    x -= f.x; y -= f.y;
    const __nv_bfloat162 m = __floats2bfloat162_rn(x, y);
    f = __bfloat1622float2(m);
    const __nv_bfloat162 l = __floats2bfloat162_rn(x - f.x, y - f.y);
    a = *reinterpret_cast<const uint32_t*>(&h);
    b = *reinterpret_cast<const uint32_t*>(&m);
    c = *reinterpret_cast<const uint32_t*>(&l);
}
// the place of 16-byte piece c of row r in a tile of rows of W elements: neighbouring rows' pieces fall on different banks
template <int W> __device__ __forceinline__ int pc_at(int r, int c) {
    constexpr int P = W / 8;
    if constexpr (P >= 8) return r * W + ((c ^ (r & 7)) << 3);
    else return r * W + ((c ^ ((r / (8 / P)) & (P - 1))) << 3);
}
// Operands of three pieces each: d is the leading product, the five others down to 2^-16 of it, smallest first, are added to e.  A product of
// the tensor cores cuts its sum off where it does not fit 32 bits, so no sum is carried through many of them (8e-7 of y, 1e-7 as it is): d starts
// from zero and is added with rounding.
template <int NT, bool FIRST>
__device__ __forceinline__ void pc_mma33(float (&d)[NT][4], float (&e)[NT][4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][NT][2]) {
#pragma unroll
    for (int sum = 2; sum >= 1; --sum)
#pragma unroll
        for (int x = sum; x >= 0; --x)
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                if (FIRST && sum == 2 && x == 2) pc_mma0(e[n], a[x], b[sum - x][n][0], b[sum - x][n][1]);
                else pc_mma(e[n], a[x], b[sum - x][n][0], b[sum - x][n][1]);
            }
#pragma unroll
    for (int n = 0; n < NT; ++n) pc_mma0(d[n], a[0], b[0][n][0], b[0][n][1]);
}
template <int NT>
__device__ __forceinline__ void pc_zero(float (&d)[NT][4]) {
#pragma unroll
    for (int n = 0; n < NT; ++n) d[n][0] = d[n][1] = d[n][2] = d[n][3] = 0.f;
}
template <int NT>
__device__ __forceinline__ void pc_add(float (&d)[NT][4], const float (&e)[NT][4]) {
#pragma unroll
    for (int n = 0; n < NT; ++n) { d[n][0] += e[n][0]; d[n][1] += e[n][1]; d[n][2] += e[n][2]; d[n][3] += e[n][3]; }
}
// B fragments of NT tiles of 8 rows (the columns of the product) for the 16 columns from piece p on; rows of W elements
template <int W, int NT>
__device__ __forceinline__ void pc_rows(const bf16* tile, int row0, int p, int lane, uint32_t (&b)[NT][2]) {
#pragma unroll
    for (int n = 0; n < NT; n += 2) {
        uint32_t r[4];
        pc_ldm4(smem_u32(tile + pc_at<W>(row0 + n * 8 + (lane & 7) + ((lane >> 4) << 3), p + ((lane >> 3) & 1))), r);
        b[n][0] = r[0]; b[n][1] = r[1]; b[n + 1][0] = r[2]; b[n + 1][1] = r[3];
    }
}

}  // namespace kl
