// What the products of a few tokens share (gemm_few.cu, the few tokens' kernels of experts.cu): weight rows that go from memory into
// the registers mma.sync reads, 32 bytes a lane.
//
// Four neighbouring lanes hold 64 consecutive elements of a row, 16 each.  m16n8k16 wants of lane (g, t) the elements 2 t, 2 t + 1, 2 t + 8 and
// 2 t + 9 of rows g and g + 8 and of token g; which elements of K those are is free as long as both operands agree, so registers 2 j and
// 2 j + 1 of a lane's are its share of the j-th instruction.
#pragma once

#include "common.cuh"

namespace qt_few {

constexpr int PIECE = 16;                   // elements of a row that a lane loads at once

struct Line { uint32_t r[PIECE / 2]; };

// weights: written when the model is loaded, read once
__device__ __forceinline__ Line load_weight(const __nv_bfloat16* p) {
    Line v;
    asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v.r[0]), "=r"(v.r[1]), "=r"(v.r[2]), "=r"(v.r[3]), "=r"(v.r[4]), "=r"(v.r[5]), "=r"(v.r[6]), "=r"(v.r[7]) : "l"(p));
    return v;
}
// what an earlier kernel wrote
__device__ __forceinline__ Line load_rows(const __nv_bfloat16* p) {
    Line v;
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v.r[0]), "=r"(v.r[1]), "=r"(v.r[2]), "=r"(v.r[3]), "=r"(v.r[4]), "=r"(v.r[5]), "=r"(v.r[6]), "=r"(v.r[7]) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void mma_16x8x16(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// c[r] += rows 16 r .. 16 r + 15 of a turn times eight tokens
template <int RT>
__device__ __forceinline__ void turn_product(float (&c)[RT][4], const Line (&a)[RT][2], const Line& b) {
#pragma unroll
    for (int j = 0; j < PIECE / 4; ++j)
#pragma unroll
        for (int r = 0; r < RT; ++r)
            mma_16x8x16(c[r], a[r][0].r[2 * j], a[r][1].r[2 * j], a[r][0].r[2 * j + 1], a[r][1].r[2 * j + 1], b.r[2 * j], b.r[2 * j + 1]);
}
__device__ __forceinline__ void cluster_store4(const float* local, uint32_t rank, float4 v) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"((uint32_t)__cvta_generic_to_shared(local)), "r"(rank));
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(remote), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

}  // namespace qt_few
