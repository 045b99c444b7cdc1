// Device code shared by the GEMV kernels whose activations are mma B fragments in code order (qgemv_stream.cu, qgemv_held.cu):
// PTX helpers, weight formats, fragment order, sums of activations.
#pragma once

#include "qgemv_stream.cuh"

namespace qgemv {
namespace {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// 16-byte asynchronous copy that brings the whole 128-byte line to L2; z: only `valid` bytes are read, the rest is zero.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16z(uint32_t dst, const void* src, int valid) {
    asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid) : "memory");
}
template <int BYTES> __device__ __forceinline__ void cp_async_small(uint32_t dst, const void* src) {
    if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global.L2::128B [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void named_barrier(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait_n() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void cp_async_wait_depth(int depth) {  // all but the newest depth - 1 groups have landed (depth 2 - 4)
    if (depth == 2) cp_async_wait_n<1>();
    else if (depth == 3) cp_async_wait_n<2>();
    else cp_async_wait_n<3>();
}
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// D = A.B + C with C kept: a chain starts from a register quad that is set up once (a zero literal would be copied into
// four registers before every chain).
__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, const float (&c)[4]) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}
__device__ __forceinline__ void mma_s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, const int (&c)[4]) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]));
}
// Shared-window loads by 32-bit address: compile-time offsets fold into the instruction.
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t v; asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory"); return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
    uint2 v; asm("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory"); return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v; asm("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory"); return v;
}
__device__ __forceinline__ float lds_half(uint32_t a) {
    uint16_t v; asm("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory"); return __half2float(__ushort_as_half(v));
}
__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
    unsigned long long v; asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory"); return v;
}
__device__ __forceinline__ uint32_t lo16(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x5410); }
__device__ __forceinline__ uint32_t hi16(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x7632); }

// 16-byte piece c of weight row r of a slot sits at piece position c ^ row_swizzle(r): the rows a shared-memory read
// touches together (2 for 16-byte, 4 for 8-byte, 8 for 4-byte reads) then fall into different banks.
__device__ __forceinline__ int row_swizzle(int r) { return ((r & 1) << 2) | (r & 2) | ((r >> 2) & 1); }

constexpr uint32_t kOnesF16 = 0x3C003C00u, kOnesU8 = 0x01010101u;

template <int FMT> struct Fmt {
    static constexpr int BITS = FMT <= kInt2G64 ? 2 : 4;
    static constexpr int NG = FMT == kInt2G64 || FMT == kInt4G64 ? 2 : FMT == kInt4G32 ? 4 : 1;   // scale groups per 128 columns
    static constexpr int KB = BITS == 2 ? 4 : 2;                  // 128-column blocks per slot
    static constexpr int W = BITS == 2 ? 2 : 4;                   // code words per lane, row and block
    static constexpr int WG = W / NG;                             // ... per scale group
};

// Two 16-byte pieces of x (16 consecutive columns) in fragment order: INT4 pairs columns (j, j+4) of each piece, INT2 pairs
// (j, j+8) of both, which is how the codes sit in the two halves of a masked word.
template <int BITS>
__device__ __forceinline__ void to_frag_order(uint4& a, uint4& b) {
    if constexpr (BITS == 4) {
        a = make_uint4(lo16(a.x, a.z), lo16(a.y, a.w), hi16(a.x, a.z), hi16(a.y, a.w));
        b = make_uint4(lo16(b.x, b.z), lo16(b.y, b.w), hi16(b.x, b.z), hi16(b.y, b.w));
    } else {
        const uint4 p = make_uint4(lo16(a.x, b.x), lo16(a.z, b.z), hi16(a.x, b.x), hi16(a.z, b.z));
        b = make_uint4(lo16(a.y, b.y), lo16(a.w, b.w), hi16(a.y, b.y), hi16(a.w, b.w));
        a = p;
    }
}

// Sum of x over each scale group of the block, for this lane's activation columns 2t and 2t+1.
template <int FMT>
__device__ __forceinline__ void group_sums(const uint32_t (&fr)[16], const float (&zero)[4], float2 (&sx)[Fmt<FMT>::NG]) {
    constexpr int PER = 8 / Fmt<FMT>::NG;             // B pairs per group
#pragma unroll
    for (int j = 0; j < Fmt<FMT>::NG; ++j) {
        float a[4];
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const uint32_t b0 = fr[(j * PER + i) * 2], b1 = fr[(j * PER + i) * 2 + 1];
            if (i == 0) mma_f16(a, kOnesF16, kOnesF16, kOnesF16, kOnesF16, b0, b1, zero);
            else mma_f16(a, kOnesF16, kOnesF16, kOnesF16, kOnesF16, b0, b1);
        }
        sx[j] = make_float2(a[0], a[1]);
    }
}

__device__ __forceinline__ float4 lds128f(uint32_t a) {
    float4 v; asm("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory"); return v;
}
template <bool BF16>
__device__ __forceinline__ void widen8(const uint4& v, float* f) {
    using XT = typename Act16<BF16>::T;
    const XT* e = reinterpret_cast<const XT*>(&v);
#pragma unroll
    for (int q = 0; q < 8; ++q) f[q] = Act16<BF16>::to_float(e[q]);
}
// Exponent of a block's largest magnitude (given as float bits), limited to where 2^(30 - e) and 2^(e - 29) are normal.
__device__ __forceinline__ int block_exponent(uint32_t bits) { return max(-96, (int)(bits >> 23) - 127); }
__device__ __forceinline__ float pow2f(int e) { return __int_as_float((e + 127) << 23); }
constexpr uint32_t kInfBits = 0x7f800000u;

}  // namespace
}  // namespace qgemv
