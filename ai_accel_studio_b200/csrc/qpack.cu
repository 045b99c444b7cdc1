// Groupwise INT2 / INT4 quantisation of a weight matrix: scale search, codes and packing in one pass.
//
// The torch expression of the same algorithm (kernels/groupwise_int2.py, groupwise_int4.py) makes a temporary of the
// matrix's size for every step of every candidate scale -- some 150 passes over memory at 13 candidates.  Here a group's
// weights stay in registers: 16 consecutive columns per lane (times V for groups above 128), 2 - 8 lanes per group.  Bound
// by instruction issue, not by HBM: 126 M warp instructions for 4096 x 4096 INT2, 18 per weight and candidate, at 63 % of the
// issue slots with 12 warps an SM.
// Measured, 4096 x 4096 INT2 with activation statistics (B200): torch expression 17.7 ms; 349 us with a decision per weight
// by quotient or estimate; 228 us with the decision per candidate as below.
//
// Results are the expression's own: every operation is rounded as there (IEEE division, no contraction), and the squared
// errors are added in the order in which the framework's reduction adds a contiguous row (four neighbours, then a binary
// tree), so equal candidates are resolved alike.  Quotients are only computed for a candidate with an estimate too close to
// a decision boundary to be sure (margins an order above the estimates' error); everywhere else |w| / s is estimated, and
// the error follows from magnitudes alone: levels are symmetric.
#include "qgemv_common.cuh"

namespace qgemv {
namespace {

constexpr float kThird = 0.3333333432674408f;         // float32(1/3)

// Index of the closest level of x in (-1, -1/3, 1/3, 1), the first one on ties of the rounded distances.
__device__ __noinline__ int closest_exact(float x) {
    const float d0 = fabsf(__fsub_rn(x, -1.0f)), d1 = fabsf(__fsub_rn(x, -kThird)), d2 = fabsf(__fsub_rn(x, kThird)), d3 = fabsf(__fsub_rn(x, 1.0f));
    int c = 0;
    float best = d0;
    if (d1 < best) { best = d1; c = 1; }
    if (d2 < best) { best = d2; c = 2; }
    if (d3 < best) c = 3;
    return c;
}
__device__ __noinline__ int round4_exact(float w, float s) {
    return (int)fminf(fmaxf(rintf(__fdiv_rn(w, s)), -8.0f), 7.0f);
}
// Code of w at scale s, exactly as the torch expression rounds it.
template <int BITS>
__device__ __forceinline__ int code_exact(float w, float s, bool clamp1) {
    if constexpr (BITS == 2) {
        float x = __fdiv_rn(w, s);
        if (clamp1) x = fminf(fmaxf(x, -1.0f), 1.0f);
        return closest_exact(x);
    } else {
        return round4_exact(w, s);
    }
}
template <int BITS> __device__ __forceinline__ float level_of(int c) {
    if constexpr (BITS == 2) return c == 0 ? -1.0f : c == 1 ? -kThird : c == 2 ? kThird : 1.0f;
    else return (float)c;
}
// Magnitude of a = |w| quantised at scale cand (cand3 = cand / 3, edge = 2 / 3 cand, inv ~ 1 / cand), and by how much a
// misses the nearest decision boundary (INT2: in units of w, INT4: of cand).  INT2's boundary at 0 (level -1/3 wins the tie)
// changes the sign only of values that are handled apart (`tiny`).
template <int BITS>
__device__ __forceinline__ float magnitude(float a, float w, float cand, float cand3, float edge, float inv, float& margin) {
    if constexpr (BITS == 2) {
        margin = fminf(margin, fabsf(a - edge));
        return a > edge ? cand : cand3;
    } else {
        const float t = a * inv, r = (t + 12582912.0f) - 12582912.0f;      // round to nearest even
        margin = fminf(margin, fabsf(fabsf(t - r) - 0.5f));
        return __fmul_rn(fminf(r, w < 0.0f ? 8.0f : 7.0f), cand);
    }
}
constexpr float kMargin = 1e-5f;

// max(x, 1e-8) that leaves NaN as it is, as the framework's clamp does.
__device__ __forceinline__ float at_least_tiny(float x) { return x < 1e-8f ? 1e-8f : x; }

template <int DT> __device__ __forceinline__ float load_w(const void* w, size_t i) {
    if constexpr (DT == QGEMV_F16) return __half2float(static_cast<const __half*>(w)[i]);
    else if constexpr (DT == QGEMV_BF16) return __bfloat162float(static_cast<const __nv_bfloat16*>(w)[i]);
    else return static_cast<const float*>(w)[i];
}

// lg lanes per group, each 16 consecutive columns of every 128 (V of them).
template <int BITS, int V, int DT>
__global__ void __launch_bounds__(256) pack_kernel(const void* __restrict__ w, long long ldw, int n, int k, int ng, int group, int lg,
                                                   const float* __restrict__ rms, const float* __restrict__ factors, int steps,
                                                   uint8_t* __restrict__ packed, __half* __restrict__ scales, bool vec, bool vec_rms) {
    const long long groups = (long long)n * ng;
    const int per_block = 256 / lg;
    const int sub = threadIdx.x / lg, l = threadIdx.x - sub * lg;
    const long long trips = (groups + per_block - 1) / per_block;
    const int row_bytes = ng * group * BITS / 8;
    for (long long trip = blockIdx.x; trip < trips; trip += gridDim.x) {
        const long long gi = min(trip * per_block + sub, groups - 1);       // the last block repeats a group: shuffles stay converged
        const int row = (int)(gi / ng), grp = (int)(gi - (long long)row * ng);
        float f[V][16], aw[V][16], tiny = 3.0e38f;                          // tiny: smallest magnitude that is not zero
        uint32_t peak_bits = 0;                                             // largest magnitude; by its bits, above which NaN's are
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int k0 = grp * group + v * 128 + l * 16;
            if (vec && k0 + 16 <= k) {
                if constexpr (DT == QGEMV_F32) {
                    const float4* src = reinterpret_cast<const float4*>(static_cast<const float*>(w) + (size_t)row * ldw + k0);
#pragma unroll
                    for (int q = 0; q < 4; ++q) { const float4 a = src[q]; f[v][q * 4] = a.x; f[v][q * 4 + 1] = a.y; f[v][q * 4 + 2] = a.z; f[v][q * 4 + 3] = a.w; }
                } else {
                    const uint4* src = reinterpret_cast<const uint4*>(static_cast<const __half*>(w) + (size_t)row * ldw + k0);
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const uint4 a = src[q];
#pragma unroll
                        for (int e = 0; e < 8; ++e) f[v][q * 8 + e] = load_w<DT>(&a, e);
                    }
                }
            } else {
#pragma unroll
                for (int e = 0; e < 16; ++e) f[v][e] = k0 + e < k ? load_w<DT>(w, (size_t)row * ldw + k0 + e) : 0.0f;
            }
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                peak_bits = max(peak_bits, __float_as_uint(fabsf(f[v][e])));
                tiny = f[v][e] != 0.0f ? fminf(tiny, fabsf(f[v][e])) : tiny;
            }
            if (rms) {
                const bool whole = k0 + 16 <= k && vec_rms;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
                    const int c = k0 + q * 4;
                    if (whole) a = __ldg(reinterpret_cast<const float4*>(rms + c));
                    else { if (c < k) a.x = rms[c]; if (c + 1 < k) a.y = rms[c + 1]; if (c + 2 < k) a.z = rms[c + 2]; if (c + 3 < k) a.w = rms[c + 3]; }
                    aw[v][q * 4] = at_least_tiny(__fmul_rn(a.x, a.x)); aw[v][q * 4 + 1] = at_least_tiny(__fmul_rn(a.y, a.y));
                    aw[v][q * 4 + 2] = at_least_tiny(__fmul_rn(a.z, a.z)); aw[v][q * 4 + 3] = at_least_tiny(__fmul_rn(a.w, a.w));
                }
            }
        }
        for (int o = 1; o < lg; o <<= 1) peak_bits = max(peak_bits, __shfl_xor_sync(0xffffffffu, peak_bits, o));
        const float peak = __uint_as_float(peak_bits), base = at_least_tiny(BITS == 2 ? peak : __fmul_rn(peak, 1.0f / 7.0f));
        float chosen = base;
        if (rms) {
            float best = 0.0f;
            for (int s = 0; s < steps; ++s) {
                const float cand = __fmul_rn(base, factors[s]);
                const float div = BITS == 2 ? fmaxf(cand, 1e-8f) : cand, inv = __fdividef(1.0f, div);
                const float cand3 = __fmul_rn(kThird, cand), edge = 0.6666667f * div;
                float e4[4][4];                        // [neighbour quadruple][element]: the framework's per-thread accumulators
                float margin = BITS == 2 ? tiny : 1.0f;
#pragma unroll
                for (int v = 0; v < V; ++v)
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        const float a = fabsf(f[v][e]);
                        const float d = __fsub_rn(magnitude<BITS>(a, f[v][e], cand, cand3, edge, inv, margin), a);
                        const float x = __fmul_rn(__fmul_rn(d, d), aw[v][e]);
                        e4[e >> 2][e & 3] = v == 0 ? x : __fadd_rn(e4[e >> 2][e & 3], x);
                    }
                if (margin < (BITS == 2 ? kMargin * div : kMargin)) {       // rare: this lane's columns again, by quotients
#pragma unroll 1
                    for (int e = 0; e < 16; ++e) {
                        float x = 0.0f;
#pragma unroll
                        for (int v = 0; v < V; ++v) {
                            float w1 = 0.0f, b = 0.0f;
#pragma unroll
                            for (int i = 0; i < 16; ++i) if (i == e) { w1 = f[v][i]; b = aw[v][i]; }
                            const float d = __fsub_rn(__fmul_rn(level_of<BITS>(code_exact<BITS>(w1, div, false)), cand), w1);
                            const float y = __fmul_rn(__fmul_rn(d, d), b);
                            x = v == 0 ? y : __fadd_rn(x, y);
                        }
#pragma unroll
                        for (int i = 0; i < 16; ++i) if (i == e) e4[i >> 2][i & 3] = x;
                    }
                }
                float t[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) t[q] = __fadd_rn(__fadd_rn(__fadd_rn(e4[q][0], e4[q][1]), e4[q][2]), e4[q][3]);
                float err = __fadd_rn(__fadd_rn(t[0], t[1]), __fadd_rn(t[2], t[3]));
                for (int o = 1; o < lg; o <<= 1) err = __fadd_rn(err, __shfl_xor_sync(0xffffffffu, err, o));
                if (s == 0 || err < best) { best = err; chosen = cand; }
            }
        }
        if (l == 0) scales[(size_t)row * ng + grp] = __float2half_rn(chosen);
#pragma unroll
        for (int v = 0; v < V; ++v) {
            uint32_t word[BITS == 2 ? 1 : 2];
#pragma unroll
            for (int i = 0; i < (BITS == 2 ? 1 : 2); ++i) {
                word[i] = 0;
#pragma unroll
                for (int e = 0; e < 32 / BITS; ++e) {
                    const int c = code_exact<BITS>(f[v][i * (32 / BITS) + e], chosen, true) + (BITS == 4 ? 8 : 0);
                    word[i] |= (uint32_t)c << (BITS * e);
                }
            }
            uint8_t* out = packed + (size_t)row * row_bytes + (size_t)(grp * group + v * 128 + l * 16) * BITS / 8;
            if constexpr (BITS == 2) *reinterpret_cast<uint32_t*>(out) = word[0];
            else *reinterpret_cast<uint2*>(out) = make_uint2(word[0], word[1]);
        }
    }
}

}  // namespace
}  // namespace qgemv

using namespace qgemv;

extern "C" int qgemv_pack(int bits, const void* w, int64_t ldw, int w_dtype, int n, int k, int group, const float* rms, const float* factors,
                          int steps, uint8_t* packed, void* scales, void* stream) {
    if (!w || !packed || !scales || n < 1 || k < 1 || ldw < k || (bits != 2 && bits != 4) || w_dtype < QGEMV_F16 || w_dtype > QGEMV_F32 ||
        (rms && (!factors || steps < 1))) {
        set_error("qgemv_pack: null pointer, non-positive size or bad type");
        return QGEMV_ERR_BAD_ARG;
    }
    const int v = group <= 128 ? 1 : group / 128, lg = group <= 128 ? group / 16 : 8;
    if (group < 16 || group % 16 || (group <= 128 ? (lg & (lg - 1)) != 0 : group % 128 != 0 || (v != 2 && v != 4))) {
        set_error("qgemv_pack: group=%d (16, 32, 64, 128, 256 and 512 are built)", group);
        return QGEMV_ERR_SHAPE;
    }
    if (reinterpret_cast<uintptr_t>(packed) % 8) { set_error("qgemv_pack: packed must be 8-byte aligned"); return QGEMV_ERR_ALIGN; }
    const int ng = (k + group - 1) / group;
    const int esize = w_dtype == QGEMV_F32 ? 4 : 2;
    const bool vec = reinterpret_cast<uintptr_t>(w) % 16 == 0 && ldw * esize % 16 == 0;
    const long long trips = ((long long)n * ng + 256 / lg - 1) / (256 / lg);
    const int grid = (int)(trips < 148 * 16 ? trips : 148 * 16);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    __half* sc = static_cast<__half*>(scales);
#define QP(B, V, D) pack_kernel<B, V, D><<<grid, 256, 0, s>>>(w, ldw, n, k, ng, group, lg, rms, factors, steps, packed, sc, vec, reinterpret_cast<uintptr_t>(rms) % 16 == 0)
#define QP_D(B, V) do { if (w_dtype == QGEMV_F16) QP(B, V, QGEMV_F16); else if (w_dtype == QGEMV_BF16) QP(B, V, QGEMV_BF16); else QP(B, V, QGEMV_F32); } while (0)
#define QP_V(B) do { if (v == 1) QP_D(B, 1); else if (v == 2) QP_D(B, 2); else QP_D(B, 4); } while (0)
    if (bits == 2) QP_V(2); else QP_V(4);
#undef QP_V
#undef QP_D
#undef QP
    return check_launch("pack_kernel");
}
