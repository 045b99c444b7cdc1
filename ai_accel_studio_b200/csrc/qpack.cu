// Groupwise INT2 / INT4 quantisation of a weight matrix: scale search, codes and packing in one pass.
//
// The torch expression of the same algorithm (kernels/groupwise_int2.py, groupwise_int4.py) makes a temporary of the
// matrix's size for every step of every candidate scale -- some 150 passes over memory at 13 candidates.  Here a group's
// weights stay in registers: 16 consecutive columns per lane (times V for groups above 128), 2 - 8 lanes per group.  Bound
// by instructions, not by HBM: 8192 x 8192 INT2 takes 202 M warp instructions at 70 % of the issue slots with 28 warps an SM,
// INT4 358 M at 78 % with 21 (groups of 128).
// Measured, 4096 x 4096 with activation statistics (B200): torch expression 17.7 ms; INT2 225 us with a decision per weight and
// candidate, 74 us as below; INT4 172 and 105; without statistics 41 and 22 - 23.  More than 16 candidates, all compared exactly: 40 of INT2
// 532 and 360, of INT4 449 and 430.
//
// Results are the expression's own: where it matters every operation is rounded as there (IEEE division, no contraction), and
// the squared errors are added in the order in which the framework's reduction adds a contiguous row (four neighbours, then a
// binary tree), so equal candidates are resolved alike.  But it rarely matters.  The candidates' errors are estimated first --
// INT2: from a histogram of the weights over all candidates' decision boundaries, one pass instead of thirteen; INT4: candidate by
// candidate, without looking at how close a decision was -- and only candidates that the estimate cannot tell apart are compared
// by the exact sums (exact_search).  Codes likewise: a quotient only where the estimate is too close to a decision boundary.
#include "qgemv_common.cuh"

namespace qgemv {
namespace {

constexpr float kThird = 0.3333333432674408f;         // float32(1/3)
constexpr float kMagic = 12582912.0f;                 // 1.5 * 2^23: adding and subtracting it rounds to an integer

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
// Distance of w from its level at scale cand (cand3 = cand / 3, edge = 2 / 3 cand, inv ~ 1 / cand), up to its sign, and in `miss` how near w
// comes to a decision boundary: INT2 the smallest distance from one, INT4 the largest distance of |w| / cand from an integer.
// INT2's boundary at 0 (level -1/3 wins the tie) changes the sign only of values that are handled apart (kTiny).
template <int BITS>
__device__ __forceinline__ float distance(float w, float cand, float cand3, float edge, float inv, float& miss) {
    if constexpr (BITS == 2) {
        const float a = fabsf(w);
        miss = fminf(miss, fabsf(a - edge));
        return __fsub_rn(a > edge ? cand : cand3, a);
    } else {
        const float t = w * inv, r = (t + kMagic) - kMagic;                // round to nearest even
        miss = fmaxf(miss, fabsf(t - r));
        return __fsub_rn(__fmul_rn(fminf(fmaxf(r, -8.0f), 7.0f), cand), w);
    }
}
// Closer to a boundary than this (of the scale) the quotient decides.  INT2: quotient, distances and edge are rounded within 2e-7; INT4: the
// last boundary is 7.5, where products with a reciprocal from reciprocal() and quotients differ by up to 3 units of 2^-24, 1.4e-6.  A positive quotient of 2^-25 and more is nearer to the level
// 1/3 than to -1/3 after rounding, too: only below kTiny may the first one win.
template <int BITS> constexpr float kMargin = BITS == 2 ? 1e-6f : 2e-6f;
constexpr float kTiny = 6e-8f;

// 1 / x within 2^-24 of itself (1e-8 <= x < 2^126).
__device__ __forceinline__ float reciprocal(float x) {
    const float near = __fdividef(1.0f, x);            // within 2^-22
    return fmaf(fmaf(-x, near, 1.0f), near, near);
}

// Code of w at scale s (edge = 2 / 3 s, inv ~ 1 / s) by estimate; false if it is too close to a decision boundary to be sure.
template <int BITS>
__device__ __forceinline__ bool code_estimate(float w, float s, float edge, float inv, int& c) {
    const float a = fabsf(w);
    if constexpr (BITS == 2) {
        const int hi = a > edge ? 1 : 0;
        c = a == 0.0f ? 1 : w < 0.0f ? 1 - hi : 2 + hi;                    // level -1/3 wins the tie at zero
        return (a == 0.0f || a > kTiny * s) && fabsf(a - edge) > kMargin<2> * s;
    } else {
        const float t = a * inv, r = (t + kMagic) - kMagic;
        c = w < 0.0f ? -(int)fminf(r, 8.0f) : (int)fminf(r, 7.0f);
        return fabsf(fabsf(t - r) - 0.5f) > kMargin<4> && t < 65536.0f;
    }
}

// Candidates whose estimated errors exceed the smallest one by no more than kErrorShare of it plus kEnergyShare of the group's energy
// N = sum of aw w^2 are compared by their exact errors E.  What separates estimates and exact errors (u = 2^-24):
// INT4: the expression rounds the level times the candidate, which can change E by 2 u sqrt(E N), 4 u sqrt(E N) <= 28 u E + u N / 7 for two
//   candidates; it decides by a rounded quotient, the estimate by a reciprocal within u, so that a weight within 16 u of a decision
//   boundary may get the other level, which changes its term by 128 u; the sums' roundings come to a few u E.  (With 1e-5 E alone, no N and
//   a reciprocal within 4 u, the best of two candidates was dropped whose levels lie on either side of a weight, close to it.)
// INT2: the estimate is a sum of terms of up to 12.5 N + 4 E altogether, since the weights below a decision boundary enter by
//   aw s^2 / 9 <= 2 aw (s / 3 - |w|)^2 + 2 aw w^2.  They are sums of up to 16 V + 17 steps, whose roundings (not their bound, which is
//   tenfold) come to 1 - 1.5 u of a term: some 4 u E + 12 u N between two candidates, a tenth of what is allowed for.  A weight on the wrong side of a
//   boundary lies within 25 u of it and changes its term by 50 u aw w^2.
constexpr float kErrorShare = 1e-5f;
template <int BITS> constexpr float kEnergyShare = BITS == 4 ? 1e-8f : 1e-5f;
constexpr int kMaxFast = 16;                          // most candidates of a search by estimates

// First candidate, and candidates per unit, if they are evenly spaced, ascending and positive; else {0, 0}.  A lane checks one of at most
// kMaxFast, so that small matrices wait for one load, not for a row of them.  All lanes of the warp call it.
__device__ __forceinline__ float2 even_grid(const float* factors, int steps) {
    const float f0 = factors[0], h = (factors[steps - 1] - f0) / (float)max(steps - 1, 1);
    const int s = min((int)(threadIdx.x & 31), steps - 1);
    const bool even = steps > 1 && f0 > 0.0f && h > 1e-3f && fabsf(factors[s] - (f0 + s * h)) <= 5e-7f * factors[steps - 1];
    return __all_sync(0xffffffffu, even) ? make_float2(f0, 1.0f / h) : make_float2(0.0f, 0.0f);
}

// max(x, 1e-8) that leaves NaN as it is, as the framework's clamp does.
__device__ __forceinline__ float at_least_tiny(float x) { return x < 1e-8f ? 1e-8f : x; }

template <int DT> __device__ __forceinline__ float load_w(const void* w, size_t i) {
    if constexpr (DT == QGEMV_F16) return __half2float(static_cast<const __half*>(w)[i]);
    else if constexpr (DT == QGEMV_BF16) return __bfloat162float(static_cast<const __nv_bfloat16*>(w)[i]);
    else return static_cast<const float*>(w)[i];
}

struct PackArgs {
    const void* w;            long long ldw;
    const float* rms;         const float* factors;           // factors NULL: evenly spaced, made by every block itself
    float first, last, spacing;
    uint8_t* packed;          __half* scales;
    int n, k, ng, group, lg, steps;           // lg: lanes per group, each 16 consecutive columns of every 128
    bool vec, vec_rms;                        // 16-byte loads of w, rms
};

// Sixteen weights of a row from column k0, zero past the last one.
template <int DT>
__device__ __forceinline__ void load_weights(const PackArgs& p, int row, int k0, float (&f)[16]) {
    if (p.vec && k0 + 16 <= p.k) {
        if constexpr (DT == QGEMV_F32) {
            const float4* src = reinterpret_cast<const float4*>(static_cast<const float*>(p.w) + (size_t)row * p.ldw + k0);
#pragma unroll
            for (int q = 0; q < 4; ++q) { const float4 a = src[q]; f[q * 4] = a.x; f[q * 4 + 1] = a.y; f[q * 4 + 2] = a.z; f[q * 4 + 3] = a.w; }
        } else {
            const uint4* src = reinterpret_cast<const uint4*>(static_cast<const __half*>(p.w) + (size_t)row * p.ldw + k0);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const uint4 a = src[q];
#pragma unroll
                for (int e = 0; e < 8; ++e) f[q * 8 + e] = load_w<DT>(&a, e);
            }
        }
    } else {
#pragma unroll
        for (int e = 0; e < 16; ++e) f[e] = k0 + e < p.k ? load_w<DT>(p.w, (size_t)row * p.ldw + k0 + e) : 0.0f;
    }
}
// What the squared errors of four columns from c count: the square of the statistics, at least 1e-8.
__device__ __forceinline__ float4 load_energy(const PackArgs& p, int c) {
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p.vec_rms && c + 4 <= p.k) a = __ldg(reinterpret_cast<const float4*>(p.rms + c));
    else { if (c < p.k) a.x = p.rms[c]; if (c + 1 < p.k) a.y = p.rms[c + 1]; if (c + 2 < p.k) a.z = p.rms[c + 2]; if (c + 3 < p.k) a.w = p.rms[c + 3]; }
    return make_float4(at_least_tiny(__fmul_rn(a.x, a.x)), at_least_tiny(__fmul_rn(a.y, a.y)), at_least_tiny(__fmul_rn(a.z, a.z)), at_least_tiny(__fmul_rn(a.w, a.w)));
}

// A lane's share of the squared errors of a candidate, decided by quotients: weights and statistics are loaded one by one, because the
// callers have them in registers, which cannot be indexed.
template <int BITS, int V, int DT>
__device__ __noinline__ float error_by_quotients(const PackArgs& p, int row, int k0, float cand, float div) {
    float t[4];
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
        float sum = 0.0f;
#pragma unroll 1
        for (int e = 0; e < 4; ++e) {
            float x = 0.0f;
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const int k = k0 + v * 128 + q * 4 + e;
                const float w = k < p.k ? load_w<DT>(p.w, (size_t)row * p.ldw + k) : 0.0f, a = k < p.k ? p.rms[k] : 0.0f;
                const float d = __fsub_rn(__fmul_rn(level_of<BITS>(code_exact<BITS>(w, div, false)), cand), w);
                const float y = __fmul_rn(__fmul_rn(d, d), at_least_tiny(__fmul_rn(a, a)));
                x = v == 0 ? y : __fadd_rn(x, y);
            }
            sum = e == 0 ? x : __fadd_rn(sum, x);
        }
        if (q == 0) t[0] = sum; else if (q == 1) t[1] = sum; else if (q == 2) t[2] = sum; else t[3] = sum;
    }
    return __fadd_rn(__fadd_rn(t[0], t[1]), __fadd_rn(t[2], t[3]));
}

// The best of the candidates in `mine`, by errors in which every operation is rounded as in the expression.  `visit`: the
// candidates of all groups of the warp (the shuffles need it converged).  Out of line, with loads of its own: of
// normal weights in groups of 128, one group in 700 (INT2, 13 candidates) or in 12 000 (INT4, 11) needs it, and its registers
// would halve the number of warps.  A column's terms are added up as they are made: kept until it is known whether a decision was
// close, they would not fit the registers beside weights and energies.
template <int BITS, int V, int DT>
__device__ __noinline__ float exact_search(const PackArgs& p, const float* factors, int row, int k0, float base, uint32_t visit, uint32_t mine, bool every) {
    float f[V][16], aw[V][16], tiny = 3.0e38f;         // tiny: smallest magnitude that is not zero
#pragma unroll
    for (int v = 0; v < V; ++v) {
        load_weights<DT>(p, row, k0 + v * 128, f[v]);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 a = load_energy(p, k0 + v * 128 + q * 4);
            aw[v][q * 4] = a.x; aw[v][q * 4 + 1] = a.y; aw[v][q * 4 + 2] = a.z; aw[v][q * 4 + 3] = a.w;
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) tiny = f[v][e] != 0.0f ? fminf(tiny, fabsf(f[v][e])) : tiny;
    }
    const int steps = p.steps, lg = p.lg;
    float best = 0.0f, chosen = base;
    bool first = true;
#pragma unroll 1
    for (int s = 0; s < steps; ++s) {
        if (!every && !(visit >> s & 1)) continue;
        const float cand = __fmul_rn(base, factors[s]);
        const float div = BITS == 2 ? fmaxf(cand, 1e-8f) : cand, inv = BITS == 2 ? 0.0f : reciprocal(div);
        const float cand3 = __fmul_rn(kThird, cand), edge = 0.6666667f * div;
        float miss = BITS == 2 ? 3.0e38f : 0.0f, t[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)                    // the framework's per-thread accumulators: four neighbours, V of each
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float x = 0.0f;
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    const float d = distance<BITS>(f[v][q * 4 + e], cand, cand3, edge, inv, miss);
                    const float y = __fmul_rn(__fmul_rn(d, d), aw[v][q * 4 + e]);
                    x = v == 0 ? y : __fadd_rn(x, y);
                }
                t[q] = e == 0 ? x : __fadd_rn(t[q], x);
            }
        float err = __fadd_rn(__fadd_rn(t[0], t[1]), __fadd_rn(t[2], t[3]));
        const bool unsure = BITS == 2 ? miss < kMargin<2> * div || tiny < kTiny * div : miss > 0.5f - kMargin<4>;
        if (unsure) err = error_by_quotients<BITS, V, DT>(p, row, k0, cand, div);       // rare
        for (int o = 1; o < lg; o <<= 1) err = __fadd_rn(err, __shfl_xor_sync(0xffffffffu, err, o));
        if (!every && !(mine >> s & 1)) continue;
        if (first || err < best) { best = err; chosen = cand; }
        first = false;
    }
    return chosen;
}

// Blocks of an SM, by registers: what a thread keeps is its weights.  4096 x 4096 fp16 with these / with one block fewer, us: INT4 groups of 128
// 106 / 114, 256 95 / 111; INT2 512 76 / 80.  INT2 up to 256 spills 208 bytes of stores a thread and more with one block more than
// here: 128 72.5 against 67, 64 81 against 77, 1024 x 1024 13.1 against 9.6.
__host__ __device__ constexpr int pack_blocks(int bits, int v) { return v == 1 ? 3 : v == 2 ? 2 : bits == 2 ? 2 : 1; }

// SEARCH: there are statistics, the scale is searched for.
template <int BITS, int V, int DT, bool SEARCH>
__global__ void __launch_bounds__(256, pack_blocks(BITS, V)) pack_kernel(const __grid_constant__ PackArgs p) {
    __shared__ float2 bins[SEARCH && BITS == 2 ? (kMaxFast + 1) * 256 : 1];        // INT2: [bin][thread], (sum aw, sum aw |w|) of the thread's columns
    [[maybe_unused]] float2* const mine = bins + (SEARCH && BITS == 2 ? threadIdx.x : 0);
    const int lg = p.lg, steps = p.steps;
    // Evenly spaced candidates as torch.linspace spaces them (from both ends, one rounding), without a launch that makes them.
    __shared__ float spaced[SEARCH ? QGEMV_PACK_MAX_SPACED : 1];
    const float* factors = p.factors;
    if (SEARCH && !factors) {
        const int s = threadIdx.x;
        if (s < steps) spaced[s] = s < steps / 2 || steps == 1 ? __fmaf_rn(p.spacing, (float)s, p.first) : __fmaf_rn(-p.spacing, (float)(steps - 1 - s), p.last);
        __syncthreads();
        factors = spaced;
    }
    float2 grid = make_float2(0.0f, 0.0f);
    if (SEARCH && steps <= kMaxFast) grid = even_grid(factors, steps);
    const long long groups = (long long)p.n * p.ng;
    const int per_block = 256 / lg;
    const int sub = threadIdx.x / lg, l = threadIdx.x - sub * lg;
    const long long trips = (groups + per_block - 1) / per_block;
    const int row_bytes = p.ng * p.group * BITS / 8;
    auto row_of = [&](long long i) { return groups < 0x80000000ll ? (int)((uint32_t)i / (uint32_t)p.ng) : (int)(i / p.ng); };
    for (long long trip = blockIdx.x; trip < trips; trip += gridDim.x) {
        const long long gi = min(trip * per_block + sub, groups - 1);       // the last block repeats a group: shuffles stay converged
        const int row = row_of(gi), grp = (int)(gi - (long long)row * p.ng), k0 = grp * p.group + l * 16;
        if (trip + gridDim.x < trips) {                // the next trip's weights to L2 meanwhile
            const long long gn = min((trip + gridDim.x) * per_block + sub, groups - 1);
            const int rn = row_of(gn), kn = (int)(gn - (long long)rn * p.ng) * p.group + l * 16;
            if (kn < p.k) asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const char*>(p.w) + ((size_t)rn * p.ldw + kn) * (DT == QGEMV_F32 ? 4 : 2)));
        }
        float f[V][16];
        uint32_t peak_bits = 0;                                             // largest magnitude; by its bits, above which NaN's are
#pragma unroll
        for (int v = 0; v < V; ++v) {
            load_weights<DT>(p, row, k0 + v * 128, f[v]);
#pragma unroll
            for (int e = 0; e < 16; ++e) peak_bits = max(peak_bits, __float_as_uint(fabsf(f[v][e])));
        }
        for (int o = 1; o < lg; o <<= 1) peak_bits = max(peak_bits, __shfl_xor_sync(0xffffffffu, peak_bits, o));
        const float peak = __uint_as_float(peak_bits), base = at_least_tiny(BITS == 2 ? peak : __fmul_rn(peak, 1.0f / 7.0f));
        float chosen = base;
        if constexpr (SEARCH) {
            // ---- which candidates can have the smallest error (a bit each), by estimates -------------------------
            uint32_t contenders = 0xffffffffu;
            const bool fast = grid.y > 0.0f;
            if (fast) {
                float lowest = 3.0e38f;
                if constexpr (BITS == 2) {
                    // The error of a candidate s follows from A = sum aw and B = sum aw |w| over |w| > 2/3 s: those take the level s,
                    // the others s / 3.  A histogram over all candidates' boundaries gives every A and B in one pass.
                    const float c1 = 1.5f * grid.y / base, c0 = 0.5f - grid.x * grid.y;      // rounds to the number of boundaries below
                    __syncwarp();                       // the group's lanes have read the previous group's sums
                    for (int s = 0; s <= steps; ++s) mine[s * 256] = make_float2(0.0f, 0.0f);
                    float energy = 0.0f;
#pragma unroll
                    for (int v = 0; v < V; ++v)
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const float4 x4 = load_energy(p, k0 + v * 128 + q * 4);
                            const float x[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const float a = fabsf(f[v][q * 4 + e]), xa = x[e] * a, t = fminf(fmaxf(fmaf(a, c1, c0), 0.0f), (float)steps);
                                float2* const at = mine + (__float_as_int(t + kMagic) - __float_as_int(kMagic)) * 256;
                                const float2 h = *at;
                                *at = make_float2(h.x + x[e], h.y + xa);
                                energy = fmaf(xa, a, energy);
                            }
                        }
                    for (int o = 1; o < lg; o <<= 1) energy += __shfl_xor_sync(0xffffffffu, energy, o);
                    // sums from the top: lane l adds bin hi - l over the group's lanes, a scan over the lanes does the rest
                    float2* const lane0 = mine - l;
                    float2 carry = make_float2(0.0f, 0.0f);
                    __syncwarp();
                    for (int hi = steps; hi >= 0; hi -= lg) {
                        const int b = hi - l;
                        float2 r = make_float2(0.0f, 0.0f);
                        if (b >= 0)
                            for (int i = 0; i < lg; ++i) { const float2 h = lane0[b * 256 + ((l + i) & (lg - 1))]; r.x += h.x; r.y += h.y; }
                        for (int o = 1; o < lg; o <<= 1) {
                            const float x = __shfl_up_sync(0xffffffffu, r.x, o, lg), y = __shfl_up_sync(0xffffffffu, r.y, o, lg);
                            if (l >= o) { r.x += x; r.y += y; }
                        }
                        r.x += carry.x; r.y += carry.y;
                        carry = make_float2(__shfl_sync(0xffffffffu, r.x, lg - 1, lg), __shfl_sync(0xffffffffu, r.y, lg - 1, lg));
                        __syncwarp();
                        if (b >= 0) lane0[b * 256] = r;
                    }
                    __syncwarp();
                    auto error = [&](int s) {           // carry: the totals
                        const float2 r = lane0[(s + 1) * 256];
                        const float cand = base * factors[s], third = cand * kThird, ra = carry.x - r.x, rb = carry.y - r.y;
                        return fmaf(cand, fmaf(cand, r.x, -2.0f * r.y), fmaf(third, fmaf(third, ra, -2.0f * rb), energy));
                    };
                    for (int s = l; s < steps; s += lg) lowest = fminf(lowest, error(s));
                    for (int o = 1; o < lg; o <<= 1) lowest = fminf(lowest, __shfl_xor_sync(0xffffffffu, lowest, o));
                    const float reach = lowest + (kErrorShare * lowest + kEnergyShare<BITS> * energy);
                    contenders = 0;
                    for (int s = l; s < steps; s += lg) contenders |= (error(s) <= reach ? 1u : 0u) << s;
                    for (int o = 1; o < lg; o <<= 1) contenders |= __shfl_xor_sync(0xffffffffu, contenders, o);
                    // No estimate: out of range; sums of aw that overflowed where those of aw w^2 did not; candidates below 1e-8,
                    // where the expression divides by 1e-8 instead and so has other decision boundaries.
                    if (!(energy > 1e-30f && energy < 1e30f && lowest < 1e30f && base * grid.x >= 1e-8f) || !contenders) contenders = 0xffffffffu;
                } else {
                    float count[V][16], energy = 0.0f;  // what the columns count
#pragma unroll
                    for (int v = 0; v < V; ++v)
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const float4 x = load_energy(p, k0 + v * 128 + q * 4);
                            count[v][q * 4] = x.x; count[v][q * 4 + 1] = x.y; count[v][q * 4 + 2] = x.z; count[v][q * 4 + 3] = x.w;
#pragma unroll
                            for (int e = 0; e < 4; ++e) energy = fmaf(count[v][q * 4 + e] * f[v][q * 4 + e], f[v][q * 4 + e], energy);
                        }
                    for (int o = 1; o < lg; o <<= 1) energy += __shfl_xor_sync(0xffffffffu, energy, o);
                    const float always = kEnergyShare<BITS> * energy;
                    contenders = 0;
#pragma unroll 1
                    for (int s = 0; s < steps; ++s) {
                        const float cand = base * factors[s], inv = reciprocal(cand);
                        float e0 = 0.0f, e1 = 0.0f;
#pragma unroll
                        for (int v = 0; v < V; ++v)
#pragma unroll
                            for (int e = 0; e < 16; ++e) {
                                const float a = fabsf(f[v][e]), r = fminf(fmaf(a, inv, kMagic) - kMagic, f[v][e] < 0.0f ? 8.0f : 7.0f);
                                const float d = fmaf(r, cand, -a);
                                if (e & 1) e1 = fmaf(d * count[v][e], d, e1); else e0 = fmaf(d * count[v][e], d, e0);
                            }
                        float err = e0 + e1;
                        for (int o = 1; o < lg; o <<= 1) err += __shfl_xor_sync(0xffffffffu, err, o);
                        // all within reach of the lowest so far; a lower one drops those that it has left behind.  What stays of a slow
                        // descent is compared by exact errors, too, which cannot change the choice.
                        if (err <= lowest + (kErrorShare * lowest + always))
                            contenders = (lowest <= err + (kErrorShare * err + always) ? contenders : 0u) | 1u << s;
                        lowest = fminf(lowest, err);
                    }
                    if (!(lowest > 1e-30f && lowest < 1e30f)) contenders = 0xffffffffu;
                }
            }
            const bool decided = fast && __popc(contenders) == 1;
            if (decided) chosen = __fmul_rn(base, factors[__ffs(contenders) - 1]);
            const uint32_t visit = __reduce_or_sync(0xffffffffu, decided ? 0u : contenders);
            if (visit) {
                const float exact = exact_search<BITS, V, DT>(p, factors, row, k0, base, visit, contenders, !fast);
                if (!decided) chosen = exact;
            }
        }
        if (l == 0) p.scales[(size_t)row * p.ng + grp] = __float2half_rn(chosen);
        const float edge = 0.6666667f * chosen, inv = BITS == 2 ? 0.0f : reciprocal(chosen);
#pragma unroll
        for (int v = 0; v < V; ++v) {
            uint32_t word[BITS == 2 ? 1 : 2], unsure = 0;
#pragma unroll
            for (int i = 0; i < (BITS == 2 ? 1 : 2); ++i) {
                word[i] = 0;
#pragma unroll
                for (int e = 0; e < 32 / BITS; ++e) {
                    const int at = i * (32 / BITS) + e;
                    int c;
                    if (!code_estimate<BITS>(f[v][at], chosen, edge, inv, c)) unsure |= 1u << at;
                    word[i] |= (uint32_t)(c + (BITS == 4 ? 8 : 0)) << (BITS * e);
                }
            }
#pragma unroll 1
            for (; unsure; unsure &= unsure - 1) {     // rare: by the quotient
                const int e = __ffs(unsure) - 1, at = (BITS * e) & 31;
                float w1 = 0.0f;
#pragma unroll
                for (int i = 0; i < 16; ++i) if (i == e) w1 = f[v][i];
                const uint32_t c = (uint32_t)(code_exact<BITS>(w1, chosen, true) + (BITS == 4 ? 8 : 0)) << at;
                const uint32_t keep = ~((BITS == 2 ? 3u : 15u) << at);
                if (BITS == 4 && e >= 8) word[BITS == 2 ? 0 : 1] = (word[BITS == 2 ? 0 : 1] & keep) | c;
                else word[0] = (word[0] & keep) | c;
            }
            uint8_t* out = p.packed + (size_t)row * row_bytes + (size_t)(k0 + v * 128) * BITS / 8;
            if constexpr (BITS == 2) *reinterpret_cast<uint32_t*>(out) = word[0];
            else *reinterpret_cast<uint2*>(out) = make_uint2(word[0], word[1]);
        }
    }
}

}  // namespace
}  // namespace qgemv

using namespace qgemv;

static int run_pack(int bits, const void* w, int64_t ldw, int w_dtype, int n, int k, int group, const float* rms, const float* factors, float first,
                    float last, int steps, uint8_t* packed, void* scales, void* stream) {
    if (!w || !packed || !scales || n < 1 || k < 1 || ldw < k || (bits != 2 && bits != 4) || w_dtype < QGEMV_F16 || w_dtype > QGEMV_F32 ||
        (rms && (steps < 1 || (!factors && steps > QGEMV_PACK_MAX_SPACED)))) {
        set_error("qgemv_pack: null pointer, non-positive size, bad type or too many candidates");
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
    const int most = 148 * pack_blocks(bits, v);       // as many blocks as are resident
    const int grid = (int)(trips < most ? trips : most);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const PackArgs a{w, ldw, rms, factors, first, last, steps > 1 ? (last - first) / (float)(steps - 1) : 0.0f, packed, static_cast<__half*>(scales), n, k, ng, group, lg, steps, vec, reinterpret_cast<uintptr_t>(rms) % 16 == 0};
#define QP(B, V, D) do { if (rms) pack_kernel<B, V, D, true><<<grid, 256, 0, s>>>(a); else pack_kernel<B, V, D, false><<<grid, 256, 0, s>>>(a); } while (0)
#define QP_D(B, V) do { if (w_dtype == QGEMV_F16) QP(B, V, QGEMV_F16); else if (w_dtype == QGEMV_BF16) QP(B, V, QGEMV_BF16); else QP(B, V, QGEMV_F32); } while (0)
#define QP_V(B) do { if (v == 1) QP_D(B, 1); else if (v == 2) QP_D(B, 2); else QP_D(B, 4); } while (0)
    if (bits == 2) QP_V(2); else QP_V(4);
#undef QP_V
#undef QP_D
#undef QP
    return check_launch("pack_kernel");
}

extern "C" int qgemv_pack(int bits, const void* w, int64_t ldw, int w_dtype, int n, int k, int group, const float* rms, const float* factors,
                          int steps, uint8_t* packed, void* scales, void* stream) {
    if (rms && !factors) { set_error("qgemv_pack: rms needs factors"); return QGEMV_ERR_BAD_ARG; }
    return run_pack(bits, w, ldw, w_dtype, n, k, group, rms, factors, 0.0f, 0.0f, steps, packed, scales, stream);
}

extern "C" int qgemv_pack_spaced(int bits, const void* w, int64_t ldw, int w_dtype, int n, int k, int group, const float* rms, float first, float last,
                                 int steps, uint8_t* packed, void* scales, void* stream) {
    return run_pack(bits, w, ldw, w_dtype, n, k, group, rms, nullptr, first, last, steps, packed, scales, stream);
}
