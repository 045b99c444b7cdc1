// The kernels of a decode step between the packed GEMVs: see include/qdecode_b200.h.
//
// All of them are latency-sized (tens of kilobytes to a few megabytes per launch): what matters is
// one launch per step of the layer, coalesced 8 / 16-byte accesses, enough CTAs for the attention
// to spread the cache over the SMs, and no waiting between CTAs (the attention's slices meet through
// an arrival counter: whoever comes last merges).
#include <atomic>
#include <type_traits>

#include "qgemv_common.cuh"
#include "../../include/qdecode_b200.h"

namespace qgemv {
namespace {

template <bool BF16> __device__ __forceinline__ float r16(float v) {
    return Act16<BF16>::to_float(Act16<BF16>::from_float(v));
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ---------------------------------------------------------------------------------------------
// residual update + RMS normalisation: one CTA per row, a thread for every 8 elements up to 1024 of them.  A chain of
// latencies (h and delta from L2, two reductions, the store), so the norm's weight, which comes from DRAM, is fetched before
// the preceding kernel has finished, and one barrier is all that the threads meet at.
// ---------------------------------------------------------------------------------------------
constexpr int kNormMaxThreads = 1024;
constexpr int kNormMaxVec = 2;                    // 8-element vectors per thread: hidden <= 1024 * 2 * 8

template <bool BF16>
__global__ void __launch_bounds__(kNormMaxThreads) rmsnorm_kernel(void* h_, long long ldh, const void* delta_, long long ldd,
                                                                  const void* w_, void* y_, long long ldy, int hidden, float eps) {
    using T = typename Act16<BF16>::T;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int row = blockIdx.x, tid = threadIdx.x, threads = blockDim.x, nvec = hidden >> 3;
    T* h = static_cast<T*>(h_) + (size_t)row * ldh;
    const T* delta = delta_ ? static_cast<const T*>(delta_) + (size_t)row * ldd : nullptr;
    const T* w = static_cast<const T*>(w_);
    T* y = static_cast<T*>(y_) + (size_t)row * ldy;
    __shared__ float red[32];

    uint4 wv[kNormMaxVec];
#pragma unroll
    for (int i = 0; i < kNormMaxVec; ++i)
        if (tid + i * threads < nvec) wv[i] = __ldg(reinterpret_cast<const uint4*>(w) + tid + i * threads);
    asm volatile("griddepcontrol.wait;" ::: "memory");

    uint4 hv[kNormMaxVec], dv[kNormMaxVec];
#pragma unroll
    for (int i = 0; i < kNormMaxVec; ++i) {
        const int v = tid + i * threads;
        if (v < nvec) {
            hv[i] = *reinterpret_cast<const uint4*>(h + v * 8);
            if (delta) dv[i] = *reinterpret_cast<const uint4*>(delta + v * 8);
        }
    }
    float sq = 0.0f;
#pragma unroll
    for (int i = 0; i < kNormMaxVec; ++i) {
        const int v = tid + i * threads;
        if (v < nvec) {
            T* he = reinterpret_cast<T*>(&hv[i]);
            if (delta) {
                const T* de = reinterpret_cast<const T*>(&dv[i]);
#pragma unroll
                for (int q = 0; q < 8; ++q) he[q] = Act16<BF16>::from_float(Act16<BF16>::to_float(he[q]) + Act16<BF16>::to_float(de[q]));
                *reinterpret_cast<uint4*>(h + v * 8) = hv[i];
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const float f = Act16<BF16>::to_float(he[q]);
                sq = fmaf(f, f, sq);
            }
        }
    }
    sq = warp_sum(sq);
    if ((tid & 31) == 0) red[tid >> 5] = sq;
    __syncthreads();
    const int lane = tid & 31;
    const float inv = rsqrtf(warp_sum(lane < threads >> 5 ? red[lane] : 0.0f) / (float)hidden + eps);
#pragma unroll
    for (int i = 0; i < kNormMaxVec; ++i) {
        const int v = tid + i * threads;
        if (v < nvec) {
            const T* he = reinterpret_cast<const T*>(&hv[i]);
            const T* we = reinterpret_cast<const T*>(&wv[i]);
            uint4 ov;
            T* oe = reinterpret_cast<T*>(&ov);
#pragma unroll
            for (int q = 0; q < 8; ++q)
                oe[q] = Act16<BF16>::from_float(Act16<BF16>::to_float(we[q]) * r16<BF16>(Act16<BF16>::to_float(he[q]) * inv));
            *reinterpret_cast<uint4*>(y + v * 8) = ov;
        }
    }
}

// ---------------------------------------------------------------------------------------------
// rotary embedding + cache append: one CTA per (head, sequence); heads = q heads, k heads, v heads
// ---------------------------------------------------------------------------------------------
template <bool BF16>
__global__ void __launch_bounds__(128) rope_append_kernel(void* q_, long long ldq, const void* k_, long long ldk,
                                                          const void* v_, long long ldv, const void* cos_, const void* sin_,
                                                          int table_rows, const long long* pos_, void* kc_, void* vc_,
                                                          int hq, int hkv, int d, int max_len, int* status) {
    using T = typename Act16<BF16>::T;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const long long pos = *pos_;
    if (pos < 0 || pos >= max_len || pos >= table_rows) {
        if (status && threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0) atomicExch(status, 1);
        return;
    }
    const int head = blockIdx.x, b = blockIdx.y, j = threadIdx.x, half = d >> 1;
    if (j >= half) return;
    const T* cs = static_cast<const T*>(cos_) + (size_t)pos * d;
    const T* sn = static_cast<const T*>(sin_) + (size_t)pos * d;
    auto rotate = [&](const T* src, T* dst) {
        const float lo = Act16<BF16>::to_float(src[j]), hi = Act16<BF16>::to_float(src[j + half]);
        // out[j] = r(r(x[j] cos[j]) + r(-x[j + d/2] sin[j])),  out[j + d/2] = r(r(x[j + d/2] cos[j + d/2]) + r(x[j] sin[j + d/2]))
        const float a = r16<BF16>(lo * Act16<BF16>::to_float(cs[j])) + r16<BF16>(-hi * Act16<BF16>::to_float(sn[j]));
        const float c = r16<BF16>(hi * Act16<BF16>::to_float(cs[j + half])) + r16<BF16>(lo * Act16<BF16>::to_float(sn[j + half]));
        dst[j] = Act16<BF16>::from_float(a);
        dst[j + half] = Act16<BF16>::from_float(c);
    };
    if (head < hq) {
        T* q = static_cast<T*>(q_) + (size_t)b * ldq + (size_t)head * d;
        rotate(q, q);
    } else if (head < hq + hkv) {
        const int kh = head - hq;
        const T* k = static_cast<const T*>(k_) + (size_t)b * ldk + (size_t)kh * d;
        T* dst = static_cast<T*>(kc_) + (((size_t)b * hkv + kh) * max_len + (size_t)pos) * d;
        rotate(k, dst);
    } else {
        const int vh = head - hq - hkv;
        const T* v = static_cast<const T*>(v_) + (size_t)b * ldv + (size_t)vh * d;
        T* dst = static_cast<T*>(vc_) + (((size_t)b * hkv + vh) * max_len + (size_t)pos) * d;
        dst[j] = v[j];
        dst[j + half] = v[j + half];
    }
}

// ---------------------------------------------------------------------------------------------
// attention of one query token per sequence: grid (slice, kv head, sequence), 8 warps per CTA, 16 positions per warp and turn
// ---------------------------------------------------------------------------------------------
constexpr int kAttWarps = 8;
constexpr int kAttMaxSlices = 16;
constexpr int kAttBlock = 16;                    // positions of a warp's turn
constexpr int kAttSlice = kAttWarps * kAttBlock; // one turn of a CTA
constexpr int kAttMaxHeads = 8;                  // query heads per kv head
constexpr int kAttCluster = 8;                   // slices of a cluster: what every device can place

// Slices the sequence axis is cut into where they meet through global memory: as many CTAs as fit the SMs one each, each with a turn's positions at
// least.  Meeting there (fence, counter, reading the parts back) costs 2.5 us, a turn well under 1 to 1.7: shorter slices only pay the former, and a
// second wave (9 slices for 32 (sequence, kv head) pairs) measured slower than more turns.
inline int attention_slices(int batch, int kv_heads, int max_len) {
    const int ctas = batch * kv_heads, by_len = max_len / kAttSlice;
    int s = 148 / ctas;
    s = s > kAttMaxSlices ? kAttMaxSlices : s;
    s = s > by_len ? by_len : s;
    return s < 1 ? 1 : s;
}

__device__ __forceinline__ uint32_t transpose8(uint32_t v) {
    uint32_t r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}

// c += A (16 x 16, row) B (16 x 8, col), both of the activation type.
template <bool BF16>
__device__ __forceinline__ void mma16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if constexpr (BF16)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
// A float of the same shared variable in CTA `rank` of the cluster.
__device__ __forceinline__ float load_peer(const float* mine, int rank) {
    float v;
    asm volatile("{ .reg .u32 a; mapa.shared::cluster.u32 a, %1, %2; ld.shared::cluster.f32 %0, [a]; }"
                 : "=f"(v) : "r"((uint32_t)__cvta_generic_to_shared(mine)), "r"(rank) : "memory");
    return v;
}

template <bool BF16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    const typename Act16<BF16>::T a = Act16<BF16>::from_float(lo), b = Act16<BF16>::from_float(hi);
    return (uint32_t)*reinterpret_cast<const unsigned short*>(&a) | (uint32_t)*reinterpret_cast<const unsigned short*>(&b) << 16;
}

// Lane t of a quad holds, of a row of D elements, the eight from 32 c + 8 t in word c of v: so the partner of every element
// under the rotation (D / 2 away) is the same lane's, D / 64 words further on.  The tables' words lie alike.
template <int D, bool BF16>
__device__ __forceinline__ void rotate_row(uint4 (&v)[D / 32], const uint4 (&cos_)[D / 32], const uint4 (&sin_)[D / 32]) {
    using T = typename Act16<BF16>::T;
    constexpr int H = D / 64;
#pragma unroll
    for (int c = 0; c < H; ++c) {
        T* lo = reinterpret_cast<T*>(&v[c]);
        T* hi = reinterpret_cast<T*>(&v[c + H]);
        const T* cl = reinterpret_cast<const T*>(&cos_[c]);
        const T* ch = reinterpret_cast<const T*>(&cos_[c + H]);
        const T* sl = reinterpret_cast<const T*>(&sin_[c]);
        const T* sh = reinterpret_cast<const T*>(&sin_[c + H]);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float a = Act16<BF16>::to_float(lo[q]), b = Act16<BF16>::to_float(hi[q]);
            lo[q] = Act16<BF16>::from_float(r16<BF16>(a * Act16<BF16>::to_float(cl[q])) + r16<BF16>(-b * Act16<BF16>::to_float(sl[q])));
            hi[q] = Act16<BF16>::from_float(r16<BF16>(b * Act16<BF16>::to_float(ch[q])) + r16<BF16>(a * Act16<BF16>::to_float(sh[q])));
        }
    }
}

// What the fused form adds: the new token's key and value rows, the rotary tables.
struct NewToken {
    const void* k; long long ldk;
    const void* v; long long ldv;
    const void* cos; const void* sin;
    int table_rows; int* status;
    bool wide;                                    // the tables' rows are on 16 bytes
};

// With the lanes of a warp along D this kernel spent its time in shuffles (five per position and query head: 36 us for 4
// sequences x 8 kv heads x 8 query heads over 1088 positions, 17 MB).  Here a warp takes 16 positions of a kv head for all
// its query heads: scores are mma m16n8k16 of 16 keys with up to 8 queries, and the values' turn is a second one, their
// transposition done in registers (movmatrix).  Keys and values go from global memory straight to fragments, 16 bytes a lane.
// The weights of the softmax enter the second product as a sum of two fp16 (three bf16) numbers, 22 (24) bits, so that no
// precision is lost against fp32 weights.  With it and the announcement to L2, fp16, in a chain of launches over caches that
// come from DRAM, rope and append included: 34.3 -> 12.1 us at the size above, 11.6 -> 7.6 us for 8 kv heads x 4 over 577
// positions, 7.1 -> 5.1 us for 2 x 7 of 64 elements over 162.  What is left is the chain position -> rows -> products ->
// softmax -> meeting, and the launch.  The slices of a sequence meet in the shared memory of a cluster where the device can place that, and what does not hang on
// the position (queries, new key and value) is asked for before it has arrived, the tables' rows 16 bytes at a time: 7.6 -> 6.2 us, 5.1 -> 4.1 and, at the
// first size, 12.4 -> 12.0.  One CTA per SM: with registers for two (128) the rotation spilled, 18.4 us above.
// ROPE: the queries are rotated on their way to fragments; the warp whose turn holds the new position takes that row from the
// projections instead of the cache, rotates the key, and writes both to the cache.
template <int D, bool BF16, bool ROPE>
__global__ void __launch_bounds__(kAttWarps * 32, 1) attention_kernel(const void* q_, long long ldq, void* kc_, void* vc_,
                                                                   const long long* pos_, void* out_, long long ldo, int heads, int hkv,
                                                                   int max_len, float scale, float* parts, int* counters, bool wide, bool clustered,
                                                                   const NewToken nt) {
    using T = typename Act16<BF16>::T;
    constexpr int C = D / 32;                     // 16-byte words of a row per lane
    constexpr int SPLIT = BF16 ? 3 : 2;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int slice = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z, slices = gridDim.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    T* kbase = static_cast<T*>(kc_) + ((size_t)b * hkv + kvh) * (size_t)max_len * D + t * 8;
    T* vbase = static_cast<T*>(vc_) + ((size_t)b * hkv + kvh) * (size_t)max_len * D + t * 8;
    int s0, s1;
    auto cut = [&](long long pos) {
        const long long len = pos < 0 ? 0 : pos >= max_len ? max_len : pos + 1;
        const int per = (int)((len + slices - 1) / slices + kAttBlock - 1) / kAttBlock * kAttBlock;
        s0 = min(slice * per, (int)len);
        s1 = min(s0 + per, (int)len);
    };
    // The cache rows go to L2 while the projections still run: only an announcement, so neither a position nor rows that
    // are not final yet can do harm.
    cut(*static_cast<const volatile long long*>(pos_));
    for (int p = s0 + warp * kAttBlock + (lane & 15); p < s1; p += kAttWarps * kAttBlock) {
        const T* row = (lane < 16 ? kbase : vbase) + (size_t)p * D - t * 8;
#pragma unroll
        for (int c = 0; c < D; c += 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + c));
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    auto load_row = [&](const T* row, uint4 (&v)[C]) {      // row points at the lane's first element
#pragma unroll
        for (int c = 0; c < C; ++c) {
            if (wide) {
                v[c] = *reinterpret_cast<const uint4*>(row + c * 32);
            } else {
                const uint2 x = *reinterpret_cast<const uint2*>(row + c * 32), y = *reinterpret_cast<const uint2*>(row + c * 32 + 4);
                v[c] = make_uint4(x.x, x.y, y.x, y.y);
            }
        }
    };
    auto store_row = [&](T* row, const uint4 (&v)[C]) {
#pragma unroll
        for (int c = 0; c < C; ++c) {
            if (wide) {
                *reinterpret_cast<uint4*>(row + c * 32) = v[c];
            } else {
                *reinterpret_cast<uint2*>(row + c * 32) = make_uint2(v[c].x, v[c].y);
                *reinterpret_cast<uint2*>(row + c * 32 + 4) = make_uint2(v[c].z, v[c].w);
            }
        }
    };
    auto clear = [&](uint4 (&v)[C]) {
#pragma unroll
        for (int c = 0; c < C; ++c) v[c] = make_uint4(0u, 0u, 0u, 0u);
    };

    // What does not hang on the position first: the queries, the new key and value (every warp, one will want them).
    uint4 qf[C], nk[C], nv[C];                    // head g of the group; the new row
    clear(qf);
    const long long pos = *static_cast<const volatile long long*>(pos_);
    if (g < heads) load_row(static_cast<const T*>(q_) + (size_t)b * ldq + (size_t)(kvh * heads + g) * D + t * 8, qf);
    if constexpr (ROPE) {
        load_row(static_cast<const T*>(nt.k) + (size_t)b * nt.ldk + (size_t)kvh * D + t * 8, nk);
        load_row(static_cast<const T*>(nt.v) + (size_t)b * nt.ldv + (size_t)kvh * D + t * 8, nv);
    }
    cut(pos);
    bool append = false;
    uint4 cs[C], sn[C];
    if constexpr (ROPE) {
        append = pos >= 0 && pos < max_len && pos < nt.table_rows;
        if (!append && nt.status && tid == 0) atomicExch(nt.status, 1);
        if (append) {
            const T* const cr = static_cast<const T*>(nt.cos) + (size_t)pos * D + t * 8;
            const T* const sr = static_cast<const T*>(nt.sin) + (size_t)pos * D + t * 8;
#pragma unroll
            for (int c = 0; c < C; ++c) {
                if (nt.wide) {
                    cs[c] = *reinterpret_cast<const uint4*>(cr + c * 32);
                    sn[c] = *reinterpret_cast<const uint4*>(sr + c * 32);
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        reinterpret_cast<T*>(&cs[c])[e] = cr[c * 32 + e];
                        reinterpret_cast<T*>(&sn[c])[e] = sr[c * 32 + e];
                    }
                }
            }
        }
    }

    uint4 ka[C], kb[C], va[C], vb[C];             // positions p + g and p + g + 8 of the turn
    auto fetch = [&](int p) {
        const int pa = p + g, pb = p + g + 8;
        clear(ka); clear(kb); clear(va); clear(vb);
        if (pa < s1 && !(append && pa == (int)pos)) { load_row(kbase + (size_t)pa * D, ka); load_row(vbase + (size_t)pa * D, va); }
        if (pb < s1 && !(append && pb == (int)pos)) { load_row(kbase + (size_t)pb * D, kb); load_row(vbase + (size_t)pb * D, vb); }
    };
    auto take_new = [&](int p) {                  // the turn's new row, if it has it
        if constexpr (ROPE) {
            if (append && p <= (int)pos && (int)pos < p + kAttBlock && (int)pos < s1) {
                const bool na = p + g == (int)pos, nb = p + g + 8 == (int)pos;
                if (na || nb) {
                    store_row(kbase + (size_t)pos * D, nk);
                    store_row(vbase + (size_t)pos * D, nv);
                }
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    if (na) { ka[c] = nk[c]; va[c] = nv[c]; }
                    if (nb) { kb[c] = nk[c]; vb[c] = nv[c]; }
                }
            }
        }
        __syncwarp();
    };
    int p = s0 + warp * kAttBlock;
    if (p < s1) fetch(p);                         // before anything waits for the queries
    if constexpr (ROPE) {
        if (append && (int)pos >= s0 && (int)pos < s1 && ((int)pos - s0) / kAttBlock % kAttWarps == warp) rotate_row<D, BF16>(nk, cs, sn);      // its turn will come here
        if (append) rotate_row<D, BF16>(qf, cs, sn);
    }
    if (p < s1) take_new(p);
    float m0 = -1.0e30f, m1 = -1.0e30f, l0 = 0.0f, l1 = 0.0f;      // heads 2t, 2t + 1; the sums of this lane's positions
    float o[D / 16][4];                           // rows: elements, see below; columns: heads 2t, 2t + 1
#pragma unroll
    for (int i = 0; i < D / 16; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[i][e] = 0.0f;

    while (p < s1) {
        const bool ia = p + g < s1, ib = p + g + 8 < s1;
        float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};    // positions p + g (0, 1), p + g + 8 (2, 3); heads 2t, 2t + 1
#pragma unroll
        for (int c = 0; c < C; ++c) {
            mma16<BF16>(s, ka[c].x, kb[c].x, ka[c].y, kb[c].y, qf[c].x, qf[c].y);
            mma16<BF16>(s, ka[c].z, kb[c].z, ka[c].w, kb[c].w, qf[c].z, qf[c].w);
        }
        s[0] = ia ? s[0] * scale : -1.0e30f; s[1] = ia ? s[1] * scale : -1.0e30f;
        s[2] = ib ? s[2] * scale : -1.0e30f; s[3] = ib ? s[3] * scale : -1.0e30f;
        float x0 = fmaxf(s[0], s[2]), x1 = fmaxf(s[1], s[3]);
#pragma unroll
        for (int off = 4; off < 32; off <<= 1) {
            x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, off));
            x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, off));
        }
        const float n0 = fmaxf(m0, x0), n1 = fmaxf(m1, x1);
        const float f0 = __expf(m0 - n0), f1 = __expf(m1 - n1);
        m0 = n0; m1 = n1;
        float w[4] = {ia ? __expf(s[0] - n0) : 0.0f, ia ? __expf(s[1] - n1) : 0.0f, ib ? __expf(s[2] - n0) : 0.0f, ib ? __expf(s[3] - n1) : 0.0f};
        l0 = fmaf(l0, f0, w[0] + w[2]);
        l1 = fmaf(l1, f1, w[1] + w[3]);
        uint32_t pw[SPLIT][2];                    // [part][positions 0 - 7, 8 - 15], transposed: head g, positions 2t, 2t + 1
#pragma unroll
        for (int i = 0; i < SPLIT; ++i) {
            pw[i][0] = transpose8(pack2<BF16>(w[0], w[1]));
            pw[i][1] = transpose8(pack2<BF16>(w[2], w[3]));
#pragma unroll
            for (int e = 0; e < 4; ++e) w[e] -= r16<BF16>(w[e]);
        }
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const uint32_t wa[4] = {va[c].x, va[c].y, va[c].z, va[c].w}, wb[4] = {vb[c].x, vb[c].y, vb[c].z, vb[c].w};
#pragma unroll
            for (int j = 0; j < 2; ++j) {         // word w of a lane's eight elements: row r of the transposed block is element 32 c + 8 (r / 2) + 2 w + r % 2
                float (&acc)[4] = o[c * 2 + j];
                acc[0] *= f0; acc[1] *= f1; acc[2] *= f0; acc[3] *= f1;
                const uint32_t a0 = transpose8(wa[2 * j]), a1 = transpose8(wa[2 * j + 1]), a2 = transpose8(wb[2 * j]), a3 = transpose8(wb[2 * j + 1]);
#pragma unroll
                for (int i = 0; i < SPLIT; ++i) mma16<BF16>(acc, a0, a1, a2, a3, pw[i][0], pw[i][1]);
            }
        }
        p += kAttWarps * kAttBlock;
        if (p < s1) { fetch(p); take_new(p); }
    }
#pragma unroll
    for (int off = 4; off < 32; off <<= 1) {
        l0 += __shfl_xor_sync(0xffffffffu, l0, off);
        l1 += __shfl_xor_sync(0xffffffffu, l1, off);
    }

    // the CTA's warps meet in shared memory
    __shared__ float sm_m[kAttWarps][kAttMaxHeads], sm_l[kAttWarps][kAttMaxHeads];
    __shared__ float sm_o[kAttWarps][kAttMaxHeads][D];
    __shared__ float cl_m[kAttMaxHeads], cl_l[kAttMaxHeads], cl_o[kAttMaxHeads * D];      // of the CTA, for its cluster
    __shared__ int is_last;
    const int active = max(1, min(kAttWarps, (s1 - s0 + kAttBlock - 1) / kAttBlock));      // warps that had a turn
    if (warp < active) {
        if (g == 0) {
            sm_m[warp][2 * t] = m0; sm_m[warp][2 * t + 1] = m1;
            sm_l[warp][2 * t] = l0; sm_l[warp][2 * t + 1] = l1;
        }
#pragma unroll
        for (int i = 0; i < D / 16; ++i) {
            const int d = (i >> 1) * 32 + (g >> 1) * 8 + (i & 1) * 4 + (g & 1);
            if (2 * t < heads) { sm_o[warp][2 * t][d] = o[i][0]; sm_o[warp][2 * t][d + 2] = o[i][2]; }
            if (2 * t + 1 < heads) { sm_o[warp][2 * t + 1][d] = o[i][1]; sm_o[warp][2 * t + 1][d + 2] = o[i][3]; }
        }
    }
    __syncthreads();
    constexpr int STRIDE = D + 4;                 // floats per (slice, head): m, l, two unused, o[D] (16-byte aligned)
    T* out = static_cast<T*>(out_) + (size_t)b * ldo + (size_t)kvh * heads * D;
    float* mine = parts + ((((size_t)b * hkv + kvh) * slices + slice) * heads) * STRIDE;
    for (int i = tid; i < heads * D; i += kAttWarps * 32) {
        const int h = i / D, dd = i - h * D;
        float mm = sm_m[0][h];
        for (int w = 1; w < active; ++w) mm = fmaxf(mm, sm_m[w][h]);
        float acc = 0.0f, ll = 0.0f;
        for (int w = 0; w < active; ++w) {
            const float f = __expf(sm_m[w][h] - mm);
            acc = fmaf(sm_o[w][h][dd], f, acc);
            ll = fmaf(sm_l[w][h], f, ll);
        }
        if (slices == 1) {
            out[i] = Act16<BF16>::from_float(ll > 0.0f ? acc * (1.0f / ll) : 0.0f);
        } else if (clustered) {
            cl_o[i] = acc;
            if (dd == 0) { cl_m[h] = mm; cl_l[h] = ll; }
        } else {
            mine[h * STRIDE + 4 + dd] = acc;
            if (dd == 0) { mine[h * STRIDE] = mm; mine[h * STRIDE + 1] = ll; }
        }
    }
    if (slices == 1) return;
    if (clustered) {                              // the slices are a cluster: each CTA makes a share of the results, from the shared memory of all, in order
        cluster_barrier();
        for (int i = slice * (kAttWarps * 32) + tid; i < heads * D; i += slices * (kAttWarps * 32)) {
            const int h = i / D;
            float mv[kAttCluster], lv[kAttCluster], ov[kAttCluster];
#pragma unroll
            for (int s = 0; s < kAttCluster; ++s) {
                mv[s] = -1.0e30f; lv[s] = ov[s] = 0.0f;
                if (s < slices) { mv[s] = load_peer(&cl_m[h], s); lv[s] = load_peer(&cl_l[h], s); ov[s] = load_peer(&cl_o[i], s); }
            }
            float mm = mv[0];
#pragma unroll
            for (int s = 1; s < kAttCluster; ++s) mm = fmaxf(mm, mv[s]);
            float ll = 0.0f, acc = 0.0f;
#pragma unroll
            for (int s = 0; s < kAttCluster; ++s) {
                const float f = __expf(mv[s] - mm);
                ll = fmaf(lv[s], f, ll);
                acc = fmaf(ov[s], f, acc);
            }
            out[i] = Act16<BF16>::from_float(ll > 0.0f ? acc * (1.0f / ll) : 0.0f);
        }
        cluster_barrier();                        // nobody leaves before the others have read its sums
        return;
    }
    // arrival: the last CTA of this (sequence, kv head) merges the slices; nobody waits
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        const int old = atomicAdd(counters + b * hkv + kvh, 1);
        is_last = old == slices - 1;
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    // Every load of the merge is independent of the others and issued before the first use: one
    // trip to L2 per head instead of one per slice.  A warp takes a head; a lane takes 4 output elements.
    const float* all = parts + (((size_t)b * hkv + kvh) * slices) * heads * STRIDE;
    const bool has_o = lane * 4 < D;
    for (int h = warp; h < heads; h += kAttWarps) {
        float mv[kAttMaxSlices], lv[kAttMaxSlices];
        float4 ov[kAttMaxSlices];
#pragma unroll
        for (int s = 0; s < kAttMaxSlices; ++s) {
            mv[s] = -1.0e30f; lv[s] = 0.0f; ov[s] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (s < slices) {
                const float* pp = all + ((size_t)s * heads + h) * STRIDE;
                const float2 ml = __ldcg(reinterpret_cast<const float2*>(pp));
                mv[s] = ml.x; lv[s] = ml.y;
                if (has_o) ov[s] = __ldcg(reinterpret_cast<const float4*>(pp + 4) + lane);
            }
        }
        float mm = -1.0e30f;
#pragma unroll
        for (int s = 0; s < kAttMaxSlices; ++s) mm = fmaxf(mm, mv[s]);
        float ll = 0.0f;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int s = 0; s < kAttMaxSlices; ++s) {
            const float f = __expf(mv[s] - mm);
            ll = fmaf(lv[s], f, ll);
            acc.x = fmaf(ov[s].x, f, acc.x); acc.y = fmaf(ov[s].y, f, acc.y);
            acc.z = fmaf(ov[s].z, f, acc.z); acc.w = fmaf(ov[s].w, f, acc.w);
        }
        if (has_o) {
            const float inv = ll > 0.0f ? 1.0f / ll : 0.0f;
            uint2 packed;
            T* pe = reinterpret_cast<T*>(&packed);
            pe[0] = Act16<BF16>::from_float(acc.x * inv); pe[1] = Act16<BF16>::from_float(acc.y * inv);
            pe[2] = Act16<BF16>::from_float(acc.z * inv); pe[3] = Act16<BF16>::from_float(acc.w * inv);
            *reinterpret_cast<uint2*>(out + h * D + lane * 4) = packed;
        }
    }
    if (tid == 0) counters[b * hkv + kvh] = 0;       // ready for the next launch (stream order makes it visible)
}

// ---------------------------------------------------------------------------------------------
// silu(gate) * up
// ---------------------------------------------------------------------------------------------
template <bool BF16>
__global__ void __launch_bounds__(256) silu_mul_kernel(const void* g_, long long ldg, const void* u_, long long ldu, void* y_,
                                                       long long ldy, int width, bool vec) {
    using T = typename Act16<BF16>::T;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int row = blockIdx.y;
    const T* g = static_cast<const T*>(g_) + (size_t)row * ldg;
    const T* u = static_cast<const T*>(u_) + (size_t)row * ldu;
    T* y = static_cast<T*>(y_) + (size_t)row * ldy;
    auto one = [](T gv, T uv) {
        const float gf = Act16<BF16>::to_float(gv);
        return Act16<BF16>::from_float(r16<BF16>(gf / (1.0f + __expf(-gf))) * Act16<BF16>::to_float(uv));
    };
    if (vec) {
        for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < (width >> 3); v += gridDim.x * blockDim.x) {
            const uint4 gv = *reinterpret_cast<const uint4*>(g + v * 8), uv = *reinterpret_cast<const uint4*>(u + v * 8);
            const T* ge = reinterpret_cast<const T*>(&gv);
            const T* ue = reinterpret_cast<const T*>(&uv);
            uint4 ov;
            T* oe = reinterpret_cast<T*>(&ov);
#pragma unroll
            for (int q = 0; q < 8; ++q) oe[q] = one(ge[q], ue[q]);
            *reinterpret_cast<uint4*>(y + v * 8) = ov;
        }
    } else {
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < width; i += gridDim.x * blockDim.x) y[i] = one(g[i], u[i]);
    }
}

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

// Launch with the programmatic-stream-serialisation attribute: the kernels above release their
// successor at entry and wait for their predecessor before they touch memory.
template <typename... KArgs, typename... Args>
int launch_clusters(const char* what, void (*kern)(KArgs...), dim3 grid, dim3 block, int cluster, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    (void)cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
    return check_launch(what);
}
template <typename... KArgs, typename... Args>
int launch_pdl(const char* what, void (*kern)(KArgs...), dim3 grid, dim3 block, cudaStream_t s, Args... args) {
    return launch_clusters(what, kern, grid, block, 1, s, args...);
}

template <bool ROPE>
int launch_attention(bool bf16, int head_dim, dim3 grid, cudaStream_t s, const void* q, long long ldq, void* kc, void* vc, const long long* pos,
                     void* out, long long ldo, int heads, int hkv, int max_len, float scale, float* parts, int* counters, bool wide, bool clustered,
                     const NewToken& nt) {
    const dim3 block(kAttWarps * 32);
#define QDEC_ATT(D, B) launch_clusters("attention_kernel", attention_kernel<D, B, ROPE>, grid, block, clustered ? (int)grid.x : 1, s, q, ldq, kc, vc, pos, out, ldo, heads, hkv, \
                                  max_len, scale, parts, counters, wide, clustered, nt)
    if (head_dim == 64) return bf16 ? QDEC_ATT(64, true) : QDEC_ATT(64, false);
    return bf16 ? QDEC_ATT(128, true) : QDEC_ATT(128, false);
#undef QDEC_ATT
}

// Clusters of `size` CTAs that the device places at a time, by the largest of the kernels (all take an SM to themselves).
int attention_clusters(int size) {
    static std::atomic<int> known[64][kAttCluster + 1];      // + 1
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { (void)cudaGetLastError(); return 0; }
    int n = known[dev][size].load(std::memory_order_relaxed) - 1;
    if (n >= 0) return n;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(size);
    cfg.blockDim = dim3(kAttWarps * 32);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = size;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, attention_kernel<128, true, true>, &cfg) != cudaSuccess) { (void)cudaGetLastError(); n = 0; }
    known[dev][size].store(n + 1, std::memory_order_relaxed);
    return n;
}

// Slices of a cluster, 0 where the global meeting is better.  The meeting in shared memory costs some 1 us (one slice 3.1 us, two 4.1, chains over 112
// positions of 64 elements), so slices pay from about 192 positions on and down to 24 each: 8 instead of 5 over 576 positions of 8 heads x 128 6.2 against
// 7.0 us (global meeting 7.6), instead of 1 over 300 4.2 against 5.6 (7.2).  As many as the device places at once for all (sequence, kv head) pairs: the
// next larger ones go in two waves (16 pairs: 6 slices 10.3 us, 7 18.9).  More slices of the other kind win where a CTA of the cluster gets so many turns more
// that they outweigh the meeting, us: 2 x 64 elements, 3072 positions 7.0 in the cluster, 7.5 in 16 slices; 4072 8.3 and 7.9; 8 x 128, 1772 8.3 and 9.0,
// 2072 8.5 and 8.1; 16 x 128 (6 slices against 8) 1072 8.3 and 8.1, 372 5.9 and 9.6.
int cluster_slices(int batch, int kv_heads, int head_dim, int max_len) {
    if (max_len < 192) return 0;
    const int pairs = batch * kv_heads, global = attention_slices(batch, kv_heads, max_len);
    for (int c = kAttCluster; c >= 2; --c) {
        if (attention_clusters(c) < pairs) continue;
        const float turns = (float)max_len / kAttSlice * (1.0f / c - 1.0f / global);        // more of them than in global slices
        return turns <= (c < kAttCluster ? 0.15f : head_dim == 64 ? 1.5f : 0.7f) ? c : 0;
    }
    return 0;
}

size_t attention_parts_floats(int batch, int q_heads, int kv_heads, int head_dim, int max_len) {
    const int slices = attention_slices(batch, kv_heads, max_len);
    return (size_t)batch * q_heads * slices * (head_dim + 4);
}

}  // namespace
}  // namespace qgemv

using namespace qgemv;

extern "C" int qdec_rmsnorm(void* h, int64_t ldh, const void* delta, int64_t ldd, const void* weight, void* y, int64_t ldy,
                            int rows, int hidden, float eps, int dtype, void* stream) {
    if (!h || !weight || !y || rows < 1 || hidden < 8) { set_error("qdec_rmsnorm: null pointer or non-positive size"); return QGEMV_ERR_BAD_ARG; }
    if (dtype != QGEMV_F16 && dtype != QGEMV_BF16) { set_error("qdec_rmsnorm: dtype must be fp16 or bf16"); return QGEMV_ERR_BAD_ARG; }
    if (hidden % 8 || hidden > kNormMaxThreads * kNormMaxVec * 8) { set_error("qdec_rmsnorm: hidden=%d must be a multiple of 8, at most %d", hidden, kNormMaxThreads * kNormMaxVec * 8); return QGEMV_ERR_SHAPE; }
    if (ldh < hidden || ldy < hidden || (delta && ldd < hidden)) { set_error("qdec_rmsnorm: a leading dimension is smaller than hidden"); return QGEMV_ERR_SHAPE; }
    if (!aligned16(h) || !aligned16(y) || !aligned16(weight) || (delta && !aligned16(delta)) || ldh % 8 || ldy % 8 || (delta && ldd % 8)) {
        set_error("qdec_rmsnorm: rows must be 16-byte aligned");
        return QGEMV_ERR_ALIGN;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int vecs = hidden / 8, threads = vecs >= kNormMaxThreads ? kNormMaxThreads : (vecs + 31) / 32 * 32;
    if (dtype == QGEMV_BF16)
        return launch_pdl("rmsnorm_kernel", rmsnorm_kernel<true>, dim3(rows), dim3(threads), s, h, (long long)ldh, delta, (long long)ldd, weight, y, (long long)ldy, hidden, eps);
    return launch_pdl("rmsnorm_kernel", rmsnorm_kernel<false>, dim3(rows), dim3(threads), s, h, (long long)ldh, delta, (long long)ldd, weight, y, (long long)ldy, hidden, eps);
}

extern "C" int qdec_rope_append(void* q, int64_t ldq, const void* k, int64_t ldk, const void* v, int64_t ldv,
                                const void* cos_table, const void* sin_table, int table_rows, const int64_t* pos,
                                void* kcache, void* vcache, int batch, int q_heads, int kv_heads, int head_dim, int max_len,
                                int32_t* status, int dtype, void* stream) {
    if (!q || !k || !v || !cos_table || !sin_table || !pos || !kcache || !vcache) { set_error("qdec_rope_append: null pointer"); return QGEMV_ERR_BAD_ARG; }
    if (batch < 1 || q_heads < 1 || kv_heads < 1 || max_len < 1 || table_rows < 1) { set_error("qdec_rope_append: non-positive size"); return QGEMV_ERR_BAD_ARG; }
    if (dtype != QGEMV_F16 && dtype != QGEMV_BF16) { set_error("qdec_rope_append: dtype must be fp16 or bf16"); return QGEMV_ERR_BAD_ARG; }
    if (head_dim < 2 || head_dim % 2 || head_dim > 256) { set_error("qdec_rope_append: head_dim=%d must be even, at most 256", head_dim); return QGEMV_ERR_SHAPE; }
    if (ldq < (int64_t)q_heads * head_dim || ldk < (int64_t)kv_heads * head_dim || ldv < (int64_t)kv_heads * head_dim) { set_error("qdec_rope_append: a leading dimension is smaller than its row"); return QGEMV_ERR_SHAPE; }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const dim3 grid(q_heads + 2 * kv_heads, batch), block(128);
    const long long* p = reinterpret_cast<const long long*>(pos);
    if (dtype == QGEMV_BF16)
        return launch_pdl("rope_append_kernel", rope_append_kernel<true>, grid, block, s, q, (long long)ldq, k, (long long)ldk, v, (long long)ldv,
                          cos_table, sin_table, table_rows, p, kcache, vcache, q_heads, kv_heads, head_dim, max_len, status);
    return launch_pdl("rope_append_kernel", rope_append_kernel<false>, grid, block, s, q, (long long)ldq, k, (long long)ldk, v, (long long)ldv,
                      cos_table, sin_table, table_rows, p, kcache, vcache, q_heads, kv_heads, head_dim, max_len, status);
}

extern "C" size_t qdec_attention_workspace_bytes(int batch, int q_heads, int kv_heads, int head_dim, int max_len) {
    if (batch < 1 || q_heads < 1 || kv_heads < 1 || head_dim < 1 || max_len < 1) return 0;
    const size_t parts = attention_parts_floats(batch, q_heads, kv_heads, head_dim, max_len) * sizeof(float);
    const size_t counters = ((size_t)batch * kv_heads * sizeof(int) + 255) / 256 * 256;
    return counters + (parts + 255) / 256 * 256;
}

namespace {
// Argument checks and launch shared by the two forms; `nt.k` == NULL: attention alone.
int run_attention(const char* name, const void* q, int64_t ldq, void* kcache, void* vcache, const int64_t* pos, void* out, int64_t ldo, int batch,
                  int q_heads, int kv_heads, int head_dim, int max_len, float scale, void* workspace, size_t workspace_bytes, int dtype,
                  const NewToken& nt, void* stream) {
    if (!q || !kcache || !vcache || !pos || !out || !workspace) { set_error("%s: null pointer", name); return QGEMV_ERR_BAD_ARG; }
    if (batch < 1 || q_heads < 1 || kv_heads < 1 || max_len < 1) { set_error("%s: non-positive size", name); return QGEMV_ERR_BAD_ARG; }
    if (dtype != QGEMV_F16 && dtype != QGEMV_BF16) { set_error("%s: dtype must be fp16 or bf16", name); return QGEMV_ERR_BAD_ARG; }
    if (head_dim != 64 && head_dim != 128) { set_error("%s: head_dim=%d (64 and 128 are built)", name, head_dim); return QGEMV_ERR_SHAPE; }
    if (q_heads % kv_heads || q_heads / kv_heads > kAttMaxHeads) { set_error("%s: %d query heads over %d kv heads (a group of 1..8 is built)", name, q_heads, kv_heads); return QGEMV_ERR_SHAPE; }
    if (ldq < (int64_t)q_heads * head_dim || ldo < (int64_t)q_heads * head_dim) { set_error("%s: a leading dimension is smaller than its row", name); return QGEMV_ERR_SHAPE; }
    if (batch > 65535 || kv_heads > 65535) { set_error("%s: batch and kv_heads are grid dimensions (at most 65535)", name); return QGEMV_ERR_TOO_LARGE; }
    const size_t need = qdec_attention_workspace_bytes(batch, q_heads, kv_heads, head_dim, max_len);
    if (workspace_bytes < need) { set_error("%s: workspace of %zu bytes required (got %zu)", name, need, workspace_bytes); return QGEMV_ERR_WORKSPACE; }
    auto rows = [](const void* p, int64_t ld, size_t a) { return reinterpret_cast<uintptr_t>(p) % a == 0 && ld * 2 % (int64_t)a == 0; };
    auto all = [&](size_t a) {
        return rows(q, ldq, a) && rows(kcache, 0, a) && rows(vcache, 0, a) && (!nt.k || (rows(nt.k, nt.ldk, a) && rows(nt.v, nt.ldv, a)));
    };
    if (reinterpret_cast<uintptr_t>(workspace) % 256 || !all(8) || !rows(out, ldo, 8)) {
        set_error("%s: workspace must be 256-byte aligned, q, out, new rows and the caches 8-byte aligned", name);
        return QGEMV_ERR_ALIGN;
    }
    int* counters = static_cast<int*>(workspace);
    float* parts = reinterpret_cast<float*>(static_cast<char*>(workspace) + ((size_t)batch * kv_heads * sizeof(int) + 255) / 256 * 256);
    const int cluster = cluster_slices(batch, kv_heads, head_dim, max_len);
    const dim3 grid(cluster ? cluster : attention_slices(batch, kv_heads, max_len), kv_heads, batch);
    return (nt.k ? launch_attention<true> : launch_attention<false>)(dtype == QGEMV_BF16, head_dim, grid, static_cast<cudaStream_t>(stream), q, ldq, kcache,
        vcache, reinterpret_cast<const long long*>(pos), out, ldo, q_heads / kv_heads, kv_heads, max_len, scale, parts, counters, all(16), cluster != 0, nt);
}
}  // namespace

extern "C" int qdec_attention(const void* q, int64_t ldq, const void* kcache, const void* vcache, const int64_t* pos,
                              void* out, int64_t ldo, int batch, int q_heads, int kv_heads, int head_dim, int max_len,
                              float scale, void* workspace, size_t workspace_bytes, int dtype, void* stream) {
    return run_attention("qdec_attention", q, ldq, const_cast<void*>(kcache), const_cast<void*>(vcache), pos, out, ldo, batch, q_heads, kv_heads,
                         head_dim, max_len, scale, workspace, workspace_bytes, dtype, NewToken{}, stream);
}

extern "C" int qdec_rope_attention(const void* q, int64_t ldq, const void* k, int64_t ldk, const void* v, int64_t ldv,
                                   const void* cos_table, const void* sin_table, int table_rows, const int64_t* pos,
                                   void* kcache, void* vcache, void* out, int64_t ldo, int batch, int q_heads, int kv_heads,
                                   int head_dim, int max_len, float scale, void* workspace, size_t workspace_bytes,
                                   int32_t* status, int dtype, void* stream) {
    if (!k || !v || !cos_table || !sin_table || table_rows < 1) { set_error("qdec_rope_attention: null pointer or empty table"); return QGEMV_ERR_BAD_ARG; }
    if (ldk < (int64_t)kv_heads * head_dim || ldv < (int64_t)kv_heads * head_dim) { set_error("qdec_rope_attention: a leading dimension is smaller than its row"); return QGEMV_ERR_SHAPE; }
    return run_attention("qdec_rope_attention", q, ldq, kcache, vcache, pos, out, ldo, batch, q_heads, kv_heads, head_dim, max_len, scale, workspace,
                         workspace_bytes, dtype, NewToken{k, ldk, v, ldv, cos_table, sin_table, table_rows, status, aligned16(cos_table) && aligned16(sin_table)}, stream);
}

extern "C" int qdec_silu_mul(const void* gate, int64_t ldg, const void* up, int64_t ldu, void* y, int64_t ldy,
                             int rows, int width, int dtype, void* stream) {
    if (!gate || !up || !y || rows < 1 || width < 1) { set_error("qdec_silu_mul: null pointer or non-positive size"); return QGEMV_ERR_BAD_ARG; }
    if (dtype != QGEMV_F16 && dtype != QGEMV_BF16) { set_error("qdec_silu_mul: dtype must be fp16 or bf16"); return QGEMV_ERR_BAD_ARG; }
    if (ldg < width || ldu < width || ldy < width) { set_error("qdec_silu_mul: a leading dimension is smaller than width"); return QGEMV_ERR_SHAPE; }
    if (rows > 65535) { set_error("qdec_silu_mul: at most 65535 rows"); return QGEMV_ERR_TOO_LARGE; }
    const bool vec = width % 8 == 0 && aligned16(gate) && aligned16(up) && aligned16(y) && ldg % 8 == 0 && ldu % 8 == 0 && ldy % 8 == 0;
    const int units = vec ? width / 8 : width;
    int blocks = (units + 255) / 256;
    blocks = blocks < 1 ? 1 : blocks > 148 * 4 ? 148 * 4 : blocks;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const dim3 grid(blocks, rows), block(256);
    if (dtype == QGEMV_BF16)
        return launch_pdl("silu_mul_kernel", silu_mul_kernel<true>, grid, block, s, gate, (long long)ldg, up, (long long)ldu, y, (long long)ldy, width, vec);
    return launch_pdl("silu_mul_kernel", silu_mul_kernel<false>, grid, block, s, gate, (long long)ldg, up, (long long)ldu, y, (long long)ldy, width, vec);
}
