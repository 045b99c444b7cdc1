// Geometry of the streaming GEMV: how the weight rows, K and the warps are cut for a given problem, and the launch.
#include "qgemv_stream.cuh"

namespace qgemv {

int sm_count() {
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { (void)cudaGetLastError(); return 148; }
    if (cached[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) { (void)cudaGetLastError(); n = 148; }
        cached[dev] = n;
    }
    return cached[dev];
}

namespace {
int log2_exact(int v) { int s = 0; while ((1 << s) < v) ++s; return (1 << s) == v ? s : -1; }

}  // namespace

int stream_format(int bits, int group) {
    if (bits == 2 && group == 64) return kInt2G64;
    if (bits == 4 && group == 32) return kInt4G32;
    if (bits == 4 && group == 64) return kInt4G64;
    if (group % 128 || log2_exact(group / 128) < 0) return -1;
    return bits == 2 ? kInt2G128 : kInt4G128;
}

namespace {

bool al(const void* q, size_t a) { return reinterpret_cast<uintptr_t>(q) % a == 0; }
int up_to(int v, int a) { return (v + a - 1) / a * a; }
int cdiv(int a, int b) { return (a + b - 1) / b; }

constexpr int kCodesPerSlot[5] = {512, 512, 256, 256, 256};
constexpr int kBlocksPerSlot[5] = {4, 4, 2, 2, 2};               // 128-column blocks
constexpr int kGroupsPerBlock[5] = {1, 2, 1, 2, 4};

// Instructions of a warp per tile and slot, and per slot and row block (fetching activations), by path and format: counted
// from the main loop.  A whole launch executes about half as many again (14336 x 4096 INT2, 16 rows: 7.7 M warp instructions by
// counter, 5 M by these), so only their ratios to each other and to the bytes matter here.
constexpr int kTileCost[2][5] = {{220, 260, 110, 130, 170}, {320, 400, 170, 210, 300}};
constexpr int kSlotCost[2][5] = {{180, 180, 110, 110, 110}, {220, 240, 130, 140, 150}};

constexpr int kMaxJobs = 32;                          // CTAs of a split that compute residual projections

// Lays out one matrix for `ctas` CTAs of `nw` warps and `cap` bytes of shared memory; false if it does not fit.
// What is chosen: K splits between CTAs (S), warps along K (wk; the others along the rows), tiles per row block (T), ring
// depth.  Estimated clocks of a CTA: the larger of its stream (HBM gives an SM 23 bytes a clock, less when the ring keeps
// under 40 KB in flight) and its instructions (four schedulers, measured 0.55 per clock), a third of the smaller, and 2500
// for a hand-over between splits.
bool plan_segment(const qgemv_problem& p, int m, int mode, bool bf16, int nw, int ctas, int cap, size_t split_floats, size_t word_floats, StreamSeg& out, int& smem_out) {
    const int fmt = out.fmt, cps = kCodesPerSlot[fmt], nb = mode == 2 ? 2 : 1;
    const bool digits = mode == 0;
    const int tiles = cdiv(p.n, kStreamTileRows), rtiles = cdiv(p.rank, kStreamTileRows);
    out.ns = cdiv(out.row_bytes, kSlotRowBytes);
    out.mp = up_to(m, 2);
    out.upitch = up_to(p.rank * 2, 16);
    const int first = 1;
    long long best = -1;
    for (int S = first; S <= 32 && S <= ctas && S <= out.ns; ++S) {
        if (best >= 0 && S > first + 3) break;
        StreamSeg s = out;
        s.ns_split = cdiv(s.ns, S);
        s.ksplit = cdiv(s.ns, s.ns_split);
        if (s.ksplit != S) continue;
        const int R = ctas / S;
        s.rows_per = R >= tiles ? kStreamTileRows : cdiv(p.n, R);
        if (p.act == QGEMV_ACT_SILU_MUL) s.rows_per = up_to(s.rows_per, kStreamTileRows);
        s.groups = cdiv(p.n, s.rows_per);
        const int nt = cdiv(s.rows_per, kStreamTileRows);
        s.rows_pad = nt * kStreamTileRows;
        s.np = up_to(s.ns_split * cps / 8, 16);
        s.nu_magic = (int)(0xffffffffu / (unsigned)(s.np / 2) + 1u);
        s.xpitch = up_to(s.np * 16, 128) + 32;
        // residual projections: K parts of t_rounds * 256 columns, one warp each
        s.t_parts = s.t_parts_split = 0; s.t_rounds = 1;
        size_t words = 0;
        if (p.rank > 0) {
            const int slice = s.ns_split * cps < p.k_original ? s.ns_split * cps : p.k_original;
            for (;; s.t_rounds *= 2) {
                s.t_parts_split = cdiv(slice, kProjectionK * s.t_rounds);
                s.t_parts = s.t_parts_split * S;
                words = (size_t)s.t_parts * p.rank * m;
                // in the first CTAs of a split: they start first.  One of them may still wait for words of a later one that is
                // not resident yet; every wait is bounded, and running out is reported by the workspace's status word.
                if ((words <= 1024 && rtiles * s.t_parts_split <= (s.groups < kMaxJobs ? s.groups : kMaxJobs)) || s.t_parts_split == 1) break;
            }
        }
        if (words * 2 + 2 > word_floats || (S > 1 && (size_t)S * p.n * s.mp > split_floats)) continue;
        int off = digits ? s.np / 16 * m * 512 : m * s.xpitch;
        s.off_up = off;   off = up_to(off + (digits || bf16 ? s.np / 16 * m * 4 : 0), 16);
        s.off_xo = off;   off += s.noc ? m * (s.noc * 64 + 16) : 0;
        s.off_upo = off;  off = up_to(off + (bf16 ? s.noc * m * 4 : 0), 128);
        s.off_ow = off;   off += (s.noc + 1) / 2 * s.rows_pad * kSlotRowBytes;
        s.off_u = off;    off += p.rank ? s.rows_pad * s.upitch : 0;
        s.off_bias = off; off = up_to(off + (p.bias ? s.rows_pad * 2 : 0), 16);
        s.off_tt = off;   off = up_to(off + s.upitch / 2 * s.mp * 4, 128);
        const int fixed = off;
        for (s.wk = 1; s.wk <= nw && s.wk <= s.ns_split; s.wk *= 2) {
            s.wr = nw / s.wk;
            s.tiles_w = cdiv(nt, s.wr);
            const int q = cdiv(s.ns_split, s.wk);
            for (s.T = 1; s.T <= kMaxTiles && s.T <= s.tiles_w; ++s.T) {
                s.nrb = cdiv(s.tiles_w, s.T);
                s.sx_bytes = mode != 0 && s.nrb > 1 ? q * kBlocksPerSlot[fmt] * kGroupsPerBlock[fmt] * nb * 32 : 0;
                s.off_sx = fixed;
                s.off_part = fixed + nw * s.sx_bytes;
                s.off_ring = up_to(s.off_part + s.wk * s.rows_pad * s.mp * 4, 128);
                const int batches = s.nrb * q;
                int smem = 0;
                for (s.depth = batches < 2 ? 2 : batches < kMaxDepth ? batches : kMaxDepth; s.depth >= 2; --s.depth) {
                    smem = s.off_ring + nw * s.depth * s.T * kSlotBytes;
                    if (smem <= cap) break;
                }
                if (s.depth < 2) continue;
                const long long ring = (long long)nw * s.depth * s.T * kSlotBytes, bytes = (long long)s.rows_per * s.ns_split * kSlotRowBytes;
                long long stream = bytes / 23;
                if (ring < bytes && ring < 40 * 1024) stream = stream * (40 * 1024) / ring;
                const long long instr = (long long)batches * (kTileCost[mode != 0][fmt] * s.T * (mode == 2 ? 3 : 2) / 2 + kSlotCost[mode != 0][fmt]);
                const long long issue = instr * nw * 100 / (4 * 55);
                const long long cost = (stream > issue ? stream + issue / 3 : issue + stream / 3) + (S > 1 ? 2500 : 0) + s.wk * 10;
                if (best < 0 || cost < best) { best = cost; out = s; smem_out = smem; }
            }
        }
    }
    return best >= 0;
}

}  // namespace

bool plan_stream(const qgemv_problem& p, size_t partial_floats, StreamPlan* out) {
    *out = StreamPlan{};
    StreamArgs& a = out->args;
    StreamSeg& s = a.seg;
    const int m = p.m;
    if (m < 1 || m > 16 || !al(p.x, 16)) return false;
    const int mode = m > 8 ? 2 : m > 2 ? 1 : 0, sms = sm_count();
    const bool bf16 = p.x_dtype == QGEMV_BF16;
    s.fmt = stream_format(p.bits, p.group);
    if (s.fmt < 0 || !al(p.packed, 16) || p.ldp % 16 || p.outliers > kStreamMaxOutliers || p.rank > kMaxRank || !al(p.scales, 2)) return false;
    s.w = p.packed; s.ldw = p.ldp;
    s.sc = static_cast<const __half*>(p.scales); s.lds = p.lds;
    s.bias = static_cast<const __half*>(p.bias);
    s.oidx = p.outlier_idx; s.ow = static_cast<const __half*>(p.outlier_w); s.ldow = p.ldow;
    s.ru = static_cast<const __half*>(p.res_u); s.ldu = p.ldu;
    s.rv = static_cast<const __half*>(p.res_v); s.ldv = p.ldv;
    s.y = p.y; s.ldy = p.ldy;
    s.n = p.n; s.act = p.act;
    s.row_bytes = (int)((long long)p.k_padded * p.bits / 8);
    s.ng = p.k_padded / p.group;
    s.gshift = p.group >= 128 ? log2_exact(p.group / 128) : 0;
    s.oc = p.outliers; s.noc = cdiv(p.outliers, 32);
    s.rank = p.rank;
    // a slot's scales of a row as one aligned copy of 4, 8 or 16 bytes
    const int count = kBlocksPerSlot[s.fmt] * kGroupsPerBlock[s.fmt] >> s.gshift, halves = count < 2 ? 2 : count;
    if (al(p.scales, halves * 2) && p.lds % halves == 0) s.flags |= kSegScaleAligned;
    if (p.outliers && al(p.outlier_w, 16) && p.ldow % 8 == 0 && p.outliers % 8 == 0) s.flags |= kSegOutlierAligned;
    if (p.rank && al(p.res_v, 16) && p.ldv % 8 == 0) s.flags |= kSegVAligned;
    if (p.rank && al(p.res_u, 16) && p.ldu % 8 == 0 && p.rank % 8 == 0) s.flags |= kSegUAligned;
    // Split sums from the start of the scratch; words of residual projections in a region of their own at its end, below
    // the one of the other kernels: a word is recognised by its launch tag, and no other data, nor tags of another count,
    // may ever be taken for one.
    if (partial_floats < kTPartFloats + kStreamWordFloats) return false;
    const size_t floor = partial_floats - kTPartFloats - kStreamWordFloats, tail = partial_floats - kTPartFloats;
    // Half-SM CTAs let two launches of a chain share an SM (the next one fetches its weights while this one runs); a
    // whole-SM CTA has 16 warps and a deep ring: for few rows of activations it pays once a launch streams so much that its
    // start and end no longer count, for more than 8 rows (whose fragments need the registers) always.
    const bool big = (size_t)p.n * s.row_bytes / sms >= 400 * 1024, first = m > 4 || big;
    for (int t = 0; t < (m > 8 ? 1 : 2); ++t) {
        const bool whole = t == 0 ? first : !first;
        const int nw = mode == 2 || !whole ? 8 : 16, cap = whole ? kStreamMaxSmem : kHalfSmem;
        int smem = 0;
        if (!plan_segment(p, m, mode, bf16, nw, sms, cap, floor, tail - floor, s, smem)) continue;
        const int ctas = s.groups * s.ksplit;
        if (ctas > 256) continue;
        out->t_off = kWsPartialOff + ((tail - (size_t)s.t_parts * s.rank * m * 2) & ~(size_t)1) * sizeof(float);
        out->part_off = kWsPartialOff;
        out->cnt_off = kWsCounterOff;
        a.x = p.x; a.ldx = p.ldx; a.m = m; a.korig = p.k_original; a.nw = nw;
        a.xaligned = p.ldx % 8 == 0 ? 1 : 0;
        a.debug = p.debug;
        out->epoch = s.rank > 0;
        out->grid = ctas; out->threads = (nw + 1) * 32; out->smem = smem; out->mode = mode;
        out->ok = true;
        return true;
    }
    return false;
}

template <int MODE, bool BF16> int launch_stream_mode(const StreamArgs& a, bool dependent, int grid, int threads, int smem, cudaStream_t s);

int launch_stream(StreamPlan& plan, bool bf16, bool dependent, void* workspace, cudaStream_t s) {
    StreamArgs& a = plan.args;
    char* ws = static_cast<char*>(workspace);
    int* cnt = reinterpret_cast<int*>(ws + kWsCounterOff);
    a.status = cnt + kWsStatusIdx;
    a.epoch = plan.epoch ? reinterpret_cast<unsigned long long*>(cnt + kWsStreamEpochIdx) : nullptr;
    a.seg.tparts = reinterpret_cast<unsigned long long*>(ws + plan.t_off);
    a.seg.partial = reinterpret_cast<float*>(ws + plan.part_off);
    a.seg.counters = reinterpret_cast<int*>(ws + plan.cnt_off);
    decltype(&launch_stream_mode<0, false>) fn[3][2] = {{launch_stream_mode<0, false>, launch_stream_mode<0, true>},
                                                        {launch_stream_mode<1, false>, launch_stream_mode<1, true>},
                                                        {launch_stream_mode<2, false>, launch_stream_mode<2, true>}};
    return fn[plan.mode][bf16 ? 1 : 0](a, dependent, plan.grid, plan.threads, plan.smem, s);
}

}  // namespace qgemv
