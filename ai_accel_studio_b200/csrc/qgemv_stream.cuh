// Declarations of the streaming GEMV shared by its planner / launcher (qgemv_plan.cu) and its kernel (qgemv_stream.cu).
#pragma once
#include "qgemv_common.cuh"

namespace qgemv {

constexpr int kStreamTileRows = 16;    // weight rows of one mma tile
constexpr int kStreamMaxOutliers = 256;
constexpr int kStreamMaxSmem = 232448; // 227 KB: one CTA per SM

constexpr int kSlotRowBytes = 128;     // bytes of one weight row in a ring slot
constexpr int kTileBytes = kStreamTileRows * kSlotRowBytes;
constexpr int kSlotBytes = kTileBytes + kStreamTileRows * 16;   // the weights of a tile and 16 bytes of scales per row
constexpr int kMaxTiles = 2;           // tiles a warp keeps accumulators for (one row block)
constexpr int kMaxDepth = 4;           // ring depth in batches (one batch = one slot per tile of a row block)
constexpr int kHalfSmem = 115712;      // 113 KB: two CTAs per SM, so that the next launch is resident while this one runs
constexpr size_t kStreamWordFloats = size_t(1) << 17;     // scratch kept for {value, launch tag} words, in 32-bit units
constexpr int kProjectionK = 256;      // K columns of one round of an in-kernel residual projection

// Weight formats: packed codes by the scale groups per 128-column block.
enum StreamFormat { kInt2G128 = 0, kInt2G64 = 1, kInt4G128 = 2, kInt4G64 = 3, kInt4G32 = 4 };

// The weight matrix of a launch: its operands and how it is cut.
struct StreamSeg {
    const uint8_t* w;         long long ldw;      // weight rows, leading dimension in bytes
    const __half* sc;         long long lds;
    const __half* bias;
    const int32_t* oidx;
    const __half* ow;         long long ldow;
    const __half* ru;         long long ldu;
    const __half* rv;         long long ldv;
    void* y;                  long long ldy;
    unsigned long long* tparts;                   // {value, launch tag} words of the residual projections
    float* partial;                               // fp32 sums of a K split: [split][row][m]
    int* counters;                                // arrivals per row group of a K split
    int n, fmt, row_bytes, act;
    int ng, gshift;                               // scale groups per row; log2(group / 128) for groups of 128 and more
    int oc, noc;                                  // outlier columns, blocks of 32 of them
    int rank, t_parts, t_parts_split, t_rounds;   // residual: K parts (all / per split), rounds of kProjectionK columns per part
    int flags;
    // geometry
    int groups, ksplit, rows_per;                 // row groups, K splits, rows of one row group
    int ns, ns_split;                             // weight slots per row, and per K split
    int wk, wr;                                   // warps along K, warps along the rows
    int tiles_w, nrb, T, depth;                   // tiles per warp, row blocks per warp, tiles per row block, ring depth
    int np, nu_magic;                             // 8-column pieces of x per activation row held in shared memory; divisor np / 2
    int xpitch;                                   // bytes between two activation rows in shared memory
    int sx_bytes;                                 // one warp's table of group sums
    int off_up, off_xo, off_upo, off_ow, off_sx, off_part, off_u, off_bias, off_tt, off_ring;   // shared memory (x starts at 0)
    int rows_pad, mp, upitch;
};
enum { kSegScaleAligned = 1, kSegOutlierAligned = 2, kSegVAligned = 4, kSegUAligned = 8 };

struct StreamArgs {
    const void* x;            long long ldx;
    int m, korig, nw;
    int xaligned, debug;
    int* status;                                  // wait-timeout status word
    unsigned long long* epoch;                    // launches of the workspace with residual projections, times 256
    StreamSeg seg;
};

// The plan of a launch: everything but the addresses that change from call to call (x, y, scratch).
struct StreamPlan {
    bool ok, epoch;
    int grid, threads, smem, mode;                // mode: 0 integer path (1 - 2 rows), 1 fp16 path (to 8), 2 (to 16)
    size_t t_off, part_off, cnt_off;              // bytes from the workspace base
    StreamArgs args;
};
int sm_count();                                       // of the current device
int stream_format(int bits, int group);               // -1: not built
// `partial_floats`: capacity of the workspace's scratch area.
bool plan_stream(const qgemv_problem& p, size_t partial_floats, StreamPlan* out);
// `dependent`: may start before the preceding kernel of the stream has finished (the weights are final).
int launch_stream(StreamPlan& plan, bool bf16, bool dependent, void* workspace, cudaStream_t s);

}  // namespace qgemv
