// K2 for lists of problems of one shape with M <= 128 (and most single ones): the W4A16 GEMM on tcgen05 with the dequantised weights as the
// tensor-memory operand, tiles taken whole or cut between CTAs.
//
// No counterpart kernel exists in the reference (its INT4 support stops at the stand-alone dequantisation kernels,
// src/t0/quant_kernels.rs:53-171).  y[m,n] = sum_k a[m,k] * w[k,n],  w = RNE_bf16((q - z) * s),  fp32 accumulate.
//
// The work is a list of chunks, 256 columns x 64 k, problem by problem, tile by tile, k last; every CTA (one per SM) takes an
// equal contiguous range of it, and its warps go through that in pairs of chunks:
//   * one warp fetches the packed words, scales and zero points of a pair into a ring of raw stages (tile-major weights: a 16 KiB piece, plain copies; row
//     layout: TMA boxes) and its activations into another (two boxes; rows up to M rounded to 16; rows beyond M are zero-filled);
//   * sixteen warps, eight to a pair in turn, turn the words into bf16 (one LOP3 per nibble pair: 0x4300 | q is the bf16 128+q, minus 128+z, times s -
//     bit-identical to the oracle because (q-z)*s is rounded once) and put them straight into tensor memory (tcgen05.st): the
//     weights are the 128-row A operand, two halves of 128 columns of y;
//   * two warps, one per half, issue 8 tcgen05.mma (128 x M' x 16, M' = M rounded to 16) a pair with the activations as the B operand in shared
//     memory.  The accumulator is y transposed: lane = column of y, tensor-memory column = row of y;
//   * four warps empty the accumulators of the tiles that end inside the range (two sets where M <= 64, so that the next tile goes on meanwhile); the
//     last tile is emptied by the sixteen.
// A tile that lies wholly in one range is stored from tensor memory.  A tile cut by range boundaries is finished by the warps that
// reach it last: see there.
//
// Whole tiles per CTA leave SMs idle where the tiles are few or just over a multiple of them: two problems of N = 11008 are 86 tiles on 148
// SMs.  A launch takes its tiles whole or cut, or leaves a single problem to the clusters of w4a16_umma.cu: `w4a16_umma_plan` weighs them.
// What bounds it is the dequantisation's instructions (0.28 us a chunk up to M = 64; two pipes that take one per two cycles are half busy, the schedulers two
// thirds) and at M = 128 the UMMAs beside them (0.34; 0.27 of tensor work), and per launch with cut tiles 3 to 7 us for handing in and adding their parts.
// Two problems of N = 11008, K = 4096 at M = 32 / 128, in bursts of a few milliseconds: 24.4 / 29.1 us with one issuing warp, one loading by boxes and the sixteen
// emptying every tile; 20.9 / 26.6 with two issuing warps, predicated; 18.8 / 26.3 with warps that empty the accumulators; 18.4 / 24.7 in pairs, and with
// activations three pairs behind at M = 128 (25.7 in step).  In long blocks, where the clock settles, M = 128 takes 31.9 us (34.6 with one issuing warp).
#include "w4a16_common.cuh"

using namespace t0;
using namespace t0::w4;

namespace {

constexpr uint32_t kUmDqWarps = 16;
// + the warps that empty accumulators, issue and load.  The serial ones share a scheduler with dequantising warps and work through a chain of instructions per
// pair, so the chains are kept short: predicated instructions on uniform values, running addresses, no divisions.
constexpr uint32_t kUmEpWarp0 = kUmDqWarps, kUmEpWarps = 4;  // empty the accumulators of all but the last tile of a range, one per tensor-memory lane quadrant
constexpr uint32_t kUmIssueWarp = kUmEpWarp0 + kUmEpWarps, kUmLoadWarp = kUmIssueWarp + 2;     // (two issuing warps)
constexpr uint32_t kUmThreads = (kUmLoadWarp + 1) * 32;     // (a warp more, even an idle one, adds 0.3 us to a launch)
constexpr uint32_t kUmXBytes = 6 * 128 * kUmBK * 2;         // activations, in stages of two chunks: three at M = 128, four at M <= 96
constexpr uint32_t kUmMaxXStages = 4;
// Tensor memory (512 columns): accumulators 2 x 128 columns, then four A stages of 2 halves x 4 k-steps x 8 columns.
constexpr uint32_t kUmTmemCols = 512;
constexpr uint32_t kUmABase = 256;                          // first column of the A stages
constexpr uint32_t kUmAStageCols = 128;                     // of two chunks: [chunk][half][k-step] x 8
constexpr uint32_t kUmAStages = 2;                          // one to a set of eight warps
constexpr uint32_t kUmScaleOff = 2 * 8 * kUmBN * 4, kUmScaleStride = 1024, kUmRawStage = kUmScaleOff + 2 * kUmScaleStride;      // words of two chunks, then scales and zero points
constexpr uint32_t kUmRawStages = 6;                        // raw weight stages of two chunks: 106 KB in flight per SM (an even number: a set of warps has every second one)
// (more than half an SM's shared memory: the kernel takes all 512 tensor-memory columns, so two of its CTAs must never share an SM)
constexpr uint32_t kUmSmem = kUmRawStages * kUmRawStage + kUmXBytes + 512 + 1024;
constexpr uint32_t kUmMinChunks = 4;                        // a CTA's range is at least this long where sums may be: below it the finish costs more than the range
constexpr size_t kUmCounterBytes = 16 * 1024;               // one word per CTA and dequantisation warp (up to 256 CTAs)

struct UmParams {
    int* status;
    uint32_t* counters;      // [grid][16]: arrivals at the tile that CTA begins and does not complete; zero between launches
    float* pieces;           // [grid][2][rows][256]: partial sums of the cut tiles (slot 0 = the CTA's first piece)
    uint64_t wait_limit_ns;
    uint32_t M, N;
    uint32_t rows;           // M rounded up to 16: width of the UMMAs and height of the activation boxes
    uint32_t n_tiles, n_chunks;
    uint32_t total;          // chunks of the launch, shared out evenly (less than 2^24)
    uint32_t whole;          // shared out by tiles instead: no tile is cut
    uint32_t tiles;          // of the launch: total / n_chunks
    uint32_t per_group;      // chunks per scale / zero-point row
    uint32_t x_stages;       // stages of activations
    UmDiv by_grid, by_total, by_chunks, by_tiles, by_group;   // the CTAs, total, n_chunks, n_tiles, per_group
    uint32_t off_scales, off_zeros;   // tile-major weights: where in a problem's buffer they begin, in units of 16 bytes
};

// First chunk of a CTA's range, and the CTA whose range holds a chunk (at most 256 CTAs and 2^24 chunks, so that products fit 32 bits; whole tiles: 2^23 tiles).
__device__ __forceinline__ uint32_t um_begin(uint32_t cta, const UmParams& p) {
    return p.whole ? um_div(cta * p.tiles, p.by_grid) * p.n_chunks : um_div(cta * p.total, p.by_grid);
}
__device__ __forceinline__ uint32_t um_owner(uint32_t chunk, const UmParams& p) { return um_div((chunk + 1) * gridDim.x - 1, p.by_total); }

// kTiled: weights in the tile-major layout (3-D maps: column in tile, row, tile), else the row layout; kProblems: room for so many problems
template <bool kTiled, uint32_t kProblems>
__global__ void __launch_bounds__(kUmThreads, 1)
w4a16_umma_cut_kernel(const UmParams p, const __grid_constant__ UmGroup<kProblems, kTiled> group) {
    constexpr uint32_t kMaps = kTiled ? 1 : 4;                // tensor maps of a problem, the activations' last
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t raw_ring = smem;
    const uint32_t x_ring = smem + kUmRawStages * kUmRawStage;           // activations: [rows][64 k] bf16, 128-byte swizzle, per stage
    const uint32_t bars = x_ring + kUmXBytes;
    const uint32_t raw_full = bars, raw_empty = bars + 8 * kUmRawStages;
    const uint32_t a_full = raw_empty + 8 * kUmRawStages, a_empty = a_full + 8 * 2 * kUmAStages;     // [128-column half][stage]
    const uint32_t x_full = a_empty + 8 * 2 * kUmAStages, x_empty = x_full + 8 * kUmMaxXStages;
    const uint32_t acc_full = x_empty + 8 * kUmMaxXStages, acc_empty = acc_full + 16;                // [accumulator set]
    const uint32_t tail_full = acc_empty + 16;               // the range's last piece is complete
    const uint32_t x_bytes = p.rows * kUmBK * 2, x_stages = p.x_stages;
    __shared__ uint32_t tmem_holder;
    __shared__ int s_abort;
    volatile int* abort_flag = &s_abort;
    const uint32_t tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;
    const uint32_t n_chunks = p.n_chunks;
    const uint32_t u0 = um_begin(blockIdx.x, p), u1 = um_begin(blockIdx.x + 1, p);
    const uint32_t acc_sets = p.rows <= 64 ? 2 : 1;          // accumulators of 128 columns a half: two sets, taken in turn, where a tile needs no more than half of them

    if (tid == 0) {
        for (uint32_t s = 0; s < kUmRawStages; ++s) {
            ptx::mbar_init(raw_full + 8 * s, 1);
            ptx::mbar_init(raw_empty + 8 * s, kUmDqWarps / 2);
        }
        for (uint32_t s = 0; s < 2 * kUmAStages; ++s) {
            ptx::mbar_init(a_full + 8 * s, kUmDqWarps / 4);       // the four warps that dequantise this half of the chunk
            ptx::mbar_init(a_empty + 8 * s, 1);
        }
        for (uint32_t s = 0; s < x_stages; ++s) {
            ptx::mbar_init(x_full + 8 * s, 1);
            ptx::mbar_init(x_empty + 8 * s, 2);
        }
        for (uint32_t s = 0; s < 2; ++s) {
            ptx::mbar_init(acc_full + 8 * s, 2);
            ptx::mbar_init(acc_empty + 8 * s, kUmEpWarps);
        }
        ptx::mbar_init(tail_full, 2);
        s_abort = 0;
        ptx::fence_barrier_init();
        ptx::fence_proxy_async_smem();
        for (uint32_t i = 0; i < kMaps; ++i) ptx::tma_prefetch_desc(&group.maps[kMaps * um_div(um_div(u0, p.by_chunks), p.by_tiles) + i]);
    }
    if (warp == kUmIssueWarp) {
        ptx::tmem_alloc(ptx::smem_u32(&tmem_holder), kUmTmemCols);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    ptx::tc_fence_after_sync();
    constexpr uint32_t tmem_base = 0;    // all columns are allocated: tensor-memory addresses are constants
    ptx::grid_launch_dependents();
    // where the range begins: tile and chunk, problem, row of scales
    const uint32_t per_group = p.per_group;
    const uint32_t item0 = um_div(u0, p.by_chunks), c0 = u0 - item0 * n_chunks, prob0 = um_div(item0, p.by_tiles), tile0 = item0 - prob0 * p.n_tiles;
    const uint32_t at0 = u0 - prob0 * n_chunks * p.n_tiles, row0 = um_div(at0, p.by_group), in_row0 = at0 - row0 * per_group;
    ptx::grid_dependency_wait();

    // The chunks of a range are taken in pairs, an even chunk of a tile and the next one; a pair is short where the range begins or ends inside it, or the tile
    // with an odd number.  Chunk i of a pair has place i of its stages.  Every role walks the pairs so: n chunks, the first of them i0.
    struct Pairs {
        uint32_t u, c, i0, n;                        // chunk of the launch, chunk of the tile
    };
    auto first_pair = [&]() { Pairs w; w.u = u0; w.c = c0; w.i0 = w.c & 1; w.n = min(min(2 - w.i0, n_chunks - w.c), u1 - u0); return w; };
    auto next_pair = [&](Pairs& w) {
        w.u += w.n; w.c += w.n;
        if (w.c == n_chunks) w.c = 0;
        w.i0 = 0;                                    // (all but the first begin at an even chunk)
        w.n = min(min(2u, n_chunks - w.c), u1 - w.u);
    };
    // The serial roles walk with their whole warp and let one elected lane issue: see ptx::mbar_wait_warp.
    if (warp == kUmLoadWarp) {
        // -------------------------------------------------------------- raw weights, scales and zero points; activations (one box per chunk, rows beyond M are zero)
        // Weights have six stages, activations three or four.  With three (M > 96) the activations follow the weights at that distance once these are full, so
        // that weights are not asked for late: 2 x (128 x 11008 x 4096) 25.7 us in step, 24.7 so.  With four the longer chain of this warp costs more: 2 x (64 x
        // 1024 x 4096) 12.6 and 12.8.
        uint32_t stage = 0, phase = 0, xs = 0, xphase = 0, x_dst = x_ring;
        uint32_t prob = prob0, tile = tile0, at = at0, row = row0, in_row = in_row0;      // at: chunk of the problem, row: its row of scales
        uint32_t x_prob = prob0, x_tile = tile0;
        const uint32_t rows_a_pair = per_group & 1 ? 2 : 1;
        Pairs w = first_pair(), wx = w;
        for (uint32_t j = 0; wx.u < u1; ++j) {
            const uint32_t issue = ptx::elect_one();
            if (w.u < u1) {
                if (!ptx::mbar_wait_warp(raw_empty + 8 * stage, phase ^ 1, abort_flag, p.wait_limit_ns)) {
                    if (lane == 0) atomicCAS(p.status, 0, kStatusProducerTimeout | (int)(w.u & 0xFFFFFF));
                    break;
                }
                const uint32_t fb = raw_full + 8 * stage, dst = raw_ring + stage * kUmRawStage;
                ptx::fence_proxy_async_smem();       // the stage was read through the generic proxy, the copies write it through the async proxy
                // a scale row for each chunk, or (group a multiple of two chunks) one for both, in place 0
                const uint32_t rows = rows_a_pair == 1 ? 1 : w.n, i0 = rows_a_pair == 1 ? 0 : w.i0, step = in_row + 1 == per_group ? 1 : 0;      // to the second chunk's row
                ptx::mbar_arrive_expect_tx_if(issue, fb, w.n * (8 * kUmBN * 4) + rows * (kUmBN * 2 + kUmBN / 2));
                if constexpr (kTiled) {
                    // the words of a problem lie one behind the other in the order of its chunks, its scales and zero points likewise
                    const uint8_t* base = group.base[prob];
                    ptx::bulk_load_if(issue, dst + w.i0 * (8 * kUmBN * 4), base + (size_t)at * (8 * kUmBN * 4), w.n * (8 * kUmBN * 4), fb);
                    for (uint32_t k = 0; k < rows; ++k) {
                        ptx::bulk_load_if(issue, dst + kUmScaleOff + (i0 + k) * kUmScaleStride, base + (size_t)p.off_scales * 16 + (size_t)(row + k * step) * (kUmBN * 2), kUmBN * 2, fb);
                        ptx::bulk_load_if(issue, dst + kUmScaleOff + (i0 + k) * kUmScaleStride + kUmBN * 2, base + (size_t)p.off_zeros * 16 + (size_t)(row + k * step) * (kUmBN / 2), kUmBN / 2, fb);
                    }
                } else {
                    const CUtensorMap* const mw = &group.maps[4 * prob];
                    const uint32_t grp = row - um_div(tile * n_chunks, p.by_group);
                    for (uint32_t k = 0; k < w.n; ++k)
                        ptx::tma_load_2d_if(issue, dst + (w.i0 + k) * (8 * kUmBN * 4), mw, fb, (int32_t)(tile * kUmBN), (int32_t)((w.c + k) * (kUmBK / 8)));
                    for (uint32_t k = 0; k < rows; ++k) {
                        ptx::tma_load_2d_if(issue, dst + kUmScaleOff + (i0 + k) * kUmScaleStride, mw + 1, fb, (int32_t)(tile * kUmBN), (int32_t)(grp + k * step));
                        ptx::tma_load_2d_if(issue, dst + kUmScaleOff + (i0 + k) * kUmScaleStride + kUmBN * 2, mw + 2, fb, (int32_t)(tile * (kUmBN / 8)), (int32_t)(grp + k * step));
                    }
                }
                at += w.n;
                in_row += w.n;
                while (in_row >= per_group) { in_row -= per_group; ++row; }
                if (w.c + w.n == n_chunks && ++tile == p.n_tiles) { tile = 0; ++prob; at = row = in_row = 0; }
                if (++stage == kUmRawStages) { stage = 0; phase ^= 1; }
                next_pair(w);
                if (x_stages < kUmMaxXStages && j >= x_stages && j < kUmRawStages) continue;
            }
            if (!ptx::mbar_wait_warp(x_empty + 8 * xs, xphase ^ 1, abort_flag, p.wait_limit_ns)) {
                if (lane == 0) atomicCAS(p.status, 0, kStatusProducerTimeout | 0x400000 | (int)(wx.u & 0x3FFFFF));
                break;
            }
            const CUtensorMap* const mx = &group.maps[kMaps * x_prob + kMaps - 1];
            ptx::mbar_arrive_expect_tx_if(issue, x_full + 8 * xs, wx.n * x_bytes);
            ptx::tma_load_3d_if(issue, x_dst + wx.i0 * x_bytes, mx, x_full + 8 * xs, (int32_t)(wx.c * kUmBK), 0, 0);
            ptx::tma_load_3d_if(issue & (wx.n >> 1), x_dst + x_bytes, mx, x_full + 8 * xs, (int32_t)((wx.c + 1) * kUmBK), 0, 0);
            __syncwarp();
            if (wx.c + wx.n == n_chunks && ++x_tile == p.n_tiles) { x_tile = 0; ++x_prob; }
            x_dst += 2 * x_bytes;
            if (++xs == x_stages) { xs = 0; xphase ^= 1; x_dst = x_ring; }
            next_pair(wx);
        }
    } else if (warp >= kUmIssueWarp) {
        // -------------------------------------------------------------- UMMA issuers, one per half of the columns: per chunk 4 k-steps of M 128 x N rows x K 16
        const uint32_t idesc = ptx::make_idesc_bf16_f32(128, p.rows, 0u), t = warp - kUmIssueWarp;
        const uint32_t my_full = a_full + 8 * kUmAStages * t, my_empty = a_empty + 8 * kUmAStages * t;
        const uint32_t x0 = (x_ring & 0x3FFFFu) >> 4, a_cols = kUmABase + t * 32;      // (addresses enter a descriptor in 16-byte units)
        uint32_t set = 0, aphase = 0, xs = 0, xphase = 0, x = x0, piece = 0;           // set: whose A stages, 2 set and 2 set + 1, are next
        uint32_t acc = t * 128, more = 0;                                              // the piece's accumulator, empty so far or not
        for (Pairs w = first_pair(); w.u < u1; next_pair(w)) {
            if (!ptx::mbar_wait_warp(x_full + 8 * xs, xphase, abort_flag, p.wait_limit_ns) ||
                !ptx::mbar_wait_warp(my_full + 8 * set, aphase, abort_flag, p.wait_limit_ns)) {
                if (lane == 0) atomicCAS(p.status, 0, kStatusMmaTimeout | (int)(w.u & 0x7FFFFF));
                break;
            }
            ptx::tc_fence_after_sync();
            const uint32_t issue = ptx::elect_one();
#pragma unroll
            for (uint32_t i = 0; i < 2; ++i) {
                if (i < w.i0 || i >= w.i0 + w.n) continue;
                const uint32_t a = a_cols + set * kUmAStageCols + i * 64, xi = x + i * (x_bytes / 16);
                ptx::umma_bf16_ts_if(issue, acc, a, xi, idesc, more);
#pragma unroll
                for (uint32_t k4 = 1; k4 < kUmBK / 16; ++k4) ptx::umma_bf16_ts_if<true>(issue, acc, a + k4 * 8, xi + k4 * 2, idesc);
                more = 1;
            }
            ptx::umma_commit_if(issue, my_empty + 8 * set);
            ptx::umma_commit_if(issue, x_empty + 8 * xs);
            if (w.c + w.n == n_chunks || w.u + w.n == u1) {
                // the piece is complete; on to the next one's accumulators, which the epilogue warps must have emptied
                // (the last one has a barrier of its own: the dequantising warps come to it without having waited for the pieces before, so that the phase of a
                // shared one would not tell them which piece is complete)
                ptx::umma_commit_if(issue, w.u + w.n == u1 ? tail_full : acc_full + 8 * (acc_sets == 2 ? piece & 1 : 0));
                __syncwarp();
                ++piece;
                const uint32_t s = acc_sets == 2 ? piece & 1 : 0, use = acc_sets == 2 ? piece >> 1 : piece;
                if (w.u + w.n < u1 && use > 0 && !ptx::mbar_wait_warp(acc_empty + 8 * s, (use - 1) & 1, abort_flag, p.wait_limit_ns)) {
                    if (lane == 0) atomicCAS(p.status, 0, kStatusMmaTimeout | 0x800000);
                    break;
                }
                ptx::tc_fence_after_sync();
                acc = t * 128 + s * 64;
                more = 0;
            }
            __syncwarp();
            aphase ^= set;
            set ^= 1;
            x += 2 * (x_bytes / 16);
            if (++xs == x_stages) { xs = 0; xphase ^= 1; x = x0; }
        }
    } else {
        const uint32_t q = warp & 3, lane_base = (q * 32) << 16;             // lane quadrant
        const bool dq = warp < kUmDqWarps;
        bool ok = true;
        if (dq) {
            // ---------------------------------------------------------- sixteen warps: dequantise into tensor memory
            // Eight warps take two chunks of the range, a raw stage, the other eight the next two: a thread has one column and all eight words of a chunk, so
            // that what stands around the arithmetic is paid once per eight words.  They go on over the ends of tiles.
            const uint32_t t = (warp >> 2) & 1, h = warp >> 3;               // 128-column half of the tile, which of the two sets
            const uint32_t n = t * 128 + q * 32 + lane;                      // this thread's column of the tile
            uint32_t mask, magic;
            asm volatile("mov.b32 %0, 0x000F000F;" : "=r"(mask));
            asm volatile("mov.b32 %0, 0x43004300;" : "=r"(magic));
            const uint32_t my_full = a_full + 8 * (kUmAStages * t + h), my_empty = a_empty + 8 * (kUmAStages * t + h);
            const uint32_t lane_w = raw_ring + n * 4, lane_s = raw_ring + kUmScaleOff + n * 2, lane_z = raw_ring + kUmScaleOff + kUmBN * 2 + (n >> 3) * 4;
            const uint32_t a_col = tmem_base + lane_base + kUmABase + h * kUmAStageCols + t * 32;
            const uint32_t second = per_group & 1 ? kUmScaleStride : 0;      // where the second chunk's scales and zero points are: its own, or the first one's
            uint32_t rs = h, rphase = 0, aphase = 0;
            Pairs w = first_pair();
            if (h) next_pair(w);
            for (; w.u < u1; next_pair(w), next_pair(w)) {
                // The A stage is free once the UMMAs of this set's pair before have read it.  (Waited for here and not before the stores: values that
                // live across a wait are moved once more to where the store takes them.)
                ok = ptx::mbar_wait(raw_full + 8 * rs, rphase, abort_flag, p.wait_limit_ns) &&
                     ptx::mbar_wait(my_empty, aphase ^ 1, abort_flag, p.wait_limit_ns);
                if (!ok) {
                    if (lane == 0) atomicCAS(p.status, 0, kStatusEpilogueTimeout | (int)(w.u & 0x3FFFFF));
                    break;
                }
                ptx::tc_fence_after_sync();
                const uint32_t off = rs * kUmRawStage;
                // (both chunks, also where a pair is short: what comes of the bytes that happen to be there is not used)
#pragma unroll
                for (uint32_t i = 0; i < 2; ++i) {
                    uint32_t words[8];
#pragma unroll
                    for (uint32_t j = 0; j < 8; ++j) words[j] = um_lds32(lane_w + off + (8 * i + j) * (kUmBN * 4));
                    const uint32_t sbits = um_lds16(lane_s + off + i * second), zword = um_lds32(lane_z + off + i * second);
                    const uint32_t zz = ((zword >> ((n & 7) * 4)) & 0xFu) * 0x00010001u + 0x43004300u;     // bf16x2 (128+z, 128+z)
                    const uint32_t ss = sbits * 0x00010001u;                                               // (s, s)
                    uint32_t r[32];                            // k order: (0,1) (2,3) ..., two consecutive k per tensor-memory column
#pragma unroll
                    for (uint32_t j = 0; j < 8; ++j) {
                        uint32_t d[4];
                        um_dequant_word(words[j], mask, magic, zz, ss, kTiled, d);
#pragma unroll
                        for (uint32_t e = 0; e < 4; ++e) r[4 * j + e] = d[e];
                    }
                    ptx::tmem_st_32x32b_x32(a_col + i * 64, r);
                }
                ptx::tmem_st_wait();
                ptx::tc_fence_before_sync();
                __syncwarp();
                ptx::mbar_arrive_if(my_full, lane == 0);
                ptx::mbar_arrive_if(raw_empty + 8 * rs, lane == 0);
                aphase ^= 1;
                rs += 2;
                if (rs >= kUmRawStages) { rs -= kUmRawStages; rphase ^= 1; }
            }
        }
        // ------------------------------------------------------------------ accumulators to y, or to the parts of cut tiles
        // The last tile of a range is emptied by the sixteen warps, which have nothing else left to do, those before it by the four epilogue warps while the
        // sixteen go on.  Either way a tile is sixteen blocks, of 32 columns x half of the rows: block b has lane quadrant b % 4, column half (b / 4) % 2 and
        // row half b / 8.  A dequantising warp does one block, an epilogue warp the four of its quadrant.
        //
        // A tile cut by range boundaries: each of its CTAs holds a partial sum over a part of K.  A block is finished by whichever CTA gets to it
        // last.  A ticket is taken first (low half of the block's counter); all but the last then store their part and count it as
        // written (high half).  The last one waits for those counts: whoever it waits for holds a ticket, so is running,
        // and the tiles before in their range can only wait for CTAs further down.  It adds the parts in k order whoever it is:
        // repeated calls agree bit for bit.
        const uint32_t last_item = um_div(u1 - 1, p.by_chunks), n_pieces = last_item - item0 + 1, n_blocks = dq ? 1 : 4;
        const uint32_t u_last = n_pieces == 1 ? u0 : last_item * n_chunks;
        const uint32_t row4s = p.rows / 8;                                   // float4s of a block a lane holds, four rows of its column each
        const size_t piece_f4 = (size_t)p.rows * (kUmBN / 4);
        uint32_t piece = dq ? n_pieces - 1 : 0;
        for (uint32_t u = dq ? u_last : u0; ok && u < (dq ? u1 : u_last); ++piece) {
            const uint32_t item = item0 + piece, tile_u0 = item * n_chunks, tile_u1 = tile_u0 + n_chunks, u_end = min(u1, tile_u1);
            const bool cut = u != tile_u0 || u_end != tile_u1;
            const uint32_t set = acc_sets == 2 ? piece & 1 : 0, use = acc_sets == 2 ? piece >> 1 : piece;
            u = u_end;
            uint32_t c_first = 0, first_slot = 0, n_parts = 1, ticket = 0;   // lane i has the ticket of block i
            uint32_t* counter = nullptr;
            if (cut) {
                c_first = um_owner(tile_u0, p);
                n_parts = um_owner(tile_u1 - 1, p) - c_first + 1;
                first_slot = um_begin(c_first, p) < tile_u0 ? 1u : 0u;       // its range began in the tile before: this is not its first piece
                counter = p.counters + c_first * kUmDqWarps + (dq ? warp : q + 4 * (lane & 3));
                if (lane < n_blocks) ticket = atomicAdd(counter, 1u) & 0xFFFFu;        // (its round trip passes under the last UMMAs)
            }
            if (!ptx::mbar_wait(dq ? tail_full : acc_full + 8 * set, dq ? 0 : use & 1, abort_flag, p.wait_limit_ns)) {
                if (lane == 0) atomicCAS(p.status, 0, kStatusEpilogueTimeout | 0xC00000);
                break;
            }
            ptx::tc_fence_after_sync();
            __syncwarp();
            const uint32_t hand_in = __ballot_sync(0xFFFFFFFFu, lane < n_blocks && ticket + 1 != n_parts);
            // 32 columns of the accumulator (rows m0 .. of y) for this warp's columns of y; a narrow tile's columns beyond its rows are not used
            auto load_rows = [&](uint32_t b, uint32_t m0, float (&v)[32]) {
                uint32_t r[32];
                ptx::tmem_ld_32x32b_x32(tmem_base + lane_base + ((b >> 2) & 1) * 128 + set * 64 + m0, r);
                ptx::tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
            };
#pragma unroll 1
            for (uint32_t i = 0; i < n_blocks; ++i) {
                if (!(hand_in >> i & 1)) continue;
                const uint32_t b = dq ? warp : q + 4 * i;
                float4* mine = (float4*)p.pieces + ((size_t)blockIdx.x * 2 + (piece == 0 ? 0 : 1)) * piece_f4 + (size_t)b * row4s * 32 + lane;
#pragma unroll 1
                for (uint32_t r4 = 0; r4 < row4s; r4 += 8) {
                    float v[32];
                    load_rows(b, (b >> 3) * (p.rows / 2) + 4 * r4, v);
#pragma unroll
                    for (uint32_t j = 0; j < 8; ++j)
                        if (r4 + j < row4s) __stcg(mine + (r4 + j) * 32, make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]));
                }
            }
            ptx::tc_fence_before_sync();
            __syncwarp();
            const bool all_in = hand_in == (1u << n_blocks) - 1;
            if (!dq && all_in) ptx::mbar_arrive_if(acc_empty + 8 * set, lane == 0);        // nothing is left to read: the UMMAs may go on
            if (hand_in >> lane & 1) {
                __threadfence();                       // the block is visible before it is counted
                atomicAdd(counter, 0x10000u);
            }
            const uint32_t prob = um_div(item, p.by_tiles);
            float* const y_out = group.y[prob];
#pragma unroll 1
            for (uint32_t i = 0; ok && i < n_blocks; ++i) {
                if (hand_in >> i & 1) continue;
                const uint32_t b = dq ? warp : q + 4 * i, m_begin = (b >> 3) * (p.rows / 2), m_end = min(p.M, m_begin + p.rows / 2);
                if (n_parts > 1) {
                    uint32_t good = 1;
                    if (lane == i) {
                        uint64_t t_start = 0;
                        for (uint32_t spin = 1; (um_ld_acquire(counter) >> 16) + 1 != n_parts; ++spin) {
                            if ((spin & 0x3F) == 0) {
                                const uint64_t now = ptx::globaltimer_ns();
                                if (t_start == 0) t_start = now;
                                if (*abort_flag || now - t_start > p.wait_limit_ns) { *abort_flag = 1; good = 0; break; }
                            }
                        }
                        if (good) *counter = 0;            // ready for the next launch
                        else atomicCAS(p.status, 0, kStatusEpilogueTimeout | 0xE00000);
                    }
                    __syncwarp();                          // orders the other lanes' loads of the parts after that lane's acquire (a shuffle does not)
                    ok = __shfl_sync(0xFFFFFFFFu, good, i) != 0;
                    if (!ok) break;
                }
                const uint32_t col = (item - prob * p.n_tiles) * kUmBN + ((b >> 2) & 1) * 128 + q * 32 + lane;
                // Thirty-two rows at a time, part after part in k order.  What this costs is the round trips of the parts' loads, so eight of a lane's
                // 16-byte loads are under way together.
#pragma unroll 1
                for (uint32_t r4 = 0; r4 < row4s; r4 += 8) {
                    const uint32_t m0 = m_begin + 4 * r4;
                    float sum[32];
                    if (n_parts == 1) {
                        load_rows(b, m0, sum);
                    } else {
#pragma unroll
                        for (uint32_t j = 0; j < 32; ++j) sum[j] = 0.0f;
#pragma unroll 1
                        for (uint32_t part = 0; part < n_parts; ++part) {
                            float f[32];
                            const uint32_t cta = c_first + part;
                            if (cta == blockIdx.x) {
                                load_rows(b, m0, f);
                            } else {
                                const float4* theirs = (const float4*)p.pieces + ((size_t)cta * 2 + (part == 0 ? first_slot : 0u)) * piece_f4 + (size_t)b * row4s * 32 + lane;
#pragma unroll
                                for (uint32_t j = 0; j < 8; ++j) {
                                    const float4 x = r4 + j < row4s ? __ldcg(theirs + (r4 + j) * 32) : make_float4(0.f, 0.f, 0.f, 0.f);
                                    f[4 * j] = x.x; f[4 * j + 1] = x.y; f[4 * j + 2] = x.z; f[4 * j + 3] = x.w;
                                }
                            }
#pragma unroll
                            for (uint32_t j = 0; j < 32; ++j) sum[j] += f[j];
                        }
                    }
                    if (col < p.N) {
#pragma unroll
                        for (uint32_t j = 0; j < 32; ++j)
                            if (m0 + j < m_end) y_out[(size_t)(m0 + j) * p.N + col] = sum[j];
                    }
                }
            }
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (!dq && !all_in) ptx::mbar_arrive_if(acc_empty + 8 * set, lane == 0);
        }
    }

    __syncwarp();
    if (*abort_flag) {
        // give copies and UMMAs already in flight time to land before shared and tensor memory go away
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    if (warp == kUmIssueWarp) {
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc(tmem_base, kUmTmemCols);
    }
}

}  // namespace

namespace t0 {

// Counters and partial sums of a launch of one CTA per SM at M = 128: what any launch needs at most.
size_t w4a16_umma_scratch_bytes(const t0_runtime* rt) { return kUmCounterBytes + (size_t)rt->sm_count * 2 * 128 * kUmBN * sizeof(float); }

// Makes room for them, once, when the runtime is made: no call allocates, and none stalls the stream for it.  The counters start at zero.
int w4a16_umma_reserve(t0_runtime* rt) {
    const size_t need = w4a16_umma_scratch_bytes(rt);
    if (need <= rt->scratch_um.size) return T0_OK;
    int rc = ensure_scratch(rt, rt->scratch_um, need);
    if (rc != T0_OK) return rc;
    const cudaError_t e = cudaMemsetAsync(rt->scratch_um.ptr, 0, kUmCounterBytes, rt->stream);
    if (e != cudaSuccess) {                // counters that may hold anything: no buffer then
        cudaFree(rt->scratch_um.ptr);
        rt->scratch_um = Scratch();
        return fail(T0_ERR_CUDA, "clearing the counters of cut tiles: %s", cudaGetErrorString(e));
    }
    return T0_OK;
}

static uint32_t cut_grid(uint32_t sms, uint64_t items, uint32_t n_chunks) {
    const uint32_t ctas = std::min<uint32_t>(sms, kUmCounterBytes / (kUmDqWarps * sizeof(uint32_t)));
    uint32_t grid = (uint32_t)std::min<uint64_t>(std::max<uint64_t>(1, items * n_chunks / kUmMinChunks), ctas);
    if (items * 2 <= ctas) {
        // Few tiles: whole parts of a tile per CTA, at most four, where that leaves few CTAs idle - a CTA then has one piece to hand in, and
        // a tile is not cut into more parts than pay.
        const uint32_t parts = std::max<uint32_t>(1, std::min<uint32_t>({4u, ctas / (uint32_t)items, n_chunks / kUmMinChunks}));
        if (parts == 4 || parts * kUmMinChunks * 2 > n_chunks || items * parts * 5 >= ctas * 4ull) grid = (uint32_t)items * parts;
    }
    return grid;
}

// How to share out the tiles of `count` problems: the fastest form, by times in microseconds fitted to 402 launches of M = 17 ... 128, 4 ... 224 tiles and
// K = 768 ... 8192, each timed in both forms (the faster one by the times is within 0.3 % of the better one in the mean; the fit of before the last changes to this
// kernel was 2.6 % off).  A chunk takes 0.28 us up to M = 64 and 0.34 (cut) or 0.32 (whole) at M = 128; handing in and adding parts adds 3 to 7 us with M.  Measured, whole tiles /
// cut: 4 x (17 x 14336 x 2048) 21.5 / 22.4, 4 x (64 x 4096 x 2048) 13.5 / 12.5; one problem as clusters / cut: 17 x 16384 x 8192 46.8 / 24.3, 100 x 14336 x 1024
// 13.4 / 15.5, 128 x 16384 x 2048 17.8 / 16.2.  (4 x (17 x 14336 x 2048): cut all the same, for the shorter sums.)
// `cluster_split`: into how many parts the cluster form would cut K (1: one problem that has tiles enough; 0: a list); `cluster_rounds`: in how many rounds
// its clusters fit on the GPU (the GPCs hold 33 of four CTAs, not 37: 128 x 9472 x 4096 36.4 us in two rounds of clusters, 20.7 cut).
//
// Cut tiles of more than 64 rows whose parts are not the same number to each (56 tiles on 148 CTAs) take 2.0 to 2.7 us more than that, which matters beside clusters: a chunk
// of one accumulator set, and up to four parts to a tile.  260 single problems that the times without it would move from clusters to cut tiles, weights not in
// L2: 9 were slower so, by up to 7 % (93 x 14112 x 1536 16.8 us cut, 15.6 as clusters; 85 x 14784 x 1152 16.1 and 14.1), with it 2 of 247, by up to 2 %.
//
// Clusters are left only for a gain of more than 8 % (they share no memory between launches, so that a recorded launch gives the same bits), whole tiles for
// none at all, nor for a loss of up to 3 % (their sums are the longest).
//
// The times choose only among forms whose sums are no longer than the library has made them for the problem, since the tensor cores' error grows with
// the length of an accumulation.  One problem: its pieces are no longer than the parts of the clusters (K = 768: four of 3 chunks, where the grid
// above would make three of 4; 39 x 3264 x 768 12.4 us as clusters, 9.2 so).  Tiles that would be cut by the times of the kernel as it was before two warps
// issued its UMMAs (0.42 to 0.52 us a chunk either way), and lists that would be by those of before its roles walked converged (0.63 us a chunk whole, 0.67 cut, 14.4 us
// for the parts), stay cut where that makes their sums shorter: both fits are kept for this alone.
// Three of 70 x 2320 x 1280, whole / cut: 10.7 / 13.1 us, 1.06e-6 / 2.4e-7 off the exact result with sums of 20 / 5 chunks; two of 84 x 4352 x 1280
// 11.0 / 13.6 us; 120 x 19352 x 2944 21.3 / 20.9 us, 2.7e-6 / 1.1e-6.
// Gives the form, and for cut tiles the number of CTAs in *ctas.
int w4a16_umma_form(uint32_t sms, uint32_t M, uint32_t N, uint32_t K, uint32_t count, uint32_t cluster_split, uint32_t cluster_rounds, uint32_t* ctas) {
    const uint64_t items = (uint64_t)ceil_div(N, kUmBN) * count;
    const uint32_t n_chunks = K / kUmBK;
    const int other = cluster_split > 1 ? kUmClusters : kUmWhole;
    uint32_t grid = cut_grid(sms, items, n_chunks);
    if (other == kUmClusters && (items * n_chunks + grid - 1) / grid > ceil_div(n_chunks, cluster_split)) grid = (uint32_t)items * cluster_split;
    *ctas = grid;
    if (items % grid == 0 || items * n_chunks >= (1u << 24)) return other;
    const double per_cta = (double)items * n_chunks / grid;
    const double rounds = (double)((items + sms - 1) / sms);
    const bool cluster_form = other == kUmClusters;
    const uint32_t parts = std::max(1u, cluster_split);
    if (cluster_split == 0 && per_cta * 0.67 + 14.4 <= 0.97 * (rounds * n_chunks * 0.63 + 4.0)) return kUmCut;
    if (ceil_div(n_chunks, parts) > items * n_chunks / grid) {       // (the first CTA's range begins with a tile: cut, no sum needs to be longer than that range)
        const double chunk = 0.42 + 0.0008 * M;
        const double uncut = cluster_form ? cluster_rounds * (ceil_div(n_chunks, parts) * 0.495 + 8.2) + 2.0 : rounds * n_chunks * chunk + 4.2;
        if (per_cta * chunk + 6.2 + 0.055 * M + (grid >= sms ? 2.0 : 0.0) <= 0.97 * uncut) return kUmCut;
    }
    const double wide = M > 64 ? M - 64.0 : 0.0;
    const double uneven = cluster_form && M > 64 && grid % items ? 2.3 : 0.0;
    const double cut = per_cta * (0.288 - 0.00037 * M + 0.00176 * wide) + 6.0 + 0.049 * M + (grid >= sms ? 1.35 : 0.0) + uneven;
    const double without = cluster_form ? cluster_rounds * (ceil_div(n_chunks, parts) * 0.497 + 5.1 + 0.0018 * M) + 5.1
                                                : rounds * n_chunks * (0.285 - 0.0001 * M + 0.0008 * wide) + 3.3 + 0.021 * M;
    return cut > (cluster_form ? 0.92 : 1.03) * without ? other : kUmCut;
}

// The form of a launch.  Cut tiles need room for their parts, and run only in launches of the runtime's own stream, whose launches run one after the
// other: a recorded launch may be replayed beside others, which would share its counters and parts.
int w4a16_umma_plan(t0_runtime* rt, uint32_t M, uint32_t N, uint32_t K, uint32_t count, uint32_t cluster_split, uint32_t cluster_rounds, uint32_t* ctas) {
    const int other = cluster_split > 1 ? kUmClusters : kUmWhole;
    if (w4a16_umma_form((uint32_t)rt->sm_count, M, N, K, count, cluster_split, cluster_rounds, ctas) != kUmCut) return other;
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(rt->stream, &capturing) != cudaSuccess || capturing != cudaStreamCaptureStatusNone) return other;
    return rt->scratch_um.ptr ? kUmCut : other;      // (a runtime made while there was no memory for the parts: the other forms need none)
}

uint32_t w4a16_umma_cut_rows(uint32_t M) { return (M + 15) & ~15u; }

// `group` holds the maps (activation boxes of w4a16_umma_cut_rows(M) rows), buffers and outputs of `count` problems of one shape.  `cut_ctas`: tiles cut between so
// many CTAs, w4a16_umma_plan has made room for their parts; 0: every CTA takes whole tiles.  Tile-major weights: `off_scales` and `off_zeros` are the offsets of these.
template <uint32_t kProblems, bool kTiled>
int launch_w4a16_umma_cut(t0_runtime* rt, const UmGroup<kProblems, kTiled>& group, uint32_t M, uint32_t N, uint32_t K, uint32_t group_size, uint32_t count, uint32_t cut_ctas,
                          size_t off_scales, size_t off_zeros) {
    auto kern = w4a16_umma_cut_kernel<kTiled, kProblems>;
    static bool attr_set[64] = {};
    if (rt->device >= 64) return fail(T0_ERR_INVALID, "device ordinal out of range");
    if (!attr_set[rt->device]) {
        T0_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kUmSmem));
        attr_set[rt->device] = true;
    }
    UmParams p;
    memset(&p, 0, sizeof p);
    p.status = rt->d_status;
    const uint64_t limit = rt->wait_limit_ns.load(std::memory_order_relaxed);
    p.wait_limit_ns = limit ? limit : ptx::kWaitLimitNs;
    p.M = M; p.N = N;
    p.rows = w4a16_umma_cut_rows(M);
    p.n_tiles = ceil_div(N, kUmBN);
    p.n_chunks = K / kUmBK;
    const uint64_t items = (uint64_t)p.n_tiles * count;
    if (items * p.n_chunks > 0x7FFFFFFFull || items > (1u << 23)) return fail(T0_ERR_UNSUPPORTED, "too many tiles");
    const uint32_t grid = cut_ctas ? cut_ctas : (uint32_t)std::min<uint64_t>(items, std::min(rt->sm_count, 256));
    p.total = (uint32_t)(items * p.n_chunks);
    p.whole = cut_ctas ? 0 : 1;
    p.tiles = (uint32_t)items;
    p.per_group = group_size / kUmBK;
    p.x_stages = std::min(kUmMaxXStages, kUmXBytes / (2 * p.rows * kUmBK * 2));
    p.by_grid = um_divisor(grid); p.by_total = um_divisor(p.total); p.by_chunks = um_divisor(p.n_chunks); p.by_tiles = um_divisor(p.n_tiles);
    p.by_group = um_divisor(p.per_group);
    if (off_zeros / 16 > 0xFFFFFFFFull) return fail(T0_ERR_UNSUPPORTED, "weights too large");
    p.off_scales = (uint32_t)(off_scales / 16); p.off_zeros = (uint32_t)(off_zeros / 16);
    if (cut_ctas) {
        p.counters = (uint32_t*)rt->scratch_um.ptr;
        p.pieces = (float*)((uint8_t*)rt->scratch_um.ptr + kUmCounterBytes);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(kUmThreads, 1, 1);
    cfg.dynamicSmemBytes = kUmSmem;
    cfg.stream = rt->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    static const bool use_pdl = getenv("T0_NO_PDL") == nullptr;
    cfg.numAttrs = use_pdl ? 1 : 0;
    cudaError_t le = cudaLaunchKernelEx(&cfg, kern, p, group);
    if (le != cudaSuccess) return fail(T0_ERR_CUDA, "W4A16 kernel launch failed: %s", cudaGetErrorString(le));
    rt->launches.fetch_add(1);
    return T0_OK;
}

template int launch_w4a16_umma_cut<1, false>(t0_runtime*, const UmGroup<1, false>&, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, size_t, size_t);
template int launch_w4a16_umma_cut<1, true>(t0_runtime*, const UmGroup<1, true>&, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, size_t, size_t);
template int launch_w4a16_umma_cut<kUmMaxGroup, false>(t0_runtime*, const UmGroup<kUmMaxGroup, false>&, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, size_t, size_t);
template int launch_w4a16_umma_cut<kUmMaxGroup, true>(t0_runtime*, const UmGroup<kUmMaxGroup, true>&, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, size_t, size_t);

}  // namespace t0
