// Internal launch interface between the runtime (runtime.cu) and the sm_100a kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "common.h"

namespace t0 {

// Error word written by a kernel whose bounded wait expired: role in the top byte.
enum : int { kStatusOk = 0, kStatusProducerTimeout = 0x01000000, kStatusMmaTimeout = 0x02000000, kStatusEpilogueTimeout = 0x03000000 };

struct GemmLaunch {
    const void* x;        // bf16 [M,K]; [K,M] with at
    const void* b;        // bf16 [N,K] (NT) or [K,N] (NN)
    void* y;              // f32 [M,N] (or planes) / bf16 [M,N]
    const float* bias;    // f32 [N] or null
    uint32_t m, n, k;
    uint32_t ldx, ldb;    // row strides in elements (0 = dense)
    uint32_t tile_n;      // 32/64/128/256
    uint32_t split_k;     // >= 1
    bool cluster;         // single-CTA kernel, 1 < split_k <= kMaxClusterParts: the parts meet in clusters, the result is complete in y
    bool halves;          // tile_n <= 128: sums of half the length, added in f32
    uint64_t plane_stride;  // elements between split planes
    bool nn, out_bf16, swap_grid;
    bool at;              // x is given transposed, [K,M] with M contiguous (row stride ldx, 0 = M); only together with nn
    uint8_t epilogue;     // T0_EPI_*
    uint8_t n_ops;        // TileIR chain (overrides epilogue when > 0)
    uint8_t ops[T0_TILE_MAX_EPILOGUE];
    float scale, clamp_min, clamp_max;
    int* status;          // device error word
    unsigned long long* probe;   // optional device buffer of two words (cycles, ns) written by CTA 0
    uint32_t n_sms;
    uint64_t wait_limit_ns;      // 0 = the default limit (ptx::kWaitLimitNs)
    bool drop_load;              // self-test: CTA 0's producer leaves out its first load, so a bounded wait must run out
    // Gathered output (multi-GPU): the product is also stored to n_peer_y other f32 [M,N] buffers, normally other GPUs'
    // memory mapped into this process.  Needs the TMA-store epilogue for every chunk: f32 output, N % 32 == 0, 16-byte aligned
    // bases, no split-K.  peer_map_slot = device memory for kMaxPeerY tensor maps (128-byte aligned) that stays untouched
    // until the launch has finished.
    void* peer_y[7];
    uint32_t n_peer_y;
    void* peer_map_slot;
    bool peer_maps_staged;       // the slot already holds the maps of exactly these destinations and this shape
};
constexpr uint32_t kMaxPeerY = 7;

// Launches the tcgen05 GEMM. Requirements (checked): x and b 16-byte aligned, row strides and
// K / split_k multiples of 8 elements, K % split_k == 0.  Returns a T0_* code.
int launch_gemm_sm100(const GemmLaunch& g, cudaStream_t stream);

constexpr uint32_t kMaxClusterParts = 8;       // the portable cluster size
// How many clusters of 1 .. kMaxClusterParts CTAs (the index), one CTA per SM, run at once on the current device.
const uint32_t* gemm_clusters_at_once();

// The CTA-pair form (cta_group::2; 256 x 256 tiles, or 256 x 128 when tile_n <= 128); NT, and NN with 256-wide tiles.
int launch_gemm_sm100_pair(const GemmLaunch& g, cudaStream_t stream);
uint32_t gemm_pair_smem_bytes(uint32_t pair_n);

// Split-K inside one launch: the split_k CTAs of an output tile form a cluster and add their partial sums through
// distributed shared memory (same sum, in split order, as planes + reduction).  NT layout, split_k 2 / 4 / 8, tile_n 64 / 128.
bool gemm_splitk_cluster_supported(const GemmLaunch& g);
int launch_gemm_sm100_splitk(const GemmLaunch& g, cudaStream_t stream);
// Several problems of ONE shape and configuration (only x, b and y differ) in one launch of the same kernel: the clusters walk
// the tiles of all the problems, so launch, prologue and drain are paid once and the exchange of one tile overlaps the main
// loop of the next.  The problems run concurrently: no y may be an input of another.  At most kMaxGroupedGemms per launch.
constexpr uint32_t kMaxGroupedGemms = 32;
int launch_gemm_sm100_splitk_grouped(const GemmLaunch* gs, uint32_t count, cudaStream_t stream);
// The same for shapes that need no split-K once several problems fill the GPU: the single-CTA kernel, NT, tile width 64 / 128.
int launch_gemm_sm100_grouped(const GemmLaunch* gs, uint32_t count, cudaStream_t stream);

// The kernel a product runs on when the caller fixes nothing: CTA pairs or single CTAs, the tile width, and into how many parts K is
// cut (single CTAs in clusters; added in the same launch).
struct GemmChoice {
    uint32_t tile_n, parts;
    bool pair, halves;
};
// No accumulation is longer than k / min_split: the tensor cores' error grows with the length of the sum (about 1e-9 of the result per
// term), so a shape whose configuration (auto_select) cuts K keeps sums at least that short, in parts or in two accumulators.  Nor is one longer than
// the library has made it for the shape before (kSums in cost_model.cpp).  parts = 0:
// nothing here does that (many tiles and a deep cut); the configuration itself is to be taken.
GemmChoice choose_gemm(uint32_t m, uint32_t n, uint32_t k, bool nn, bool out_bf16, uint32_t min_split, uint32_t n_sms, const uint32_t* clusters_at_once);

// t0_cached_auto_select, saying whether the environment forces the configuration (T0_FORCE_CFG).
int cached_config(uint32_t m, uint32_t k, uint32_t n, t0_gemm_config* out, bool* forced);

// y[i] = sum_s planes[s][i] in split order, then the epilogue; K4.
int launch_splitk_reduce(const float* planes, void* y, const float* bias, uint32_t m, uint32_t n, uint32_t split_k,
                         bool out_bf16, uint8_t epilogue, uint8_t n_ops, const uint8_t* ops, float scale, float clamp_min,
                         float clamp_max, cudaStream_t stream);

// dst[r][0..dst_cols) = src[r][0..cols) zero-extended, 16-bit elements (staging copy for shapes TMA cannot address).  dst_cols is a
// multiple of 8 and dst 16-byte aligned; src and cols are anything.
struct PadCopy {
    const uint16_t* src;
    uint16_t* dst;
    uint32_t rows, cols, dst_cols;
};
// Up to two copies in one launch (rows = 0: none).
int launch_pad_copy_u16(const PadCopy& a, const PadCopy& b, cudaStream_t stream);

int launch_fill_uniform_bf16(void* dst, uint64_t n, uint64_t seed, uint64_t first, cudaStream_t stream);
int launch_fill_u32(void* dst, uint64_t n, uint64_t seed, uint64_t first, cudaStream_t stream);
int launch_fill_range_bf16(void* dst, uint64_t n, uint64_t seed, uint64_t first, float lo, float hi, cudaStream_t stream);

// Shared-memory footprint of the GEMM pipeline for a tile width.
uint32_t gemm_stage_count(uint32_t tile_n);
uint32_t gemm_smem_bytes(uint32_t tile_n);

// Scratch of the fused W4A16 kernels: the arrival-counter region, and counters plus two pieces per CTA for a grid of `ctas`.
size_t w4a16_counter_region_bytes();
size_t w4a16_fixed_scratch_bytes(uint32_t ctas);

}  // namespace t0
