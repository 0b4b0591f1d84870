// K2 for single problems of 16 < M <= 128 with few column tiles: the fused W4A16 GEMM on tcgen05, weights in the row layout (packed[K/8][N],
// scales[K/G][N], zeros[K/G][N/8]) or the tile-major layout, dequantisation in the main loop, no K x N scratch matrix; and the choice between this
// kernel and the one of w4a16_umma_cut.cu, which takes lists and the other single problems.
//
// No counterpart kernel exists in the reference (its INT4 support stops at the stand-alone dequantisation kernels,
// src/t0/quant_kernels.rs:53-171).  y[m,n] = sum_k a[m,k] * w[k,n],  w = RNE_bf16((q - z) * s),  fp32 accumulate.
//
// One CTA owns a 256-column tile of y and a range of K; the CTAs that share a tile form a cluster and add their partial
// sums through distributed shared memory (split order, deterministic), as the split-K GEMM does.  Per 64-deep k chunk:
//   * one warp fetches the chunk's packed words (8 rows x 256 columns), its scales and zero points with three TMA boxes
//     into a ring of raw stages, another the chunk's activations into the operand ring;
//   * sixteen dequantisation warps turn the words into bf16 (one LOP3 per nibble pair: 0x4300 | q is the bf16 128+q,
//     minus 128+z, times s - bit-identical to the oracle because (q-z)*s is rounded once) and write them as the UMMA's B
//     operand: 256 rows (n) x 64 k, K-major, 128-byte swizzle.  A packed word holds eight consecutive k of one column
//     and the nibble pairs come out as (k, k+4); four byte permutes put them back into k order, so that the activations
//     (the 128-row A operand) can come straight from global memory through TMA (rows beyond M are zero-filled);
//   * a third serial warp issues four tcgen05.mma (128 x 256 x 16) per chunk into a 128 x 256 fp32 accumulator in tensor memory.
// At the end the sixteen warps read the accumulator, park it in shared memory (over the rings, idle by then), exchange
// across the cluster and store.  Every wait is bounded.
#include "w4a16_common.cuh"

using namespace t0;
using namespace t0::w4;

namespace {

constexpr uint32_t kUmDqWarps = 16;
// + the warps that fetch weights and activations and the one that issues the UMMAs; each walks whole and lets one elected lane issue
// (ptx::mbar_wait_warp), which shortens the serial chain that sets a chunk's pace.
constexpr uint32_t kUmRawWarp = kUmDqWarps, kUmXWarp = kUmDqWarps + 1, kUmIssueWarp = kUmDqWarps + 2;
constexpr uint32_t kUmThreads = (kUmDqWarps + 3) * 32;
constexpr uint32_t kUmRawStages = 6;
constexpr uint32_t kUmAbStages = 3;
constexpr uint32_t kUmBBytes = kUmBN * kUmBK * 2;           // 32 KiB
constexpr uint32_t kUmABytes = 128 * kUmBK * 2;             // 16 KiB
constexpr uint32_t kUmRingBytes = kUmRawStages * kUmRawStride + kUmAbStages * (kUmABytes + kUmBBytes);   // 202752
constexpr uint32_t kUmPitch = kUmBN + 4;                    // floats per parked row
constexpr uint32_t kUmParkBytes = 128 * kUmPitch * 4;       // 133120, over the rings
static_assert(kUmParkBytes <= kUmRingBytes, "the parked accumulator must fit over the rings");
constexpr uint32_t kUmSmem = kUmRingBytes + 512 + 1024;
constexpr uint32_t kUmTmemCols = 256;

struct UmParams {
    float* y;
    int* status;
    uint64_t wait_limit_ns;
    uint32_t M, N;
    uint32_t group;          // k per scale / zero-point row (a multiple of 64)
    uint32_t n_tiles, n_chunks, split;
    uint32_t tiled;          // the weights are in the tile-major layout (3-D maps: column in tile, row, tile) instead of the row layout
};

__device__ __forceinline__ uint32_t um_cluster_id() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t um_n_clusters() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%nclusterid.x;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void um_sts128(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__global__ void __launch_bounds__(kUmThreads, 1)
w4a16_umma_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_s,
                  const __grid_constant__ CUtensorMap map_z, const __grid_constant__ CUtensorMap map_a, const UmParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t raw_ring = smem;
    const uint32_t a_ring = smem + kUmRawStages * kUmRawStride;
    const uint32_t b_ring = a_ring + kUmAbStages * kUmABytes;
    const uint32_t park = smem;                                   // [128][260] f32 over the rings, used when they are idle
    const uint32_t bars = smem + kUmRingBytes;
    const uint32_t raw_full = bars, raw_empty = bars + 8 * kUmRawStages;
    const uint32_t ab_full = raw_empty + 8 * kUmRawStages, ab_empty = ab_full + 8 * kUmAbStages;
    const uint32_t acc_full = ab_empty + 8 * kUmAbStages, acc_empty = acc_full + 8;
    const uint32_t parked_bar = acc_empty + 8, read_bar = parked_bar + 8;
    __shared__ uint32_t tmem_holder;
    __shared__ int s_abort;
    volatile int* abort_flag = &s_abort;

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t split = ptx::cluster_ctarank();
    const uint32_t c_begin = (uint32_t)((uint64_t)split * p.n_chunks / p.split), c_end = (uint32_t)((uint64_t)(split + 1) * p.n_chunks / p.split);
    const uint32_t my_chunks = c_end - c_begin;

    if (tid == 0) {
        for (uint32_t s = 0; s < kUmRawStages; ++s) {
            ptx::mbar_init(raw_full + 8 * s, 1);
            ptx::mbar_init(raw_empty + 8 * s, kUmDqWarps / 2);    // the eight warps of the group that dequantises the chunk
        }
        for (uint32_t s = 0; s < kUmAbStages; ++s) {
            ptx::mbar_init(ab_full + 8 * s, kUmDqWarps / 2 + 1);  // eight warps' weights + the activations' bytes (producer)
            ptx::mbar_init(ab_empty + 8 * s, 1);
        }
        ptx::mbar_init(acc_full, 1);
        ptx::mbar_init(acc_empty, kUmDqWarps);
        ptx::mbar_init(parked_bar, kUmDqWarps * p.split);
        ptx::mbar_init(read_bar, kUmDqWarps * p.split);
        s_abort = 0;
        ptx::fence_barrier_init();
        ptx::fence_proxy_async_smem();
        ptx::tma_prefetch_desc(&map_w);
        ptx::tma_prefetch_desc(&map_s);
        ptx::tma_prefetch_desc(&map_z);
        ptx::tma_prefetch_desc(&map_a);
    }
    if (warp == kUmIssueWarp) {
        ptx::tmem_alloc(ptx::smem_u32(&tmem_holder), kUmTmemCols);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    ptx::cluster_sync_all();          // every CTA's barriers exist before anyone signals across the cluster
    ptx::tc_fence_after_sync();
    const uint32_t tmem_base = tmem_holder;
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();

    if (warp == kUmRawWarp) {
        // ------------------------------------------------------------ weights: three TMA boxes per chunk
        uint32_t stage = 0, phase = 0, iter = 0;
        bool ok = true;
        for (uint32_t tile = um_cluster_id(); ok && tile < p.n_tiles; tile += um_n_clusters(), ++iter) {
            // the rings double as the parking area: the previous tile's copy must have been read by the whole cluster
            if (iter > 0 && !__all_sync(0xFFFFFFFFu, ptx::mbar_wait_cluster(read_bar, (iter - 1) & 1, abort_flag, p.wait_limit_ns))) {
                if (lane == 0) atomicCAS(p.status, 0, kStatusProducerTimeout | 0x800000);
                break;
            }
            const uint32_t n0 = tile * kUmBN;
            for (uint32_t c = c_begin; c < c_end; ++c) {
                if (!ptx::mbar_wait_warp(raw_empty + 8 * stage, phase ^ 1, abort_flag, p.wait_limit_ns)) {
                    if (lane == 0) atomicCAS(p.status, 0, kStatusProducerTimeout | (int)(c & 0xFFFFFF));
                    ok = false;
                    break;
                }
                const uint32_t fb = raw_full + 8 * stage, dst = raw_ring + stage * kUmRawStride;
                const uint32_t grp = c * kUmBK / p.group;
                if (ptx::elect_one()) {
                    ptx::fence_proxy_async_smem();           // the stage was read through the generic proxy, the copies write it through the async proxy
                    ptx::mbar_arrive_expect_tx(fb, kUmRawBytes);
                    if (p.tiled) {
                        // tile-major layout: the chunk's 8 KB of words are contiguous, as are its scales and zero points
                        ptx::tma_load_3d(dst, &map_w, fb, 0, (int32_t)(c * (kUmBK / 8)), (int32_t)tile);
                        ptx::tma_load_3d(dst + 8 * kUmBN * 4, &map_s, fb, 0, (int32_t)grp, (int32_t)tile);
                        ptx::tma_load_3d(dst + 8 * kUmBN * 4 + kUmBN * 2, &map_z, fb, 0, (int32_t)grp, (int32_t)tile);
                    } else {
                        ptx::tma_load_2d(dst, &map_w, fb, (int32_t)n0, (int32_t)(c * (kUmBK / 8)));
                        ptx::tma_load_2d(dst + 8 * kUmBN * 4, &map_s, fb, (int32_t)n0, (int32_t)grp);
                        ptx::tma_load_2d(dst + 8 * kUmBN * 4 + kUmBN * 2, &map_z, fb, (int32_t)(n0 / 8), (int32_t)grp);
                    }
                }
                __syncwarp();
                if (++stage == kUmRawStages) { stage = 0; phase ^= 1; }
            }
        }
    } else if (warp == kUmXWarp) {
        // ------------------------------------------------------------ activations: one 128-row box per chunk, as soon as the UMMAs that read the
        // operand stage are done
        uint32_t as = 0, aphase = 0, iter = 0;
        bool ok = true;
        for (uint32_t tile = um_cluster_id(); ok && tile < p.n_tiles; tile += um_n_clusters(), ++iter) {
            if (iter > 0 && !__all_sync(0xFFFFFFFFu, ptx::mbar_wait_cluster(read_bar, (iter - 1) & 1, abort_flag, p.wait_limit_ns))) break;
            for (uint32_t c = c_begin; c < c_end; ++c) {
                if (!ptx::mbar_wait_warp(ab_empty + 8 * as, aphase ^ 1, abort_flag, p.wait_limit_ns)) {
                    if (lane == 0) atomicCAS(p.status, 0, kStatusProducerTimeout | 0x400000 | (int)(c & 0x3FFFFF));
                    ok = false;
                    break;
                }
                if (ptx::elect_one()) {
                    ptx::fence_proxy_async_smem();           // the rings were the parking area of the previous tile (generic proxy)
                    ptx::mbar_arrive_expect_tx(ab_full + 8 * as, kUmABytes);
                    ptx::tma_load_3d(a_ring + as * kUmABytes, &map_a, ab_full + 8 * as, (int32_t)(c * kUmBK), 0, 0);
                }
                __syncwarp();
                if (++as == kUmAbStages) { as = 0; aphase ^= 1; }
            }
        }
    } else if (warp == kUmIssueWarp) {
        // ------------------------------------------------------------ UMMA issuer
        constexpr uint32_t kIdesc = ptx::make_idesc_bf16_f32(128, kUmBN, 0u);
        uint32_t stage = 0, phase = 0, iter = 0;
        bool ok = true;
        for (uint32_t tile = um_cluster_id(); ok && tile < p.n_tiles; tile += um_n_clusters(), ++iter) {
            if (iter > 0 && !ptx::mbar_wait_warp(acc_empty, (iter - 1) & 1, abort_flag, p.wait_limit_ns)) {
                if (lane == 0) atomicCAS(p.status, 0, kStatusMmaTimeout | 0x800000);
                break;
            }
            ptx::tc_fence_after_sync();
            for (uint32_t c = 0; c < my_chunks; ++c) {
                if (!ptx::mbar_wait_warp(ab_full + 8 * stage, phase, abort_flag, p.wait_limit_ns)) {
                    if (lane == 0) atomicCAS(p.status, 0, kStatusMmaTimeout | (int)(c & 0x7FFFFF));
                    ok = false;
                    break;
                }
                ptx::tc_fence_after_sync();
                const uint32_t a_addr = a_ring + stage * kUmABytes, b_addr = b_ring + stage * kUmBBytes;
                if (ptx::elect_one()) {
#pragma unroll
                    for (uint32_t k4 = 0; k4 < kUmBK / 16; ++k4) {
                        const uint64_t da = ptx::make_smem_desc(a_addr + k4 * 32, 16, 1024);
                        const uint64_t db = ptx::make_smem_desc(b_addr + k4 * 32, 16, 1024);
                        ptx::umma_bf16_ss(tmem_base, da, db, kIdesc, (c | k4) != 0 ? 1u : 0u);
                    }
                    ptx::umma_commit(ab_empty + 8 * stage);
                }
                __syncwarp();
                if (++stage == kUmAbStages) { stage = 0; phase ^= 1; }
            }
            if (ok && ptx::elect_one()) ptx::umma_commit(acc_full);
            __syncwarp();
        }
    } else {
        // ------------------------------------------------------------ sixteen warps: dequantise, then the epilogue
        // Two groups of eight warps take alternate chunks: a warp's chain per chunk (wait, loads, arithmetic, stores, proxy
        // fence, arrive) is longer than the UMMAs of a chunk, so with all sixteen warps on the same chunk that chain, not any
        // unit, set the pace; two chunks in flight hide it.  A thread owns one column of the tile and all eight word rows.
        const uint32_t grp = warp >> 3, n = (warp & 7) * 32 + lane;
        uint32_t mask, magic;
        asm volatile("mov.b32 %0, 0x000F000F;" : "=r"(mask));
        asm volatile("mov.b32 %0, 0x43004300;" : "=r"(magic));
        uint32_t iter = 0, t_base = 0;                              // t_base: chunks of earlier tiles (ring positions run on across tiles)
        bool ok = true;
        const uint32_t b_off = (n >> 3) * 1024 + (n & 7) * 128;
        for (uint32_t tile = um_cluster_id(); tile < p.n_tiles; tile += um_n_clusters(), ++iter, t_base += my_chunks) {
            const uint32_t n0 = tile * kUmBN;
            if (ok && iter > 0 && !ptx::mbar_wait_cluster(read_bar, (iter - 1) & 1, abort_flag, p.wait_limit_ns)) {
                if (lane == 0) atomicCAS(p.status, 0, kStatusEpilogueTimeout | 0x400000);
                ok = false;
            }
            for (uint32_t ci = 0; ok && ci < my_chunks; ++ci) {
                const uint32_t t = t_base + ci;
                if ((t & 1u) != grp) continue;
                const uint32_t rs = t % kUmRawStages, rphase = (t / kUmRawStages) & 1u, as = t % kUmAbStages, aphase = (t / kUmAbStages) & 1u;
                if (!ptx::mbar_wait(raw_full + 8 * rs, rphase, abort_flag, p.wait_limit_ns)) {
                    if (lane == 0) atomicCAS(p.status, 0, kStatusEpilogueTimeout | (int)(ci & 0x3FFFFF));
                    ok = false;
                    break;
                }
                const uint32_t raw = raw_ring + rs * kUmRawStride;
                uint32_t words[8];
#pragma unroll
                for (uint32_t i = 0; i < 8; ++i) words[i] = um_lds32(raw + i * (kUmBN * 4) + n * 4);
                const uint32_t sbits = um_lds16(raw + 8 * kUmBN * 4 + n * 2);
                const uint32_t zword = um_lds32(raw + 8 * kUmBN * 4 + kUmBN * 2 + (n >> 3) * 4);
                const uint32_t zz = ((zword >> ((n & 7) * 4)) & 0xFu) * 0x00010001u + 0x43004300u;     // bf16x2 (128+z, 128+z)
                const uint32_t ss = sbits * 0x00010001u;                                               // (s, s)
                if (!ptx::mbar_wait(ab_empty + 8 * as, aphase ^ 1, abort_flag, p.wait_limit_ns)) {
                    if (lane == 0) atomicCAS(p.status, 0, kStatusEpilogueTimeout | 0x800000 | (int)(ci & 0x3FFFFF));
                    ok = false;
                    break;
                }
                const uint32_t b_stage = b_ring + as * kUmBBytes + b_off;
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j) {
                    const uint32_t wd = words[j];
                    uint32_t v[4];
                    um_dequant_word(wd, mask, magic, zz, ss, p.tiled, v);
                    um_sts128(b_stage + ((j ^ (n & 7)) << 4), v[0], v[1], v[2], v[3]);
                }
                // The UMMAs read these bytes through the async proxy.  The warp's writes are ordered before lane 0 by the warp
                // barrier; lane 0's proxy fence and release-arrive then publish them (one fence per warp instead of 32:
                // the fence is the most expensive instruction of the chunk).
                __syncwarp();
                if (lane == 0) {
                    ptx::fence_proxy_async_smem();
                    ptx::mbar_arrive(raw_empty + 8 * rs);
                    ptx::mbar_arrive(ab_full + 8 * as);
                }
            }
            // ---- epilogue: the accumulator of this CTA's part of K
            if (ok && !ptx::mbar_wait(acc_full, iter & 1, abort_flag, p.wait_limit_ns)) {
                if (lane == 0) atomicCAS(p.status, 0, kStatusEpilogueTimeout | 0xC00000);
                ok = false;
            }
            if (!ok) break;
            ptx::tc_fence_after_sync();
            const uint32_t q = warp & 3, cg = warp >> 2;             // tensor-memory lane quarter, 64-column group
            const uint32_t row_in = q * 32 + lane;
            // park (the rings are idle: every chunk has been consumed), tell the cluster, wait for everyone
#pragma unroll 1
            for (uint32_t h = 0; h < 2; ++h) {
                uint32_t r[32];
                ptx::tmem_ld_32x32b_x32(tmem_base + ((q * 32) << 16) + cg * 64 + h * 32, r);
                ptx::tmem_ld_wait();
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j)
                    um_sts128(park + (row_in * kUmPitch + cg * 64 + h * 32 + 4 * j) * 4, r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
            }
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                ptx::mbar_arrive(acc_empty);
                for (uint32_t s = 0; s < p.split; ++s) ptx::mbar_arrive_cluster(ptx::mapa(parked_bar, s));
            }
            if (!ptx::mbar_wait_cluster(parked_bar, iter & 1, abort_flag, p.wait_limit_ns)) {
                if (lane == 0) atomicCAS(p.status, 0, kStatusEpilogueTimeout | 0xD00000);
                ok = false;
                break;
            }
            {
                // this CTA's column slice of the tile (whole float4s), every row; splits added in split order
                const uint32_t slice_w = ((kUmBN / p.split + 3) / 4) * 4;
                const uint32_t s_begin = split * slice_w, s_end = min(kUmBN, s_begin + slice_w);
                const uint32_t f4_per_row = s_end > s_begin ? (s_end - s_begin) / 4 : 0;
                const uint32_t items = 128 * f4_per_row;
                const bool vec = ((uintptr_t)p.y & 15) == 0 && p.N % 4 == 0;   // (any N with tile-major weights)
                constexpr uint32_t kU = 2;
                for (uint32_t i0 = tid; i0 < items; i0 += kU * kUmDqWarps * 32) {
                    float4 part[kU][4];
#pragma unroll
                    for (uint32_t u = 0; u < kU; ++u) {
                        const uint32_t i = i0 + u * kUmDqWarps * 32;
                        const uint32_t row = i / f4_per_row, c4 = i - row * f4_per_row;
#pragma unroll
                        for (uint32_t s = 0; s < 4; ++s)
                            part[u][s] = (i < items && s < p.split) ? ptx::ld_cluster_f4(ptx::mapa(park + (row * kUmPitch + s_begin + c4 * 4) * 4, s))
                                                                    : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
#pragma unroll
                    for (uint32_t u = 0; u < kU; ++u) {
                        const uint32_t i = i0 + u * kUmDqWarps * 32;
                        if (i >= items) break;
                        const uint32_t row = i / f4_per_row, c4 = i - row * f4_per_row;
                        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                        for (uint32_t s = 0; s < 4; ++s)
                            if (s < p.split) { acc.x += part[u][s].x; acc.y += part[u][s].y; acc.z += part[u][s].z; acc.w += part[u][s].w; }
                        const uint32_t col = n0 + s_begin + c4 * 4;
                        if (row >= p.M || col >= p.N) continue;
                        float* dst = p.y + (size_t)row * p.N + col;
                        if (vec && col + 4 <= p.N) *(float4*)dst = acc;
                        else {
                            const float o[4] = {acc.x, acc.y, acc.z, acc.w};
                            for (uint32_t j = 0; j < 4 && col + j < p.N; ++j) dst[j] = o[j];
                        }
                    }
                }
            }
            __syncwarp();
            if (lane == 0)
                for (uint32_t s = 0; s < p.split; ++s) ptx::mbar_arrive_cluster(ptx::mapa(read_bar, s));      // this warp has read every copy
        }
    }

    // ---------------------------------------------------------------- common exit
    __syncwarp();
    if (*abort_flag) {
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    ptx::cluster_sync_all();          // no CTA's shared memory goes away while a peer may still read its copy or signal its barriers
    if (warp == kUmIssueWarp) {
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc(tmem_base, kUmTmemCols);
    }
}

// ------------------------------------------------------------------ tile-major weight layout
//
// The row layout puts the 8 KB of packed words a CTA needs per chunk in eight 1 KB pieces 4N bytes apart; HBM serves that
// pattern at about a third of its copy bandwidth, which is then what bounds these kernels (not the arithmetic, not the
// UMMAs).  The tile-major layout stores every 256-column tile as a matrix of its own, so a chunk's words, scales and zero
// points are each one contiguous piece:
//   words  [T][K/8][256] u32, scales [T][K/G][256] bf16, zero points [T][K/G][32] u32, T = ceil(N / 256), columns past N zero;
//   within a word code k sits in nibble (k >> 1) + 4 (k & 1).
struct TiledLayout { size_t off_words, off_scales, off_zeros, total; uint32_t tiles, rows, groups; };

TiledLayout tiled_layout(uint32_t K, uint32_t N, uint32_t group) {
    TiledLayout L;
    L.tiles = ceil_div(N, kUmBN); L.rows = K / 8; L.groups = K / group;
    L.off_words = 0;
    L.off_scales = (size_t)L.tiles * L.rows * kUmBN * 4;
    L.off_zeros = L.off_scales + (size_t)L.tiles * L.groups * kUmBN * 2;
    L.total = L.off_zeros + (size_t)L.tiles * L.groups * (kUmBN / 8) * 4;
    return L;
}

// Row layout -> tile-major layout: one thread per output word / scale / zero-point word.
__global__ void w4_to_tiled_kernel(const uint32_t* __restrict__ packed, const uint16_t* __restrict__ scales, const uint32_t* __restrict__ zeros,
                                   uint8_t* __restrict__ out, uint32_t N, uint32_t nz, TiledLayout L) {
    const uint64_t n_words = (uint64_t)L.tiles * L.rows * kUmBN;
    const uint64_t n_scales = (uint64_t)L.tiles * L.groups * kUmBN;
    const uint64_t n_zwords = (uint64_t)L.tiles * L.groups * (kUmBN / 8);
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_words + n_scales + n_zwords; i += stride) {
        if (i < n_words) {
            const uint32_t c = (uint32_t)(i % kUmBN);
            const uint64_t r = i / kUmBN;
            const uint32_t row = (uint32_t)(r % L.rows), tile = (uint32_t)(r / L.rows);
            const uint32_t n = tile * kUmBN + c;
            // code k of the word moves to nibble (k >> 1) + 4 (k & 1): the kernels pull nibbles i and i + 4 out together as one
            // bf16 pair, which is then (k, k + 1) with k = 2i, the order the UMMA operand wants, with no byte permutes
            uint32_t w = n < N ? packed[(size_t)row * N + n] : 0u, v = 0;
#pragma unroll
            for (uint32_t kk = 0; kk < 8; ++kk) v |= ((w >> (4 * kk)) & 0xFu) << (4 * ((kk >> 1) + 4 * (kk & 1)));
            ((uint32_t*)(out + L.off_words))[i] = v;
        } else if (i < n_words + n_scales) {
            const uint64_t j = i - n_words;
            const uint32_t c = (uint32_t)(j % kUmBN);
            const uint64_t r = j / kUmBN;
            const uint32_t g = (uint32_t)(r % L.groups), tile = (uint32_t)(r / L.groups);
            const uint32_t n = tile * kUmBN + c;
            ((uint16_t*)(out + L.off_scales))[j] = n < N ? scales[(size_t)g * N + n] : (uint16_t)0;
        } else {
            const uint64_t j = i - n_words - n_scales;
            const uint32_t wz = (uint32_t)(j % (kUmBN / 8));
            const uint64_t r = j / (kUmBN / 8);
            const uint32_t g = (uint32_t)(r % L.groups), tile = (uint32_t)(r / L.groups);
            const uint32_t n0 = tile * kUmBN + wz * 8;
            ((uint32_t*)(out + L.off_zeros))[j] = n0 < N ? zeros[(size_t)g * nz + (n0 >> 3)] : 0u;
        }
    }
}

}  // namespace

namespace t0 {

// w4a16_umma_cut.cu
int w4a16_umma_plan(t0_runtime* rt, uint32_t M, uint32_t N, uint32_t K, uint32_t count, uint32_t cluster_split, uint32_t cluster_rounds, uint32_t* ctas);
uint32_t w4a16_umma_cut_rows(uint32_t M);
template <uint32_t kProblems, bool kTiled>
int launch_w4a16_umma_cut(t0_runtime* rt, const UmGroup<kProblems, kTiled>& group, uint32_t M, uint32_t N, uint32_t K, uint32_t group_size, uint32_t count, uint32_t cut_ctas,
                          size_t off_scales, size_t off_zeros);

static t0_w4a16_args um_args(uint64_t a, uint64_t packed, uint64_t scales, uint64_t zeros, uint64_t y, uint32_t M, uint32_t N, uint32_t K, uint32_t group) {
    t0_w4a16_args q;
    memset(&q, 0, sizeof q);
    q.a = a; q.packed = packed; q.scales = scales; q.zeros = zeros; q.y = y; q.m = M; q.n = N; q.k = K; q.group = group;
    return q;
}

// Whether the fused tcgen05 kernel takes this W4A16 problem.
bool w4a16_umma_supported(uint64_t a, uint64_t packed, uint64_t scales, uint64_t zeros, uint64_t y, uint32_t M, uint32_t N, uint32_t K, uint32_t group) {
    if (M == 0 || M > 128 || N % 32 || K == 0 || K % kUmBK || group == 0 || group % kUmBK || K % group) return false;
    if (((a | packed | scales | zeros) & 15) != 0 || (y & 3) != 0) return false;
    return true;
}

// The four tensor maps of one problem: packed words, scales, zero points, and the activations (K-major boxes
// of 64 k x a_rows, 128-byte swizzle, rows beyond M read as zero).
static int um_maps(uint64_t a, uint64_t packed, uint64_t scales, uint64_t zeros, uint32_t M, uint32_t N, uint32_t K, uint32_t group, CUtensorMap* out4, uint32_t a_rows = 128) {
    int rc = gemm::make_map_2d_plain(&out4[0], (const void*)packed, 4, K / 8, N, kUmBN, kUmBK / 8);
    if (rc == T0_OK) rc = gemm::make_map_2d_plain(&out4[1], (const void*)scales, 2, K / group, N, kUmBN, 1);
    if (rc == T0_OK) rc = gemm::make_map_2d_plain(&out4[2], (const void*)zeros, 4, K / group, N / 8, kUmBN / 8, 1);
    if (rc == T0_OK) rc = gemm::make_map_kmajor(&out4[3], (const void*)a, M, K, K, 1, a_rows);
    return rc;
}

// The same four maps over the tile-major buffer: 3-D views (column in tile, row, tile).
static int um_maps_tiled(uint64_t a, uint64_t tiled, uint32_t M, uint32_t N, uint32_t K, uint32_t group, CUtensorMap* out4, uint32_t a_rows = 128) {
    const TiledLayout L = tiled_layout(K, N, group);
    const uint8_t* base = (const uint8_t*)tiled;
    int rc = gemm::make_map_3d_plain(&out4[0], base + L.off_words, 4, kUmBN, L.rows, L.tiles, kUmBN * 4, (uint64_t)L.rows * kUmBN * 4, kUmBN, kUmBK / 8);
    if (rc == T0_OK) rc = gemm::make_map_3d_plain(&out4[1], base + L.off_scales, 2, kUmBN, L.groups, L.tiles, kUmBN * 2, (uint64_t)L.groups * kUmBN * 2, kUmBN, 1);
    if (rc == T0_OK) rc = gemm::make_map_3d_plain(&out4[2], base + L.off_zeros, 4, kUmBN / 8, L.groups, L.tiles, (kUmBN / 8) * 4, (uint64_t)L.groups * (kUmBN / 8) * 4, kUmBN / 8, 1);
    if (rc == T0_OK) rc = gemm::make_map_kmajor(&out4[3], (const void*)a, M, K, K, 1, a_rows);
    return rc;
}

static bool um_tiled_supported(uint64_t a, uint64_t tiled, uint64_t y, uint32_t M, uint32_t N, uint32_t K, uint32_t group) {
    if (M == 0 || M > 128 || N == 0 || K == 0 || K % kUmBK || group == 0 || group % kUmBK || K % group) return false;
    return ((a | tiled) & 15) == 0 && (y & 3) == 0;
}

// How many clusters of `split` CTAs the device holds at once.  Makes the kernel ready for a launch.
static int um_clusters_at_once(t0_runtime* rt, uint32_t split, uint32_t* clusters) {
    static bool attr_set[64] = {};
    static int max_clusters[64][5] = {};
    if (rt->device >= 64) return fail(T0_ERR_INVALID, "device ordinal out of range");
    if (!attr_set[rt->device]) {
        T0_CUDA(cudaFuncSetAttribute(w4a16_umma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kUmSmem));
        attr_set[rt->device] = true;
    }
    if (!max_clusters[rt->device][split]) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = split; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
        cfg.gridDim = dim3(split * ((uint32_t)rt->sm_count / split), 1, 1);
        cfg.blockDim = dim3(kUmThreads, 1, 1);
        cfg.dynamicSmemBytes = kUmSmem;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int n = 0;
        cudaError_t e = cudaOccupancyMaxActiveClusters(&n, w4a16_umma_kernel, &cfg);
        if (e != cudaSuccess || n <= 0) { cudaGetLastError(); n = (int)((uint32_t)rt->sm_count / split) * 3 / 4; }
        max_clusters[rt->device][split] = std::max(n, 1);
    }
    *clusters = (uint32_t)max_clusters[rt->device][split];
    return T0_OK;
}

static int um_launch(t0_runtime* rt, const CUtensorMap* m4, UmParams p, uint32_t split, uint32_t clusters_at_once) {
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kUmThreads, 1, 1);
    cfg.dynamicSmemBytes = kUmSmem;
    cfg.stream = rt->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = split; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    p.split = split;
    static const bool use_pdl = getenv("T0_NO_PDL") == nullptr;
    const uint32_t clusters = std::min(p.n_tiles, clusters_at_once);
    cfg.gridDim = dim3(clusters * split, 1, 1);
    cfg.numAttrs = use_pdl ? 2 : 1;
    cudaError_t le = cudaLaunchKernelEx(&cfg, w4a16_umma_kernel, m4[0], m4[1], m4[2], m4[3], p);
    if (le != cudaSuccess) return fail(T0_ERR_CUDA, "W4A16 kernel launch failed: %s", cudaGetErrorString(le));
    rt->launches.fetch_add(1);
    return T0_OK;
}

static UmParams um_params(t0_runtime* rt, uint64_t y, uint32_t M, uint32_t N, uint32_t K, uint32_t group) {
    UmParams p;
    memset(&p, 0, sizeof p);
    p.y = (float*)y; p.status = rt->d_status;
    const uint64_t limit = rt->wait_limit_ns.load(std::memory_order_relaxed);
    p.wait_limit_ns = limit ? limit : ptx::kWaitLimitNs;
    p.M = M; p.N = N; p.group = group;
    p.n_tiles = ceil_div(N, kUmBN);
    p.n_chunks = K / kUmBK;
    return p;
}

// The maps, buffer and output of problem i of a launch on the kernel that takes whole tiles or cuts them (w4a16_umma_cut.cu).
template <uint32_t kProblems, bool kTiled>
static int um_group_entry(UmGroup<kProblems, kTiled>& grp, uint32_t i, const t0_w4a16_args& a) {
    const uint32_t rows = w4a16_umma_cut_rows(a.m);
    grp.y[i] = (float*)a.y;
    if constexpr (kTiled) {
        grp.base[i] = (const uint8_t*)a.packed;
        return gemm::make_map_kmajor(&grp.maps[i], (const void*)a.a, a.m, a.k, a.k, 1, rows);
    } else {
        return um_maps(a.a, a.packed, a.scales, a.zeros, a.m, a.n, a.k, a.group, &grp.maps[4 * i], rows);
    }
}

// `count` problems of one shape in one launch, which run concurrently.
template <bool kTiled>
static int um_launch_list(t0_runtime* rt, const t0_w4a16_args* args, uint32_t count, uint32_t cut_ctas) {
    static UmGroup<kUmMaxGroup, kTiled> grp;     // up to 16.6 KB: kept off the stack, filled under the lock, copied by the launch
    static std::mutex grp_mu;
    std::lock_guard<std::mutex> lock(grp_mu);
    for (uint32_t i = 0; i < count; ++i) {
        int rc = um_group_entry(grp, i, args[i]);
        if (rc != T0_OK) return rc;
    }
    TiledLayout L = {};                              // (the row layout's scales and zero points have maps)
    if constexpr (kTiled) L = tiled_layout(args[0].k, args[0].n, args[0].group);
    return launch_w4a16_umma_cut(rt, grp, args[0].m, args[0].n, args[0].k, args[0].group, count, cut_ctas, L.off_scales, L.off_zeros);
}

template <bool kTiled>
static int um_launch_single(t0_runtime* rt, const t0_w4a16_args& a, uint32_t cut_ctas) {
    UmGroup<1, kTiled> one;
    int rc = um_group_entry(one, 0, a);
    if (rc != T0_OK) return rc;
    TiledLayout L = {};
    if constexpr (kTiled) L = tiled_layout(a.k, a.n, a.group);
    return launch_w4a16_umma_cut(rt, one, a.m, a.n, a.k, a.group, 1, cut_ctas, L.off_scales, L.off_zeros);
}

static int um_launch_one(t0_runtime* rt, const t0_w4a16_args& a, bool tiled) {
    // as many parts of K as fill the machine (the parts of a tile form a cluster of at most four CTAs)
    const uint32_t n_tiles = ceil_div(a.n, kUmBN);
    const uint32_t split = std::min(std::max<uint32_t>(1, std::min<uint32_t>(4, (uint32_t)rt->sm_count / std::max<uint32_t>(1, n_tiles))), a.k / kUmBK);
    uint32_t ctas, clusters = 1;
    int rc = split > 1 ? um_clusters_at_once(rt, split, &clusters) : T0_OK;
    if (rc != T0_OK) return rc;
    const int plan = w4a16_umma_plan(rt, a.m, a.n, a.k, 1, split, ceil_div(n_tiles, clusters), &ctas);
    if (plan != kUmClusters) {
        const uint32_t cut_ctas = plan == kUmCut ? ctas : 0;
        return tiled ? um_launch_single<true>(rt, a, cut_ctas) : um_launch_single<false>(rt, a, cut_ctas);
    }
    UmParams p = um_params(rt, a.y, a.m, a.n, a.k, a.group);
    p.tiled = tiled ? 1 : 0;
    CUtensorMap m4[4];
    rc = tiled ? um_maps_tiled(a.a, a.packed, a.m, a.n, a.k, a.group, m4) : um_maps(a.a, a.packed, a.scales, a.zeros, a.m, a.n, a.k, a.group, m4);
    if (rc != T0_OK) return rc;
    return um_launch(rt, m4, p, split, clusters);
}

int launch_w4a16_umma(t0_runtime* rt, uint64_t a, uint64_t packed, uint64_t scales, uint64_t zeros, uint64_t y, uint32_t M, uint32_t N, uint32_t K,
                      uint32_t group) {
    const t0_w4a16_args one = um_args(a, packed, scales, zeros, y, M, N, K, group);
    return um_launch_one(rt, one, false);
}

int launch_w4a16_umma_tiled(t0_runtime* rt, uint64_t a, uint64_t tiled, uint64_t y, uint32_t M, uint32_t N, uint32_t K, uint32_t group) {
    const t0_w4a16_args one = um_args(a, tiled, 0, 0, y, M, N, K, group);
    return um_launch_one(rt, one, true);
}

static int um_launch_grouped(t0_runtime* rt, const t0_w4a16_args* args, uint32_t count, bool tiled) {
    if (count == 0) return T0_OK;
    if (count > kUmMaxGroup) return fail(T0_ERR_INVALID, "at most %u problems per grouped launch (got %u)", kUmMaxGroup, count);
    const t0_w4a16_args& a0 = args[0];
    for (uint32_t i = 0; i < count; ++i) {
        const t0_w4a16_args& a = args[i];
        if (a.m != a0.m || a.n != a0.n || a.k != a0.k || a.group != a0.group) return fail(T0_ERR_INVALID, "grouped launch: problem %u differs from problem 0 in shape", i);
        if (!(tiled ? um_tiled_supported(a.a, a.packed, a.y, a.m, a.n, a.k, a.group) : w4a16_umma_supported(a.a, a.packed, a.scales, a.zeros, a.y, a.m, a.n, a.k, a.group)))
            return fail(T0_ERR_UNSUPPORTED, "grouped launch: problem %u is not a shape of the fused tcgen05 kernel", i);
    }
    uint32_t ctas;
    const int plan = w4a16_umma_plan(rt, a0.m, a0.n, a0.k, count, 0, 0, &ctas);
    const uint32_t cut_ctas = plan == kUmCut ? ctas : 0;
    return tiled ? um_launch_list<true>(rt, args, count, cut_ctas) : um_launch_list<false>(rt, args, count, cut_ctas);
}

int launch_w4a16_umma_tiled_grouped(t0_runtime* rt, const t0_w4a16_args* args, uint32_t count) { return um_launch_grouped(rt, args, count, true); }

int launch_w4a16_umma_grouped(t0_runtime* rt, const t0_w4a16_args* args, uint32_t count) { return um_launch_grouped(rt, args, count, false); }

}  // namespace t0

extern "C" {

size_t t0_w4_tiled_bytes(uint32_t K, uint32_t N, uint32_t group) {
    if (K == 0 || N == 0 || group == 0 || K % kUmBK || group % kUmBK || K % group) return 0;
    return tiled_layout(K, N, group).total;
}

int t0_w4_to_tiled(t0_runtime* rt, uint64_t packed, uint64_t scales, uint64_t zeros, uint64_t out, uint32_t K, uint32_t N, uint32_t group) {
    int rc = check_rt(rt);
    if (rc != T0_OK) return rc;
    if (!packed || !scales || !zeros || !out) return fail(T0_ERR_INVALID, "null device pointer");
    if (K == 0 || N == 0 || group == 0 || K % kUmBK || group % kUmBK || K % group)
        return fail(T0_ERR_UNSUPPORTED, "the tile-major layout needs K %% 64 == 0 and group %% 64 == 0 with group | K (K=%u, group=%u)", K, group);
    if (out & 127) return fail(T0_ERR_INVALID, "the output buffer must be 128-byte aligned");
    DeviceGuard guard(rt->device);
    const TiledLayout L = tiled_layout(K, N, group);
    const uint64_t n = L.total / 2;
    const uint32_t grid = (uint32_t)std::min<uint64_t>((n + 255) / 256, 148ull * 16);
    w4_to_tiled_kernel<<<grid, 256, 0, rt->stream>>>((const uint32_t*)packed, (const uint16_t*)scales, (const uint32_t*)zeros, (uint8_t*)out, N, (N + 7) / 8, L);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(T0_ERR_CUDA, "layout conversion launch failed: %s", cudaGetErrorString(e));
    rt->launches.fetch_add(1);
    return T0_OK;
}

int t0_w4a16_gemm_tiled(t0_runtime* rt, uint64_t a, uint64_t tiled, uint64_t y, uint32_t M, uint32_t N, uint32_t K, uint32_t group) {
    int rc = check_rt(rt);
    if (rc != T0_OK) return rc;
    if (M == 0 || N == 0) return T0_OK;
    if (!a || !tiled || !y) return fail(T0_ERR_INVALID, "null device pointer");
    if (!um_tiled_supported(a, tiled, y, M, N, K, group))
        return fail(T0_ERR_UNSUPPORTED, "shape M=%u N=%u K=%u group=%u: needs M <= 128, K %% 64 == 0, group %% 64 == 0, group | K, a and the weights 16-byte aligned", M, N, K, group);
    DeviceGuard guard(rt->device);
    return launch_w4a16_umma_tiled(rt, a, tiled, y, M, N, K, group);
}

int t0_w4a16_gemm_tiled_grouped(t0_runtime* rt, const t0_w4a16_args* args, size_t count) {
    int rc = check_rt(rt);
    if (rc != T0_OK) return rc;
    if (!args && count) return fail(T0_ERR_INVALID, "null arguments");
    for (size_t i = 0; i < count; ++i) {
        const t0_w4a16_args& a = args[i];
        if (a.m == 0 || a.n == 0) return fail(T0_ERR_INVALID, "grouped launch: problem %zu is empty", i);
        if (!a.a || !a.packed || !a.y) return fail(T0_ERR_INVALID, "null device pointer in problem %zu", i);
        if (!um_tiled_supported(a.a, a.packed, a.y, a.m, a.n, a.k, a.group))
            return fail(T0_ERR_UNSUPPORTED, "problem %zu: needs M <= 128, K %% 64 == 0, group %% 64 == 0, group | K, a and the weights 16-byte aligned", i);
        // the problems run at the same time: no output may be an activation or the output of another problem
        const uint64_t y_lo = a.y, y_hi = a.y + (uint64_t)a.m * a.n * 4;
        for (size_t j = 0; j < count; ++j) {
            if (j == i) continue;
            const t0_w4a16_args& b = args[j];
            const uint64_t by_hi = b.y + (uint64_t)b.m * b.n * 4, ba_hi = b.a + (uint64_t)b.m * b.k * 2;
            if ((y_lo < by_hi && b.y < y_hi) || (y_lo < ba_hi && b.a < y_hi))
                return fail(T0_ERR_INVALID, "grouped launch: the output of problem %zu overlaps the activations or the output of problem %zu (the problems run concurrently)", i, j);
        }
    }
    DeviceGuard guard(rt->device);
    // runs of equal shapes share a launch (up to 32 problems each)
    size_t i = 0;
    while (i < count) {
        size_t n = 1;
        while (i + n < count && n < kUmMaxGroup && args[i + n].m == args[i].m && args[i + n].n == args[i].n && args[i + n].k == args[i].k && args[i + n].group == args[i].group) ++n;
        rc = n == 1 ? launch_w4a16_umma_tiled(rt, args[i].a, args[i].packed, args[i].y, args[i].m, args[i].n, args[i].k, args[i].group)
                    : launch_w4a16_umma_tiled_grouped(rt, args + i, (uint32_t)n);
        if (rc != T0_OK) return rc;
        i += n;
    }
    return T0_OK;
}

}  // extern "C"

