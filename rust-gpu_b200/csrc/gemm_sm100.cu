// K1 — dense bf16 GEMM for sm_100a: y[M,N] = x[M,K] * op(b), fp32 accumulation in tensor memory.
//
// Replaces the reference's generated RDNA kernels (src/t0/gemm_gen.rs:668-1438 generate_lds_db and
// src/t0/tile_ir.rs:887-2459 lower_gemm).  Same contract: bf16 operands, NT (b = WT[N,K]) or NN
// (b = B[K,N]) layout, f32 output, optional split-K planes at y + id*M*N (gemm_gen.rs:447-448),
// ragged M/N/K handled by zero fill and predicated stores (tile_ir.rs:1142-1203,3699-3717), fused
// epilogues (gemm_gen.rs:40-49, tile_ir.rs:3406-3533).
//
// Structure (one persistent CTA per SM, 192 threads):
//   warp 0      TMA producer: 128B-swizzled tiles of A (128 x 64) and B (BN x 64) into a ring of stages
//   warp 1      UMMA issuer: four tcgen05.mma (128 x BN x 16) per stage, accumulator in tensor memory;
//               owns the tensor-memory allocation (two accumulator buffers of BN columns)
//   warps 2..5  epilogue: tcgen05.ld the finished accumulator, apply the epilogue, store to global,
//               while the issuer already fills the other accumulator buffer
// The producer and the issuer walk with their whole warp and one elected lane issues (see ptx::mbar_wait_warp): nanoseconds per 64-deep k block at
// BN = 128 / 64 / 32: 310 / 302 / 298 as a single diverged lane, 255 / 242 / 234 so.  With copies and UMMAs predicated instead of branched around 204 / 152 / 108,
// where the same measurement (the slope from K = 2048 to 8192, 144 tiles) gives 227 / 234 / 232 for the branch.
// All inter-role hand-offs are mbarriers; every wait is bounded and a wait that expires writes an
// error word the host turns into an error (no trap, no unbounded spin).
#include "kernels.h"
#include "ptx_sm100.cuh"
#include <type_traits>
#include "gemm_common.cuh"


namespace t0 {

namespace {

using namespace gemm;
constexpr uint32_t kThreads = 192;

__host__ __device__ constexpr uint32_t stages_for(uint32_t bn) { return bn == 256 ? 4 : bn == 128 ? 6 : 8; }

// The k blocks of a part of K: of a plane (a third map dimension), or, where the launch adds the parts itself, a range of the whole K.
struct KRange { uint32_t first, end, z; };
template <bool kCluster>
__device__ __forceinline__ KRange k_range(uint32_t split, const KParams& p) {
    if (!kCluster) return {0, p.kb_per_split, split};
    return {split * p.kb_per_split / p.split_k, (split + 1) * p.kb_per_split / p.split_k, 0};      // (kb_per_split is all of K here)
}

// First k block of a part's second accumulator (the end of the part when it has only one).
template <uint32_t kAccs>
__device__ __forceinline__ uint32_t k_mid(const KRange& kr, const KParams& p) {
    return kAccs == 2 && p.halves ? kr.first + (kr.end - kr.first + 1) / 2 : kr.end;
}
// Four columns of one row of the result.
__device__ __forceinline__ void store4(const KParams& p, bool vec, uint32_t row, uint32_t col, const float (&o)[4]) {
    if (row >= p.M) return;
    const size_t off = (size_t)row * p.N + col;
    if (vec) {
        if (p.out_bf16) {
            const __nv_bfloat162 h[2] = {__floats2bfloat162_rn(o[0], o[1]), __floats2bfloat162_rn(o[2], o[3])};
            *(uint2*)((__nv_bfloat16*)p.y + off) = *(const uint2*)h;
        } else {
            *(float4*)((float*)p.y + off) = make_float4(o[0], o[1], o[2], o[3]);
        }
        return;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (col + j >= p.N) break;
        if (p.out_bf16) ((__nv_bfloat16*)p.y)[off + j] = __float2bfloat16_rn(o[j]);
        else ((float*)p.y)[off + j] = o[j];
    }
}

// The sums of a tile's parts as the CTAs of a cluster have parked them ([quarter][4 columns][32 rows] float4, the same layout in each):
// items `first` .. `end` - 1 of `units` column units of the quarters that have rows, kItems of them and kParts parts under way at a time.
// A lane reads its row.  Stored so, an instruction would touch 32 rows, 16 bytes of each; kItems lanes exchange their items first, so that it
// writes 32 / kItems rows, kItems * 16 bytes of each.  688 x 1152 x 3136 in two parts, with bias: 20.1 us without this and with the epilogue
// applied unit by unit, 16.7 so (18.2 when the parts went through L2 to the CTA that finished last).
template <uint32_t BN, uint32_t kItems, uint32_t kParts>
__device__ __forceinline__ void add_parked(const KParams& p, uint32_t park, uint32_t first, uint32_t end, uint32_t units, uint32_t row0, uint32_t col0, uint32_t lane) {
    const bool vec = p.N % 4 == 0 && ((uintptr_t)p.y & 15) == 0;      // four columns of a row start on a 16-byte (bf16: 8-byte) boundary
#pragma unroll 1
    for (uint32_t i0 = first; i0 < end; i0 += kItems) {
        float4 f[kItems][kParts];
#pragma unroll
        for (uint32_t e = 0; e < kItems; ++e) {
            const uint32_t i = i0 + e < end ? i0 + e : i0, quarter = i / units, unit = i - quarter * units;
#pragma unroll
            for (uint32_t s = 0; s < kParts; ++s)
                if (s < p.split_k) f[e][s] = ptx::ld_cluster_f4(ptx::mapa(park + quarter * (BM * BN) + unit * 512 + lane * 16, s));
        }
        float o[kItems][4];
#pragma unroll
        for (uint32_t e = 0; e < kItems; ++e) {
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) o[e][j] = 0.0f;
#pragma unroll
            for (uint32_t s = 0; s < kParts; ++s)
                if (s < p.split_k) { o[e][0] += f[e][s].x; o[e][1] += f[e][s].y; o[e][2] += f[e][s].z; o[e][3] += f[e][s].w; }
        }
        const uint32_t quarter = i0 / units, unit = i0 - quarter * units, row = row0 + quarter * 32;
        if (i0 + kItems <= end && unit + kItems <= units) {            // (warp-uniform) all of one quarter
            apply_epilogue(*(float (*)[kItems * 4])o, col0 + unit * 4, p);
            // item e of lane l goes to item l % kItems of lane l - l % kItems + e, a bit at a time
#pragma unroll
            for (uint32_t bit = 1; bit < kItems; bit *= 2) {
                const bool upper = lane & bit;
#pragma unroll
                for (uint32_t e = 0; e < kItems; ++e) {
                    if (e & bit) continue;
#pragma unroll
                    for (uint32_t j = 0; j < 4; ++j) {
                        const float got = __shfl_xor_sync(0xFFFFFFFFu, upper ? o[e][j] : o[e + bit][j], bit);
                        if (upper) o[e][j] = got;
                        else o[e + bit][j] = got;
                    }
                }
            }
#pragma unroll
            for (uint32_t e = 0; e < kItems; ++e) store4(p, vec, row + lane / kItems * kItems + e, col0 + (unit + lane % kItems) * 4, o[e]);
            continue;
        }
#pragma unroll
        for (uint32_t e = 0; e < kItems; ++e) {
            const uint32_t i = i0 + e;
            if (i >= end) break;
            apply_epilogue(o[e], col0 + i % units * 4, p);
            store4(p, vec, row0 + i / units * 32 + lane, col0 + i % units * 4, o[e]);
        }
    }
}

// Grouped launch: operand and output maps and the output addresses of up to kMaxGroupedGemms problems of one shape (12.5 KB
// of kernel parameters).
struct GroupOperands3 {
    CUtensorMap maps[3 * kMaxGroupedGemms];     // A, B, Y of problem i at 3i, 3i + 1, 3i + 2
    void* y[kMaxGroupedGemms];
};

// B_MN = B is given as B[K,N] (N contiguous), A_MN = A is given as A[K,M] (M contiguous): boxes of 64(k) x 64 columns, read by the
// UMMA through MN-major descriptors.
// kCluster = the parts of a tile's K are the CTAs of a cluster, one tile each: they add their sums through distributed shared memory.
template <uint32_t BN, bool B_MN, bool kGrouped = false, bool A_MN = false, bool kCluster = false>
__global__ void __launch_bounds__(kThreads, 1)
gemm_bf16_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                         const __grid_constant__ CUtensorMap map_y, const KParams p,
                         const __grid_constant__ std::conditional_t<kGrouped, GroupOperands3, NoGroup> group) {
    constexpr uint32_t kStages = stages_for(BN);
    constexpr uint32_t kBStageBytes = BN * BK * 2;
    constexpr uint32_t kStageBytes = kAStageBytes + kBStageBytes;
    // Two accumulator buffers.  Up to 128 columns a buffer holds two accumulators: with p.halves the first and second half of a part's
    // k blocks are summed apart and added in f32 by the epilogue, which halves the length of the tensor cores' sums and so their error.
    constexpr uint32_t kAccs = BN <= 128 ? 2 : 1;
    constexpr uint32_t kTmemCols = 2 * BN * kAccs;   // 128..512, a power of two
    constexpr uint32_t kIdesc = ptx::make_idesc_bf16_f32(BM, BN, B_MN ? 1u : 0u, A_MN ? 1u : 0u);

    extern __shared__ uint8_t smem_raw[];
    // 128-byte swizzled tiles need 1024-byte alignment
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* a_tiles = smem;
    uint8_t* b_tiles = smem + kStages * kAStageBytes;
    uint8_t* epi_stage = smem + kStages * kStageBytes;          // 4 warps x 2 blocks of kEpiStageBytes; 1024-byte aligned
    uint64_t* bars = (uint64_t*)(epi_stage + 8 * kEpiStageBytes);
    uint64_t* full_bar = bars;                       // [kStages] TMA bytes landed
    uint64_t* empty_bar = bars + kStages;            // [kStages] UMMAs finished reading the stage
    uint64_t* tmem_full_bar = bars + 2 * kStages;    // [2] accumulator complete
    uint64_t* tmem_empty_bar = bars + 2 * kStages + 2;  // [2] accumulator drained by the epilogue
    uint64_t* parked_bar = bars + 2 * kStages + 4;      // kCluster: every epilogue warp of the cluster has parked its rows
    uint32_t* tmem_holder = (uint32_t*)(bars + 2 * kStages + 5);
    volatile int* abort_flag = (volatile int*)(tmem_holder + 1);

    const uint32_t warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0);     // (the shuffle tells the compiler that a role is the whole warp's)
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t work_per_problem = p.tiles_m * p.tiles_n * p.split_k;
    uint32_t total_work = work_per_problem;                 // a grouped launch walks the tiles of all its problems, problem-major
    if constexpr (kGrouped) total_work = work_per_problem * p.n_problems;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kStages; ++s) {
            ptx::mbar_init(ptx::smem_u32(&full_bar[s]), 1);
            ptx::mbar_init(ptx::smem_u32(&empty_bar[s]), 1);
        }
        for (uint32_t b = 0; b < 2; ++b) {
            ptx::mbar_init(ptx::smem_u32(&tmem_full_bar[b]), 1);
            ptx::mbar_init(ptx::smem_u32(&tmem_empty_bar[b]), 4);   // one arrival per epilogue warp
        }
        if constexpr (kCluster) ptx::mbar_init(ptx::smem_u32(parked_bar), 4 * p.split_k);
        *abort_flag = 0;
        ptx::fence_barrier_init();
        ptx::fence_proxy_async_smem();
        ptx::tma_prefetch_desc(&map_a);
        ptx::tma_prefetch_desc(&map_b);
        if (p.tma_store) ptx::tma_prefetch_desc(&map_y);
    }
    if (warp == 1) {
        ptx::tmem_alloc(ptx::smem_u32(tmem_holder), kTmemCols);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    if constexpr (kCluster) ptx::cluster_sync_all();          // every CTA's barriers exist before anyone signals across the cluster
    ptx::tc_fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xFFFFFFFFu, *tmem_holder, 0);
    const uint32_t a_smem = ptx::smem_u32(a_tiles), b_smem = ptx::smem_u32(b_tiles), full = ptx::smem_u32(full_bar), empty = ptx::smem_u32(empty_bar);
    // everything above touched only shared and tensor memory; global memory comes after the previous grid is done
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();
    ClockProbe probe;
    probe.begin(p);

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer: the whole warp walks, one lane issues
        {
            uint32_t stage = 0, phase = 0;
            bool ok = true;
            for (uint32_t w = blockIdx.x; ok && w < total_work; w += gridDim.x) {
                uint32_t prob = 0, item = w;
                if constexpr (kGrouped) { prob = w / work_per_problem; item = w - prob * work_per_problem; }
                const WorkItem wi = decode_work(item, p);
                const CUtensorMap* ma = &map_a;
                const CUtensorMap* mb = &map_b;
                if constexpr (kGrouped) { ma = &group.maps[3 * prob]; mb = &group.maps[3 * prob + 1]; }
                const KRange kr = k_range<kCluster>(wi.split, p);
                for (uint32_t kb = kr.first; kb < kr.end; ++kb) {
                    if (!ptx::mbar_wait_warp(empty + 8 * stage, phase ^ 1, abort_flag, p.wait_limit_ns)) {
                        if (lane == 0) atomicCAS(p.status, 0, kStatusProducerTimeout | (int)(w & 0xFFFFFF));
                        ok = false;
                        break;
                    }
                    const uint32_t fb = full + 8 * stage, a_dst = a_smem + stage * kAStageBytes, b_dst = b_smem + stage * kBStageBytes;
                    // self-test of the failure path: this stage is never filled, so the issuer's bounded wait must run out
                    if (p.drop_load && blockIdx.x == 0 && w == 0 && kb == 0) { if (++stage == kStages) { stage = 0; phase ^= 1; } continue; }
                    const uint32_t issue = ptx::elect_one();
                    ptx::mbar_arrive_expect_tx_if(issue, fb, kStageBytes);
                    if constexpr (!A_MN) {
                        ptx::tma_load_3d_if(issue, a_dst, ma, fb, (int32_t)(kb * BK), (int32_t)(wi.m_blk * BM), (int32_t)kr.z);
                    } else {
#pragma unroll
                        for (uint32_t j = 0; j < BM / 64; ++j)
                            ptx::tma_load_3d_if(issue, a_dst + j * (BK * 128), ma, fb, (int32_t)(wi.m_blk * BM + j * 64), (int32_t)(kb * BK), (int32_t)kr.z);
                    }
                    if constexpr (!B_MN) {
                        ptx::tma_load_3d_if(issue, b_dst, mb, fb, (int32_t)(kb * BK), (int32_t)(wi.n_blk * BN), (int32_t)kr.z);
                    } else {
                        // B[K,N]: one 64(k) x 64(n) box per 64 columns; each box is an [k][128 B] block
#pragma unroll
                        for (uint32_t j = 0; j < BN / 64; ++j)
                            ptx::tma_load_3d_if(issue, b_dst + j * (BK * 128), mb, fb, (int32_t)(wi.n_blk * BN + j * 64), (int32_t)(kb * BK), (int32_t)kr.z);
                    }
                    __syncwarp();
                    if (++stage == kStages) { stage = 0; phase ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ UMMA issuer: the whole warp walks, one lane issues
        {
            uint32_t stage = 0, phase = 0, iter = 0;
            const uint32_t a_desc = ptx::smem_desc_lo(a_smem, A_MN ? BK * 128 : 16), b_desc = ptx::smem_desc_lo(b_smem, B_MN ? BK * 128 : 16);
            bool ok = true;
            for (uint32_t w = blockIdx.x; ok && w < total_work; w += gridDim.x, ++iter) {
                const uint32_t buf = iter & 1, acc_phase = (iter >> 1) & 1;
                if (!ptx::mbar_wait_warp(ptx::smem_u32(&tmem_empty_bar[buf]), acc_phase ^ 1, abort_flag, p.wait_limit_ns)) {
                    if (lane == 0) atomicCAS(p.status, 0, kStatusMmaTimeout | (int)(w & 0xFFFFFF));
                    break;
                }
                ptx::tc_fence_after_sync();
                const KRange kr = k_range<kCluster>(w % p.split_k, p);
                const uint32_t kb_mid = k_mid<kAccs>(kr, p);
                uint32_t tmem_d = tmem_base + buf * BN * kAccs;
                for (uint32_t kb = kr.first; kb < kr.end; ++kb) {
                    if (!ptx::mbar_wait_warp(full + 8 * stage, phase, abort_flag, p.wait_limit_ns)) {
                        if (lane == 0) atomicCAS(p.status, 0, kStatusMmaTimeout | 0x800000 | (int)(w & 0x7FFFFF));
                        ok = false;
                        break;
                    }
                    ptx::tc_fence_after_sync();
                    if (kb == kb_mid) tmem_d += BN;
                    // K-major, 128B swizzle: 8-row groups 1024 B apart; a 16-element K step is 32 B.  MN-major: 64-column atoms 8 KiB apart, 8-row k
                    // groups 1024 B apart; a K step is two groups.
                    const uint32_t issue = ptx::elect_one(), a = a_desc + stage * (kAStageBytes / 16), b = b_desc + stage * (kBStageBytes / 16);
                    ptx::umma_bf16_ss_if(issue, tmem_d, a, b, kIdesc, kb != kr.first && kb != kb_mid);
#pragma unroll
                    for (uint32_t k4 = 1; k4 < BK / 16; ++k4) ptx::umma_bf16_ss_if(issue, tmem_d, a + k4 * (A_MN ? 128 : 2), b + k4 * (B_MN ? 128 : 2), kIdesc, 1u);
                    ptx::umma_commit_if(issue, empty + 8 * stage);
                    __syncwarp();
                    if (++stage == kStages) { stage = 0; phase ^= 1; }
                }
                if (ok && ptx::elect_one()) ptx::umma_commit(ptx::smem_u32(&tmem_full_bar[buf]));
                __syncwarp();
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue (warps 2..5)
        const uint32_t quarter = warp & 3;   // tensor-memory lanes 32*quarter .. +31 belong to this warp
        uint32_t iter = 0, n_stores = 0;     // n_stores: this warp's committed TMA stores, see store_chunk
        for (uint32_t w = blockIdx.x; w < total_work; w += gridDim.x, ++iter) {
            uint32_t prob = 0, item = w;
            if constexpr (kGrouped) { prob = w / work_per_problem; item = w - prob * work_per_problem; }
            const WorkItem wi = decode_work(item, p);
            void* y_out = p.y;
            const CUtensorMap* my = &map_y;
            if constexpr (kGrouped) { y_out = group.y[prob]; my = &group.maps[3 * prob + 2]; }
            const uint32_t buf = iter & 1, acc_phase = (iter >> 1) & 1;
            const uint32_t row_base = wi.m_blk * BM + quarter * 32;
            if constexpr (kCluster) {
                // the tile's bias into L1 under the main loop: the warps would wait for it once for every few columns they add
                if (p.bias && lane * 32 < BN && wi.n_blk * BN + lane * 32 < p.N) ptx::prefetch_l1(p.bias + wi.n_blk * BN + lane * 32);
            }
            if (!ptx::mbar_wait(ptx::smem_u32(&tmem_full_bar[buf]), acc_phase, abort_flag, p.wait_limit_ns)) {
                if (lane == 0) atomicCAS(p.status, 0, kStatusEpilogueTimeout | (int)(w & 0xFFFFFF));
                break;
            }
            ptx::tc_fence_after_sync();
            const KRange kr = k_range<kCluster>(wi.split, p);
            const bool two_accs = k_mid<kAccs>(kr, p) < kr.end;
            const uint32_t tmem_acc = tmem_base + ((quarter * 32) << 16) + buf * BN * kAccs;
            if constexpr (kCluster) {
                // Split-K with a complete result: the CTAs of the cluster hold the parts of one tile.  Every warp parks its rows' sums in its
                // CTA's shared memory, over the ring that is idle by then, and tells every CTA.  The tile is then shared out evenly over all
                // the warps of the cluster, whatever its rows and columns; the parts are added in split order, the same sums as the planes
                // form.  Nothing but the operands and the result is in global memory, so launches may run beside one another, recorded or not.
                // What bounds it is latency: park, signal, and one or two round trips of remote reads, about 3 us with the cluster's start.
                // 16 x 2048 x 2048: 8.8 us, 10.9 with the parts added through L2 by the CTA that finishes last, 20.0 as clusters of
                // eight that do not all run at once; 128 x 4096 x 4096 (32 clusters of four): 15.6 us, 16.9 with column slices read row by row.
                const uint32_t park = ptx::smem_u32(smem);
#pragma unroll 1
                for (uint32_t c = 0; c < BN / 32 && row_base < p.M; ++c) {
                    uint32_t r[32];
                    load_acc<BN>(tmem_acc + c * 32, two_accs, r);
#pragma unroll
                    for (uint32_t j = 0; j < 8; ++j)
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(park + quarter * (BM * BN) + (c * 8 + j) * 512 + lane * 16), "r"(r[4 * j]),
                                     "r"(r[4 * j + 1]), "r"(r[4 * j + 2]), "r"(r[4 * j + 3])
                                     : "memory");
                }
                __syncwarp();
                if (lane == 0)
                    for (uint32_t s = 0; s < p.split_k; ++s) ptx::mbar_arrive_cluster(ptx::mapa(ptx::smem_u32(parked_bar), s));
                if (!ptx::mbar_wait_cluster(ptx::smem_u32(parked_bar), 0, abort_flag, p.wait_limit_ns)) {
                    if (lane == 0) atomicCAS(p.status, 0, kStatusEpilogueTimeout | 0x800000 | (int)(w & 0x7FFFFF));
                    break;
                }
                const uint32_t row0 = wi.m_blk * BM, col0 = wi.n_blk * BN;
                const uint32_t units = (min(BN, p.N - col0) + 3) / 4;
                const uint32_t items = (min(BM, p.M - row0) + 31) / 32 * units;
                const uint32_t worker = wi.split * 4 + warp - 2, first = worker * items / (4 * p.split_k), end = (worker + 1) * items / (4 * p.split_k);
                if (p.split_k <= 4) add_parked<BN, 4, 4>(p, park, first, end, units, row0, col0, lane);
                else add_parked<BN, 2, 8>(p, park, first, end, units, row0, col0, lane);
                break;                                   // a cluster has one tile
            }
#pragma unroll 1
            for (uint32_t c = 0; c < BN / 32; ++c) {
                const uint32_t col0 = wi.n_blk * BN + c * 32;
                if (col0 >= p.N) break;   // warp-uniform
                uint32_t r[32];
                load_acc<BN>(tmem_acc + c * 32, two_accs, r);
                store_chunk(p, r, row_base, lane, c, col0, wi.split, epi_stage + quarter * 2 * kEpiStageBytes, n_stores,
                            p.tma_store ? my : nullptr, y_out);
            }
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&tmem_empty_bar[buf]));
        }
        if (p.tma_store && lane == 0) ptx::bulk_wait_group_all();   // this warp's stores are complete before shared memory goes away
    }

    // ---------------------------------------------------------------- common exit
    __syncwarp();
    probe.end(p);
    if (*abort_flag) {
        // give copies and UMMAs already in flight time to land before shared and tensor memory go away
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    if constexpr (kCluster) ptx::cluster_sync_all();          // no CTA's shared memory goes away while a peer may still read it or signal its barrier
    if (warp == 1) {
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc(tmem_base, kTmemCols);
    }
}

// ------------------------------------------------------------------ host side

template <uint32_t BN, bool B_MN, bool kGrouped = false, bool A_MN = false, bool kCluster = false>
int launch_instance(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& my, const KParams& p, uint32_t grid, cudaStream_t stream,
                    const std::conditional_t<kGrouped, GroupOperands3, NoGroup>& group = {}) {
    auto kern = gemm_bf16_tcgen05_kernel<BN, B_MN, kGrouped, A_MN, kCluster>;
    const uint32_t smem = gemm_smem_bytes(BN);
    static bool attr_set[64] = {};   // per instantiation, per device
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return fail(T0_ERR_CUDA, "cudaFuncSetAttribute(smem=%u): %s", smem, cudaGetErrorString(e));
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    cudaError_t e = launch_pdl_clusters(kern, grid, kCluster ? p.split_k : 1, kThreads, smem, stream, ma, mb, my, p, group);
    if (e != cudaSuccess) return fail(T0_ERR_CUDA, "GEMM kernel launch failed: %s", cudaGetErrorString(e));
    return T0_OK;
}

}  // namespace

// The SMs of a GPC hold whole clusters only, and GPCs differ in size: 148 SMs hold 15 clusters of eight, not 18 (a B200 reports 74, 45, 33,
// 26, 22, 15, 15 for two to eight).  Behind a kernel whose blocks leave one by one, clusters of odd size do not pack as well (44 clusters of
// three: 12.2 us behind one of their own, 17.6 behind a conversion; 40: no difference), so the table stays below that for them.  Where
// the device's own figure is lower, it counts.
const uint32_t* gemm_clusters_at_once() {
    static uint32_t table[64][kMaxClusterParts + 1] = {};
    static std::mutex mu;
    static const uint32_t safe[kMaxClusterParts + 1] = {0, 148, 74, 40, 33, 24, 20, 14, 15};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return safe;
    std::lock_guard<std::mutex> lock(mu);
    if (!table[dev][1]) {
        auto kern = gemm_bf16_tcgen05_kernel<64, false, false, false, true>;
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm_smem_bytes(64));
        for (uint32_t size = 2; size <= kMaxClusterParts; ++size) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute attr;
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim = {size, 1, 1};
            cfg.gridDim = dim3(size * 148, 1, 1);
            cfg.blockDim = dim3(kThreads, 1, 1);
            cfg.dynamicSmemBytes = gemm_smem_bytes(64);
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) { cudaGetLastError(); n = 1; }
            table[dev][size] = std::min((uint32_t)n, safe[size]);
        }
        table[dev][1] = safe[1];
    }
    return table[dev];
}

uint32_t gemm_stage_count(uint32_t tile_n) { return stages_for(snap_tile_n(tile_n)); }

uint32_t gemm_smem_bytes(uint32_t tile_n) {
    const uint32_t bn = snap_tile_n(tile_n);
    // tiles + barriers/holder (256 B) + the epilogue warps' staging chunks + slack for the 1024-byte alignment of the dynamic segment
    return stages_for(bn) * (kAStageBytes + bn * BK * 2) + 256 + 8 * kEpiStageBytes + 1024;
}

int launch_gemm_sm100(const GemmLaunch& g, cudaStream_t stream) {
    if (g.m == 0 || g.n == 0) return T0_OK;
    if (g.k == 0) return fail(T0_ERR_INVALID, "K must be positive");
    // parts of K: planes of the output (and of the operand maps), or, where the launch adds them itself, ranges of the whole K
    const bool parts = g.cluster && g.split_k > 1;
    const uint32_t planes = parts || g.split_k == 0 ? 1 : g.split_k, split = parts ? g.split_k : planes;
    if (g.k % planes) return fail(T0_ERR_UNSUPPORTED, "K=%u not divisible by split_k=%u", g.k, split);
    const uint32_t kps = g.k / planes;
    if (parts && (split > kMaxClusterParts || split > ceil_div(g.k, BK)))
        return fail(T0_ERR_UNSUPPORTED, "split-K in one launch: %u parts of %u k blocks", split, ceil_div(g.k, BK));
    const uint32_t ldx = g.ldx ? g.ldx : (g.at ? g.m : g.k);
    const uint32_t ldb = g.ldb ? g.ldb : (g.nn ? g.n : g.k);
    if (g.at && !g.nn) return fail(T0_ERR_UNSUPPORTED, "a transposed first operand goes with B[K,N]");
    if ((ldx % 8) || (ldb % 8) || (planes > 1 && (kps % 8)))
        return fail(T0_ERR_UNSUPPORTED, "row strides (%u, %u) and, with split-K, K per split (%u) must be multiples of 8 for the TMA path", ldx, ldb, kps);
    if (((uintptr_t)g.x & 15) || ((uintptr_t)g.b & 15)) return fail(T0_ERR_UNSUPPORTED, "operand pointers must be 16-byte aligned");
    const uint32_t bn = snap_tile_n(g.tile_n);
    if (g.nn && bn < 64) return fail(T0_ERR_UNSUPPORTED, "NN layout needs tile_n >= 64");

    KParams p;
    memset(&p, 0, sizeof p);
    p.wait_limit_ns = g.wait_limit_ns ? g.wait_limit_ns : ptx::kWaitLimitNs; p.drop_load = g.drop_load ? 1 : 0;
    p.y = g.y; p.bias = g.bias; p.status = g.status; p.probe = g.probe; p.trace = nullptr; p.plane_stride = g.plane_stride;
    p.M = g.m; p.N = g.n; p.K = g.k;
    p.tiles_m = ceil_div(g.m, BM); p.tiles_n = ceil_div(g.n, bn); p.split_k = split;
    p.kb_per_split = ceil_div(kps, BK);
    p.swap_grid = g.swap_grid ? 1 : 0; p.raster_group = 8;
    p.out_bf16 = g.out_bf16 ? 1 : 0; p.epilogue = g.epilogue; p.n_ops = g.n_ops;
    p.scale = g.scale; p.clamp_min = g.clamp_min; p.clamp_max = g.clamp_max;
    memcpy(p.ops, g.ops, sizeof p.ops);
    p.halves = g.halves ? 1 : 0;

    CUtensorMap ma, mb;
    int rc = g.at ? make_map_nmajor(&ma, g.x, g.m, ldx, kps, planes) : make_map_kmajor(&ma, g.x, g.m, ldx, kps, planes, BM);
    if (rc != T0_OK) return rc;
    rc = g.nn ? make_map_nmajor(&mb, g.b, g.n, ldb, kps, planes) : make_map_kmajor(&mb, g.b, g.n, ldb, kps, planes, bn);
    if (rc != T0_OK) return rc;

    const uint64_t total = (uint64_t)p.tiles_m * p.tiles_n * split;
    if (total > 0x7FFFFFFFull) return fail(T0_ERR_UNSUPPORTED, "too many tiles");
    const uint32_t grid = (uint32_t)(parts ? total : std::min<uint64_t>(total, g.n_sms ? g.n_sms : 148));
    CUtensorMap my = ma;   // a valid map either way; only read when p.tma_store is set
    if (tma_output_ok(g, planes, bn)) {
        rc = make_map_out(&my, g.y, g.m, g.n, planes, g.plane_stride, g.out_bf16);
        if (rc != T0_OK) return rc;
        p.tma_store = 1;
    }
    rc = stage_peer_maps(g, p, split, stream);
    if (rc != T0_OK) return rc;

    if (parts) {
        if (g.at && bn <= 128)
            return bn == 64 ? launch_instance<64, true, false, true, true>(ma, mb, my, p, grid, stream)
                            : launch_instance<128, true, false, true, true>(ma, mb, my, p, grid, stream);
        if (g.at) return fail(T0_ERR_UNSUPPORTED, "no cluster form for a transposed first operand with 256-wide tiles");
        if (g.nn) {
            switch (bn) {
                case 64: return launch_instance<64, true, false, false, true>(ma, mb, my, p, grid, stream);
                case 128: return launch_instance<128, true, false, false, true>(ma, mb, my, p, grid, stream);
                default: return launch_instance<256, true, false, false, true>(ma, mb, my, p, grid, stream);
            }
        }
        switch (bn) {
            case 32: return launch_instance<32, false, false, false, true>(ma, mb, my, p, grid, stream);
            case 64: return launch_instance<64, false, false, false, true>(ma, mb, my, p, grid, stream);
            case 128: return launch_instance<128, false, false, false, true>(ma, mb, my, p, grid, stream);
            default: return launch_instance<256, false, false, false, true>(ma, mb, my, p, grid, stream);
        }
    }
    if (g.at) {
        switch (bn) {
            case 64: return launch_instance<64, true, false, true>(ma, mb, my, p, grid, stream);
            case 128: return launch_instance<128, true, false, true>(ma, mb, my, p, grid, stream);
            default: return launch_instance<256, true, false, true>(ma, mb, my, p, grid, stream);
        }
    }
    if (g.nn) {
        switch (bn) {
            case 64: return launch_instance<64, true>(ma, mb, my, p, grid, stream);
            case 128: return launch_instance<128, true>(ma, mb, my, p, grid, stream);
            default: return launch_instance<256, true>(ma, mb, my, p, grid, stream);
        }
    }
    switch (bn) {
        case 32: return launch_instance<32, false>(ma, mb, my, p, grid, stream);
        case 64: return launch_instance<64, false>(ma, mb, my, p, grid, stream);
        case 128: return launch_instance<128, false>(ma, mb, my, p, grid, stream);
        default: return launch_instance<256, false>(ma, mb, my, p, grid, stream);
    }
}

// Several problems of one shape, no split-K, NT layout, 64- or 128-wide tiles, in one launch: the persistent CTAs walk the
// tiles of all the problems (see kernels.h).  Every problem must qualify for the TMA path (16-byte aligned operands, K % 8).
int launch_gemm_sm100_grouped(const GemmLaunch* gs, uint32_t count, cudaStream_t stream) {
    if (!gs || count == 0) return T0_OK;
    if (count > kMaxGroupedGemms) return fail(T0_ERR_INVALID, "at most %u problems per grouped launch (got %u)", kMaxGroupedGemms, count);
    const GemmLaunch& g0 = gs[0];
    if (g0.m == 0 || g0.n == 0) return T0_OK;
    const uint32_t bn = snap_tile_n(g0.tile_n);
    if (g0.nn || (g0.split_k > 1) || (bn != 64 && bn != 128) || g0.k == 0 || g0.k % 8 || g0.n_peer_y)
        return fail(T0_ERR_UNSUPPORTED, "grouped launch: NT layout, no split-K, tile width 64 or 128, K a positive multiple of 8");
    const uint32_t ldx = g0.ldx ? g0.ldx : g0.k, ldb = g0.ldb ? g0.ldb : g0.k;
    if ((ldx % 8) || (ldb % 8)) return fail(T0_ERR_UNSUPPORTED, "grouped launch: row strides must be multiples of 8");
    KParams p;
    memset(&p, 0, sizeof p);
    p.wait_limit_ns = g0.wait_limit_ns ? g0.wait_limit_ns : ptx::kWaitLimitNs;
    p.y = g0.y; p.bias = g0.bias; p.status = g0.status; p.probe = g0.probe;
    p.M = g0.m; p.N = g0.n; p.K = g0.k;
    p.tiles_m = ceil_div(g0.m, BM); p.tiles_n = ceil_div(g0.n, bn); p.split_k = 1;
    p.kb_per_split = ceil_div(g0.k, BK);
    p.swap_grid = g0.swap_grid ? 1 : 0; p.raster_group = 8;
    p.out_bf16 = g0.out_bf16 ? 1 : 0; p.epilogue = g0.epilogue; p.n_ops = g0.n_ops;
    p.scale = g0.scale; p.clamp_min = g0.clamp_min; p.clamp_max = g0.clamp_max;
    memcpy(p.ops, g0.ops, sizeof p.ops);
    p.n_problems = count;
    bool tma_store = true;
    for (uint32_t i = 0; i < count; ++i) tma_store = tma_store && tma_output_ok(gs[i], 1, bn);
    p.tma_store = tma_store ? 1 : 0;
    static GroupOperands3 group;         // 12.5 KB: kept off the stack, filled under the lock, copied by the launch
    static std::mutex group_mu;
    std::lock_guard<std::mutex> lock(group_mu);
    for (uint32_t i = 0; i < count; ++i) {
        const GemmLaunch& g = gs[i];
        if (g.m != g0.m || g.n != g0.n || g.k != g0.k || g.ldx != g0.ldx || g.ldb != g0.ldb || g.tile_n != g0.tile_n || g.split_k != g0.split_k ||
            g.nn != g0.nn || g.out_bf16 != g0.out_bf16 || g.swap_grid != g0.swap_grid || g.epilogue != g0.epilogue || g.n_ops != g0.n_ops ||
            memcmp(g.ops, g0.ops, sizeof g.ops) != 0 || g.scale != g0.scale || g.clamp_min != g0.clamp_min || g.clamp_max != g0.clamp_max ||
            g.bias != g0.bias)
            return fail(T0_ERR_INVALID, "grouped launch: problem %u differs from problem 0 in shape or configuration", i);
        if (!g.x || !g.b || !g.y) return fail(T0_ERR_INVALID, "grouped launch: null pointer in problem %u", i);
        if (((uintptr_t)g.x & 15) || ((uintptr_t)g.b & 15)) return fail(T0_ERR_UNSUPPORTED, "grouped launch: operands of problem %u are not 16-byte aligned", i);
        int rc = make_map_kmajor(&group.maps[3 * i], g.x, g.m, ldx, g.k, 1, BM);
        if (rc == T0_OK) rc = make_map_kmajor(&group.maps[3 * i + 1], g.b, g.n, ldb, g.k, 1, bn);
        if (rc != T0_OK) return rc;
        group.maps[3 * i + 2] = group.maps[3 * i];          // a valid map either way; only read when p.tma_store is set
        if (tma_store) {
            rc = make_map_out(&group.maps[3 * i + 2], g.y, g.m, g.n, 1, 0, g.out_bf16);
            if (rc != T0_OK) return rc;
        }
        group.y[i] = g.y;
    }
    const uint64_t total = (uint64_t)p.tiles_m * p.tiles_n * count;
    if (total > 0x7FFFFFFFull) return fail(T0_ERR_UNSUPPORTED, "too many tiles");
    const uint32_t grid = (uint32_t)std::min<uint64_t>(total, g0.n_sms ? g0.n_sms : 148);
    return bn == 128 ? launch_instance<128, false, true>(group.maps[0], group.maps[1], group.maps[2], p, grid, stream, group)
                     : launch_instance<64, false, true>(group.maps[0], group.maps[1], group.maps[2], p, grid, stream, group);
}

}  // namespace t0
