// Constants and device helpers shared by the fused W4A16 kernels (row-layout kernels in w4a16.cu, streaming-layout kernel
// in w4a16_stream.cu): the band / step geometry, the work split, the bf16x2 dequantisation primitives.
#pragma once

#include <cuda_bf16.h>

#include "runtime_internal.h"
#include "gemm_common.cuh"

namespace t0 {
namespace w4 {

constexpr int kWarps = 16;               // consumer warps; one more warp feeds them through TMA
constexpr int kThreads = (kWarps + 1) * 32;
constexpr int kSlabCols = 32;            // columns one warp owns
constexpr int kBandSlabs = 8;            // slabs side by side in a CTA: 256 columns = 1 KiB of every packed row
constexpr int kBandCols = kSlabCols * kBandSlabs;
constexpr int kSlices = kWarps / kBandSlabs;   // k slices of 64 per step
constexpr int kUnitK = kSlices * 64;     // k depth of one step of the CTA: 128
constexpr int kStages = 8;               // steps in flight per CTA (TMA ring)
constexpr int kARecord = 288;            // bytes per 8-k activation record (256 + 32: conflict-free quad reads)
constexpr int kWeightBytes = (kUnitK / 8) * kBandCols * 4;   // 16 packed rows x 1 KiB
constexpr int kScaleBytes = kBandCols * 2;
constexpr int kZeroBytes = (kBandCols / 8) * 4;
constexpr int kStageBytes = kWeightBytes + kScaleBytes + kZeroBytes + 128;   // 17152, keeps every stage 128-byte aligned
constexpr int kRedBytes = kWarps * 16 * 33 * 4;
constexpr int kPieceFloats = 16 * kBandCols;
constexpr int kMaxAUnits = 12;           // steps of activations staged at a time (54 KiB)
constexpr size_t kMaxSmem = 128 + (size_t)kStages * kStageBytes + kRedBytes + 256 + (size_t)kMaxAUnits * (kUnitK / 8) * kARecord;
constexpr size_t kCounterRegion = 16 * 1024;   // arrival counters: up to 4096 bands (N <= 1048576)

struct W4Params {
    const uint16_t* a;
    float* y;
    float* partials;     // [grid][2][16*256]
    int* counters;       // [n_bands], zero between calls
    int* status;         // error word of the runtime (bounded waits)
    uint32_t M, N, K;
    uint32_t units_per_group;   // group / 128: steps that share one row of scales and zero points
    uint32_t n_bands, ksteps, total_units;
    uint32_t a_units;    // steps of activations the shared-memory area holds (max steps of one CTA)
    unsigned long long* stamps;   // optional trace: 4 nanosecond stamps per CTA (entry, staged, loop done, exit)
};

__device__ __forceinline__ uint32_t owner_of(uint32_t unit, uint32_t grid, uint32_t total) {
    return (uint32_t)((((uint64_t)unit + 1) * grid - 1) / total);
}
__device__ __forceinline__ uint32_t range_begin(uint32_t cta, uint32_t grid, uint32_t total) {
    return (uint32_t)((uint64_t)cta * total / grid);
}

__device__ __forceinline__ uint32_t bf16x2_sub(uint32_t a, uint32_t b) {
    __nv_bfloat162 r = __hsub2(*(__nv_bfloat162*)&a, *(__nv_bfloat162*)&b);
    return *(uint32_t*)&r;
}
__device__ __forceinline__ uint32_t bf16x2_mul(uint32_t a, uint32_t b) {
    __nv_bfloat162 r = __hmul2(*(__nv_bfloat162*)&a, *(__nv_bfloat162*)&b);
    return *(uint32_t*)&r;
}

__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// (x & mask) | magic in one LOP3; mask and magic must sit in registers (the instruction takes one immediate at most)
__device__ __forceinline__ uint32_t and_or(uint32_t x, uint32_t mask, uint32_t magic) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(x), "r"(mask), "r"(magic));
    return r;
}

// The tcgen05 kernels (w4a16_umma.cu, w4a16_umma_cut.cu): a chunk of the raw weights is 8 packed rows x 256 columns, their scales and
// zero points.
constexpr uint32_t kUmBN = 256;                             // columns of y per tile
constexpr uint32_t kUmBK = 64;                              // k per chunk: one 128-byte swizzle atom of bf16
constexpr uint32_t kUmRawBytes = 8 * kUmBN * 4 + kUmBN * 2 + (kUmBN / 8) * 4;      // 8832: words, scales, zero points
constexpr uint32_t kUmRawStride = 9216;                     // keeps every stage 1024-byte aligned

__device__ __forceinline__ uint32_t um_lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t um_lds16(uint32_t addr) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr) : "memory");
    return v;
}

__device__ __forceinline__ uint32_t um_ld_acquire(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Division by a number the host knows: the quotient by a product with floor((2^32 - 1) / d), at most two short.  Every CTA divides a few times before its first
// load, on the way of the whole launch, and a division takes 150 cycles.
struct UmDiv {
    uint32_t d, m;
};
inline UmDiv um_divisor(uint32_t d) { return {d, 0xFFFFFFFFu / d}; }
__device__ __forceinline__ uint32_t um_div(uint32_t a, const UmDiv& by) {
    uint32_t q = __umulhi(a, by.m), r = a - q * by.d;
    if (r >= by.d) { ++q; r -= by.d; }
    return r >= by.d ? q + 1 : q;
}

// The eight codes of a packed word as bf16x2 pairs in k order, (0,1) (2,3) (4,5) (6,7): (code | 0x4300) is the bf16 128 + code, so minus (128 + z),
// times s, is (q - z) * s rounded once.  zz = (128 + z) and ss = s, both halves alike.
__device__ __forceinline__ void um_dequant_word(uint32_t wd, uint32_t mask, uint32_t magic, uint32_t zz, uint32_t ss, bool tiled, uint32_t (&o)[4]) {
    const uint32_t v0 = bf16x2_mul(bf16x2_sub(and_or(wd, mask, magic), zz), ss);            // row layout: k 0, 4
    const uint32_t v1 = bf16x2_mul(bf16x2_sub(and_or(wd >> 4, mask, magic), zz), ss);       // k 1, 5
    const uint32_t v2 = bf16x2_mul(bf16x2_sub(and_or(wd >> 8, mask, magic), zz), ss);       // k 2, 6
    const uint32_t v3 = bf16x2_mul(bf16x2_sub(and_or(wd >> 12, mask, magic), zz), ss);      // k 3, 7
    if (tiled) {                           // tile-major words are stored so that the pairs come out in k order
        o[0] = v0; o[1] = v1; o[2] = v2; o[3] = v3;
    } else {
        o[0] = __byte_perm(v0, v1, 0x5410);
        o[1] = __byte_perm(v2, v3, 0x5410);
        o[2] = __byte_perm(v0, v1, 0x7632);
        o[3] = __byte_perm(v2, v3, 0x7632);
    }
}

// The tensor maps and outputs of up to kProblems problems of one shape, in the kernel parameters: row layout, four maps each (weights, scales, zero points,
// activations); tile-major layout, the activations' alone and the buffer, which is copied from without one (4.6 KB for a list).  A launch copies its
// parameters: a single call in a block of its own size 4.2 us on the host instead of 5.0, 20 x 14336 x 2048 waited for 24.8 instead of 26.0.
constexpr uint32_t kUmMaxGroup = 32;
template <uint32_t kProblems, bool kTiled>
struct UmGroup {
    CUtensorMap maps[(kTiled ? 1 : 4) * kProblems];
    float* y[kProblems];
    const uint8_t* base[kTiled ? kProblems : 1];
};

// How a launch shares out its tiles: the parts of a tile's K over the CTAs of a cluster (one problem); whole tiles per CTA; equal ranges of the
// list of chunks, tiles cut where ranges end.
enum { kUmClusters, kUmWhole, kUmCut };

// Trace buffer of the T0_W4_TRACE debugging aid: freed on every path out of the entry point that made it.
struct StampBuffer {
    unsigned long long* d = nullptr;
    size_t words = 0;
    int make(uint32_t grid) {
        words = (size_t)grid * 8;
        T0_CUDA(cudaMalloc(&d, words * sizeof(unsigned long long)));
        T0_CUDA(cudaMemset(d, 0, words * sizeof(unsigned long long)));
        return T0_OK;
    }
    ~StampBuffer() { if (d) cudaFree(d); }
};

}  // namespace w4
}  // namespace t0
