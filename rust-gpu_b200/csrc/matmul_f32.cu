// The framework-facing f32 entries over the bf16 GEMM: Ignis `matmul` and its backward helpers, and the
// `BlasLib::gemm` / `gemv` facade.
//
// Reference: src/ignis/ops/bf16_matmul.rs — `matmul(x[M,K] f32, w[K,N] f32) -> y[M,N] f32` (:33-59) runs
// `dispatch_gemm_forward` (:162-207): read x and w back to the host, round to bf16 (nearest even, :371-372), transpose w,
// pad everything to tile multiples, upload, GEMM, un-pad with a copy kernel (:318-348).  `gemm_backward_data` (:216-262)
// is dX = dY * W^T, `gemm_backward_weight` (:264-312) is dW = X^T * dY, `matmul_with_wt_bf16` (:93-133) takes the weight
// already transposed and in bf16.  src/universal/math/mod.rs:24-47 is the BLAS trait, math/blas.rs:18-100 its CPU body.
//
// Here the conversion of both operands is one pass on the device (f32 -> bf16, rows padded to whole 16-byte units) and the GEMM
// reads them where they lie: w as B[K,N], X^T for dW as A[K,M], so nothing is ever transposed; ragged edges are handled by
// TMA zero fill and clipped stores, and nothing is copied back or round-tripped through the host.
#include "runtime_internal.h"
#include "gemm_common.cuh"

using namespace t0;

namespace {

__device__ __forceinline__ uint16_t bf16_rne_bits(float v) {
    // bf16_matmul.rs:371-372: (bits + 0x7FFF + ((bits >> 16) & 1)) >> 16
    const uint32_t bits = __float_as_uint(v);
    return (uint16_t)((bits + 0x7FFFu + ((bits >> 16) & 1u)) >> 16);
}

// One operand of a conversion launch: dst[r * ld_dst + c] = bf16(src[r * ld_src + c]), c < cols, in units of eight destination
// elements of one row (ld_dst is a multiple of 8 and dst 16-byte aligned; columns from cols to ld_dst are written as zero).
struct CvtOperand {
    const float* src;
    uint16_t* dst;
    uint32_t rows, cols, ld_src, ld_dst;
};

__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) { return (uint32_t)bf16_rne_bits(lo) | ((uint32_t)bf16_rne_bits(hi) << 16); }

__device__ __forceinline__ void cvt_unit(const CvtOperand& o, bool vec, uint32_t r, uint32_t c) {
    const float* s = o.src + (size_t)r * o.ld_src + c;
    float v[8];
    if (vec) {
        const float4 lo = __ldcs((const float4*)s), hi = __ldcs((const float4*)s + 1);      // the f32 source is read once
        v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w; v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
    } else {
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) v[i] = c + i < o.cols ? s[i] : 0.0f;
    }
    *(uint4*)(o.dst + (size_t)r * o.ld_dst + c) = make_uint4(bf16_pair(v[0], v[1]), bf16_pair(v[2], v[3]), bf16_pair(v[4], v[5]), bf16_pair(v[6], v[7]));
}

// Both operands of a product in one launch, whatever their strides and alignment: two 16-byte loads and one 16-byte store per unit.  Bound by memory.  It starts under
// the tail of the kernel before it and lets the product start under its own (programmatic dependent launch); until the wait
// returns it touches no global memory, since the kernel before may still write the sources or read the scratch.
// A training step of a 1024 -> 4096 layer on 2048 rows ran six conversion launches, one of them transposing: 127 us; with one
// launch per product and X^T read by the tensor cores as it lies, 105 us.
__global__ void __launch_bounds__(256) cvt_operands_kernel(const CvtOperand a, const CvtOperand b) {
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const CvtOperand& o = i == 0 ? a : b;
        const bool vec = (o.cols % 8 == 0) && (o.ld_src % 4 == 0) && ((uintptr_t)o.src & 15) == 0;
        const uint32_t per_row = o.ld_dst / 8;
        const uint64_t units = (uint64_t)o.rows * per_row;
        for (; u < units; u += stride) {
            const uint32_t r = units >> 32 ? (uint32_t)(u / per_row) : (uint32_t)u / per_row;      // a 64-bit division only where it is needed
            cvt_unit(o, vec, r, (uint32_t)(u - (uint64_t)r * per_row) * 8);
        }
        u -= units;
    }
}

// The same for operands without gaps between their rows, which is what the matmul entries have whenever the rows are whole units: unit u of the
// launch is unit u of a, then of b, so there is nothing to divide and nothing to branch on.  Bound by memory, and the loads in flight are what feeds
// it: 2048 threads an SM with 32 bytes each.  More bytes a thread cost registers, and with them threads beside the product that is still
// running (two units 32 registers and no gain, four 80 registers and 10 % of a step lost); sixteen blocks an SM instead of the eight that fit
// give the next one to whichever SM is free first.  Half as many blocks as fit: 111 us for the step below.
// kKeep: plain loads (not the read-only path, whose lines may be older than the launch that wrote them), so that a source that the next products convert again is still in L2; without it evict-first loads (cvt_keeps).
// Steps on 2048 rows of a 1024 -> 4096 layer 94.0 -> 86.9 us, 256 rows 40.1 -> 36.1, 4096 rows of 4096 -> 4096 (evict-first) 375.6 -> 373.1.
template <bool kKeep>
__global__ void __launch_bounds__(256, 8) cvt_dense_kernel(const float* sa, uint16_t* da, const float* sb, uint16_t* db, uint32_t units_a, uint32_t units) {
    ptx::grid_launch_dependents();
    const uint32_t stride = gridDim.x * blockDim.x;
    uint32_t u = blockIdx.x * blockDim.x + threadIdx.x;
    ptx::grid_dependency_wait();
    for (; u < units; u += stride) {
        const bool second = u >= units_a;
        const uint32_t i = second ? u - units_a : u;
        const float4* s = (const float4*)(second ? sb : sa) + 2 * (size_t)i;
        const float4 lo = kKeep ? s[0] : __ldcs(s), hi = kKeep ? s[1] : __ldcs(s + 1);
        ((uint4*)(second ? db : da))[i] = make_uint4(bf16_pair(lo.x, lo.y), bf16_pair(lo.z, lo.w), bf16_pair(hi.x, hi.y), bf16_pair(hi.z, hi.w));
    }
}

// c[i][j] = alpha * t[i][j] + beta * c[i][j]   (blas.rs:56: alpha * sum + beta * c)
__global__ void axpby_kernel(const float* __restrict__ t, float* __restrict__ c, uint32_t m, uint32_t n, uint32_t ldc, float alpha, float beta) {
    const uint64_t total = (uint64_t)m * n;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const uint32_t r = (uint32_t)(i / n), j = (uint32_t)(i - (uint64_t)r * n);
        float* dst = c + (size_t)r * ldc + j;
        // beta == 0 must not read c (BLAS convention; the reference multiplies, which propagates NaN from garbage)
        *dst = beta == 0.0f ? alpha * t[i] : alpha * t[i] + beta * *dst;
    }
}

// y[i] = alpha * sum_j a[i*lda + j] * x[j*incx] + beta * y[i*incy]: one warp per row, f32 throughout (blas.rs:77-100)
__global__ void gemv_f32_kernel(const float* __restrict__ a, const float* __restrict__ x, float* __restrict__ y, uint32_t m, uint32_t n,
                                uint32_t lda, uint32_t incx, uint32_t incy, float alpha, float beta) {
    const uint32_t warps_per_block = blockDim.x >> 5, lane = threadIdx.x & 31;
    for (uint32_t row = blockIdx.x * warps_per_block + (threadIdx.x >> 5); row < m; row += gridDim.x * warps_per_block) {
        float sum = 0.0f;
        for (uint32_t j = lane; j < n; j += 32) sum = fmaf(a[(size_t)row * lda + j], x[(size_t)j * incx], sum);
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
        if (lane == 0) {
            float* dst = y + (size_t)row * incy;
            *dst = beta == 0.0f ? alpha * sum : alpha * sum + beta * *dst;
        }
    }
}

uint32_t blocks_for(uint64_t n, uint32_t per_block, uint32_t sms) {
    const uint64_t want = (n + per_block - 1) / per_block;
    return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(want, (uint64_t)sms * 8));
}

uint32_t pitch(uint32_t cols) { return (cols + 7) & ~7u; }      // row stride of a converted operand: whole 16-byte units for the TMA maps

// The bf16 copy of src[rows][cols] (row stride ld_src) goes to `dense`, or, where rows have to be padded, to `padded` (the buffer of the
// padded operand copies of the bf16 entries): makes room and describes the conversion.
int plan_cvt(t0_runtime* rt, Scratch& dense, Scratch& padded, uint64_t src, uint32_t rows, uint32_t cols, uint32_t ld_src, CvtOperand* o) {
    Scratch& s = pitch(cols) == cols ? dense : padded;
    int rc = ensure_scratch(rt, s, std::max<size_t>((size_t)rows * pitch(cols) * 2, 16));
    if (rc != T0_OK) return rc;
    *o = CvtOperand{(const float*)src, (uint16_t*)s.ptr, rows, cols, ld_src, pitch(cols)};
    return T0_OK;
}

// No gaps between rows, whole units, 16-byte loads.
bool dense(const CvtOperand& o) { return o.rows == 0 || (o.ld_src == o.cols && o.ld_dst == o.cols && ((uintptr_t)o.src & 15) == 0); }

// Sources of up to half of the L2 (63 of 126 MB) and their bf16 copies fit in it together, so keeping the sources costs the product nothing and a step's later
// conversions find them: 38.5 -> 36.1 us for the 256-row step above.  Larger ones would push the copies out (4096 rows: 376.9 us kept, 373.1 evict-first).
bool cvt_keeps(uint64_t source_bytes) { return source_bytes <= 63ull << 20; }

// `b` may have no rows (one operand only).
int launch_cvt(t0_runtime* rt, const CvtOperand& a, const CvtOperand& b) {
    const uint64_t units = (uint64_t)a.rows * (a.ld_dst / 8) + (uint64_t)b.rows * (b.ld_dst / 8);
    if (units == 0) return T0_OK;
    cudaError_t e;
    if (dense(a) && dense(b) && units < (1u << 31)) {       // thread indices stay below 2^32
        const uint32_t units_a = (uint32_t)((uint64_t)a.rows * (a.ld_dst / 8));
        const uint32_t grid = (uint32_t)std::min<uint64_t>((units + 255) / 256, (uint64_t)rt->sm_count * 16);
        e = cvt_keeps(units * 32) ? gemm::launch_pdl(cvt_dense_kernel<true>, grid, 256, 0, rt->stream, a.src, a.dst, b.src, b.dst, units_a, (uint32_t)units)
                                  : gemm::launch_pdl(cvt_dense_kernel<false>, grid, 256, 0, rt->stream, a.src, a.dst, b.src, b.dst, units_a, (uint32_t)units);
    } else {
        e = gemm::launch_pdl(cvt_operands_kernel, blocks_for(units, 256, rt->sm_count), 256, 0, rt->stream, a, b);
    }
    if (e != cudaSuccess) return fail(T0_ERR_CUDA, "f32 -> bf16 conversion launch failed: %s", cudaGetErrorString(e));
    rt->launches.fetch_add(1);
    return T0_OK;
}

// y[m,n] = bf16(a) * bf16(b): both operands converted in one launch, then the product.  a is [m,k], or [k,m] with `at`; b is [k,n]
// with `nn`, else [n,k].
int product(t0_runtime* rt, uint64_t a, uint32_t lda, bool at, uint64_t b, uint32_t ldb, bool nn, uint64_t y, uint32_t m, uint32_t n, uint32_t k) {
    CvtOperand oa, ob;
    int rc = at ? plan_cvt(rt, rt->scratch_cvt_a, rt->scratch_a, a, k, m, lda, &oa) : plan_cvt(rt, rt->scratch_cvt_a, rt->scratch_a, a, m, k, lda, &oa);
    if (rc == T0_OK) rc = nn ? plan_cvt(rt, rt->scratch_cvt_b, rt->scratch_b, b, k, n, ldb, &ob) : plan_cvt(rt, rt->scratch_cvt_b, rt->scratch_b, b, n, k, ldb, &ob);
    if (rc == T0_OK) rc = launch_cvt(rt, oa, ob);
    if (rc != T0_OK) return rc;
    return gemm_strided(rt, (uint64_t)(uintptr_t)oa.dst, oa.ld_dst, at, (uint64_t)(uintptr_t)ob.dst, ob.ld_dst, nn, y, m, n, k);
}

int check_ptrs(t0_runtime* rt, std::initializer_list<uint64_t> ptrs) {
    int rc = check_rt(rt);
    if (rc != T0_OK) return rc;
    for (uint64_t p : ptrs)
        if (!p) return fail(T0_ERR_INVALID, "null device pointer");
    return T0_OK;
}

}  // namespace

extern "C" {

int t0_matmul_f32(t0_runtime* rt, uint64_t x, uint64_t w, uint64_t y, uint32_t m, uint32_t k, uint32_t n) {
    int rc = check_ptrs(rt, {x, w, y});
    if (rc != T0_OK) return rc;
    if (m == 0 || n == 0) return T0_OK;
    DeviceGuard guard(rt->device);
    return product(rt, x, k, false, w, n, true, y, m, n, k);         // y = x * w, w read as B[K,N]
}

int t0_matmul_f32_with_wt_bf16(t0_runtime* rt, uint64_t x, uint64_t wt_bf16, uint64_t y, uint32_t m, uint32_t k, uint32_t n) {
    int rc = check_ptrs(rt, {x, wt_bf16, y});
    if (rc != T0_OK) return rc;
    if (m == 0 || n == 0) return T0_OK;
    DeviceGuard guard(rt->device);
    CvtOperand oa, none = {};
    rc = plan_cvt(rt, rt->scratch_cvt_a, rt->scratch_a, x, m, k, k, &oa);
    if (rc == T0_OK) rc = launch_cvt(rt, oa, none);
    if (rc != T0_OK) return rc;
    return gemm_strided(rt, (uint64_t)(uintptr_t)oa.dst, oa.ld_dst, false, wt_bf16, 0, false, y, m, n, k);
}

int t0_matmul_f32_backward_data(t0_runtime* rt, uint64_t dy, uint64_t w, uint64_t dx, uint32_t m, uint32_t k, uint32_t n) {
    int rc = check_ptrs(rt, {dy, w, dx});
    if (rc != T0_OK) return rc;
    if (m == 0 || k == 0) return T0_OK;
    DeviceGuard guard(rt->device);
    return product(rt, dy, n, false, w, n, false, dx, m, k, n);      // dX[M,K] = dY[M,N] * W[K,N]^T: contraction over N
}

int t0_matmul_f32_backward_weight(t0_runtime* rt, uint64_t x, uint64_t dy, uint64_t dw, uint32_t m, uint32_t k, uint32_t n) {
    int rc = check_ptrs(rt, {x, dy, dw});
    if (rc != T0_OK) return rc;
    if (k == 0 || n == 0) return T0_OK;
    DeviceGuard guard(rt->device);
    return product(rt, x, k, true, dy, n, true, dw, k, n, m);        // dW[K,N] = X^T[K,M] * dY[M,N]: contraction over M, X read as it lies
}

int t0_blas_gemm_f32(t0_runtime* rt, uint32_t m, uint32_t n, uint32_t k, float alpha, uint64_t a, uint32_t lda, uint64_t b, uint32_t ldb,
                     float beta, uint64_t c, uint32_t ldc) {
    int rc = check_ptrs(rt, {a, b, c});
    if (rc != T0_OK) return rc;
    if (m == 0 || n == 0) return T0_OK;
    if (lda < k || ldb < n || ldc < n) return fail(T0_ERR_INVALID, "leading dimensions (%u, %u, %u) smaller than the rows they stride (%u, %u, %u)", lda, ldb, ldc, k, n, n);
    DeviceGuard guard(rt->device);
    const bool direct = alpha == 1.0f && beta == 0.0f && ldc == n;
    uint64_t t = c;
    if (!direct) {
        rc = ensure_scratch(rt, rt->scratch_cvt_c, (size_t)m * n * 4);
        if (rc != T0_OK) return rc;
        t = (uint64_t)(uintptr_t)rt->scratch_cvt_c.ptr;
    }
    rc = product(rt, a, lda, false, b, ldb, true, t, m, n, k);
    if (rc != T0_OK || direct) return rc;
    axpby_kernel<<<blocks_for((uint64_t)m * n, 1024, rt->sm_count), 256, 0, rt->stream>>>((const float*)t, (float*)c, m, n, ldc, alpha, beta);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(T0_ERR_CUDA, "axpby launch failed: %s", cudaGetErrorString(e));
    rt->launches.fetch_add(1);
    return T0_OK;
}

int t0_blas_gemv_f32(t0_runtime* rt, uint32_t m, uint32_t n, float alpha, uint64_t a, uint32_t lda, uint64_t x, uint32_t incx, float beta,
                     uint64_t y, uint32_t incy) {
    int rc = check_ptrs(rt, {a, x, y});
    if (rc != T0_OK) return rc;
    if (m == 0) return T0_OK;
    if (lda < n || incx == 0 || incy == 0) return fail(T0_ERR_INVALID, "lda=%u < n=%u or a zero increment", lda, n);
    DeviceGuard guard(rt->device);
    gemv_f32_kernel<<<blocks_for(m, 8, rt->sm_count), 256, 0, rt->stream>>>((const float*)a, (const float*)x, (float*)y, m, n, lda, incx, incy, alpha, beta);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(T0_ERR_CUDA, "gemv launch failed: %s", cudaGetErrorString(e));
    rt->launches.fetch_add(1);
    return T0_OK;
}

}  // extern "C"
