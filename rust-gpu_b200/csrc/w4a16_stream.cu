// K2, streaming form: the fused W4A16 GEMM for M <= 16 on weights in the streaming layout, one persistent launch for a
// whole list of problems.
//
// No counterpart kernel exists in the reference (its INT4 support stops at the stand-alone dequantisation kernels,
// src/t0/quant_kernels.rs:53-171); the batching idea is the reference's DispatchQueue (src/t0/prefill_dispatch.rs:61-206):
// a decode step submits one projection after another and waits once.
//
// y[m,n] = sum_k a[m,k] * w[k,n],  w = RNE_bf16((q - z) * s),  fp32 accumulate.  The int4 weights are ~97 % of the bytes,
// so the kernel is organised around streaming them exactly once at HBM rate:
//   * weights come in the layout of t0_w4_prepack: per (256-column band, 128-deep k step) one contiguous 16 KiB tile whose
//     words are in 16 x 16 fragment order; a "unit" is one such tile.  The units of ALL problems of a launch form
//     one list, cut into equal contiguous ranges, one per CTA (one CTA per SM), so that launch, pipeline fill and the band
//     fix-up at the end of a range are paid once per launch instead of once per problem;
//   * one warp streams the range into a ring of stages: per step the 16 KiB tile, its scales and zero points (three bulk copies) and
//     the step's activations (two TMA boxes of 16 rows x 64 k, 128-byte swizzle, rows beyond M read as zero);
//   * sixteen warps dequantise, eight of them (32 columns each) per step in turn: nibble pairs become bf16x2 with one LOP3 (0x4300 | q is the
//     bf16 128+q), minus (128+z), times s - bit-identical to the oracle because (q-z)*s is rounded once - and every word IS the 16 x 16
//     fragment that tcgen05.st.16x128b puts into tensor memory, where the weights are the 128-row A operand;
//   * two warps, one per half of the band's columns, issue tcgen05.mma 128 x 16 x 16, the activations being the B operand in shared memory as TMA
//     delivers them.  The accumulator is y transposed (lane = column of y).  Four accumulators, by k step modulo four, keep the sums as short as
//     they were on mma.sync (two warps with two accumulators each);
//   * four warps empty the accumulators: a band that lies wholly inside a range is stored directly; a band shared by several CTAs is finished by
//     whichever CTA arrives last (per-band arrival counter, partial pieces in scratch, added in k order: deterministic, repeated calls agree bit
//     for bit); no CTA ever waits for another.  The loading warp counts a range's leading partial band in meanwhile.
// What bounds the loop is instructions: a step takes about 940 cycles, of which its 2975 warp instructions need 744 to issue (1920 are the dequantisation, 15 per packed
// word, on two pipes that take one per two cycles: 512 cycles of theirs at the least), then HBM (710).  Everything else was taken off the dequantising warps' schedulers: with mma.sync the
// products and the activation fragments were theirs as well.  Two problems of M = 1, N = 11008, K = 4096: 18.6 us with mma.sync, 16.8 so; four of M = 16,
// N = 14336: 53.3 and 35.9.  On the way there: one issuing warp, its instructions behind a branch and not predicated, a division per step in
// the producer, waits between the arithmetic and its stores: 38.3 at M = 16.  Tried and taken back: three groups of eight dequantising warps (35.8),
// a warp that prepares scales and zero points for them (35.9), barriers tested a step ahead (36.7).
// Every barrier wait is bounded; a wait that runs out raises the CTA's abort flag, the roles unwind, the status word is
// written and the host reports T0_ERR_TIMEOUT.
#include "w4a16_common.cuh"

using namespace t0;
using namespace t0::w4;

namespace {

constexpr int kStDqWarps = 16;                        // dequantising warps: eight to a step in turn, each with 32 columns of the band
constexpr int kStEpWarps = 4;                         // empty the accumulators (one per tensor-memory lane quadrant)
constexpr int kStProducerWarp = 0, kStIssueWarp0 = 1; // two warps issue the UMMAs, one per 128-column half of the band
constexpr int kStEpWarp0 = 3, kStDqWarp0 = kStEpWarp0 + kStEpWarps;      // (a warp more, even an idle one, adds 0.3 us to a launch)
constexpr int kStThreads = (kStDqWarp0 + kStDqWarps) * 32;
constexpr int kStMRows = 16;                          // rows of the activations the UMMAs take
constexpr int kStSzOff = kWeightBytes;                // in a stage: the tile, scales and zero points, activations
constexpr int kStXOff = kWeightBytes + 1024;
constexpr int kStXChunk = kStMRows * 128;             // 64 k of the activations
constexpr int kStStageBytes = kStXOff + 2 * kStXChunk;
constexpr int kStStages = 10;
constexpr int kStTxBytes = kWeightBytes + kScaleBytes + kZeroBytes + 2 * kStXChunk;
// Tensor memory (512 columns): the accumulators [half of the band][k step % 4] x 16, then three A stages, a step each: [half][k step] x 8 columns.
constexpr uint32_t kStTmemCols = 512;
constexpr uint32_t kStAccCols = 128;
constexpr uint32_t kStAStages = 3;
constexpr uint32_t kStAStageCols = 128;
constexpr uint32_t kStBars = 2 * kStStages + 4 * kStAStages + 5;
constexpr size_t kStSmem = 1024 + (size_t)kStStages * kStStageBytes + kStBars * 8;      // (more than half an SM's: two CTAs must never share its tensor memory)

struct StProblem {
    float* y;                  // [M][N] f32
    const uint8_t* tiles;      // [band][kstep][16][256] u32
    const uint8_t* scales_t;   // [band][K/G][256] bf16
    const uint8_t* zeros_t;    // [band][K/G][32] u32
    uint32_t M, N;
    uint32_t ksteps, units_per_group, n_bands;
    uint32_t band_begin;       // first arrival counter of this problem
    UmDiv by_ksteps, by_group; // ksteps, units_per_group
};

template <uint32_t kProblems>
struct StParams {
    float* partials;           // [grid][2][16*256]
    int* counters;             // one per band of the launch, zero between launches
    int* status;               // error word of the runtime (bounded waits)
    unsigned long long* stamps;   // optional trace: 4 nanosecond stamps per CTA (entry, first step landed, loop done, exit)
    uint64_t wait_limit_ns;
    uint32_t per_cta, rest;    // the launch's units = grid * per_cta + rest
    float cta_per_unit;        // grid / units
    UmDiv by_grid;
    uint32_t unit_begin[kProblems];   // first unit of a problem in the launch's list; beyond the last problem 2^32 - 1
    StProblem prob[kProblems];
    CUtensorMap x[kProblems];  // activations, boxes of 16 rows x 64 k (last: what every launch reads first lies together)
};
constexpr uint32_t kStMaxProblems = 32;               // problems per launch (the table travels as a kernel parameter) ...
constexpr uint32_t kStFewProblems = 8;                // ... or as a parameter of a fourth of the size: 0.4 us less on the host (5 x 512 x 512: 5.2 us of host time a launch, 4.85)

// First unit of a CTA's range, floor(cta * total / grid), and the CTA whose range holds a unit: without the 64-bit divisions, which take hundreds of cycles
// where a band is finished.
template <class Params>
__device__ __forceinline__ uint32_t st_begin(const Params& P, uint32_t cta) { return cta * P.per_cta + um_div(cta * P.rest, P.by_grid); }
template <class Params>
__device__ __forceinline__ uint32_t st_owner(const Params& P, uint32_t unit) {
    uint32_t c = (uint32_t)((float)unit * P.cta_per_unit);     // off by a CTA at most
    if (st_begin(P, c) > unit) --c;
    if (c + 1 < gridDim.x && st_begin(P, c + 1) <= unit) ++c;
    return c;
}

struct Cursor { uint32_t p, band, ks; };

// By a converged warp, of which each lane looks at a problem.  (Walking the list problem by problem, three times a launch, missed the constant cache at each:
// 32 of 1024 x 1024 at M = 1 15.1 us, 11.5 so.)
template <uint32_t kProblems>
__device__ __forceinline__ Cursor locate(const StParams<kProblems>& P, uint32_t unit) {
    static_assert(kProblems <= 32, "a lane looks at a problem");
    Cursor c;
    c.p = __popc(__ballot_sync(0xFFFFFFFFu, P.unit_begin[min(threadIdx.x & 31, kProblems - 1)] <= unit && (threadIdx.x & 31) < kProblems)) - 1;
    const uint32_t r = unit - P.unit_begin[c.p];
    c.band = um_div(r, P.prob[c.p].by_ksteps);
    c.ks = r - c.band * P.prob[c.p].ksteps;
    return c;
}

constexpr uint32_t kStFinishers = kStDqWarps * 32;    // threads that finish a cut band ...
constexpr uint32_t kStInFlight = 8;                   // ... each with so many 16-byte loads of contributors' pieces under way together

// barriers 1: the epilogue warps, 2: these and the dequantising warps, 3: the dequantising warps
__device__ __forceinline__ void st_epilogue_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kStEpWarps * 32) : "memory"); }
__device__ __forceinline__ void st_tail_sync() { asm volatile("bar.sync 2, %0;" ::"n"((kStDqWarps + kStEpWarps) * 32) : "memory"); }
__device__ __forceinline__ void st_finishers_sync() { asm volatile("bar.sync 3, %0;" ::"n"(kStFinishers) : "memory"); }
// explicit shared-space accesses: the ring's address went through an integer for alignment, so plain pointers would make
// the compiler use generic loads and 64-bit address arithmetic
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}

__device__ __forceinline__ void sts128(uint32_t addr, const uint4& v) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// Item i of a band's outputs: four columns of a row.
__device__ __forceinline__ void st_store4(const StProblem& pr, uint32_t band, uint32_t i, const float4& v) {
    const uint32_t row = i / (kBandCols / 4), col = band * kBandCols + (i % (kBandCols / 4)) * 4;
    const float o[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j)
        if (col + j < pr.N) pr.y[(size_t)row * pr.N + col + j] = o[j];
}

// The CTAs that share a cut band.  Only the first can hold the band in slot 1 of its two pieces (its range began in the band before).
struct StShare { uint32_t first, last, first_slot; };
template <class Params>
__device__ __forceinline__ StShare st_share(const Params& P, uint32_t first_unit, uint32_t ksteps) {
    StShare h;
    h.first = st_owner(P, first_unit);
    h.last = st_owner(P, first_unit + ksteps - 1);
    h.first_slot = st_begin(P, h.first) < first_unit ? 1u : 0u;
    return h;
}
template <class Params>
__device__ __forceinline__ const float* st_piece(const Params& P, const StShare& h, uint32_t cta) {
    return P.partials + ((size_t)cta * 2 + (cta == h.first ? h.first_slot : 0u)) * kPieceFloats;
}

// The CTA that contributes last to a band adds the pieces and stores; nobody waits for anybody.  By its dequantising warps: a thread has four columns of a row,
// and where that leaves threads over, up to eight of them make a sum, which add parts of the list of contributors and then, through shared memory, each
// other's: always in the same order, whoever does it.  (A band of N = 1024, K = 4096 has 32 contributors, whose pieces one thread fetches in eight round trips
// of 0.7 us.)  The shares are worked out before it is known who finishes, since a division takes longer than such a warp has then.
struct StFinish {
    StShare h;
    uint32_t p, band, items, groups, g, i, begin, end;
};
template <class Params>
__device__ __forceinline__ StFinish st_finish(const Params& P, uint32_t p, uint32_t band, uint32_t t) {
    StFinish f;
    const StProblem& pr = P.prob[p];
    f.h = st_share(P, P.unit_begin[p] + band * pr.ksteps, pr.ksteps);
    f.p = p; f.band = band;
    f.items = pr.M * (kBandCols / 4);
    const uint32_t count = f.h.last - f.h.first + 1;
    f.groups = max(1u, min(min(8u, kStFinishers / f.items), (count + kStInFlight - 1) / kStInFlight));
    f.g = f.groups > 1 ? t / f.items : 0;
    f.i = t - f.g * f.items;
    const uint32_t per = (count + f.groups - 1) / f.groups;
    f.begin = f.h.first + f.g * per;
    f.end = f.g < f.groups ? min(f.begin + per, f.h.last + 1) : 0;
    return f;
}
// The sums of kItems items of a thread over its contributors, in CTA order, one contributor after the other.
template <uint32_t kItems, class Params>
__device__ __forceinline__ void st_add_pieces(const Params& P, const StFinish& f, float4 (&sum)[kItems]) {
    constexpr uint32_t kCo = kStInFlight / kItems;
    const float4* piece = (const float4*)st_piece(P, f.h, f.begin);
#pragma unroll
    for (uint32_t j = 0; j < kItems; ++j) sum[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t c = f.begin; c < f.end; c += kCo) {
        float4 v[kCo][kItems];
#pragma unroll
        for (uint32_t b = 0; b < kCo; ++b) {
            const float4* src = (c + b == f.begin ? piece : (const float4*)(P.partials + (size_t)(c + b) * 2 * kPieceFloats)) + f.i;
#pragma unroll
            for (uint32_t j = 0; j < kItems; ++j) {
                v[b][j] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (c + b < f.end && f.i + j * kStFinishers < f.items) v[b][j] = __ldcg(src + j * kStFinishers);
            }
        }
#pragma unroll
        for (uint32_t b = 0; b < kCo; ++b)
#pragma unroll
            for (uint32_t j = 0; j < kItems; ++j) {
                sum[j].x += v[b][j].x; sum[j].y += v[b][j].y; sum[j].z += v[b][j].z; sum[j].w += v[b][j].w;
            }
    }
}
template <class Params>
__device__ __forceinline__ void st_reduce_band(const Params& P, const StFinish& f, uint32_t t, uint32_t exchange) {
    const StProblem& pr = P.prob[f.p];
    if (f.items > kStFinishers) {                     // M > 8: two items a thread (16 * 64 at most)
        float4 sum[2];
        st_add_pieces<2>(P, f, sum);
        st_store4(pr, f.band, f.i, sum[0]);
        if (f.i + kStFinishers < f.items) st_store4(pr, f.band, f.i + kStFinishers, sum[1]);
    } else {
        float4 sum[1];
        if (f.g < f.groups && f.i < f.items) {
            st_add_pieces<1>(P, f, sum);
            if (f.groups == 1) st_store4(pr, f.band, f.i, sum[0]);
            else sts128(exchange + (f.g * f.items + f.i) * 16, make_uint4(__float_as_uint(sum[0].x), __float_as_uint(sum[0].y), __float_as_uint(sum[0].z), __float_as_uint(sum[0].w)));
        }
        if (f.groups > 1) {
            st_finishers_sync();
            if (t < f.items) {
                sum[0] = make_float4(0.f, 0.f, 0.f, 0.f);
                for (uint32_t j = 0; j < f.groups; ++j) {
                    const uint4 v = lds128(exchange + (j * f.items + t) * 16);
                    sum[0].x += __uint_as_float(v.x); sum[0].y += __uint_as_float(v.y); sum[0].z += __uint_as_float(v.z); sum[0].w += __uint_as_float(v.w);
                }
                st_store4(pr, f.band, t, sum[0]);
            }
            st_finishers_sync();                      // (the exchange is free again)
        }
    }
    if (t == 0) P.counters[pr.band_begin + f.band] = 0;   // ready for the next launch
}

template <uint32_t kProblems>
__global__ void __launch_bounds__(kStThreads, 1)
w4a16_stream_kernel(const __grid_constant__ StParams<kProblems> P) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t ring = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t full_bar = ring + kStStages * kStStageBytes;          // the stage's bytes have landed
    const uint32_t empty_bar = full_bar + kStStages * 8;                 // read by eight dequantising warps and the UMMAs
    const uint32_t a_full = empty_bar + kStStages * 8;                   // A stages, [half][stage]: four warps have written their step
    const uint32_t a_empty = a_full + 2 * kStAStages * 8;
    const uint32_t acc_full = a_empty + 2 * kStAStages * 8;              // accumulators
    const uint32_t acc_empty = acc_full + 8;
    const uint32_t head_written = acc_empty + 8;                         // the epilogue warps have stored the head piece
    const uint32_t head_counted = head_written + 8;                      // it is counted in and s_head_last is valid
    const uint32_t end_near = head_counted + 8;                          // one step of the range is left to dequantise
    __shared__ uint32_t tmem_holder;
    __shared__ int s_abort, s_last, s_all, s_head_last, s_head_go;
    volatile int* abort_flag = &s_abort;

    const uint32_t tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;     // (the shuffle tells the compiler that a role is the whole warp's)
    const uint32_t U0 = st_begin(P, blockIdx.x);
    const uint32_t U1 = st_begin(P, blockIdx.x + 1);
    auto stamp = [&](int i) {
        if (P.stamps) P.stamps[blockIdx.x * 4 + i] = ptx::globaltimer_ns();
    };
    if (tid == 0) {
        for (int s = 0; s < kStStages; ++s) {
            ptx::mbar_init(full_bar + s * 8, 1);
            ptx::mbar_init(empty_bar + s * 8, kStDqWarps / 2);
        }
        for (uint32_t s = 0; s < 2 * kStAStages; ++s) {
            ptx::mbar_init(a_full + s * 8, kStDqWarps / 4);
            ptx::mbar_init(a_empty + s * 8, 1);
        }
        ptx::mbar_init(acc_full, 2);
        ptx::mbar_init(acc_empty, kStEpWarps);
        ptx::mbar_init(head_written, kStEpWarps);
        ptx::mbar_init(head_counted, 1);
        ptx::mbar_init(end_near, 1);
        s_abort = 0;
        s_last = s_all = s_head_last = 0;
        ptx::fence_barrier_init();
        ptx::fence_proxy_async_smem();
    }
    if (warp == kStIssueWarp0) {
        ptx::tmem_alloc(ptx::smem_u32(&tmem_holder), kStTmemCols);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    ptx::tc_fence_after_sync();
    constexpr uint32_t tmem_base = 0;    // all columns are allocated: tensor-memory addresses are constants
    ptx::grid_launch_dependents();
    Cursor c = locate(P, U0);
    if (warp == kStProducerWarp && lane == 0) ptx::tma_prefetch_desc(&P.x[c.p]);
    ptx::grid_dependency_wait();      // global memory is read and written only after the previous grid in the stream is done
    if (tid == 0) stamp(0);
    // What is cut at the ends of the range.  Worked out where it is needed, after a warp's loop (the empty statement keeps it there: it would take registers
    // that the loops have none of).
    struct Ends {
        Cursor first, last;
        uint32_t head_first, head_ksteps;   // first unit and steps of the first band
        bool has_head;           // A head piece: the range starts inside a band and goes on into the next one.  Counting it in (fence, atomic round trip) is the loading
                                 // warp's job, so that the epilogue warps are there for the last piece, which may come soon.
        bool tail_cut;           // the last piece (the steps of one band this CTA owns) goes on in the next CTA, or began in the one before
    };
    auto range_ends = [&]() {
        uint32_t lo = U0, hi = U1;
        asm volatile("" : "+r"(lo), "+r"(hi));
        __syncwarp();
        Ends e;
        e.first = locate(P, lo);
        e.last = locate(P, hi - 1);
        e.head_first = lo - e.first.ks;
        e.head_ksteps = P.prob[e.first.p].ksteps;
        e.has_head = e.first.ks != 0 && e.head_first + e.head_ksteps < hi;
        const uint32_t end_first = P.unit_begin[e.last.p] + e.last.band * P.prob[e.last.p].ksteps;
        e.tail_cut = end_first < lo || end_first + P.prob[e.last.p].ksteps > hi;
        return e;
    };
    // The serial roles walk with their whole warp and let one elected lane issue: see ptx::mbar_wait_warp.
    if (warp == kStProducerWarp) {
        // (A problem's tiles lie one behind the other in the order of its units, its rows of scales and zero points likewise: running addresses.  The chain of
        // this warp is kept short: with a division per step it took 800 cycles a step from the four dequantising warps it shares a scheduler with.)
        // It counts the head piece in as soon as that is written: the ring holds several steps, which the fence and the atomic's round trip do not take.
        const uint32_t head_left = P.prob[c.p].ksteps - c.ks, first_p = c.p, first_band = c.band;
        bool head_pending = c.ks != 0 && head_left < U1 - U0;
        auto count_head = [&]() {
            if (lane == 0) {
                const StShare h = st_share(P, U0 + head_left - P.prob[first_p].ksteps, P.prob[first_p].ksteps);
                __threadfence();                       // the piece is visible before this CTA is counted
                const int last = atomicAdd(&P.counters[P.prob[first_p].band_begin + first_band], 1) == (int)(h.last - h.first);
                if (last) __threadfence();
                s_head_last = last;
            }
        };
        uint32_t stage = 0, phase = 0;
        for (uint32_t u = U0; u < U1; ++c.p) {
            const StProblem& pr = P.prob[c.p];
            const uint32_t begin = P.unit_begin[c.p], at = u - begin, row = um_div(at, pr.by_group), u_stop = min(U1, begin + pr.ksteps * pr.n_bands);
            const uint8_t* tile = pr.tiles + (size_t)at * kWeightBytes;
            const uint8_t* scales = pr.scales_t + (size_t)row * kScaleBytes;
            const uint8_t* zeros = pr.zeros_t + (size_t)row * kZeroBytes;
            uint32_t in_row = at - row * pr.units_per_group, k = (at - um_div(at, pr.by_ksteps) * pr.ksteps) * kUnitK;
            if (u_stop < U1 && lane == 0) ptx::tma_prefetch_desc(&P.x[c.p + 1]);
            bool ok = true;
            for (; u < u_stop; ++u) {
                ok = ptx::mbar_wait_warp(empty_bar + stage * 8, phase ^ 1, abort_flag, P.wait_limit_ns);
                if (!ok) break;
                const uint32_t dst = ring + stage * kStStageBytes, fb = full_bar + stage * 8;
                if (ptx::elect_one()) {
                    ptx::fence_proxy_async_smem();       // the stage was read through the generic proxy, the copies write it through the async proxy
                    ptx::mbar_arrive_expect_tx(fb, kStTxBytes);
                    ptx::bulk_load(dst, tile, kWeightBytes, fb);
                    ptx::bulk_load(dst + kStSzOff, scales, kScaleBytes, fb);
                    ptx::bulk_load(dst + kStSzOff + kScaleBytes, zeros, kZeroBytes, fb);
                    ptx::tma_load_3d(dst + kStXOff, &P.x[c.p], fb, (int32_t)k, 0, 0);
                    ptx::tma_load_3d(dst + kStXOff + kStXChunk, &P.x[c.p], fb, (int32_t)k + 64, 0, 0);
                }
                __syncwarp();
                if (head_pending && ptx::mbar_test_warp(head_written, 0)) {
                    count_head();
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive(head_counted);
                    head_pending = false;
                }
                if (++stage == kStStages) { stage = 0; phase ^= 1; }
                tile += kWeightBytes;
                if (++in_row == pr.units_per_group) { in_row = 0; scales += kScaleBytes; zeros += kZeroBytes; }
                k += kUnitK;
                if (k == pr.ksteps * kUnitK) k = 0;
            }
            if (!ok) {
                if (lane == 0) atomicCAS(P.status, 0, kStatusProducerTimeout | (int)(u & 0xFFFFFF));
                break;
            }
        }
        if (head_pending) {
            if (ptx::mbar_wait_warp(head_written, 0, abort_flag, P.wait_limit_ns)) count_head(); else if (lane == 0) atomicCAS(P.status, 0, kStatusEpilogueTimeout | 0xD00000);
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(head_counted);       // (counted or not: nobody waits for what does not come)
        }
    } else if (warp < kStEpWarp0) {
        // -------------------------------------------------------------- UMMA issuers: per 64 k four k steps of M 128 x N 16 x K 16
        constexpr uint32_t idesc = ptx::make_idesc_bf16_f32(128, kStMRows, 0u);
        const uint32_t t = warp - kStIssueWarp0;
        const uint32_t my_full = a_full + t * kStAStages * 8, my_empty = a_empty + t * kStAStages * 8;
        const uint32_t x0 = ((ring + kStXOff) & 0x3FFFFu) >> 4;      // addresses enter a descriptor in 16-byte units
        uint32_t x = x0, aphase = 0, piece = 0, as = 0;
        const uint32_t acc = t * 64;
        bool ok = true;
        for (uint32_t u = U0; ok && u < U1; ++piece) {
            const uint32_t u_end = min(U1, u + P.prob[c.p].ksteps - c.ks);
            if (piece > 0 && !ptx::mbar_wait_warp(acc_empty, (piece & 1) ^ 1, abort_flag, P.wait_limit_ns)) {
                if (lane == 0) atomicCAS(P.status, 0, kStatusMmaTimeout | 0x800000);
                break;
            }
            for (uint32_t first = 1; u < u_end; ++u, first = 0) {
                // (what the dequantising warps waited for before they signal includes the activations of the step)
                if (!ptx::mbar_wait_warp(my_full + as * 8, aphase, abort_flag, P.wait_limit_ns)) {
                    if (lane == 0) atomicCAS(P.status, 0, kStatusMmaTimeout | (int)(u & 0x7FFFFF));
                    ok = false;
                    break;
                }
                ptx::tc_fence_after_sync();
                const uint32_t issue = ptx::elect_one(), a_cols = kStAccCols + t * 64 + as * kStAStageCols;
                if (first) {
#pragma unroll
                    for (uint32_t k4 = 0; k4 < 4; ++k4) ptx::umma_bf16_ts_if<false>(issue, acc + k4 * kStMRows, a_cols + k4 * 8, x + k4 * 2, idesc);
                } else {
#pragma unroll
                    for (uint32_t k4 = 0; k4 < 4; ++k4) ptx::umma_bf16_ts_if<true>(issue, acc + k4 * kStMRows, a_cols + k4 * 8, x + k4 * 2, idesc);
                }
#pragma unroll
                for (uint32_t k4 = 0; k4 < 4; ++k4) ptx::umma_bf16_ts_if<true>(issue, acc + k4 * kStMRows, a_cols + 32 + k4 * 8, x + kStXChunk / 16 + k4 * 2, idesc);
                ptx::umma_commit_if(issue, my_empty + as * 8);
                __syncwarp();
                if (++as == kStAStages) { as = 0; aphase ^= 1; }
                x = x == x0 + (kStStages - 1) * (kStStageBytes / 16) ? x0 : x + kStStageBytes / 16;
            }
            if (!ok) break;
            if (ptx::elect_one()) ptx::umma_commit(acc_full);
            __syncwarp();
            c.ks = 0;
            if (++c.band == P.prob[c.p].n_bands) { c.band = 0; ++c.p; }
        }
    } else if (warp >= kStDqWarp0) {
        // -------------------------------------------------------------- sixteen warps: dequantise into tensor memory
        const uint32_t set = (warp - kStDqWarp0) >> 3, g = lane >> 2;              // every second step; a lane has columns g + 8 i of the warp's 32
        const uint32_t pair = ((warp - kStDqWarp0) & 4) | (warp & 3);            // columns 32 pair .. + 31, those of its tensor-memory lane quadrant
        const uint32_t a_lane = (((pair & 3) * 32) << 16) + kStAccCols + (pair >> 2) * 64;
        const uint32_t my_full = a_full + (pair >> 2) * kStAStages * 8, my_empty = a_empty + (pair >> 2) * kStAStages * 8;
        uint32_t mask, magic;
        asm volatile("mov.b32 %0, 0x000F000F;" : "=r"(mask));
        asm volatile("mov.b32 %0, 0x43004300;" : "=r"(magic));
        uint32_t stage = set, phase = 0, as = set, aphase = 0;
        const uint32_t lane_w = ring + pair * 2048 + lane * 16;              // [16 column groups][2 k halves][32 lanes] uint4
        const uint32_t lane_s = ring + kStSzOff + (pair * 32 + g) * 2;
        const uint32_t lane_z = ring + kStSzOff + kScaleBytes + pair * 16;
        for (uint32_t u = U0 + set; u < U1; u += 2) {
            if (!ptx::mbar_wait(full_bar + stage * 8, phase, abort_flag, P.wait_limit_ns)) {
                if (lane == 0) atomicCAS(P.status, 0, kStatusEpilogueTimeout | (int)(u & 0x3FFFFF));
                break;
            }
            if (tid == kStDqWarp0 * 32 && u == U0) stamp(1);
            const uint32_t off = stage * kStStageBytes;
            uint4 q[2][2];                            // [k half][column group]
#pragma unroll
            for (int kh = 0; kh < 2; ++kh)
#pragma unroll
                for (int cg = 0; cg < 2; ++cg) q[kh][cg] = lds128(lane_w + off + cg * 1024 + kh * 512);
            const uint4 z4 = lds128(lane_z + off);
            uint32_t zz[4], ss[4];                    // columns g + 8 i: bf16x2 (128+z, 128+z) and (s, s)
#pragma unroll
            for (int i = 0; i < 4; ++i) ss[i] = um_lds16(lane_s + off + i * 16);
            // The A stage is free once the UMMAs of three steps ago have read it.  (Waited for here and not before the stores: values that live across
            // a wait are moved once more to where the store takes them, 64 moves a step.)
            if (!ptx::mbar_wait(my_empty + as * 8, aphase ^ 1, abort_flag, P.wait_limit_ns)) {
                if (lane == 0) atomicCAS(P.status, 0, kStatusEpilogueTimeout | 0x800000 | (int)(u & 0x3FFFFF));
                break;
            }
            ptx::tc_fence_after_sync();
            // So the step of three ago is done with its ring stage: dequantised, and its activations read.
            ptx::mbar_arrive_if(empty_bar + (stage < 3 ? stage + kStStages - 3 : stage - 3) * 8, lane == 0 && u >= U0 + 3);
            {
                const uint32_t z[4] = {z4.x, z4.y, z4.z, z4.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    zz[i] = ((z[i] >> (4 * g)) & 0xFu) * 0x00010001u + 0x43004300u;
                    ss[i] *= 0x00010001u;
                }
            }
            const uint32_t dst = a_lane + as * kStAStageCols;
#pragma unroll
            for (int kh = 0; kh < 2; ++kh) {
#pragma unroll
                for (int cg = 0; cg < 2; ++cg) {
                    const uint32_t w[4] = {q[kh][cg].x, q[kh][cg].y, q[kh][cg].z, q[kh][cg].w};
                    uint32_t r[16];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {     // one word per k step: fragment registers (columns g, g + 8) x (k 2t, 2t + 8)
                        r[4 * e + 0] = bf16x2_mul(bf16x2_sub(and_or(w[e], mask, magic), zz[2 * cg]), ss[2 * cg]);
                        r[4 * e + 1] = bf16x2_mul(bf16x2_sub(and_or(w[e] >> 4, mask, magic), zz[2 * cg + 1]), ss[2 * cg + 1]);
                        r[4 * e + 2] = bf16x2_mul(bf16x2_sub(and_or(w[e] >> 8, mask, magic), zz[2 * cg]), ss[2 * cg]);
                        r[4 * e + 3] = bf16x2_mul(bf16x2_sub(and_or(w[e] >> 12, mask, magic), zz[2 * cg + 1]), ss[2 * cg + 1]);
                    }
                    ptx::tmem_st_16x128b_x8(dst + kh * 32 + ((cg * 16u) << 16), r);
                }
            }
            ptx::tmem_st_wait();
            ptx::tc_fence_before_sync();
            __syncwarp();
            ptx::mbar_arrive_if(my_full + as * 8, lane == 0);
            as += 2;
            if (as >= kStAStages) { as -= kStAStages; aphase ^= 1; }
            stage += 2;
            if (stage >= kStStages) { stage -= kStStages; phase ^= 1; }
        }
        // The set that does not have the last step is through first, one step before the end.
        ptx::mbar_arrive_if(end_near, tid == (kStDqWarp0 + ((U1 - U0) & 1) * 8) * 32);
        if (tid == kStDqWarp0 * 32) stamp(2);
        // Finish the bands of the last and the first piece, where this CTA turned out to be the last to contribute to them.  (The last step is done with by
        // then, so the ring is free.)
        const uint32_t ft = tid - kStDqWarp0 * 32;
        const Ends e = range_ends();
        if (e.tail_cut) {
            const StFinish f = st_finish(P, e.last.p, e.last.band, ft);
            st_tail_sync();
            if (s_last) st_reduce_band(P, f, ft, ring);
        }
        if (e.has_head) {
            const StFinish f = st_finish(P, e.first.p, e.first.band, ft);
            if (ft == 0) s_head_go = ptx::mbar_wait(head_counted, 0, abort_flag, P.wait_limit_ns) && s_head_last;
            if (e.tail_cut) st_finishers_sync();
            else st_tail_sync();
            if (s_head_go) st_reduce_band(P, f, ft, ring);
        }
    } else {
        // -------------------------------------------------------------- four warps: accumulators to y, or to a piece
        const uint32_t quad = warp & 3, et = tid - kStEpWarp0 * 32;
        bool ok = true;
        uint32_t piece = 0;
        for (uint32_t u = U0; u < U1; ++piece) {
            const StProblem& pr = P.prob[c.p];
            const uint32_t first_unit = P.unit_begin[c.p] + c.band * pr.ksteps, last_unit = first_unit + pr.ksteps;   // [first, last)
            const bool whole = first_unit >= U0 && last_unit <= U1, tail = last_unit >= U1;
            const StShare h = st_share(P, first_unit, pr.ksteps);
            int* const counter = P.counters + pr.band_begin + c.band;
            float* const part = P.partials + ((size_t)blockIdx.x * 2 + (first_unit <= U0 ? 0u : 1u)) * kPieceFloats;   // slot 0: the piece with this CTA's first unit
            // The last piece is on the way of everything behind the launch.  Where its band has one more part, that lies as a rule in a range that began with it,
            // and is long there: looked for as the last step is dequantised, it is fetched and added to the accumulators at once, with no hand-in, fence and atomic.
            // (On a barrier that completes once.  These warps follow none of the ring's barriers, whose parity an earlier phase answers as well.)
            bool rest_there = false;
            float other[2][16];
            if (!whole && tail && h.last - h.first == 1) {      // (barriers are met whether or not a wait has run out)
                const uint32_t cta = h.first == blockIdx.x ? h.last : h.first;
                ok = ok && ptx::mbar_wait(end_near, 0, abort_flag, P.wait_limit_ns);
                if (et == 0) s_all = ok && um_ld_acquire((const uint32_t*)counter) != 0;
                st_epilogue_sync();
                rest_there = s_all != 0;
                if (rest_there) {
#pragma unroll
                    for (uint32_t t = 0; t < 2; ++t)
#pragma unroll
                        for (uint32_t m = 0; m < 16; ++m) other[t][m] = m < pr.M ? __ldcg(st_piece(P, h, cta) + m * kBandCols + t * 128 + quad * 32 + lane) : 0.0f;
                }
            }
            if (ok && !ptx::mbar_wait(acc_full, piece & 1, abort_flag, P.wait_limit_ns)) {
                if (lane == 0) atomicCAS(P.status, 0, kStatusEpilogueTimeout | 0xC00000);
                ok = false;
            }
            if (ok) {
                ptx::tc_fence_after_sync();
#pragma unroll
                for (uint32_t t = 0; t < 2; ++t) {
                    const uint32_t col = t * 128 + quad * 32 + lane, n = c.band * kBandCols + col;
#pragma unroll
                    for (uint32_t m0 = 0; m0 < 16; m0 += 8) {
                        if (m0 >= pr.M) break;
                        uint32_t d[4][8];
                        float v[8];
#pragma unroll
                        for (uint32_t k4 = 0; k4 < 4; ++k4) ptx::tmem_ld_32x32b_x8(tmem_base + ((quad * 32) << 16) + t * 64 + k4 * kStMRows + m0, d[k4]);
                        ptx::tmem_ld_wait();
#pragma unroll
                        for (uint32_t j = 0; j < 8; ++j)
                            v[j] = (__uint_as_float(d[0][j]) + __uint_as_float(d[1][j])) + (__uint_as_float(d[2][j]) + __uint_as_float(d[3][j]));
                        if (whole || rest_there) {
                            // (of two parts the order does not matter; the zero gives a sum of negative zeros the sign it has where the pieces are added)
                            if (rest_there) {
#pragma unroll
                                for (uint32_t j = 0; j < 8; ++j) v[j] = (0.0f + v[j]) + other[t][m0 + j];
                            }
                            if (n < pr.N) {
#pragma unroll
                                for (uint32_t j = 0; j < 8; ++j)
                                    if (m0 + j < pr.M) pr.y[(size_t)(m0 + j) * pr.N + n] = v[j];
                            }
                        } else {
#pragma unroll
                            for (uint32_t j = 0; j < 8; ++j)
                                if (m0 + j < pr.M) part[(m0 + j) * kBandCols + col] = v[j];
                        }
                    }
                }
                ptx::tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(acc_empty);
            }
            if (!whole && !tail) {
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(head_written);
            } else if (!whole) {
                st_epilogue_sync();                    // every thread's part of the piece is written ...
                if (et == 0) {
                    int last = 0;
                    if (rest_there) {
                        *counter = 0;                  // ready for the next launch
                    } else if (ok) {
                        __threadfence();               // ... and made visible before this CTA is counted
                        last = atomicAdd(counter, 1) == (int)(h.last - h.first);
                        if (last) __threadfence();
                    }
                    s_last = last;
                }
            }
            u = min(U1, last_unit);
            c.ks = 0;
            if (++c.band == pr.n_bands) { c.band = 0; ++c.p; }
        }
        const Ends e = range_ends();
        if (e.tail_cut || e.has_head) st_tail_sync();
    }

    __syncwarp();
    if (*abort_flag) {
        // give copies and UMMAs already in flight time to land before shared and tensor memory go away
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    if (warp == kStIssueWarp0) {
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc(tmem_base, kStTmemCols);
    }
    if (tid == 0) stamp(3);
}

// ------------------------------------------------------------------ streaming (tile-major) weight layout

struct PrepackLayout { size_t off_tiles, off_scales, off_zeros, total; uint32_t bands, ksteps, groups; };

PrepackLayout prepack_layout(uint32_t K, uint32_t N, uint32_t group) {
    PrepackLayout L;
    L.bands = ceil_div(N, kBandCols); L.ksteps = K / kUnitK; L.groups = K / group;
    L.off_tiles = 0;
    L.off_scales = (size_t)L.bands * L.ksteps * kWeightBytes;
    L.off_zeros = L.off_scales + (size_t)L.bands * L.groups * kScaleBytes;
    L.total = L.off_zeros + (size_t)L.bands * L.groups * kZeroBytes;
    return L;
}

// Row layout -> streaming layout.  One thread per four tile words (the four words that draw on the same four source words),
// per scale, or per word of eight zero points.  Columns past N are written as zero.
__global__ void w4_prepack_kernel(const uint32_t* __restrict__ packed, const uint16_t* __restrict__ scales, const uint32_t* __restrict__ zeros,
                                  uint8_t* __restrict__ out, uint32_t K, uint32_t N, uint32_t nz, PrepackLayout L) {
    const uint64_t n_words = (uint64_t)L.bands * L.ksteps * 16 * kBandCols / 4;      // units of four words
    const uint64_t n_scales = (uint64_t)L.bands * L.groups * kBandCols;
    const uint64_t n_zwords = (uint64_t)L.bands * L.groups * (kBandCols / 8);
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_words + n_scales + n_zwords; i += stride) {
        if (i < n_words) {
            // Word (tile, w, j, lane, e) of the fragment order: k step s = 4j + e of column tile w, lane (g, t); nibble c / c+4 =
            // codes (k, k+1) of column n = 16w + g + 8(c & 1) at k = 16s + 2t + 8(c >> 1).  The four words t = 0..3 of one
            // (tile, w, j, g, e) take nibble pair t of the same four source words (two rows x two columns).
            const uint32_t e = (uint32_t)(i & 3), g = (uint32_t)((i >> 2) & 7), j = (uint32_t)((i >> 5) & 1), w = (uint32_t)((i >> 6) & 15);
            const uint64_t tile = i >> 10;
            const uint32_t ks = (uint32_t)(tile % L.ksteps), band = (uint32_t)(tile / L.ksteps);
            const uint32_t sstep = 4 * j + e;
            const uint32_t n0 = band * kBandCols + w * 16 + g, n1 = n0 + 8;
            const size_t r0 = (size_t)(ks * (kUnitK / 8) + 2 * sstep) * N;
            uint32_t src[4];
            src[0] = n0 < N ? __ldg(packed + r0 + n0) : 0u;
            src[1] = n1 < N ? __ldg(packed + r0 + n1) : 0u;
            src[2] = n0 < N ? __ldg(packed + r0 + N + n0) : 0u;
            src[3] = n1 < N ? __ldg(packed + r0 + N + n1) : 0u;
            uint32_t* dst = (uint32_t*)(out + L.off_tiles) + ((tile << 12) | ((uint64_t)w << 8) | ((uint64_t)j << 7) | ((uint64_t)g << 4) | e);
#pragma unroll
            for (uint32_t t = 0; t < 4; ++t) {
                uint32_t v = 0;
#pragma unroll
                for (uint32_t c = 0; c < 4; ++c) {
                    const uint32_t pair = src[c] >> (8 * t);
                    v |= (pair & 0xFu) << (4 * c);
                    v |= ((pair >> 4) & 0xFu) << (4 * (c + 4));
                }
                dst[t * 4] = v;                       // lane 4g + t: sixteen bytes further on
            }
        } else if (i < n_words + n_scales) {
            const uint64_t j = i - n_words;
            const uint32_t c = (uint32_t)(j % kBandCols);
            const uint64_t row = j / kBandCols;
            const uint32_t g = (uint32_t)(row % L.groups), band = (uint32_t)(row / L.groups);
            const uint32_t n = band * kBandCols + c;
            ((uint16_t*)(out + L.off_scales))[j] = n < N ? scales[(size_t)g * N + n] : (uint16_t)0;
        } else {
            const uint64_t j = i - n_words - n_scales;
            const uint32_t wz = (uint32_t)(j % (kBandCols / 8));
            const uint64_t row = j / (kBandCols / 8);
            const uint32_t g = (uint32_t)(row % L.groups), band = (uint32_t)(row / L.groups);
            const uint32_t n0 = band * kBandCols + wz * 8;     // eight columns, aligned to a source word
            ((uint32_t*)(out + L.off_zeros))[j] = n0 < N ? zeros[(size_t)g * nz + (n0 >> 3)] : 0u;
        }
    }
}

uint32_t prepack_grid_for(uint64_t n, uint32_t block) {
    uint64_t gsz = (n + block - 1) / block;
    const uint64_t cap = 148ull * 16;
    return (uint32_t)(gsz < 1 ? 1 : (gsz > cap ? cap : gsz));
}

// One launch for up to kProblems problems (already validated).
template <uint32_t kProblems>
int launch_stream_chunk(t0_runtime* rt, const t0_w4a16_args* args, size_t count) {
    StParams<kProblems> P;                            // (up to 6.7 KB: what the kernel reads is filled in, nothing is cleared first)
    P.stamps = nullptr;
    uint64_t total = 0, bands = 0;
    PrepackLayout L = {};
    for (size_t i = 0; i < count; ++i) {
        const t0_w4a16_args& a = args[i];
        // A list is mostly of one shape: what that decides is taken from the problem before, since divisions and the encoding of a map are most of a problem's time
        // here (32 of 512 x 512: 12.6 us of host time a launch without, 11.1 so).
        const bool same_x = i > 0 && a.m == args[i - 1].m && a.k == args[i - 1].k && gemm::make_map_like(&P.x[i], P.x[i - 1], (const void*)a.a);
        int rc = same_x ? T0_OK : gemm::make_map_kmajor(&P.x[i], (const void*)a.a, a.m, a.k, a.k, 1, kStMRows);
        if (rc != T0_OK) return rc;
        if (i == 0 || a.k != args[i - 1].k || a.n != args[i - 1].n || a.group != args[i - 1].group) L = prepack_layout(a.k, a.n, a.group);
        StProblem& q = P.prob[i];
        if (i > 0 && a.k == args[i - 1].k && a.group == args[i - 1].group) {
            q = P.prob[i - 1];
        } else {
            q.ksteps = L.ksteps; q.units_per_group = a.group / kUnitK;
            q.by_ksteps = um_divisor(q.ksteps); q.by_group = um_divisor(q.units_per_group);
        }
        q.y = (float*)a.y;
        q.tiles = (const uint8_t*)a.packed + L.off_tiles;
        q.scales_t = (const uint8_t*)a.packed + L.off_scales;
        q.zeros_t = (const uint8_t*)a.packed + L.off_zeros;
        q.M = a.m; q.N = a.n; q.n_bands = L.bands;
        P.unit_begin[i] = (uint32_t)total; q.band_begin = (uint32_t)bands;
        total += (uint64_t)L.bands * L.ksteps;
        bands += L.bands;
    }
    for (size_t i = count; i < kProblems; ++i) P.unit_begin[i] = 0xFFFFFFFFu;
    if (total == 0) return T0_OK;
    if (total > 0x7FFFFFFFull || bands * sizeof(int) > kCounterRegion) return fail(T0_ERR_UNSUPPORTED, "batch too large: %llu steps, %llu bands", (unsigned long long)total, (unsigned long long)bands);
    const uint32_t grid = (uint32_t)std::min<uint64_t>(total, (uint64_t)rt->sm_count);
    const size_t need = kCounterRegion + (size_t)grid * 2 * kPieceFloats * sizeof(float);
    if (need > rt->scratch_w4.size) {
        int rc = ensure_scratch(rt, rt->scratch_w4, need);
        if (rc != T0_OK) return rc;
        T0_CUDA(cudaMemsetAsync(rt->scratch_w4.ptr, 0, kCounterRegion, rt->stream));
    }
    P.counters = (int*)rt->scratch_w4.ptr;
    P.partials = (float*)((uint8_t*)rt->scratch_w4.ptr + kCounterRegion);
    P.status = rt->d_status;
    const uint64_t limit = rt->wait_limit_ns.load(std::memory_order_relaxed);
    P.wait_limit_ns = limit ? limit : ptx::kWaitLimitNs;
    P.per_cta = (uint32_t)total / grid; P.rest = (uint32_t)total % grid; P.cta_per_unit = (float)grid / (float)total; P.by_grid = um_divisor(grid);
    static bool attr_set[64] = {};
    if (rt->device >= 64) return fail(T0_ERR_INVALID, "device ordinal out of range");
    if (!attr_set[rt->device]) {
        T0_CUDA(cudaFuncSetAttribute(w4a16_stream_kernel<kProblems>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStSmem));
        attr_set[rt->device] = true;
    }
    // T0_W4_TRACE=1: per-CTA stamps, summarised on stderr after a blocking wait (a debugging aid, off by default)
    static const bool trace = getenv("T0_W4_TRACE") != nullptr;
    StampBuffer stamps;
    if (trace) {
        int rc = stamps.make(grid);
        if (rc != T0_OK) return rc;
        P.stamps = stamps.d;
    }
    static const bool use_pdl = getenv("T0_NO_PDL") == nullptr;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(kStThreads, 1, 1);
    cfg.dynamicSmemBytes = kStSmem;
    cfg.stream = rt->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = use_pdl ? 1 : 0;
    void* launch_args[] = {&P};                       // (not by value, which would copy them once more)
    cudaError_t le = cudaLaunchKernelExC(&cfg, (const void*)w4a16_stream_kernel<kProblems>, launch_args);
    if (le != cudaSuccess) return fail(T0_ERR_CUDA, "W4A16 kernel launch failed: %s", cudaGetErrorString(le));
    rt->launches.fetch_add(1);
    if (trace) {
        std::vector<unsigned long long> h((size_t)grid * 4);
        T0_CUDA(cudaStreamSynchronize(rt->stream));
        T0_CUDA(cudaMemcpy(h.data(), stamps.d, h.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost));
        unsigned long long t_min = ~0ull, t_max = 0;
        double fill = 0, loop = 0, tail = 0;
        uint32_t slow = 0;
        for (uint32_t c = 0; c < grid; ++c) {
            t_min = std::min(t_min, h[c * 4]); t_max = std::max(t_max, h[c * 4 + 3]);
            fill += (double)(h[c * 4 + 1] - h[c * 4]); loop += (double)(h[c * 4 + 2] - h[c * 4 + 1]); tail += (double)(h[c * 4 + 3] - h[c * 4 + 2]);
            if (h[c * 4 + 3] - h[c * 4] > h[slow * 4 + 3] - h[slow * 4]) slow = c;
        }
        fprintf(stderr, "[w4a16 stream trace] %zu problems, %llu steps on %u CTAs: first entry -> last exit %.2f us; per CTA mean: first step landed after %.2f us, "
                "main loop %.2f us (%.3f us per step), flush+exit %.2f us; slowest CTA %u entered %.2f us after the first, loop %.2f us, flush+exit %.2f us\n",
                count, (unsigned long long)total, grid, (t_max - t_min) * 1e-3, fill / grid * 1e-3, loop / grid * 1e-3, loop / grid * 1e-3 / ((double)total / grid),
                tail / grid * 1e-3, slow, (h[slow * 4] - t_min) * 1e-3, (h[slow * 4 + 2] - h[slow * 4 + 1]) * 1e-3, (h[slow * 4 + 3] - h[slow * 4 + 2]) * 1e-3);
    }
    return T0_OK;
}

int check_stream_problem(const t0_w4a16_args& a) {
    if (!a.a || !a.packed || !a.y) return fail(T0_ERR_INVALID, "null device pointer");
    if (a.m > 16) return fail(T0_ERR_UNSUPPORTED, "M=%u: the streaming-layout kernel takes M <= 16; use t0_w4a16_gemm on the row layout for larger M", a.m);
    if (a.k == 0 || a.k % kUnitK || a.group == 0 || a.group % kUnitK || a.k % a.group || a.n % 8)
        return fail(T0_ERR_UNSUPPORTED, "shape K=%u N=%u group=%u: needs K %% 128 == 0, group %% 128 == 0, group | K, N %% 8 == 0", a.k, a.n, a.group);
    if ((a.a & 15) || (a.packed & 127) || (a.y & 3)) return fail(T0_ERR_INVALID, "a must be 16-byte, the weights 128-byte and y 4-byte aligned");
    return T0_OK;
}

}  // namespace

extern "C" {

size_t t0_w4_prepacked_bytes(uint32_t K, uint32_t N, uint32_t group) {
    if (K == 0 || N == 0 || group == 0 || K % kUnitK || group % kUnitK || K % group) return 0;
    return prepack_layout(K, N, group).total;
}

int t0_w4_prepack(t0_runtime* rt, uint64_t packed, uint64_t scales, uint64_t zeros, uint64_t out, uint32_t K, uint32_t N, uint32_t group) {
    int rc = check_rt(rt);
    if (rc != T0_OK) return rc;
    if (!packed || !scales || !zeros || !out) return fail(T0_ERR_INVALID, "null device pointer");
    if (K == 0 || N == 0 || group == 0 || K % kUnitK || group % kUnitK || K % group)
        return fail(T0_ERR_UNSUPPORTED, "the streaming layout needs K %% 128 == 0 and group %% 128 == 0 with group | K (K=%u, group=%u)", K, group);
    if (N % 8) return fail(T0_ERR_UNSUPPORTED, "N=%u must be a multiple of 8 (eight zero points per word)", N);
    if (out & 127) return fail(T0_ERR_INVALID, "the output buffer must be 128-byte aligned");
    DeviceGuard guard(rt->device);
    const PrepackLayout L = prepack_layout(K, N, group);
    const uint64_t n = L.total / 2;
    w4_prepack_kernel<<<prepack_grid_for(n, 256), 256, 0, rt->stream>>>((const uint32_t*)packed, (const uint16_t*)scales, (const uint32_t*)zeros,
                                                                       (uint8_t*)out, K, N, (N + 7) / 8, L);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(T0_ERR_CUDA, "prepack launch failed: %s", cudaGetErrorString(e));
    rt->launches.fetch_add(1);
    return T0_OK;
}

int t0_w4a16_gemm_prepacked_batch(t0_runtime* rt, const t0_w4a16_args* args, size_t count) {
    int rc = check_rt(rt);
    if (rc != T0_OK) return rc;
    if (!args && count) return fail(T0_ERR_INVALID, "null arguments");
    DeviceGuard guard(rt->device);
    // every problem is checked before anything is launched; empty problems are dropped
    std::vector<t0_w4a16_args> live;
    live.reserve(count);
    for (size_t i = 0; i < count; ++i) {
        if (args[i].m == 0 || args[i].n == 0) continue;
        rc = check_stream_problem(args[i]);
        if (rc != T0_OK) return rc;
        live.push_back(args[i]);
    }
    // launches of up to kStMaxProblems problems; a launch also ends where the band counters or the step index would overflow
    size_t i = 0;
    while (i < live.size()) {
        size_t n = 0;
        uint64_t bands = 0, units = 0;
        while (i + n < live.size() && n < (size_t)kStMaxProblems) {
            const PrepackLayout L = prepack_layout(live[i + n].k, live[i + n].n, live[i + n].group);
            if (n > 0 && ((bands + L.bands) * sizeof(int) > kCounterRegion || units + (uint64_t)L.bands * L.ksteps > 0x7FFFFFFFull)) break;
            bands += L.bands; units += (uint64_t)L.bands * L.ksteps;
            ++n;
        }
        rc = n <= kStFewProblems ? launch_stream_chunk<kStFewProblems>(rt, live.data() + i, n) : launch_stream_chunk<kStMaxProblems>(rt, live.data() + i, n);
        if (rc != T0_OK) return rc;
        i += n;
    }
    return T0_OK;
}

int t0_w4a16_gemm_prepacked(t0_runtime* rt, uint64_t a, uint64_t prepacked, uint64_t y, uint32_t M, uint32_t N, uint32_t K, uint32_t group) {
    t0_w4a16_args one;
    memset(&one, 0, sizeof one);
    one.a = a; one.packed = prepacked; one.y = y; one.m = M; one.n = N; one.k = K; one.group = group;
    return t0_w4a16_gemm_prepacked_batch(rt, &one, 1);
}

}  // extern "C"
