// Exact brute-force k-NN through the tensor cores: the same words as the FP32
// scan of bruteforce.cu (BruteforceRouter::batch_query,
// router/bruteforce_router.hpp:130-190), found by evaluating in FP32 only the
// few rows that can be among a query's k nearest.
//
//   1. Rows and queries are rounded to FP16 (scaled by powers of two; the rows
//      once per index, or the subset's on every call), keeping the exact norms
//      and the largest rounding residual.
//   2. bf_filter_kernel computes v = A_x + B_x q.x for every pair with
//      tcgen05.mma (FP16 operands, FP32 accumulation in TMEM), a value that
//      orders the rows as the distance does up to a bounded error E_q, and keeps
//      the smallest v of many groups of rows. The k-th smallest group minimum t
//      is at least the k-th smallest v (the minima are k different rows).
//   3. The same kernel again lists every row with v <= t + 2 E_q.
//   4. bf_rerank_kernel evaluates the listed rows in FP32 in the reference's
//      summation order, sorts them by (distance, vid) and writes the best k.
//
// Why no row is missed: let e(x) be the FP32 distance, d(x) the real one in v's
// units, |v - d| + |e - d| <= E_q for every row. The k rows behind the k smallest
// minima have e <= t + E_q, so the k-th smallest e is at most t + E_q, and a row
// among the k nearest has v <= e + E_q <= t + 2 E_q. E_q bounds, with Cauchy's
// inequality: the rounding of both operands (their exact residual norms r_q and
// the rows' largest R), the accumulation in the tensor core (2^-19 of |q||x| per
// 16 products, 32 times the unit of its FP32 accumulator), the FP32 chain of the
// distance itself, and the rounding of sqrt (distances that are equal after it).
// The accumulation's share is a margin and no documented property: against 64 bits on
// the same FP16 operands it took at most 5 % of it, at 64 to 2,048 elements of normal,
// one-signed, cancelling and widely spread values.
// A query whose list does not fit, or an index or query whose norms leave the
// range in which these bounds hold, goes to the FP32 scan: rows that are not
// finite or whose nonzero norms leave [10^-9, 10^9], queries above 10^15, and for
// dot below 2^-50, for cosine outside [10^-9, 10^9]. The lower limits keep what
// FP32 sums of squares lose to underflow (elements below 2^-74: |q| and r_q fall
// short by at most 2^-67 at 16,384 elements, R likewise) far below the 2^-14 of
// |q||x| that E_q holds for the accumulation. Squared distances need none on the
// query: there E_q holds 2^-14 of (|q| + |x|)^2, and |x| is at least 10^-9.
//
// What bounds it: at 1M x 128, 1,000 queries, k 100 the listing pass is 0.26 TFLOP
// (0.16 ms at the measured FP16 rate) and takes 0.29 ms before hits, 0.47 ms with
// them: the epilogue, 128 accumulator columns a thread and tile with two warps a
// scheduler. Sampling one row in 4 makes pass 1 0.09 ms and lists 400 rows a query;
// their FP32 step takes 0.04 ms. The whole call: 36.0 -> 0.67 ms; 37 queries over
// 40,001 of 123,457 x 96 rows 0.45 -> 0.20 ms.
#include <algorithm>
#include <cfloat>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "../../include/artea_gpu.h"
#include "bruteforce.h"
#include "common.h"
#include "internal.h"

namespace artea_gpu {
namespace {

constexpr uint32_t kTileQ = 128;          // queries of a tile: the TMEM lanes
constexpr uint32_t kTileX = 256;          // rows of a tile: accumulator columns
constexpr uint32_t kChunkK = 64;          // FP16 elements of an operand chunk: one 128-byte swizzle row
constexpr uint32_t kABytes = kTileQ * kChunkK * 2;
constexpr uint32_t kBBytes = kTileX * kChunkK * 2;
constexpr uint32_t kMaxStages = 6;        // operand stages, as many as fit
constexpr uint32_t kMaxSample = 8;
constexpr uint32_t kMaxResidentK = 6;     // chunks of the query tile kept for the whole kernel
constexpr uint32_t kThreads = 320;        // TMA warp, MMA warp, 8 epilogue warps
constexpr uint32_t kEpilogue = 256;
constexpr uint32_t kWarpCols = kTileX / 2;   // columns of an epilogue warp
constexpr uint32_t kHitBuffer = 192;      // hits a warp gathers before it appends them to the lists
constexpr uint32_t kListCap = 4096;       // survivors of a query
constexpr uint32_t kMaxGroups2 = 16384;   // group minima of a query
// Dynamic shared memory that the kernels are allowed. The limit belongs to the
// function, not to a call: one that followed a call's width could be lowered by
// another thread between a call's setting it and its launch.
constexpr uint32_t kFilterSmem = 190u * 1024u;
constexpr uint32_t kRerankSmem = 160u * 1024u;
constexpr uint32_t kSpin = 1u << 20;      // polls (each suspends for a while) before a wait counts as lost

struct FilterArgs {
    const float* a;          // rows: A, at whole tiles (infinite past n_rows)
    const float* b;          // rows: B (null: 1)
    uint32_t n_pad;          // rows up to whole tiles: entries of a and b
    uint32_t nq;
    uint32_t chunks;         // K / 64
    uint32_t stages;
    uint32_t sample;         // 1: every row; F: a tile is 256 / F rows of each of F times 256
    uint32_t row_groups;     // CTAs of a query tile
    uint32_t tiles;          // row tiles
    uint32_t per_flush;      // row tiles of a CTA between two sets of minima
    uint32_t groups;         // minima of a query
    float* minima;           // nq x groups (pass 1)
    const float* limit;      // nq: list rows with v <= limit (pass 2; null: pass 1)
    uint32_t* count;         // nq
    uint2* list;             // nq x kListCap: {row, v}
    int* error;
    const BfStats* xs;       // scale of the rows
    const float4* qinfo;     // queries: norm, residual norm, 1 / scale
    float sign;              // factor of q.x in v: -2 or -1
};

// The power of two that brings a norm to [2^13, 2^14): every element then lies
// within FP16's range and the larger ones in its normal range.
__device__ __forceinline__ float pow2_scale(float norm) {
    if (!(norm > 0.0f) || !isfinite(norm)) return 1.0f;
    int e;
    frexpf(norm, &e);
    return ldexpf(1.0f, min(max(14 - e, -100), 100));
}

__device__ __forceinline__ void tc_mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void tc_mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool tc_mbar_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < kSpin; ++i) {
        uint32_t ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap* map, uint32_t x, uint32_t y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}

// Shared-memory matrix descriptor, K-major, 128-byte swizzle: rows of 128 bytes,
// 8-row groups 1,024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    return static_cast<uint64_t>((addr & 0x3FFFFu) >> 4) | (1ull << 16) | (static_cast<uint64_t>(1024u >> 4) << 32) |
           (1ull << 46) | (2ull << 61);
}
// Instruction descriptor: FP32 accumulators, FP16 operands, both K-major.
constexpr uint32_t kIdesc = (1u << 4) | ((kTileX >> 3) << 17) | ((kTileQ >> 4) << 24);

__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, bool accumulate) {
    asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
                 " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
                 ::"r"(d), "l"(a), "l"(b), "r"(kIdesc), "r"(accumulate ? 1u : 0u) : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// 64 accumulator columns of the warp's 32 lanes, in pairs.
__device__ __forceinline__ void tmem_load64(uint32_t addr, f32x2 (&v)[32]) {
    uint32_t r[64];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(addr + 0u));
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]), "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]), "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]), "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
                 : "r"(addr + 32u));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = static_cast<f32x2>(r[2 * i]) | (static_cast<f32x2>(r[2 * i + 1]) << 32);
}
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    return static_cast<f32x2>(__float_as_uint(a)) | (static_cast<f32x2>(__float_as_uint(b)) << 32);
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// Four columns' A and B at row (rows past n_rows: A infinite, B 0; the arrays end
// with the last tile).
__device__ __forceinline__ void filter_columns(const FilterArgs& a, uint32_t row, float4* fa, float4* fb) {
    *fa = make_float4(INFINITY, INFINITY, INFINITY, INFINITY);
    *fb = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (row < a.n_pad) {
        *fa = __ldg(reinterpret_cast<const float4*>(a.a + row));
        if (a.b) *fb = __ldg(reinterpret_cast<const float4*>(a.b + row));
    }
}

// A row within a query's limit: {row, v} into the warp's buffer (a global append
// waits for its counter about 1,000 cycles), or to the list where that is full.
struct FilterHit {
    uint32_t q, row;
    float v;
};
__device__ __forceinline__ void filter_append(const FilterArgs& a, const FilterHit& h) {
    const uint32_t pos = atomicAdd(a.count + h.q, 1u);
    if (pos < kListCap) a.list[static_cast<size_t>(h.q) * kListCap + pos] = make_uint2(h.row, __float_as_uint(h.v));
}
__device__ __forceinline__ void filter_hit(const FilterArgs& a, FilterHit* hits, uint32_t* count, uint32_t q, uint32_t row,
                                        float v) {
    const FilterHit h = {q, row, v};
    const uint32_t pos = atomicAdd(count, 1u);
    if (pos < kHitBuffer) hits[pos] = h;
    else filter_append(a, h);
}

// Appends a warp's gathered hits to the lists.
__device__ __noinline__ void filter_flush(const FilterArgs& a, const FilterHit* hits, uint32_t n) {
    for (uint32_t i = threadIdx.x & 31u; i < n; i += 32u) filter_append(a, hits[i]);
    __syncwarp();
}

// One CTA: a tile of 128 queries against every row_groups-th tile of 256 rows
// (sampled tiles: 256 / F rows at the start of each of F times 256 rows, so that
// any stretch of rows is sampled evenly).
// Warp 0 loads operand chunks by TMA, warp 1 issues the MMAs into two TMEM
// accumulators in turn, warps 2-9 read an accumulator while the other fills:
// thread = query (TMEM lane), a warp takes one half of the tile's columns, 64 at a
// time. (16 epilogue warps leave 96 registers a thread, which spills.)
__global__ void __launch_bounds__(kThreads, 1) bf_filter_kernel(const __grid_constant__ CUtensorMap map_q,
                                                               const __grid_constant__ CUtensorMap map_x,
                                                               const FilterArgs a) {
    extern __shared__ __align__(1024) unsigned char tc_smem[];
    __shared__ __align__(8) uint64_t bars[2 * kMaxStages + 6];
    __shared__ uint32_t tmem_base;
    __shared__ __align__(16) float col_a[8][kWarpCols];
    __shared__ __align__(16) float col_b[8][kWarpCols];
    __shared__ FilterHit hit_buffer[8][kHitBuffer];
    __shared__ uint32_t hit_count[8];
    const uint32_t base = (smem_addr(tc_smem) + 1023u) & ~1023u;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const bool resident = a.chunks <= kMaxResidentK;
    const uint32_t stage_bytes = kBBytes + (resident ? 0u : kABytes);
    const uint32_t stages = base + (resident ? a.chunks * kABytes : 0u);
    const uint32_t bar0 = smem_addr(bars);
    const uint32_t full = bar0, empty = bar0 + 8u * kMaxStages;                  // per stage
    const uint32_t acc_full = bar0 + 16u * kMaxStages, acc_empty = acc_full + 16u;   // per accumulator
    const uint32_t q_full = acc_empty + 16u, drained = q_full + 8u;
    const uint32_t qt = blockIdx.x / a.row_groups, rg = blockIdx.x - qt * a.row_groups;
    if (tid == 0) {
        for (uint32_t s = 0; s < a.stages; ++s) {
            tc_mbar_init(full + 8u * s, 1);
            tc_mbar_init(empty + 8u * s, 1);
        }
        for (uint32_t i = 0; i < 2; ++i) {
            tc_mbar_init(acc_full + 8u * i, 1);
            tc_mbar_init(acc_empty + 8u * i, kEpilogue);
        }
        tc_mbar_init(q_full, 1);
        tc_mbar_init(drained, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_addr(&tmem_base)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;

    if (warp == 0) {
        if (lane == 0) {
            bool ok = true;
            if (resident) {
                mbar_expect(q_full, a.chunks * kABytes);
                for (uint32_t c = 0; c < a.chunks; ++c)
                    tma_load(base + c * kABytes, &map_q, c * kChunkK, qt * kTileQ, q_full);
            }
            uint32_t it = 0;
            for (uint32_t t = rg; t < a.tiles && ok; t += a.row_groups) {
                for (uint32_t c = 0; c < a.chunks && ok; ++c, ++it) {
                    const uint32_t s = it % a.stages, round = it / a.stages;
                    if (round) ok = tc_mbar_wait(empty + 8u * s, (round - 1u) & 1u);
                    if (!ok) break;
                    mbar_expect(full + 8u * s, stage_bytes);
                    const uint32_t at = stages + s * stage_bytes;
                    const uint32_t piece = kTileX / a.sample;   // the map's box: that many rows
                    for (uint32_t i = 0; i < a.sample; ++i)
                        tma_load(at + i * piece * 128u, &map_x, c * kChunkK, (t * a.sample + i) * kTileX, full + 8u * s);
                    if (!resident) tma_load(at + kBBytes, &map_q, c * kChunkK, qt * kTileQ, full + 8u * s);
                }
            }
            if (!ok) atomicCAS(a.error, 0, 1);
            // The copies in flight land before the CTA's memory is given up.
            for (uint32_t s = 0; s < a.stages && it; ++s) {
                const uint32_t used = it > s ? (it - s + a.stages - 1u) / a.stages : 0u;   // loads issued into stage s
                if (used && !tc_mbar_wait(full + 8u * s, (used - 1u) & 1u)) atomicCAS(a.error, 0, 1);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            bool ok = true;
            if (resident) ok = tc_mbar_wait(q_full, 0);
            uint32_t it = 0, n = 0;
            for (uint32_t t = rg; t < a.tiles && ok; t += a.row_groups, ++n) {
                const uint32_t buf = n & 1u, round = n >> 1;
                if (round) ok = tc_mbar_wait(acc_empty + 8u * buf, (round - 1u) & 1u);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (uint32_t c = 0; c < a.chunks && ok; ++c, ++it) {
                    const uint32_t s = it % a.stages;
                    ok = tc_mbar_wait(full + 8u * s, (it / a.stages) & 1u);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t at = stages + s * stage_bytes;
                    const uint32_t aq = resident ? base + c * kABytes : at + kBBytes;
#pragma unroll
                    for (uint32_t k = 0; k < kChunkK / 16u; ++k)
                        mma_f16(tmem + buf * kTileX, smem_desc(aq + 32u * k), smem_desc(at + 32u * k), c + k != 0u);
                    mma_commit(empty + 8u * s);
                }
                mma_commit(acc_full + 8u * buf);
            }
            // Nothing is in flight when the TMEM is given up, whatever happened above.
            mma_commit(drained);
            if (!tc_mbar_wait(drained, 0)) ok = false;
            if (!ok) atomicCAS(a.error, 0, 1);
        }
    } else {
        const uint32_t quadrant = warp & 3u, e = warp - 2u, part = e >> 2;
        const uint32_t q = qt * kTileQ + 32u * quadrant + lane;
        const bool valid = q < a.nq;
        const bool collect = a.limit != nullptr;
        const float beta = a.sign / pow2_scale(sqrtf(__uint_as_float(a.xs->max_sq))) * (valid ? a.qinfo[q].z : 0.0f);
        const f32x2 beta2 = pack2(beta, beta);
        float limit = collect && valid ? a.limit[q] : -INFINITY;
        float m[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) m[i] = INFINITY;
        uint32_t n = 0, set = 0;
        bool ok = true;
        FilterHit* hits = hit_buffer[e];
        if (lane == 0) hit_count[e] = 0;
        __syncwarp();
        // The warp's columns' A (and B), in its own shared memory: four columns a
        // lane, loaded a tile ahead. Column col of tile t is row t * stride + a fixed
        // offset.
        const uint32_t piece = kTileX / a.sample, stride = kTileX * a.sample;
        const uint32_t my_col = part * kWarpCols + 4u * lane;
        const uint32_t my_row = my_col / piece * kTileX + my_col % piece;
        float4 next_a, next_b;
        filter_columns(a, rg * stride + my_row, &next_a, &next_b);
        const float* fa = col_a[e];
        const float* fb = col_b[e];
        for (uint32_t t = rg; t < a.tiles; t += a.row_groups, ++n) {
            const uint32_t buf = n & 1u;
            __syncwarp();
            *reinterpret_cast<float4*>(&col_a[e][4u * lane]) = next_a;
            if (a.b) *reinterpret_cast<float4*>(&col_b[e][4u * lane]) = next_b;
            __syncwarp();
            const uint32_t tn = t + a.row_groups;
            if (tn < a.tiles) filter_columns(a, tn * stride + my_row, &next_a, &next_b);
            ok = ok && tc_mbar_wait(acc_full + 8u * buf, (n >> 1) & 1u);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (uint32_t c = 0; c < kWarpCols; c += 64u) {
                f32x2 v[32];   // 64 columns, in pairs
                __syncwarp();
                tmem_load64(tmem + ((32u * quadrant) << 16) + buf * kTileX + part * kWarpCols + c, v);
                if (c) {   // the values are in registers
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    tc_mbar_arrive(acc_empty + 8u * buf);
                }
                const ulonglong2* pa = reinterpret_cast<const ulonglong2*>(fa + c);
                const ulonglong2* pb = reinterpret_cast<const ulonglong2*>(fb + c);
                if (a.b) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const ulonglong2 wa = pa[i], wb = pb[i];
                        v[2 * i] = fma2(mul2(v[2 * i], beta2), wb.x, wa.x);
                        v[2 * i + 1] = fma2(mul2(v[2 * i + 1], beta2), wb.y, wa.y);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const ulonglong2 wa = pa[i];
                        v[2 * i] = fma2(v[2 * i], beta2, wa.x);
                        v[2 * i + 1] = fma2(v[2 * i + 1], beta2, wa.y);
                    }
                }
                if (!collect) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) m[i] = min3(m[i], lo32(v[i]), hi32(v[i]));
                    continue;
                }
                const uint32_t row0 = t * kTileX + part * kWarpCols + c;
                bool any = false;
#pragma unroll
                for (int b = 0; b < 4; ++b) {   // 16 columns at a time
                    float low = INFINITY;
#pragma unroll
                    for (int i = 0; i < 8; ++i) low = min3(low, lo32(v[8 * b + i]), hi32(v[8 * b + i]));
                    if (low <= limit) {   // about one in 150 for a lane at 400 of 1M
                        any = true;
                        // Mostly one column of the 16, whose v is low.
                        uint32_t bits = 0;
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            bits |= lo32(v[8 * b + i]) <= limit ? 1u << (2 * i) : 0u;
                            bits |= hi32(v[8 * b + i]) <= limit ? 2u << (2 * i) : 0u;
                        }
                        const uint32_t row = row0 + 16u * b;
                        if ((bits & (bits - 1u)) == 0u) {
                            filter_hit(a, hits, &hit_count[e], q, row + __ffs(bits) - 1u, low);
                        } else {
#pragma unroll
                            for (int i = 0; i < 16; ++i) {
                                const float w = (i & 1) ? hi32(v[8 * b + i / 2]) : lo32(v[8 * b + i / 2]);
                                if (w <= limit) filter_hit(a, hits, &hit_count[e], q, row + i, w);
                            }
                        }
                    }
                }
                if (__any_sync(0xffffffffu, any)) {
                    const uint32_t c = *reinterpret_cast<volatile uint32_t*>(&hit_count[e]);
                    __syncwarp();
                    if (c >= kHitBuffer / 2u) {
                        filter_flush(a, hits, min(c, kHitBuffer));
                        if (lane == 0) hit_count[e] = 0;
                        // A query whose list is full already goes to the scan: the rest
                        // of its rows would be appended in vain (1M x 128 equal rows,
                        // 1,000 queries, filter and scan: 49.0 -> 34.9 ms).
                        if (valid && *reinterpret_cast<volatile uint32_t*>(a.count + q) > kListCap) limit = -INFINITY;
                        __syncwarp();
                    }
                }
            }
            if (!collect && ((n + 1u) % a.per_flush == 0u || tn >= a.tiles)) {
                if (valid) {
                    const uint32_t g = (set * a.row_groups + rg) * 64u + part * 32u;
                    float4* out = reinterpret_cast<float4*>(a.minima + static_cast<size_t>(q) * a.groups + g);
#pragma unroll
                    for (int i = 0; i < 8; ++i) out[i] = make_float4(m[4 * i], m[4 * i + 1], m[4 * i + 2], m[4 * i + 3]);
                }
#pragma unroll
                for (int i = 0; i < 32; ++i) m[i] = INFINITY;
                ++set;
            }
        }
        __syncwarp();
        if (collect) filter_flush(a, hits, min(*reinterpret_cast<volatile uint32_t*>(&hit_count[e]), kHitBuffer));
        if (!ok) atomicCAS(a.error, 0, 1);
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// Largest, smallest nonzero and not finite x.x of the index.
__global__ void __launch_bounds__(256) bf_norms_kernel(const float* __restrict__ xsq, uint32_t n, BfStats* s) {
    uint32_t mx = 0, mn = 0x7f800000u, bad = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t b = __float_as_uint(xsq[i]);
        if (b >= 0x7f800000u) bad = 1;   // inf, NaN (x.x is never negative)
        mx = max(mx, b);
        if (b) mn = min(mn, b);
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    mn = __reduce_min_sync(0xffffffffu, mn);
    bad = __reduce_or_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31u) == 0u) {
        atomicMax(&s->max_sq, mx);
        atomicMin(&s->min_sq, mn);
        if (bad) atomicOr(&s->bad, 1u);
    }
}

// Queries to FP16, k_pad elements each (zeros past dim), one warp a query, with its
// norm, residual norm and 1 / scale. Each has the scale of its own norm: with one for
// the batch, one query of 10^12 times the others' norm rounded those to nothing and
// sent them to the scan. The caller's queries need no more than a float's alignment.
__global__ void __launch_bounds__(256) bf_round_queries_kernel(const float* __restrict__ q, uint32_t n, uint32_t dim,
                                                               uint32_t k_pad, __half* __restrict__ out,
                                                               float4* __restrict__ qinfo) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= n) return;   // warp-uniform
    const float* row = q + static_cast<size_t>(i) * dim;
    float sq = 0.0f;
    for (uint32_t k = lane; k < dim; k += 32) sq = fmaf(row[k], row[k], sq);
    for (int off = 16; off > 0; off >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, off);
    const float norm = sqrtf(sq), scale = pow2_scale(norm), inv = 1.0f / scale;
    float res = 0.0f;
    __half2* o = reinterpret_cast<__half2*>(out + static_cast<size_t>(i) * k_pad);
    for (uint32_t k = 2u * lane; k < k_pad; k += 64) {
        const float x = k < dim ? row[k] : 0.0f, y = k < dim ? row[k + 1u] : 0.0f;   // dim is even
        const __half2 h = __floats2half2_rn(x * scale, y * scale);
        const float2 b = __half22float2(h);
        const float e0 = x - b.x * inv, e1 = y - b.y * inv;
        res = fmaf(e0, e0, fmaf(e1, e1, res));
        o[k / 2u] = h;
    }
    for (int off = 16; off > 0; off >>= 1) res += __shfl_xor_sync(0xffffffffu, res, off);
    if (lane == 0) qinfo[i] = make_float4(norm * 1.00001f, sqrtf(res) * 1.00001f, inv, 0.0f);
}

// Rows (vecs, or those of ids) to FP16, k_pad elements each (zeros past dim), 8
// lanes a row, scaled by scale_from; the residual norms' maxima into res_max.
__global__ void __launch_bounds__(256) bf_round_kernel(const float* __restrict__ vecs, const uint32_t* __restrict__ ids,
                                                       const float* __restrict__ xsq, uint32_t n, uint32_t dim,
                                                       uint32_t k_pad, const BfStats* scale_from,
                                                       __half* __restrict__ out, BfStats* res_max) {
    const uint32_t lane = threadIdx.x & 31u, sub = lane & 7u;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const float scale = pow2_scale(sqrtf(__uint_as_float(scale_from->max_sq)));
    const float inv = 1.0f / scale;
    uint32_t mres = 0, mrel = 0;
    for (uint32_t base = 4u * ((blockIdx.x * blockDim.x + threadIdx.x) >> 5); base < n; base += 4u * warps) {
        const uint32_t i = base + (lane >> 3);
        const bool in = i < n;
        const uint32_t vid = in ? (ids ? ids[i] : i) : 0u;
        const float* row = vecs + static_cast<size_t>(vid) * dim;
        float res = 0.0f;
        uint2* o = reinterpret_cast<uint2*>(out + static_cast<size_t>(i) * k_pad);
#pragma unroll 4
        for (uint32_t k = 4u * sub; k < k_pad; k += 32u) {   // dim is a multiple of 16: fours are whole
            if (!in) continue;
            const float4 x = k < dim ? __ldg(reinterpret_cast<const float4*>(row + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
            const __half2 h0 = __floats2half2_rn(x.x * scale, x.y * scale), h1 = __floats2half2_rn(x.z * scale, x.w * scale);
            const float2 b0 = __half22float2(h0), b1 = __half22float2(h1);
            const float e0 = x.x - b0.x * inv, e1 = x.y - b0.y * inv, e2 = x.z - b1.x * inv, e3 = x.w - b1.y * inv;
            res = fmaf(e0, e0, fmaf(e1, e1, fmaf(e2, e2, fmaf(e3, e3, res))));
            uint2 w;
            w.x = *reinterpret_cast<const uint32_t*>(&h0);
            w.y = *reinterpret_cast<const uint32_t*>(&h1);
            o[k / 4u] = w;
        }
#pragma unroll
        for (int off = 4; off > 0; off >>= 1) res += __shfl_xor_sync(0xffffffffu, res, off);
        const float r = sqrtf(res) * 1.00001f;
        if (in) {
            const float norm = sqrtf(xsq[vid]);
            mres = max(mres, __float_as_uint(r));
            if (norm > 0.0f) mrel = max(mrel, __float_as_uint(r / norm * 1.00001f));
        }
    }
    mres = __reduce_max_sync(0xffffffffu, mres);
    mrel = __reduce_max_sync(0xffffffffu, mrel);
    if (lane == 0) {
        atomicMax(&res_max->max_res, mres);
        atomicMax(&res_max->max_rel, mrel);
    }
}

// A and, for cosine, B of every row for a metric, up to whole tiles (n_pad).
__global__ void __launch_bounds__(256) bf_ab_kernel(const uint32_t* __restrict__ ids, const float* __restrict__ xsq,
                                                    uint32_t n, uint32_t n_pad, int metric, float* __restrict__ a,
                                                    float* __restrict__ b) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_pad) return;
    const float nx = i < n ? xsq[ids ? ids[i] : i] : 0.0f;
    a[i] = i >= n ? INFINITY : (metric == ARTEA_GPU_COSINE || metric == ARTEA_GPU_DOT ? 0.0f : nx);
    if (b) b[i] = nx > 0.0f ? 1.0f / sqrtf(nx) : 0.0f;
}

__device__ __forceinline__ uint32_t v_key(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float key_v(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// The k-th smallest of keys[0, n) (shared memory, one CTA of 256 threads; lo, hi:
// the thread's own extremes), rounded up in its last 8 bits: found bit by bit below
// the common high bits, counting the smaller keys.
__device__ uint32_t kth_key(const uint32_t* keys, uint32_t n, uint32_t k, uint32_t lo, uint32_t hi,
                            uint32_t (*sums)[8]) {
    const uint32_t tid = threadIdx.x;
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if ((tid & 31u) == 0u) {
        sums[0][tid >> 5] = lo;
        sums[1][tid >> 5] = hi;
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        lo = min(lo, sums[0][w]);
        hi = max(hi, sums[1][w]);
    }
    __syncthreads();
    const int top = 31 - __clz((lo ^ hi) | 1u);   // the highest bit in which keys differ
    uint32_t prefix = lo & ~((2u << top) - 1u);
    for (int bit = top; bit >= 8; --bit) {
        const uint32_t cand = prefix | (1u << bit);
        uint32_t c = 0;
#pragma unroll 4
        for (uint32_t i = tid; i < n; i += 256) c += keys[i] < cand ? 1u : 0u;
        c = __reduce_add_sync(0xffffffffu, c);
        if ((tid & 31u) == 0u) sums[bit & 1][tid >> 5] = c;
        __syncthreads();
        uint32_t below = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) below += sums[bit & 1][w];
        if (below < k) prefix = cand;
    }
    return prefix | 0xffu;
}

// One CTA a query: t, at least the k-th smallest of its group minima, and the
// limit t + 2 E_q; a query outside the bounds' range gets an overfull count
// instead, which sends it to the scan.
__global__ void __launch_bounds__(256) bf_limit_kernel(const float* __restrict__ minima, uint32_t groups, uint32_t k,
                                                       const float4* __restrict__ qinfo, const BfStats* xs,
                                                       const BfStats* res_max, uint32_t k_pad, int metric,
                                                       float* __restrict__ limit, float* __restrict__ spread,
                                                       uint32_t* __restrict__ count) {
    extern __shared__ uint32_t keys[];
    __shared__ uint32_t sums[2][8];
    const uint32_t q = blockIdx.x, tid = threadIdx.x;
    uint32_t lo = 0xffffffffu, hi = 0u;
    for (uint32_t i = tid; i < groups; i += 256) {
        const uint32_t key = v_key(minima[static_cast<size_t>(q) * groups + i]);
        keys[i] = key;
        lo = min(lo, key);
        hi = max(hi, key);
    }
    const uint32_t key = kth_key(keys, groups, k, lo, hi, sums);
    if (tid == 0) {
        const float t = key_v(key);
        const float Q = qinfo[q].x, rq = qinfo[q].y;
        const float X = sqrtf(__uint_as_float(xs->max_sq)) * 1.00001f;
        const float R = __uint_as_float(res_max->max_res), rel = __uint_as_float(res_max->max_rel);
        const float g = (static_cast<float>(k_pad) / 16.0f + 32.0f) * 1.9073486e-6f;   // 2^-19 a step
        float e;
        bool safe = Q <= 1.0e15f;
        // The lower limits on Q: see the top of the file.
        if (metric == ARTEA_GPU_COSINE) {
            e = rq + (Q + rq) * rel + g * Q;
            safe = Q >= 1.0e-9f && Q <= 1.0e9f;
        } else if (metric == ARTEA_GPU_DOT) {
            e = rq * X + (Q + rq) * R + g * Q * X;
            safe = safe && Q >= 8.8817842e-16f;   // 2^-50
        } else {
            e = 2.0f * (rq * X + (Q + rq) * R) + g * (Q + X) * (Q + X);
        }
        const float two_e = 2.0f * e * 1.0001f;
        const float l = t + two_e + fabsf(t) * 2.4e-7f;
        safe = safe && isfinite(l);
        limit[q] = safe ? l : -INFINITY;
        spread[q] = two_e;
        count[q] = safe ? 0u : kListCap + 1u;
    }
}

// Sorts keys[0, p2) (a power of two; the CTA's barrier comes first) and writes the
// best k as words.
__device__ void sort_out(uint64_t* keys, uint32_t p2, uint32_t k, uint64_t* __restrict__ out) {
    const uint32_t tid = threadIdx.x;
    for (uint32_t k2 = 2; k2 <= p2; k2 <<= 1) {
        for (uint32_t j = k2 >> 1; j > 0; j >>= 1) {
            for (uint32_t i = tid; i < p2; i += 256) {
                const uint32_t p = i ^ j;
                if (p > i) {
                    const uint64_t x = keys[i], y = keys[p];
                    if ((x > y) == ((i & k2) == 0)) {
                        keys[i] = y;
                        keys[p] = x;
                    }
                }
            }
            __syncthreads();
        }
    }
    for (uint32_t i = tid; i < k; i += 256) {
        const uint64_t key = keys[i];
        uint32_t u = static_cast<uint32_t>(key >> 32);
        u = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
        out[i] = (static_cast<uint64_t>(u) << 32) | static_cast<uint32_t>(key);
    }
}

__device__ __forceinline__ uint64_t rr_key(float d, uint32_t vid) {
    return (static_cast<uint64_t>(v_key(d)) << 32) | vid;
}

// One CTA a query. The k-th smallest v of its list, u, again bounds the k-th
// smallest distance (the list holds the k smallest v of all), so only rows with v
// <= u + 2 E_q are evaluated in FP32 (4 lanes a row, the distance kernel's order),
// then sorted by (distance, vid); the best k as words. Queries whose list
// overflowed are appended to redo (redo[0]: their number).
template <int kMetric>
__global__ void __launch_bounds__(256) bf_rerank_kernel(const float* __restrict__ vecs, const float* __restrict__ xsq,
                                                        const uint32_t* __restrict__ ids, uint32_t dim,
                                                        const float* __restrict__ queries, uint32_t k,
                                                        const uint32_t* __restrict__ count,
                                                        const uint2* __restrict__ list,
                                                        const float* __restrict__ spread, uint32_t q_first,
                                                        uint32_t* __restrict__ redo, uint64_t* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char rr_smem[];
    uint64_t* keys = reinterpret_cast<uint64_t*>(rr_smem);                         // kListCap
    uint32_t* rows = reinterpret_cast<uint32_t*>(keys + kListCap);                 // kListCap
    float* qs = reinterpret_cast<float*>(rows + kListCap);                         // dim
    __shared__ uint32_t sums[2][8];
    __shared__ uint32_t kept;
    const uint32_t q = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t listed = count[q];
    if (listed > kListCap || listed < k) {   // (fewer than k cannot be: the minima's rows are listed)
        if (tid == 0) redo[1u + atomicAdd(redo, 1u)] = q_first + q;
        return;
    }
    for (uint32_t i = tid; i < dim; i += 256) qs[i] = queries[static_cast<size_t>(q) * dim + i];
    uint32_t* vk = reinterpret_cast<uint32_t*>(keys);   // the list's v keys
    const uint2* mine = list + static_cast<size_t>(q) * kListCap;
    uint32_t lo = 0xffffffffu, hi = 0u;
    for (uint32_t i = tid; i < listed; i += 256) {
        const uint32_t key = v_key(__uint_as_float(mine[i].y));
        vk[i] = key;
        lo = min(lo, key);
        hi = max(hi, key);
    }
    if (tid == 0) kept = 0;
    const uint32_t u_key = kth_key(vk, listed, k, lo, hi, sums);
    const float u = key_v(u_key);
    const float lim = u + spread[q] + fabsf(u) * 2.4e-7f;
    for (uint32_t i = tid; i < listed; i += 256)
        if (key_v(vk[i]) <= lim) rows[atomicAdd(&kept, 1u)] = mine[i].x;
    __syncthreads();
    const uint32_t n = kept;
    uint32_t p2 = 32;
    while (p2 < n) p2 <<= 1;
    for (uint32_t i = n + tid; i < p2; i += 256) keys[i] = ~0ull;
    __syncthreads();
    const float qsq = kMetric == ARTEA_GPU_COSINE ? query_sqnorm<true>(qs, dim) : 0.0f;
    const uint32_t r = lane >> 2, gi = lane & 3u;
    for (uint32_t base = warp * 8u; base < n; base += 64u) {
        const uint32_t idx = min(base + r, n - 1u);
        const uint32_t at = rows[idx];
        const uint32_t vid = ids ? ids[at] : at;
        const float* row = vecs + static_cast<size_t>(vid) * dim + 4u * gi;
        f32x2 A01 = 0ull, A23 = 0ull;
#pragma unroll 8
        for (uint32_t c = 0; c < dim; c += 16)
            accumulate<kMetric>(__ldg(reinterpret_cast<const ulonglong2*>(row + c)),
                                *reinterpret_cast<const ulonglong2*>(qs + c + 4u * gi), A01, A23);
        float d = fold16<true>(lo32(A01), hi32(A01), lo32(A23), hi32(A23));
        if (kMetric == ARTEA_GPU_EUCLIDEAN) {
            d = __fsqrt_rn(d);
        } else if (kMetric == ARTEA_GPU_DOT) {
            d = -d;
        } else if (kMetric == ARTEA_GPU_COSINE) {
            // utils/simd_distance.hpp:263-274
            const float denom = __fsqrt_rn(__fmul_rn(qsq, xsq[vid]));
            d = denom > 0.0f ? __fsub_rn(1.0f, __fdiv_rn(d, denom)) : 1.0f;
        }
        if (gi == 0u && base + r < n) keys[base + r] = rr_key(d, vid);
    }
    __syncthreads();
    sort_out(keys, p2, k, out + static_cast<size_t>(q) * k);
}

// ---------------------------------------------------------------------------
// A few queries: the same selection on the FP32 distances themselves. One pass
// writes every row's distance key (its order as an unsigned number) and each warp's
// smallest; the k-th smallest of those bounds the k-th smallest key, the rows up to
// it are listed and sorted. A row is read by 4 lanes in whole sectors. One query
// over 1M x 128 at k 100: the scan, whose CTAs each sort the first rows they meet,
// 0.98 ms; this 0.16 ms.
// ---------------------------------------------------------------------------
template <int kMetric>
__global__ void __launch_bounds__(256) bf_few_distances_kernel(const float* __restrict__ vecs,
                                                               const float* __restrict__ xsq,
                                                               const uint32_t* __restrict__ ids, uint32_t n,
                                                               uint32_t dim, const float* __restrict__ queries,
                                                               uint32_t* __restrict__ keys,
                                                               uint32_t* __restrict__ minima) {
    extern __shared__ __align__(16) unsigned char few_smem[];
    float* qs = reinterpret_cast<float*>(few_smem);
    const uint32_t q = blockIdx.y, lane = threadIdx.x & 31u, gi = lane & 3u;
    for (uint32_t i = threadIdx.x; i < dim; i += 256) qs[i] = queries[static_cast<size_t>(q) * dim + i];
    __syncthreads();
    const float qsq = kMetric == ARTEA_GPU_COSINE ? query_sqnorm<true>(qs, dim) : 0.0f;
    const uint32_t warp = blockIdx.x * 8u + (threadIdx.x >> 5), warps = gridDim.x * 8u;
    uint32_t low = 0xffffffffu;
    for (uint32_t base = warp * 8u; base < n; base += warps * 8u) {
        const uint32_t r = base + (lane >> 2);
        const bool valid = r < n;
        const uint32_t vid = valid ? (ids ? ids[r] : r) : 0u;
        const float* row = vecs + static_cast<size_t>(vid) * dim + 4u * gi;
        f32x2 A01 = 0ull, A23 = 0ull;
#pragma unroll 8
        for (uint32_t c = 0; c < dim; c += 16)
            accumulate<kMetric>(__ldg(reinterpret_cast<const ulonglong2*>(row + c)),
                                *reinterpret_cast<const ulonglong2*>(qs + c + 4u * gi), A01, A23);
        const float s = fold16<true>(lo32(A01), hi32(A01), lo32(A23), hi32(A23));
        const float d = finish_distance<kMetric, true>(s, qsq, kMetric == ARTEA_GPU_COSINE ? __ldg(xsq + vid) : 1.0f);
        if (valid && gi == 0u) {
            const uint32_t key = v_key(d);
            keys[static_cast<size_t>(q) * n + r] = key;
            low = min(low, key);
        }
    }
    low = __reduce_min_sync(0xffffffffu, low);
    if (lane == 0) minima[static_cast<size_t>(q) * warps + warp] = low;
}

__global__ void __launch_bounds__(256) bf_few_limit_kernel(const uint32_t* __restrict__ minima, uint32_t groups,
                                                           uint32_t k, uint32_t* __restrict__ limit,
                                                           uint32_t* __restrict__ count) {
    extern __shared__ uint32_t keys[];
    __shared__ uint32_t sums[2][8];
    const uint32_t q = blockIdx.x;
    uint32_t lo = 0xffffffffu, hi = 0u;
    for (uint32_t i = threadIdx.x; i < groups; i += 256) {
        const uint32_t key = minima[static_cast<size_t>(q) * groups + i];
        keys[i] = key;
        lo = min(lo, key);
        hi = max(hi, key);
    }
    const uint32_t key = kth_key(keys, groups, k, lo, hi, sums);
    if (threadIdx.x == 0) {
        limit[q] = key;
        count[q] = 0;
    }
}

__global__ void __launch_bounds__(256) bf_few_list_kernel(const uint32_t* __restrict__ keys,
                                                          const uint32_t* __restrict__ ids, uint32_t n,
                                                          const uint32_t* __restrict__ limit,
                                                          uint32_t* __restrict__ count, uint64_t* __restrict__ list) {
    const uint32_t q = blockIdx.y, lim = limit[q];
    for (uint32_t r = blockIdx.x * 256u + threadIdx.x; r < n; r += gridDim.x * 256u) {
        const uint32_t key = keys[static_cast<size_t>(q) * n + r];
        if (key > lim) continue;
        const uint32_t pos = atomicAdd(count + q, 1u);
        if (pos < kListCap)
            list[static_cast<size_t>(q) * kListCap + pos] = (static_cast<uint64_t>(key) << 32) | (ids ? ids[r] : r);
    }
}

__global__ void __launch_bounds__(256) bf_few_sort_kernel(const uint64_t* __restrict__ list,
                                                          const uint32_t* __restrict__ count, uint32_t k,
                                                          uint32_t* __restrict__ redo, uint64_t* __restrict__ out) {
    __shared__ uint64_t keys[kListCap];
    const uint32_t q = blockIdx.x, n = count[q];
    if (n > kListCap || n < k) {
        if (threadIdx.x == 0) redo[1u + atomicAdd(redo, 1u)] = q;
        return;
    }
    uint32_t p2 = 32;
    while (p2 < n) p2 <<= 1;
    for (uint32_t i = threadIdx.x; i < p2; i += 256) keys[i] = i < n ? list[static_cast<size_t>(q) * kListCap + i] : ~0ull;
    __syncthreads();
    sort_out(keys, p2, k, out + static_cast<size_t>(q) * k);
}

using FewFn = void (*)(const float*, const float*, const uint32_t*, uint32_t, uint32_t, const float*, uint32_t*,
                       uint32_t*);

FewFn few_kernel(int metric) {
    switch (metric) {
        case ARTEA_GPU_EUCLIDEAN_SQR: return bf_few_distances_kernel<ARTEA_GPU_EUCLIDEAN_SQR>;
        case ARTEA_GPU_EUCLIDEAN: return bf_few_distances_kernel<ARTEA_GPU_EUCLIDEAN>;
        case ARTEA_GPU_COSINE: return bf_few_distances_kernel<ARTEA_GPU_COSINE>;
        default: return bf_few_distances_kernel<ARTEA_GPU_DOT>;
    }
}

using RerankFn = void (*)(const float*, const float*, const uint32_t*, uint32_t, const float*, uint32_t,
                          const uint32_t*, const uint2*, const float*, uint32_t, uint32_t*, uint64_t*);

RerankFn rerank_kernel(int metric) {
    switch (metric) {
        case ARTEA_GPU_EUCLIDEAN_SQR: return bf_rerank_kernel<ARTEA_GPU_EUCLIDEAN_SQR>;
        case ARTEA_GPU_EUCLIDEAN: return bf_rerank_kernel<ARTEA_GPU_EUCLIDEAN>;
        case ARTEA_GPU_COSINE: return bf_rerank_kernel<ARTEA_GPU_COSINE>;
        default: return bf_rerank_kernel<ARTEA_GPU_DOT>;
    }
}

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn() {
    static EncodeFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &r) != cudaSuccess ||
            r != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            p = nullptr;
        }
        return reinterpret_cast<EncodeFn>(p);
    }();
    return fn;
}

bool encode(CUtensorMap* map, void* base, uint64_t rows, uint32_t k_pad, uint32_t box_rows) {
    EncodeFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {k_pad, rows};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(k_pad) * 2};
    const cuuint32_t box[2] = {kChunkK, box_rows};
    const cuuint32_t ones[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, base, dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

// A device's workspace, shared by its indexes and freed with the last of them: a
// first call on a new index would otherwise pay its allocation. The call that holds
// it waits for its kernels before it lets go; a call that finds it held allocates
// its own.
struct BfPool {
    std::mutex mu;                  // held by a call
    uint32_t indexes = 0;           // guarded by g_pools_mu
    unsigned char* d_work[2] = {};
    size_t bytes[2] = {};
};
constexpr int kMaxDevices = 64;
static std::mutex g_pools_mu;
static BfPool g_pools[kMaxDevices];

BfCache* bf_cache_create(int device, const float* d_xsq, uint32_t n, int sms) {
    auto* c = new BfCache();
    c->device = device;
    if (device < kMaxDevices) {
        std::lock_guard<std::mutex> lk(g_pools_mu);
        ++g_pools[device].indexes;
    }
    if (n == 0 || dev_alloc(&c->d_norms, 1) != ARTEA_GPU_OK) return c;   // (the scan needs no norms)
    BfStats zero = {};
    zero.min_sq = 0x7f800000u;
    if (cudaMemcpy(c->d_norms, &zero, sizeof(zero), cudaMemcpyHostToDevice) == cudaSuccess) {
        bf_norms_kernel<<<sms * 4, 256>>>(d_xsq, n, c->d_norms);
        c->norms_ready = cudaMemcpy(&c->norms, c->d_norms, sizeof(BfStats), cudaMemcpyDeviceToHost) == cudaSuccess;
    }
    cudaGetLastError();
    return c;
}

void bf_cache_destroy(BfCache* c) {
    if (!c) return;
    dev_free(c->d_norms);
    dev_free(c->d_rows);
    if (c->device < kMaxDevices) {
        BfPool& p = g_pools[c->device];
        std::lock_guard<std::mutex> lk(g_pools_mu);
        if (--p.indexes == 0) {   // no call is running: each has an index of its device
            for (int i = 0; i < 2; ++i) {
                dev_free(p.d_work[i]);
                p.bytes[i] = 0;
            }
        }
    }
    delete c;
}

BfWork::BfWork(const artea_gpu_index* ix)
    : pool(ix->device >= 0 && ix->device < kMaxDevices ? &g_pools[ix->device] : nullptr) {
    held = pool && pool->mu.try_lock();
}

int BfWork::get(int slot, size_t bytes, unsigned char** p) {
    if (!held) {
        dev_free(own[slot]);
        if (int rc = dev_alloc(&own[slot], bytes)) return rc;
        *p = own[slot];
        return ARTEA_GPU_OK;
    }
    if (pool->bytes[slot] < bytes) {
        dev_free(pool->d_work[slot]);
        pool->bytes[slot] = 0;
        if (int rc = dev_alloc(&pool->d_work[slot], bytes)) return rc;
        pool->bytes[slot] = bytes;
    }
    *p = pool->d_work[slot];
    return ARTEA_GPU_OK;
}

BfWork::~BfWork() {
    if (running) {
        cudaStreamSynchronize(stream);
        cudaGetLastError();
    }
    for (auto& p : own) dev_free(p);
    if (held) {
        for (int i = 0; i < 2; ++i) {   // a large workspace is not kept
            if (pool->bytes[i] > kBfKeepBytes) {
                dev_free(pool->d_work[i]);
                pool->bytes[i] = 0;
            }
        }
        pool->mu.unlock();
    }
}

namespace {

size_t up256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }

// The index's rows in FP16, k_pad elements each.
size_t rounded_bytes(const artea_gpu_index* ix) {
    return static_cast<size_t>(ix->nvecs) * ((ix->dim + kChunkK - 1) / kChunkK * kChunkK) * sizeof(__half);
}

// With want_rows the index's rounded rows, made once; false where the filter cannot
// be used (norms outside the bounds' range, no memory).
bool bf_prepare(const artea_gpu_index* ix, bool want_rows, int sms, cudaStream_t st) {
    BfCache* c = ix->bf;
    std::lock_guard<std::mutex> lk(c->mu);
    if (!c->norms_ready) return false;
    float mx, mn;
    std::memcpy(&mx, &c->norms.max_sq, 4);
    std::memcpy(&mn, &c->norms.min_sq, 4);
    if (c->norms.bad || !(mx >= 1.0e-18f) || !(mx <= 1.0e18f) || !(mn >= 1.0e-18f)) return false;
    if (want_rows && !c->rows_ready) {
        // Without the memory the call goes to the scan; a later one asks again.
        const uint32_t k_pad = (ix->dim + kChunkK - 1) / kChunkK * kChunkK;
        if (ix->lean || !room_for_copy(ix, rounded_bytes(ix)) ||
            dev_alloc(&c->d_rows, static_cast<size_t>(ix->nvecs) * k_pad) != ARTEA_GPU_OK)
            return false;
        bf_round_kernel<<<sms * 8, 256, 0, st>>>(ix->d_vecs, nullptr, ix->d_xsq, ix->nvecs, ix->dim, k_pad, c->d_norms,
                                                 c->d_rows, c->d_norms);
        if (cudaStreamSynchronize(st) != cudaSuccess) {   // other streams may use them next
            dev_free(c->d_rows);
            return false;
        }
        c->rows_ready = true;
    }
    return true;
}

}  // namespace

bool bf_rows_ready(const artea_gpu_index* ix) {
    std::lock_guard<std::mutex> lk(ix->bf->mu);
    return ix->bf->rows_ready;
}

uint64_t bf_rows_bytes(const artea_gpu_index* ix) { return bf_rows_ready(ix) ? rounded_bytes(ix) : 0u; }

void bf_drop_rows(const artea_gpu_index* ix) {
    std::lock_guard<std::mutex> lk(ix->bf->mu);
    dev_free(ix->bf->d_rows);
    ix->bf->rows_ready = false;
}

// Queries of a batch: bounds the workspace (16 query tiles keep every SM busy).
constexpr uint32_t kBatchQ = 2048;

int bf_tensor(const artea_gpu_index* ix, int metric, const float* d_queries, uint32_t nq, uint32_t topk,
              const uint32_t* d_subset, uint32_t n_rows, uint64_t* d_out, BfWork& work, int sms, cudaStream_t st,
              bool* used, std::vector<uint32_t>* redo) {
    *used = false;
    if (!encode_fn() || !bf_prepare(ix, d_subset == nullptr, sms, st)) {
        cudaGetLastError();
        return ARTEA_GPU_OK;
    }
    BfCache* c = ix->bf;
    const uint32_t dim = ix->dim, k_pad = (dim + kChunkK - 1) / kChunkK * kChunkK;
    const uint32_t batch = std::min(nq, kBatchQ);
    const uint32_t tiles = (n_rows + kTileX - 1) / kTileX;
    // Pass 1 samples one row in F while about k F rows then pass the limit, which
    // keeps the FP32 step small beside a pass over the rows.
    uint32_t sample = 1;
    while (sample < kMaxSample && 2u * sample * topk <= 512u && tiles / (2u * sample) >= 64u) sample *= 2;
    const uint32_t tiles_a = (tiles + sample - 1) / sample;
    // Row groups: one CTA an SM. Sets of minima: at least 8 k groups of rows where
    // the tiles allow it, so that the k nearest rows are mostly in different ones.
    auto shape = [&](uint32_t b, uint32_t* rg, uint32_t* per_flush, uint32_t* groups) {
        const uint32_t qt = (b + kTileQ - 1) / kTileQ;
        *rg = std::max(1u, std::min(tiles_a, static_cast<uint32_t>(sms) / qt));
        const uint32_t per_cta = (tiles_a + *rg - 1) / *rg;
        uint32_t sets = std::min(per_cta, std::max(1u, (8u * topk + *rg * 64u - 1) / (*rg * 64u)));
        while (sets > 1 && sets * *rg * 64u > kMaxGroups2) --sets;
        *per_flush = (per_cta + sets - 1) / sets;
        *groups = (per_cta + *per_flush - 1) / *per_flush * *rg * 64u;
    };
    uint32_t rg, per_flush, groups, most = 0;
    for (uint32_t first = 0; first < nq; first += batch) {
        shape(std::min(batch, nq - first), &rg, &per_flush, &groups);
        most = std::max(most, groups);
    }
    if (most > kMaxGroups2) return ARTEA_GPU_OK;
    // Workspace.
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t p = at;
        at = up256(at + bytes);
        return p;
    };
    const size_t o_q = take(static_cast<size_t>(batch) * k_pad * 2), o_info = take(sizeof(float4) * batch);
    const size_t o_min = take(sizeof(float) * batch * static_cast<size_t>(most));
    const size_t o_lim = take(sizeof(float) * batch), o_cnt = take(sizeof(uint32_t) * batch);
    const size_t o_spread = take(sizeof(float) * batch);
    const size_t o_list = take(sizeof(uint2) * batch * static_cast<size_t>(kListCap));
    const size_t o_redo = take(sizeof(uint32_t) * (static_cast<size_t>(nq) + 2));
    const uint32_t n_pad = tiles * kTileX;
    const size_t o_a = take(sizeof(float) * static_cast<size_t>(n_pad));
    const size_t o_b = metric == ARTEA_GPU_COSINE ? take(sizeof(float) * static_cast<size_t>(n_pad)) : 0;
    const size_t o_rows = d_subset ? take(static_cast<size_t>(n_rows) * k_pad * 2) : 0, o_rs = take(sizeof(BfStats));
    unsigned char* base = nullptr;
    if (work.get(1, at, &base) != ARTEA_GPU_OK) return ARTEA_GPU_OK;   // the scan needs less
    auto* q16 = reinterpret_cast<__half*>(base + o_q);
    auto* info = reinterpret_cast<float4*>(base + o_info);
    auto* rs = reinterpret_cast<BfStats*>(base + o_rs);
    auto* d_redo = reinterpret_cast<uint32_t*>(base + o_redo);   // count, indices..., error word last
    auto* col_a = reinterpret_cast<float*>(base + o_a);
    auto* col_b = metric == ARTEA_GPU_COSINE ? reinterpret_cast<float*>(base + o_b) : nullptr;
    int* d_error = reinterpret_cast<int*>(d_redo + nq + 1);
    CUDA_TRY(cudaMemsetAsync(d_redo, 0, sizeof(uint32_t), st));
    CUDA_TRY(cudaMemsetAsync(d_error, 0, sizeof(int), st));
    __half* x16 = c->d_rows;
    const BfStats* res = c->d_norms;
    if (d_subset) {
        x16 = reinterpret_cast<__half*>(base + o_rows);
        CUDA_TRY(cudaMemsetAsync(rs, 0, sizeof(BfStats), st));
        bf_round_kernel<<<sms * 8, 256, 0, st>>>(ix->d_vecs, d_subset, ix->d_xsq, n_rows, dim, k_pad, c->d_norms, x16,
                                                 rs);
        res = rs;
    }
    bf_ab_kernel<<<(n_pad + 255) / 256, 256, 0, st>>>(d_subset, ix->d_xsq, n_rows, n_pad, metric, col_a, col_b);
    CUtensorMap map_x, map_s, map_q;
    if (!encode(&map_x, x16, n_rows, k_pad, kTileX) || !encode(&map_s, x16, n_rows, k_pad, kTileX / sample))
        return ARTEA_GPU_OK;
    const uint32_t chunks = k_pad / kChunkK;
    const bool resident = chunks <= kMaxResidentK;
    const uint32_t kept = 1024u + (resident ? chunks * kABytes : 0u), stage = kBBytes + (resident ? 0u : kABytes);
    const uint32_t stages = std::min(kMaxStages, (kFilterSmem - kept) / stage);
    // (At least half an SM's shared memory: one CTA an SM holds all its TMEM.)
    const uint32_t smem = std::max(117u * 1024u, kept + stages * stage);
    CUDA_TRY(cudaFuncSetAttribute(reinterpret_cast<const void*>(bf_filter_kernel),
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kFilterSmem)));
    CUDA_TRY(cudaFuncSetAttribute(reinterpret_cast<const void*>(bf_limit_kernel),
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kMaxGroups2 * 4)));
    RerankFn rr = rerank_kernel(metric);
    const uint32_t rr_smem = kListCap * 12u + dim * 4u;
    if (rr_smem > kRerankSmem) return ARTEA_GPU_OK;
    CUDA_TRY(cudaFuncSetAttribute(reinterpret_cast<const void*>(rr), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(kRerankSmem)));
    for (uint32_t first = 0; first < nq; first += batch) {
        const uint32_t b = std::min(batch, nq - first);
        const float* qv = d_queries + static_cast<size_t>(first) * dim;
        shape(b, &rg, &per_flush, &groups);
        bf_round_queries_kernel<<<(b + 7) / 8, 256, 0, st>>>(qv, b, dim, k_pad, q16, info);
        if (!encode(&map_q, q16, b, k_pad, kTileQ)) return fail(ARTEA_GPU_ECUDA, "brute force: query tensor map");
        FilterArgs f;
        std::memset(&f, 0, sizeof(f));
        f.a = col_a;
        f.b = col_b;
        f.n_pad = n_pad;
        f.nq = b;
        f.chunks = chunks;
        f.stages = stages;
        f.row_groups = rg;
        f.tiles = tiles_a;
        f.sample = sample;
        f.per_flush = per_flush;
        f.groups = groups;
        f.minima = reinterpret_cast<float*>(base + o_min);
        f.count = reinterpret_cast<uint32_t*>(base + o_cnt);
        f.list = reinterpret_cast<uint2*>(base + o_list);
        f.error = d_error;
        f.xs = c->d_norms;
        f.qinfo = info;
        f.sign = metric == ARTEA_GPU_COSINE || metric == ARTEA_GPU_DOT ? -1.0f : -2.0f;
        float* limit = reinterpret_cast<float*>(base + o_lim);
        float* spread = reinterpret_cast<float*>(base + o_spread);
        const uint32_t qt = (b + kTileQ - 1) / kTileQ;
        // A CTA with fewer row tiles leaves its last sets of minima unwritten.
        CUDA_TRY(cudaMemsetAsync(f.minima, 0x7f, sizeof(float) * b * static_cast<size_t>(groups), st));
        bf_filter_kernel<<<qt * rg, kThreads, smem, st>>>(map_q, map_s, f);
        bf_limit_kernel<<<b, 256, groups * 4, st>>>(f.minima, groups, topk, info, c->d_norms, res, k_pad, metric, limit,
                                                    spread, f.count);
        f.limit = limit;
        f.sample = 1;
        f.tiles = tiles;
        f.row_groups = std::max(1u, std::min(tiles, static_cast<uint32_t>(sms) / qt));
        bf_filter_kernel<<<qt * f.row_groups, kThreads, smem, st>>>(map_q, map_x, f);
        rr<<<b, 256, rr_smem, st>>>(ix->d_vecs, ix->d_xsq, d_subset, dim, qv, topk, f.count, f.list, spread, first, d_redo,
                                    d_out + static_cast<size_t>(first) * topk);
        CUDA_TRY(cudaGetLastError());
    }
    std::vector<uint32_t> head(static_cast<size_t>(nq) + 2);
    CUDA_TRY(cudaMemcpyAsync(head.data(), d_redo, sizeof(uint32_t) * head.size(), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    if (head[nq + 1] != 0) return fail(ARTEA_GPU_EKERNEL, "brute force: a wait of the filter kernel ran out");
    redo->assign(head.begin() + 1, head.begin() + 1 + head[0]);
    *used = true;
    return ARTEA_GPU_OK;
}

int bf_few(const artea_gpu_index* ix, int metric, const float* d_queries, uint32_t nq, uint32_t topk,
           const uint32_t* d_subset, uint32_t n_rows, uint64_t* d_out, BfWork& work, int sms, cudaStream_t st,
           bool* used, std::vector<uint32_t>* redo) {
    *used = false;
    // 8 warps a CTA, 4 CTAs an SM: 4,736 minima on 148 SMs. Each stands for two rows
    // or more; fewer than 4 k of them would list too many rows.
    const uint32_t ctas = std::min(static_cast<uint32_t>(sms) * 4u, (n_rows + 127u) / 128u), groups = ctas * 8u;
    if (groups < 4u * topk || groups > kMaxGroups2 || ix->dim * 4u > 48u * 1024u) return ARTEA_GPU_OK;
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t p = at;
        at = up256(at + bytes);
        return p;
    };
    const size_t o_keys = take(sizeof(uint32_t) * static_cast<size_t>(nq) * n_rows);
    const size_t o_min = take(sizeof(uint32_t) * static_cast<size_t>(nq) * groups);
    const size_t o_lim = take(sizeof(uint32_t) * nq), o_cnt = take(sizeof(uint32_t) * nq);
    const size_t o_list = take(sizeof(uint64_t) * static_cast<size_t>(nq) * kListCap);
    const size_t o_redo = take(sizeof(uint32_t) * (static_cast<size_t>(nq) + 1));
    unsigned char* base = nullptr;
    if (work.get(1, at, &base) != ARTEA_GPU_OK) return ARTEA_GPU_OK;   // the scan needs less
    auto* keys = reinterpret_cast<uint32_t*>(base + o_keys);
    auto* minima = reinterpret_cast<uint32_t*>(base + o_min);
    auto* limit = reinterpret_cast<uint32_t*>(base + o_lim);
    auto* count = reinterpret_cast<uint32_t*>(base + o_cnt);
    auto* list = reinterpret_cast<uint64_t*>(base + o_list);
    auto* d_redo = reinterpret_cast<uint32_t*>(base + o_redo);
    CUDA_TRY(cudaMemsetAsync(d_redo, 0, sizeof(uint32_t), st));
    few_kernel(metric)<<<dim3(ctas, nq), 256, ix->dim * 4, st>>>(ix->d_vecs, ix->d_xsq, d_subset, n_rows, ix->dim,
                                                                 d_queries, keys, minima);
    CUDA_TRY(cudaFuncSetAttribute(reinterpret_cast<const void*>(bf_few_limit_kernel),
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kMaxGroups2 * 4)));
    bf_few_limit_kernel<<<nq, 256, groups * 4, st>>>(minima, groups, topk, limit, count);
    bf_few_list_kernel<<<dim3(std::min(static_cast<uint32_t>(sms) * 4u, (n_rows + 1023u) / 1024u), nq), 256, 0, st>>>(
        keys, d_subset, n_rows, limit, count, list);
    bf_few_sort_kernel<<<nq, 256, 0, st>>>(list, count, topk, d_redo, d_out);
    CUDA_TRY(cudaGetLastError());
    std::vector<uint32_t> head(static_cast<size_t>(nq) + 1);
    CUDA_TRY(cudaMemcpyAsync(head.data(), d_redo, sizeof(uint32_t) * head.size(), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    redo->assign(head.begin() + 1, head.begin() + 1 + head[0]);
    *used = true;
    return ARTEA_GPU_OK;
}

}  // namespace artea_gpu
