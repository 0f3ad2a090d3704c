// Device side of the B200 query path: one warp searches one query.
//
// Restates, on the GPU, hierarchical_graph_router.hpp:195-248 (_query with
// RandomSeeding=false; enable_early_stop either way): entry point, greedy descent
// on levels top..1 (detail/beam_loop.hpp:129-166), beam search on level 0
// (detail/beam_loop.hpp:90-119) with StdCandidateQueue's rules
// (router/data_structures/std_candidate_queue.hpp:358-513), top-k extraction
// (std_candidate_queue.hpp:542-561).
//
// Data layout in HBM (uploaded once):
//   vecs      N x D float32, D a multiple of 16, rows 64-byte aligned
//   vinfo     N x {highest_level, local_vid} (uint2)
//   offsets   per highest-level group h: N_h*(h+1)+1 uint64 CSR offsets
//   nbrs      uint32 neighbour ids in CSR row order
//   l0row     N x uint64 level-0 row descriptor: start | length << 40
// Per search slot (one per resident warp): a spill bitset (N bits) and the
// list of ids set in it since the last clear.
//
// Shared memory per warp: the query row, the candidate queue (sorted array of
// (dist, vid|explored), 2L slots), a candidate batch and the visited hash.
#pragma once

#include <cstdint>
#include <cfloat>
#include <type_traits>
#include <cuda_runtime.h>

#include "../../include/artea_gpu.h"

namespace artea_gpu {

constexpr uint32_t kFull = 0xffffffffu;
constexpr uint32_t kExplored = 0x80000000u;
constexpr uint32_t kVidMask = 0x7fffffffu;
constexpr uint32_t kInvalidLevel = 0xffffffffu;
constexpr uint32_t kEmptySlot = 0xffffffffu;
constexpr uint32_t kCandBatch = 64;     // candidates evaluated per distance batch
constexpr uint32_t kPadRow = 64;        // ids per fixed-stride level-0 row (DeviceGraph::l0pad)
constexpr int kMaxGroups = 64;
constexpr int kRowLenShift = 40;        // l0row: start in bits 0..39, length in 40..63
constexpr unsigned long long kRowStartMask = (1ull << kRowLenShift) - 1ull;

enum : int {
    kErrNone = 0,
    kErrBadVid = 1,        // an id >= N reached the kernel
    kErrBound = 2,         // an iteration bound was exceeded
    kErrQueue = 3,         // queue capacity exceeded (cannot happen for cap >= 2L)
    kErrArgs = 4,          // per-query topk/queue outside the launch's limits
    kErrTimeout = 5,       // a bulk copy did not complete within the wait bound
};

constexpr uint32_t kStageRows = 8;          // rows per staged pass (one per row group)
constexpr uint32_t kStagePad = 4;           // words of padding per staged row (bank spread)
constexpr uint32_t kWaitBound = 1u << 22;   // mbarrier polls before a copy counts as lost

struct DeviceGraph {
    const float* __restrict__ vecs;
    const float* __restrict__ xsq;   // per-row x.x (row_sqnorm_kernel)
    const uint2* __restrict__ vinfo;
    const uint32_t* __restrict__ nbrs;
    const unsigned long long* __restrict__ l0row;
    // Level-0 rows at a fixed stride: N x kPadRow ids, 0xffffffff past the row's
    // length, so a row's ids are one dependent load away from its vid instead of
    // two (descriptor, ids). Null when some row is longer or repeats an id.
    // (1M x 128, 10,000 queries, queue 400: 13.20 -> 12.56 ms.)
    const uint32_t* __restrict__ l0pad;
    uint32_t n;
    uint32_t dim;
    uint32_t top;      // kInvalidLevel when empty
    uint32_t entry;
    uint32_t l0_unique;   // every level-0 row of <= 64 ids holds distinct ids
    const uint64_t* offsets[kMaxGroups];
};

// Trace of a search for the subsystem probes (kernels compiled with kTrace):
// per query, the level-0 expansions (vid, new candidates), the candidates'
// ids and distances in evaluation order, the cursor that seeds level 0, and
// the lengths recorded (capped at cap / rows_cap).
struct TraceArgs {
    uint32_t* ids;       // nq x cap
    float* dists;        // nq x cap
    uint2* rows;         // nq x rows_cap: (expanded vid, new candidates)
    uint2* cur;          // nq: (cursor vid, its distance bits)
    uint2* len;          // nq: (candidates, rows) recorded
    uint32_t cap;
    uint32_t rows_cap;
    uint32_t upper_only; // stop after the upper levels (the greedy descent alone)
};

struct SearchArgs {
    DeviceGraph g;
    const float* __restrict__ queries;
    uint32_t nq;
    const uint32_t* __restrict__ topk;    // may be null
    const uint32_t* __restrict__ queue;   // may be null
    uint32_t topk_default;
    uint32_t queue_default;
    uint32_t k_stride;
    uint32_t cap;                         // queue entries per warp (>= 2 * max queue)
    uint32_t vh_bits;                     // log2 of the shared-memory visited table in 16-byte units (0: none)
    uint32_t vk_bits;                     // log2 of the vid permutation space (visited_kbits)
    uint64_t* __restrict__ out;
    artea_gpu_query_stats* __restrict__ stats;   // may be null
    uint32_t* __restrict__ vis_bits;      // slots x words_per_slot
    uint32_t* __restrict__ vis_list;      // slots x list_cap
    uint64_t words_per_slot;
    uint32_t list_cap;
    uint32_t* __restrict__ next_query;    // persistent schedule work counter
    int* __restrict__ error;
    uint32_t l0_only;
    unsigned long long* __restrict__ phase_cycles;   // nq x kPhases, optional
    uint32_t coherent;        // queries/topk/queue may change while the kernel runs (serving ring)
    uint32_t early_stop;      // stop level-h greedy walks at distance <= es_thr[h]
    float es_thr[kMaxGroups]; // per-level thresholds in query distance units
    uint32_t compact;         // queue capacity may be below 2L: a query that could lose a live
                              // entry is abandoned and listed in overflow for the full-capacity rerun
    uint32_t* __restrict__ overflow;   // [count, rerun counter, query indices...] (compact only)
    uint32_t l0_pipe;         // the launch takes a kernel with the pipelined level-0 loop (needs g.l0pad)
    uint32_t pf_l2;           // pipelined loop: also prefetch the second pass's rows into L2
    const uint32_t* __restrict__ order;   // persistent schedule: query order (null: 0..nq-1)
    TraceArgs tr;             // kernels compiled with kTrace only
};

// Phase-cycle breakdown written per query when phase_cycles is set.
enum : int {
    kPhUpper = 0,     // greedy descent on levels >= 1
    kPhPop = 1,       // pop, row descriptor, first ids, next-entry prefetch
    kPhCollect = 2,   // row ids + visited test_and_set
    kPhDist = 3,      // distance batches
    kPhMerge = 4,     // queue merge
    kPhTail = 5,      // result write-out and visited clear
    kPhTotal = 6,     // whole query
    kPhPrefetchHits = 7,  // expansions whose row descriptor was prefetched
    kPhases = 8
};

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }

__device__ __forceinline__ bool entry_less(float da, uint32_t va, float db, uint32_t vb) {
    return da < db || (da == db && (va & kVidMask) < (vb & kVidMask));
}

__device__ __forceinline__ void set_error(int* error, int code) {
    atomicCAS(error, 0, code);
}

// ---------------------------------------------------------------------------
// Distances (subsystem d). 4 lanes per row, 8 rows per warp pass. Lane group
// slot g in [0,4) owns AVX-512 lanes 4g..4g+3 of the reference's 16-lane
// accumulation (utils/simd_distance.hpp:100-115): for chunk c it loads the
// float4 at element 16c+4g and FMAs into four accumulators, so each
// accumulator is exactly one reference lane's chain. The fold then follows
// GCC's _mm512_reduce_add_ps tree: lanes (i, i+8) are warp lanes g and g^2,
// lanes (i, i+4) are g and g^1, then (i, i^2) and lane0+lane1 inside a lane.
// FAST mode folds each lane's four components first (warp order).
// ---------------------------------------------------------------------------
template <bool kExact>
__device__ __forceinline__ float fold16(float a0, float a1, float a2, float a3) {
    if (kExact) {
        a0 = __fadd_rn(a0, __shfl_xor_sync(kFull, a0, 2));
        a1 = __fadd_rn(a1, __shfl_xor_sync(kFull, a1, 2));
        a2 = __fadd_rn(a2, __shfl_xor_sync(kFull, a2, 2));
        a3 = __fadd_rn(a3, __shfl_xor_sync(kFull, a3, 2));
        a0 = __fadd_rn(a0, __shfl_xor_sync(kFull, a0, 1));
        a1 = __fadd_rn(a1, __shfl_xor_sync(kFull, a1, 1));
        a2 = __fadd_rn(a2, __shfl_xor_sync(kFull, a2, 1));
        a3 = __fadd_rn(a3, __shfl_xor_sync(kFull, a3, 1));
        const float u0 = __fadd_rn(a0, a2);
        const float u1 = __fadd_rn(a1, a3);
        return __fadd_rn(u0, u1);
    } else {
        float s = (a0 + a1) + (a2 + a3);
        s += __shfl_xor_sync(kFull, s, 1);
        s += __shfl_xor_sync(kFull, s, 2);
        return s;
    }
}

__device__ __forceinline__ float4 ldg4(const float* p) {
    return __ldg(reinterpret_cast<const float4*>(p));
}

// Squared norm of the query with the reference's lane structure (the nsq1
// accumulator of utils/simd_distance.hpp:251-268), needed by cosine.
template <bool kExact>
__device__ float query_sqnorm(const float* __restrict__ q, uint32_t dim) {
    const int g = lane_id() & 3;
    float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
    #pragma unroll 1
    for (uint32_t c = 0; c < dim; c += 16) {
        const float4 v = *reinterpret_cast<const float4*>(q + c + 4 * g);
        a0 = fmaf(v.x, v.x, a0); a1 = fmaf(v.y, v.y, a1);
        a2 = fmaf(v.z, v.z, a2); a3 = fmaf(v.w, v.w, a3);
    }
    return fold16<kExact>(a0, a1, a2, a3);
}

// Per pass each lane issues up to kBlock float4 loads of its row segment
// before any arithmetic, so a D=128 row costs one memory round trip.
constexpr int kBlock = 8;

// Packed FP32x2 arithmetic (sm_100): each element is rounded on its own, as
// two scalar instructions would round it, so the exact mode is unaffected;
// the pair halves the instruction count of the accumulation.
typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float lo32(f32x2 v) { return __uint_as_float(static_cast<uint32_t>(v)); }
__device__ __forceinline__ float hi32(f32x2 v) { return __uint_as_float(static_cast<uint32_t>(v >> 32)); }

// One chunk of 4 elements (x from the row, y from the query) into the pair
// accumulators A01/A23.
template <int kMetric>
__device__ __forceinline__ void accumulate(const ulonglong2 x, const ulonglong2 y, f32x2& A01, f32x2& A23) {
    if (kMetric == ARTEA_GPU_EUCLIDEAN_SQR || kMetric == ARTEA_GPU_EUCLIDEAN) {
        const f32x2 d01 = sub2(y.x, x.x), d23 = sub2(y.y, x.y);
        A01 = fma2(d01, d01, A01);
        A23 = fma2(d23, d23, A23);
    } else {
        // dot and cosine: q.x (cosine's x.x comes from the index's row norms)
        A01 = fma2(y.x, x.x, A01);
        A23 = fma2(y.y, x.y, A23);
    }
}

// ---------------------------------------------------------------------------
// TMA row staging: one cp.async.bulk per candidate row into the warp's
// shared-memory stage, completion counted on the warp's mbarrier, so a pass
// costs one memory round trip whatever the row length.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint32_t mbar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect(uint32_t mbar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void bulk_row_copy(uint32_t dst, const float* src, uint32_t bytes, uint32_t mbar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(mbar) : "memory");
}

// Bounded wait for the phase with the given parity; false if it never came.
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
    #pragma unroll 1
    for (uint32_t i = 0; i < kWaitBound; ++i) {
        uint32_t ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(ok) : "r"(mbar), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}

struct Stage {
    float* buf;          // kStageRows rows of dim + kStagePad words (null: no staging)
    uint32_t mbar;       // shared address of the warp's mbarrier
    uint32_t phase;      // parity of the next phase to wait for
};

// ---------------------------------------------------------------------------
// Distances of rows of at most kBlock chunks. A warp issues an instruction every
// 4-8 cycles in a search (one warp a scheduler in a team, five otherwise, each one
// dependent chain), so what counts is instructions:
// lanes without a row of their own repeat the last one (the same addresses, no
// extra traffic) instead of being masked, and rows are loaded apart from the
// arithmetic, ahead of it.
// ---------------------------------------------------------------------------
template <int kMetric, bool kExact>
__device__ __forceinline__ float finish_distance(float res, float qsq, float xsq) {
    if (kMetric == ARTEA_GPU_EUCLIDEAN) return __fsqrt_rn(res);
    if (kMetric == ARTEA_GPU_DOT) return -res;
    if (kMetric == ARTEA_GPU_COSINE) {
        // utils/simd_distance.hpp:263-274
        const float denom = __fsqrt_rn(__fmul_rn(qsq, xsq));
        return denom > 0.0f ? __fsub_rn(1.0f, __fdiv_rn(res, denom)) : 1.0f;
    }
    return res;
}

// A row warp's registers for rows loaded ahead of their arithmetic: pairs, or
// single elements for wide rows (packing those into pairs would wait for every
// load in turn).
typedef f32x2 RowRegs[16];
typedef float WideRegs[32];

// Rows cvid[p, min(p + 8, cnt)) of at most kBlock chunks (kN: their number, or 0
// for nchunks), 4 lanes a row as in batch_distances; cnt > p.
template <int kN>
__device__ __forceinline__ void row8_load(const DeviceGraph& g, const uint32_t* cvid, uint32_t p, uint32_t cnt,
                                          uint32_t nchunks, RowRegs& x) {
    const uint32_t lane = static_cast<uint32_t>(lane_id());
    const uint32_t vid = cvid[min(p + (lane >> 2), cnt - 1u)];
    const float* row = g.vecs + static_cast<size_t>(vid) * g.dim + 4u * (lane & 3u);
#pragma unroll
    for (int k = 0; k < (kN ? kN : kBlock); ++k) {
        if (kN || static_cast<uint32_t>(k) < nchunks) {
            const ulonglong2 w = __ldg(reinterpret_cast<const ulonglong2*>(row + 16 * k));
            x[2 * k] = w.x;
            x[2 * k + 1] = w.y;
        }
    }
}

template <int kMetric, bool kExact, int kN>
__device__ __forceinline__ void row8_distance(const DeviceGraph& g, const float* __restrict__ q, float qsq,
                                              const uint32_t* cvid, float* cdist, uint32_t p, uint32_t cnt,
                                              uint32_t nchunks, const RowRegs& x) {
    const uint32_t lane = static_cast<uint32_t>(lane_id());
    const uint32_t idx = p + (lane >> 2);
    const float xsq = kMetric == ARTEA_GPU_COSINE ? __ldg(g.xsq + cvid[min(idx, cnt - 1u)]) : 1.0f;
    const float* qq = q + 4u * (lane & 3u);
    f32x2 A01 = 0ull, A23 = 0ull;
#pragma unroll
    for (int k = 0; k < (kN ? kN : kBlock); ++k)
        if (kN || static_cast<uint32_t>(k) < nchunks)
            accumulate<kMetric>(make_ulonglong2(x[2 * k], x[2 * k + 1]),
                                *reinterpret_cast<const ulonglong2*>(qq + 16 * k), A01, A23);
    const float res = finish_distance<kMetric, kExact>(fold16<kExact>(lo32(A01), hi32(A01), lo32(A23), hi32(A23)), qsq,
                                                       xsq);
    if (idx < cnt && (lane & 3u) == 0u) cdist[idx] = res;
}

// Loads of the next expansion's rows, issued ahead of its distance phase so
// they are in flight while the warp merges the current batch. With kRegs, the
// first pass's first block of chunks (rows cvid[0, 8), one float4 per chunk
// and lane) is loaded into x, which batch_distances then consumes (kPre);
// without, those rows' first 512 bytes are prefetched into L2 (one 128-byte
// line per lane). With l2_next, the second pass's rows (cvid[8, 16)) are
// prefetched into L2 as well.
__device__ __forceinline__ void prefetch_l2(const void* p) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

template <bool kRegs>
__device__ __forceinline__ void dist_preload(const DeviceGraph& g, const uint32_t* cvid, uint32_t cnt,
                                             RowRegs& x, bool l2_next) {
    const int lane = lane_id();
    const uint32_t r = static_cast<uint32_t>(lane) >> 2;
    const uint32_t gi = lane & 3;
    const uint32_t dim = g.dim;
    const uint32_t off = 128u * gi;   // byte offset of this lane's line in a row
    if (kRegs) {
        const uint32_t nchunks = dim >> 4;
        if (cnt) {
            if (nchunks == 8u) row8_load<8>(g, cvid, 0, cnt, nchunks, x);
            else if (nchunks == 6u) row8_load<6>(g, cvid, 0, cnt, nchunks, x);
            else row8_load<0>(g, cvid, 0, cnt, min(nchunks, static_cast<uint32_t>(kBlock)), x);
        }
    } else if (r < cnt && off < dim * 4u) {
        prefetch_l2(reinterpret_cast<const char*>(g.vecs + static_cast<size_t>(cvid[r]) * dim) + off);
    }
    if (l2_next && cnt > 8u) {
        const uint32_t r2 = 8u + r;
        if (r2 < cnt && off < dim * 4u)
            prefetch_l2(reinterpret_cast<const char*>(g.vecs + static_cast<size_t>(cvid[r2]) * dim) + off);
    }
}

// Distances for cnt candidates (ids in cvid, shared memory) into cdist, one
// pass of 8 rows at a time: passes pass0, pass0 + stride, ... (the warps of a
// cooperative search split the passes; one warp alone takes them all). With
// kPre, the first pass's first block of chunks is taken from pre (loaded by
// dist_preload<true> on the same cvid) instead of being loaded here.
// The whole batch for rows of kN chunks: about 50 instructions a pass less than the
// masked loads below (1M x 128, 10,000 queries, 96 registers: queue 100 4.30 -> 3.55
// ms, pipelined 3.60 -> 3.41; 1M x 96 cosine uneven batch 5.95 -> 5.55 ms).
template <int kMetric, bool kExact, bool kPre, int kN>
__device__ __forceinline__ void narrow_distances(const DeviceGraph& g, const float* __restrict__ q, float qsq,
                                                 const uint32_t* cvid, float* cdist, uint32_t cnt,
                                                 const RowRegs* pre) {
    RowRegs x;
    if (kPre) {
#pragma unroll
        for (int k = 0; k < 2 * kN; ++k) x[k] = (*pre)[k];
    }
    #pragma unroll 1
    for (uint32_t p = 0; p < cnt; p += 8u) {
        if (!kPre || p) row8_load<kN>(g, cvid, p, cnt, kN, x);
        row8_distance<kMetric, kExact, kN>(g, q, qsq, cvid, cdist, p, cnt, kN, x);
    }
    __syncwarp();
}

template <int kMetric, bool kExact, bool kStage, bool kPre = false, bool kSplit = false, bool kNarrow = false>
__device__ void batch_distances(const DeviceGraph& g, const float* __restrict__ q, float qsq,
                                const uint32_t* cvid, float* cdist, uint32_t cnt, Stage& st, int* error,
                                const RowRegs* pre = nullptr, uint32_t pass0 = 0,
                                uint32_t stride = 1) {
    if (!kSplit) {
        pass0 = 0;
        stride = 1;
    }
    const int lane = lane_id();
    const int r = lane >> 2;
    const int gi = lane & 3;
    const uint32_t dim = g.dim;
    const uint32_t nchunks = dim >> 4;
    const uint32_t sstride = dim + kStagePad;
    // Level 0, rows of 128 and 96 elements. The other widths up to 128 stay on the
    // masked loop: the same code with their number of chunks in a register takes more
    // of them, and the autotuner then leaves the 96-register kernels (1M rows, 10,000
    // queries, queue 100: 16 elements 2.64 -> 3.02 ms, 64 3.15 -> 3.57, 112 3.51 ->
    // 3.98, and 128 itself 2.82 -> 3.03; without the two widths' own code 128 3.75 ms).
    if (kNarrow && !kStage && !kSplit) {
        if (nchunks == 8u) return narrow_distances<kMetric, kExact, kPre, 8>(g, q, qsq, cvid, cdist, cnt, pre);
        if (nchunks == 6u) return narrow_distances<kMetric, kExact, kPre, 6>(g, q, qsq, cvid, cdist, cnt, pre);
    }
    #pragma unroll 1
    for (uint32_t p = 8u * pass0; p < cnt; p += 8u * stride) {
        const uint32_t idx = p + r;
        const bool valid = idx < cnt;
        const uint32_t vid = valid ? cvid[idx] : 0u;
        // x.x of the row, stored at index creation in this kernel's exact
        // summation order (row_sqnorm_kernel); loaded ahead of the row.
        const float xsq = (kMetric == ARTEA_GPU_COSINE && valid) ? __ldg(g.xsq + vid) : 1.0f;
        const float* row;
        if (kStage) {
            // The stage's previous contents have been read by every lane
            // (generic proxy) before the async proxy overwrites them.
            const uint32_t nrows = min(kStageRows, cnt - p);
            __syncwarp();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            if (lane == 0) mbar_expect(st.mbar, nrows * dim * 4u);
            __syncwarp();
            if (static_cast<uint32_t>(lane) < nrows)
                bulk_row_copy(smem_addr(st.buf + lane * sstride), g.vecs + static_cast<size_t>(cvid[p + lane]) * dim,
                              dim * 4u, st.mbar);
            if (!mbar_wait(st.mbar, st.phase)) {
                set_error(error, kErrTimeout);
                mbar_wait(st.mbar, st.phase);   // a second bounded wait for the copies in flight
            }
            st.phase ^= 1u;
            row = st.buf + r * sstride + 4 * gi;
        } else {
            row = g.vecs + static_cast<size_t>(vid) * dim + 4 * gi;
        }
        const float* qq = q + 4 * gi;
        f32x2 A01 = 0ull, A23 = 0ull;   // L2: diff^2; dot/cos: q*x   (+0.0f pairs)
        #pragma unroll 1
        for (uint32_t cb = 0; cb < nchunks; cb += kBlock) {
            ulonglong2 x[kBlock];
            if (kPre && p == 0 && cb == 0) {
#pragma unroll
                for (int k = 0; k < kBlock; ++k) x[k] = make_ulonglong2((*pre)[2 * k], (*pre)[2 * k + 1]);
            } else {
#pragma unroll
                for (int k = 0; k < kBlock; ++k) {
                    const ulonglong2* src = reinterpret_cast<const ulonglong2*>(row + 16 * (cb + k));
                    x[k] = (valid && cb + k < nchunks) ? (kStage ? *src : __ldg(src)) : make_ulonglong2(0ull, 0ull);
                }
            }
#pragma unroll
            for (int k = 0; k < kBlock; ++k) {
                if (cb + k < nchunks) {
                    const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(qq + 16 * (cb + k));
                    accumulate<kMetric>(x[k], y, A01, A23);
                }
            }
        }
        const float a0 = lo32(A01), a1 = hi32(A01), a2 = lo32(A23), a3 = hi32(A23);
        float res = fold16<kExact>(a0, a1, a2, a3);
        if (kMetric == ARTEA_GPU_EUCLIDEAN) {
            res = __fsqrt_rn(res);
        } else if (kMetric == ARTEA_GPU_DOT) {
            res = -res;
        } else if (kMetric == ARTEA_GPU_COSINE) {
            // utils/simd_distance.hpp:263-274
            const float denom = __fsqrt_rn(__fmul_rn(qsq, xsq));
            res = denom > 0.0f ? __fsub_rn(1.0f, __fdiv_rn(res, denom)) : 1.0f;
        }
        if (valid && gi == 0) cdist[idx] = res;
    }
    __syncwarp();
}

// Rows of more than kBlock chunks: 16 lanes a row, lane j owning the reference's
// AVX-512 lane j (element 16c + j of every chunk c), so a lane keeps 32 chunks in
// flight; two rows a pass. The fold's xor steps (8, 4, 2, 1) are fold16's tree (FAST: 1, 2,
// 4, 8, fold16<false>'s order), so distances are bit-identical.
constexpr uint32_t kWideBlock = 32;

// Block cb (in chunks) of rows cvid[p, min(p + 2, cnt)); cnt > p.
__device__ __forceinline__ void slice_load(const DeviceGraph& g, const uint32_t* cvid, uint32_t p, uint32_t cnt,
                                           WideRegs& x, uint32_t cb = 0) {
    const uint32_t lane = static_cast<uint32_t>(lane_id());
    const uint32_t left = (g.dim >> 4) - cb;
    const uint32_t vid = cvid[min(p + (lane >> 4), cnt - 1u)];
    const float* row = g.vecs + static_cast<size_t>(vid) * g.dim + (lane & 15u) + 16u * cb;
#pragma unroll
    for (int k = 0; k < static_cast<int>(kWideBlock); ++k)
        if (static_cast<uint32_t>(k) < left) x[k] = __ldg(row + 16 * k);
}

template <int kMetric, bool kExact>
__device__ __forceinline__ void slice_distance(const DeviceGraph& g, const float* __restrict__ q, float qsq,
                                              const uint32_t* cvid, float* cdist, const uint32_t* slots, uint32_t p,
                                              uint32_t cnt, WideRegs& x) {
    const uint32_t lane = static_cast<uint32_t>(lane_id());
    const uint32_t j = lane & 15u;
    const uint32_t nchunks = g.dim >> 4;
    const uint32_t idx = p + (lane >> 4);
    const float xsq = kMetric == ARTEA_GPU_COSINE ? __ldg(g.xsq + cvid[min(idx, cnt - 1u)]) : 1.0f;
    float acc = 0.0f;
    #pragma unroll 1
    for (uint32_t cb = 0; cb < nchunks; cb += kWideBlock) {
        if (cb) slice_load(g, cvid, p, cnt, x, cb);
#pragma unroll
        for (int k = 0; k < static_cast<int>(kWideBlock); ++k) {
            if (cb + k < nchunks) {
                const float y = q[16u * (cb + k) + j], v = x[k];
                if (kMetric == ARTEA_GPU_EUCLIDEAN_SQR || kMetric == ARTEA_GPU_EUCLIDEAN) {
                    const float d = __fsub_rn(y, v);
                    acc = __fmaf_rn(d, d, acc);
                } else {
                    acc = __fmaf_rn(y, v, acc);
                }
            }
        }
    }
    if (kExact) {
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(kFull, acc, off));
    } else {
#pragma unroll
        for (int off = 1; off < 16; off <<= 1) acc = __fadd_rn(acc, __shfl_xor_sync(kFull, acc, off));
    }
    const float res = finish_distance<kMetric, kExact>(acc, qsq, xsq);
    if (idx < cnt && j == 0u) cdist[slots[idx]] = res;
}

// A row warp's rows of one pass, by width (128 and 96, the benchmark's, have
// their own code).
__device__ __forceinline__ void slice_load(const DeviceGraph& g, const uint32_t* cvid, uint32_t p, uint32_t cnt,
                                           RowRegs& x) {
    const uint32_t nchunks = g.dim >> 4;
    if (nchunks == 8u) row8_load<8>(g, cvid, p, cnt, nchunks, x);
    else if (nchunks == 6u) row8_load<6>(g, cvid, p, cnt, nchunks, x);
    else row8_load<0>(g, cvid, p, cnt, nchunks, x);
}

template <int kMetric, bool kExact>
__device__ __forceinline__ void slice_distance(const DeviceGraph& g, const float* __restrict__ q, float qsq,
                                               const uint32_t* cvid, float* cdist, uint32_t p, uint32_t cnt,
                                               RowRegs& x) {
    const uint32_t nchunks = g.dim >> 4;
    if (nchunks == 8u) row8_distance<kMetric, kExact, 8>(g, q, qsq, cvid, cdist, p, cnt, nchunks, x);
    else if (nchunks == 6u) row8_distance<kMetric, kExact, 6>(g, q, qsq, cvid, cdist, p, cnt, nchunks, x);
    else row8_distance<kMetric, kExact, 0>(g, q, qsq, cvid, cdist, p, cnt, nchunks, x);
}

// ---------------------------------------------------------------------------
// Team search (warps per query > 1): a CTA of kG row warps and one queue warp
// (warp 0, the leader) searches one query. The leader publishes commands here
// and all warps meet at a named barrier. kCmdDist: every warp of the CTA takes
// the 8-row passes of a distance batch in turn (warp w: passes w, w + W, ...;
// upper levels, and level 0 of graphs without fixed-stride rows), each row by
// one warp with the same code, so distances are bit-identical to one warp's.
// kCmdLevel0: the row warps enter the level-0 loop (l0_team_rows) and leave it
// when the leader ends it. kCmdQuit: no queries are left.
// ---------------------------------------------------------------------------
enum : uint32_t { kCmdDist = 0, kCmdLevel0 = 1, kCmdQuit = 2 };

struct CoopCtl {
    const uint32_t* cvid;
    float* cdist;
    uint32_t cnt;
    float qsq;
    uint32_t cmd;
    uint32_t next;      // level 0: vertex to expand (kVidMask: the loop ends)
    uint32_t pf;        // level 0: vertex expected to be expanded after it (kVidMask: none)
    uint32_t list_n;    // level 0: ids put in the visited bitset since the last clear
    uint32_t evals;     // level 0: distance evaluations
    uint32_t row_ids;   // level 0: ids in the rows expanded
    uint32_t lead;      // helped search: the leader's warp
    uint32_t pad[3];
    // Level 0, one part of each per row warp: the unvisited ids of the expected row;
    // the new ids of the row expanded and their slots.
    uint32_t spec[kPadRow];
    uint32_t ids[kPadRow];
    uint32_t slots[kPadRow];
};
constexpr uint32_t kCoopWords = sizeof(CoopCtl) / 4;
static_assert(sizeof(CoopCtl) % 16 == 0, "the control block keeps the regions after it aligned");
constexpr int kCoopBarrier = 1;   // commands: every warp of the team waits
constexpr int kRowsBarrier = 2;   // level 0, A: the row warps have written (they do not wait)
constexpr int kNextBarrier = 3;   // level 0, B: the leader has published (it does not wait)

__device__ __forceinline__ void coop_barrier(int warps) {
    asm volatile("barrier.sync %0, %1;" ::"r"(kCoopBarrier), "r"(warps * 32) : "memory");
}
__device__ __forceinline__ void team_arrive(int barrier, int warps) {
    asm volatile("barrier.arrive %0, %1;" ::"r"(barrier), "r"(warps * 32) : "memory");
}
__device__ __forceinline__ void team_wait(int barrier, int warps) {
    asm volatile("barrier.sync %0, %1;" ::"r"(barrier), "r"(warps * 32) : "memory");
}

// kG: row warps of the team (0: one warp searches alone).
template <int kMetric, bool kExact, bool kStage, int kG>
__device__ __forceinline__ void dist_call(const DeviceGraph& g, const float* __restrict__ q, float qsq,
                                          const uint32_t* cvid, float* cdist, uint32_t cnt, Stage& st, int* error,
                                          CoopCtl* coop) {
    if (kG == 0) {
        batch_distances<kMetric, kExact, kStage>(g, q, qsq, cvid, cdist, cnt, st, error);
        return;
    }
    if (lane_id() == 0) {
        coop->cvid = cvid;
        coop->cdist = cdist;
        coop->cnt = cnt;
        coop->qsq = qsq;
        coop->cmd = kCmdDist;
    }
    coop_barrier(kG + 1);   // start
    batch_distances<kMetric, kExact, false, false, true>(g, q, qsq, cvid, cdist, cnt, st, error, nullptr, 0u, kG + 1);
    coop_barrier(kG + 1);   // done
}

// ---------------------------------------------------------------------------
// Visited set (subsystem c): exact, in two tiers.
//   1. A bucketed table in shared memory. vid -> p = (vid * odd) mod 2^kbits is
//      a bijection, so (bucket A = high tbits bits of p, quotient Q = the other
//      kbits - tbits bits) identifies vid exactly; a bucket is 4 uint16 slots
//      (8 bytes, one load), 0xFFFF marks an empty slot. When the quotient has
//      at most 14 bits, an id whose bucket A is full goes to a second bucket
//      B = A ^ alt(Q), stored as Q | 0x8000: the flag keeps it apart from
//      B's own ids (whose slots hold flag-free quotients), and B with Q gives
//      back A and so the id. Buckets only fill up, never drain, until clear():
//      an id absent from A while A has a free slot was never visited (it would
//      only have gone to B with A full), likewise for B.
//   2. The slot's bitset in HBM (atomicOr = test_and_set,
//      containers/version_tag_table.hpp:128-132), used for ids whose buckets
//      are full.
// Ids set in the bitset are listed so clear() (a version bump in the
// reference, version_tag_table.hpp:142-148) zeroes only the words it touched,
// or the whole bitset if the list overflowed. With no table (tbits == 0)
// every id goes to the bitset.
// ---------------------------------------------------------------------------
constexpr uint32_t kVisitedMul = 0x9E3779B1u;   // odd: multiplication mod 2^k is a bijection
constexpr uint32_t kAltFlag = 0x8000u;          // slot holds an id whose first bucket was full

// Permutation space of the table for a graph of n vertices and a table of
// 16 << table_log bytes (2^(table_log + 1) buckets of 8 bytes): returns kbits
// (>= log2 n and > the bucket bits), or 0 when a quotient would not fit in
// 15 bits (table too small for n).
__host__ __device__ inline uint32_t visited_kbits(uint32_t n, uint32_t table_log) {
    uint32_t kb = 1;
    #pragma unroll 1
    while (kb < 32 && (1ull << kb) < n) ++kb;
    if (table_log == 0) return kb;
    const uint32_t tbits = table_log + 1;
    if (kb < tbits + 1) kb = tbits + 1;
    return kb - tbits > 15 ? 0u : kb;
}

struct Visited {
    uint2* tab;         // shared-memory buckets (4 uint16 slots each)
    uint32_t tbits;     // log2 of the bucket count (0: no table)
    uint32_t kbits;     // log2 of the permutation space
    uint32_t kmask;     // 2^kbits - 1
    uint32_t* bits;
    uint32_t* list;
    uint32_t list_n;
    uint32_t list_cap;
    uint64_t words;
    bool global_used;
    bool list_overflow;
    uint32_t spills;
};

// One id's place in the table: its first bucket, its second (~0u when the
// quotient leaves no second choice) and its quotient.
struct TableWalk {
    uint32_t a;
    uint32_t b;
    uint32_t q;
};

__device__ __forceinline__ TableWalk table_walk(const Visited& vs, uint32_t vid) {
    const uint32_t p = (vid * kVisitedMul) & vs.kmask;
    const uint32_t qbits = vs.kbits - vs.tbits;
    TableWalk w;
    w.a = p >> qbits;
    w.q = p & ((1u << qbits) - 1u);
    // alt(Q): the second bucket's offset from the quotient's bits (0 would
    // give B == A: no second choice for that quotient).
    const uint32_t h = (w.q * 0x2545F491u) >> (32u - vs.tbits);
    w.b = (qbits <= 14 && h != 0) ? (w.a ^ h) : 0xffffffffu;
    return w;
}

// Both buckets read at once (at most one CAS): 1 if the id is present (Q in
// A, or Q | flag in B), 0 if it was inserted now (into A while A has a free
// slot, else into B), 2 if both are full (the bitset decides), -1 if another
// lane filled the chosen slot meanwhile (read again). A match in B is the id
// itself whatever A holds: (B, Q) gives back A.
__device__ __forceinline__ uint32_t zero_half(uint32_t x) {   // nonzero iff a 16-bit half of x is 0
    return (x - 0x00010001u) & ~x & 0x80008000u;
}

// A bucket's slots fill in order (low half of x first, high half of y last),
// so it is full once the last one is taken, and comparisons give the first
// free slot.
// The packed compare intrinsics are several instructions each on sm_100; a test
// is about 55 instructions this way instead of 90 (1M x 128, queue 100, 10,000
// queries: 4.34 -> 4.25 ms at 128 registers; queue 400: 14.23 -> 13.97 ms).
constexpr uint32_t kHighFree = 0xFFFF0000u;   // a word at or above: its high slot is free

__device__ __forceinline__ uint32_t bucket_match(uint2 b, uint32_t pattern) {
    return zero_half(b.x ^ pattern) | zero_half(b.y ^ pattern);
}

__device__ __forceinline__ int table_try(const Visited& vs, const TableWalk& w) {
    const bool has_b = w.b != 0xffffffffu;
    const uint2 ba = vs.tab[w.a];
    const uint2 bb = has_b ? vs.tab[w.b] : make_uint2(0u, 0u);   // full, no flagged value
    const uint32_t fq = w.q | kAltFlag;
    if (bucket_match(ba, w.q * 0x10001u) | bucket_match(bb, fq * 0x10001u)) return 1;
    uint32_t bucket = w.a, val = w.q;
    uint2 bk = ba;
    if (ba.y < kHighFree) {
        // A is full (for good): B decides.
        if (bb.y < kHighFree) return 2;
        bucket = w.b;
        val = fq;
        bk = bb;
    }
    const uint32_t wi = bk.x < kHighFree ? 1u : 0u;
    const uint32_t old = wi ? bk.y : bk.x;
    const uint32_t desired = old == 0xFFFFFFFFu ? (kHighFree | val) : ((old & 0xFFFFu) | (val << 16));
    uint32_t* word = reinterpret_cast<uint32_t*>(vs.tab + bucket) + wi;
    return atomicCAS(word, old, desired) == old ? 0 : -1;
}

// Returns 1 if vid is in the table, 0 if it was inserted now, 2 if its
// buckets are full (the bitset decides). Every retry follows a slot filled
// by another lane, so the loop ends within the 8 slots of the two buckets.
__device__ __forceinline__ int table_test_insert(const Visited& vs, uint32_t vid) {
    const TableWalk w = table_walk(vs, vid);
    #pragma unroll 1
    for (int step = 0; step < 24; ++step) {
        const int r = table_try(vs, w);
        if (r >= 0) return r;
    }
    return 2;
}

// test_and_set for one id per lane (act lanes hold distinct vids); all lanes
// call. Returns true in the lanes whose id was not yet visited.
__device__ __forceinline__ bool visited_test_and_set(Visited& vs, uint32_t vid, bool act) {
    const int lane = lane_id();
    bool is_new = false;
    bool in_bits = false;
    if (act) {
        const int t = vs.tbits ? table_test_insert(vs, vid) : 2;
        if (t == 0) {
            is_new = true;
        } else if (t == 2) {
            const uint32_t mask = 1u << (vid & 31);
            const uint32_t old = atomicOr(vs.bits + (vid >> 5), mask);
            is_new = !(old & mask);
            in_bits = is_new;
        }
    }
    const uint32_t b = __ballot_sync(kFull, in_bits);
    if (b) {
        const uint32_t pos = vs.list_n + __popc(b & ((1u << lane) - 1u));
        if (in_bits && pos < vs.list_cap) vs.list[pos] = vid;
        const uint32_t total = vs.list_n + __popc(b);
        if (total > vs.list_cap) vs.list_overflow = true;
        vs.list_n = min(total, vs.list_cap);
        vs.global_used = true;
    }
    __syncwarp();
    return is_new;
}

// set(): mark one id (all lanes call with the same vid).
__device__ __forceinline__ void visited_set(Visited& vs, uint32_t vid) {
    visited_test_and_set(vs, vid, lane_id() == 0);
}

// table_test_insert for two distinct ids per lane, the two walks
// interleaved. r0/r1 as table_test_insert's return values (-1: inactive).
__device__ __forceinline__ void table_test_insert2(const Visited& vs, uint32_t v0, bool a0, uint32_t v1, bool a1,
                                                   int* r0, int* r1) {
    const TableWalk w0 = table_walk(vs, a0 ? v0 : 0u), w1 = table_walk(vs, a1 ? v1 : 0u);
    int t0 = a0 ? -1 : -2, t1 = a1 ? -1 : -2;
    #pragma unroll 1
    for (int step = 0; step < 24 && (t0 == -1 || t1 == -1); ++step) {
        if (t0 == -1) t0 = table_try(vs, w0);
        if (t1 == -1) t1 = table_try(vs, w1);
    }
    *r0 = a0 ? (t0 < 0 ? 2 : t0) : -1;
    *r1 = a1 ? (t1 < 0 ? 2 : t1) : -1;
}

// test_and_set for two ids per lane; all the ids of the warp are distinct.
__device__ __forceinline__ void visited_test_and_set2(Visited& vs, uint32_t v0, bool a0, uint32_t v1, bool a1,
                                                      bool* new0, bool* new1) {
    const int lane = lane_id();
    int t0 = a0 ? 2 : -1, t1 = a1 ? 2 : -1;
    if (vs.tbits) table_test_insert2(vs, v0, a0, v1, a1, &t0, &t1);
    // Both bitset tests are issued before either result is used: one DRAM latency
    // an expansion in place of two (1M x 128, 10,000 queries, 4 KB table: queue 400
    // 11.6 -> 10.6 ms, queue 100 3.22 -> 3.05 ms).
    const uint32_t mask0 = 1u << (v0 & 31), mask1 = 1u << (v1 & 31);
    uint32_t old0 = ~0u, old1 = ~0u;
    if (t0 == 2) old0 = atomicOr(vs.bits + (v0 >> 5), mask0);
    if (t1 == 2) old1 = atomicOr(vs.bits + (v1 >> 5), mask1);
    const bool in0 = !(old0 & mask0), in1 = !(old1 & mask1);
    const bool n0 = t0 == 0 || in0, n1 = t1 == 0 || in1;
    const uint32_t b0 = __ballot_sync(kFull, in0), b1 = __ballot_sync(kFull, in1);
    if (b0 | b1) {
        const uint32_t lt = (1u << lane) - 1u;
        const uint32_t pos0 = vs.list_n + __popc(b0 & lt);
        const uint32_t pos1 = vs.list_n + __popc(b0) + __popc(b1 & lt);
        if (in0 && pos0 < vs.list_cap) vs.list[pos0] = v0;
        if (in1 && pos1 < vs.list_cap) vs.list[pos1] = v1;
        const uint32_t total = vs.list_n + __popc(b0) + __popc(b1);
        if (total > vs.list_cap) vs.list_overflow = true;
        vs.list_n = min(total, vs.list_cap);
        vs.global_used = true;
    }
    __syncwarp();
    *new0 = n0;
    *new1 = n1;
}

// Whether an id is unvisited, without marking it. While other warps insert, an
// id they are inserting may still read as unvisited.
__device__ __forceinline__ bool visited_open(const Visited& vs, uint32_t vid) {
    if (vs.tbits) {
        const TableWalk w = table_walk(vs, vid);
        const uint2 ba = vs.tab[w.a];
        const uint2 bb = w.b != 0xffffffffu ? vs.tab[w.b] : make_uint2(0u, 0u);
        if (bucket_match(ba, w.q * 0x10001u) | bucket_match(bb, (w.q | kAltFlag) * 0x10001u)) return false;
        if (ba.y >= kHighFree || bb.y >= kHighFree) return true;
    }
    return !((__ldcg(vs.bits + (vid >> 5)) >> (vid & 31)) & 1u);
}

// test_and_set for one id per lane of one warp of a team, other warps doing
// the same for other ids: the ids put in the bitset are listed through the
// team's shared count (which may pass list_cap: the list then overflowed).
__device__ __forceinline__ bool team_test_and_set(const Visited& vs, uint32_t* list_n, uint32_t vid, bool act) {
    bool is_new = false;
    if (act) {
        const int t = vs.tbits ? table_test_insert(vs, vid) : 2;
        is_new = t == 0;
        if (t == 2) {
            const uint32_t mask = 1u << (vid & 31);
            is_new = !(atomicOr(vs.bits + (vid >> 5), mask) & mask);
            if (is_new) {
                const uint32_t pos = atomicAdd(list_n, 1u);
                if (pos < vs.list_cap) vs.list[pos] = vid;
            }
        }
    }
    __syncwarp();
    return is_new;
}

__device__ __forceinline__ void table_reset(const Visited& vs) {
    if (vs.tbits) {
        // Two buckets per 16-byte store.
        uint4* t4 = reinterpret_cast<uint4*>(vs.tab);
        const uint32_t n = 1u << (vs.tbits - 1);
        #pragma unroll 1
        for (uint32_t i = lane_id(); i < n; i += 32) t4[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
    }
}

__device__ inline void visited_clear(Visited& vs) {
    const int lane = lane_id();
    __syncwarp();
    table_reset(vs);
    if (vs.global_used) {
        if (vs.list_overflow) {
            uint4* w4 = reinterpret_cast<uint4*>(vs.bits);
            const uint64_t n4 = vs.words / 4;
            #pragma unroll 1
            for (uint64_t i = lane; i < n4; i += 32) w4[i] = make_uint4(0, 0, 0, 0);
        } else {
            // Eight ids a lane are read before their words are written (the compiler
            // cannot move a read past a write): one latency in place of eight (1M x 128,
            // queue 400, 4 KB table: 102,000 -> 20,000 cycles a query).
            #pragma unroll 1
            for (uint32_t i = lane; i < vs.list_n; i += 256) {
                uint32_t id[8];
#pragma unroll
                for (uint32_t t = 0; t < 8; ++t) id[t] = i + 32u * t < vs.list_n ? __ldcg(vs.list + i + 32u * t) : kVidMask;
#pragma unroll
                for (uint32_t t = 0; t < 8; ++t)
                    if (id[t] != kVidMask) vs.bits[id[t] >> 5] = 0u;
            }
        }
        vs.spills++;
    }
    vs.list_n = 0;
    vs.global_used = false;
    vs.list_overflow = false;
    __threadfence_block();
    __syncwarp();
}

// Collect the not-yet-visited ids of row[start, len) (CSR order, first
// occurrence wins, marking them visited) into cvid[0, *cnt), at most
// kCandBatch of them; *consumed reports how far it got. The ids of row[0, 32)
// and row[32, 64) may be passed in preloaded (ids0/ids1, one per lane).
__device__ __forceinline__ void collect_unvisited(const DeviceGraph& g, Visited& vs, const uint32_t* __restrict__ row,
                                                  uint32_t len, uint32_t start, uint32_t* cvid, uint32_t* cnt,
                                                  uint32_t* consumed, int* error, uint32_t ids0, uint32_t ids1,
                                                  bool have_ids) {
    const int lane = lane_id();
    uint32_t c = 0;
    uint32_t i = start;
    #pragma unroll 1
    while (i < len && c + 32 <= kCandBatch) {
        const uint32_t idx = i + lane;
        const bool act = idx < len;
        uint32_t vid = 0xffffffffu;
        if (act) vid = (have_ids && i == 0) ? ids0 : (have_ids && i == 32) ? ids1 : __ldg(row + idx);
        if (act && vid >= g.n) set_error(error, kErrBadVid);
        const uint32_t peers = __match_any_sync(kFull, vid);
        const bool first = act && ((peers & ((1u << lane) - 1u)) == 0) && vid < g.n;
        const bool is_new = visited_test_and_set(vs, vid, first);
        const uint32_t b = __ballot_sync(kFull, is_new);
        if (is_new) cvid[c + __popc(b & ((1u << lane) - 1u))] = vid;
        c += __popc(b);
        i += 32;
    }
    __syncwarp();
    *cnt = c;
    *consumed = min(i, len);
}

// collect_unvisited for a whole level-0 row of at most 64 distinct ids,
// preloaded as row[lane] (ids0) and row[32 + lane] (ids1), 0xffffffff past
// len: one pass, two ids per lane. Ids are distinct, so the order in which
// lanes insert them cannot change which are new; the new ones are written to
// cvid in row order. Returns their count.
__device__ __forceinline__ uint32_t collect_row64_unique(const DeviceGraph& g, Visited& vs, uint32_t ids0,
                                                         uint32_t ids1, uint32_t len, uint32_t* cvid, int* error) {
    const int lane = lane_id();
    const bool in0 = static_cast<uint32_t>(lane) < len, in1 = static_cast<uint32_t>(lane) + 32u < len;
    if ((in0 && ids0 >= g.n) || (in1 && ids1 >= g.n)) set_error(error, kErrBadVid);
    bool n0, n1;
    visited_test_and_set2(vs, ids0, in0 && ids0 < g.n, ids1, in1 && ids1 < g.n, &n0, &n1);
    const uint32_t b0 = __ballot_sync(kFull, n0), b1 = __ballot_sync(kFull, n1);
    const uint32_t lt = (1u << lane) - 1u;
    if (n0) cvid[__popc(b0 & lt)] = ids0;
    if (n1) cvid[__popc(b0) + __popc(b1 & lt)] = ids1;
    __syncwarp();
    return __popc(b0) + __popc(b1);
}

// ---------------------------------------------------------------------------
// Candidate queue (subsystem b). Sorted ascending by (dist, vid) in shared
// memory, one 8-byte entry {vid word, dist bits} per candidate, so a search
// step, a move or a pop test is one load; bit 31 of the vid word marks
// "explored". T = the first min(n, L)
// entries. Entries past L that tie the worst distance lb are entries the
// reference evicted from its top-L heap but still holds in its unexplored
// heap; they stay expandable until lb drops. Any entry worse than lb is dead
// and trimmed. At most L entries can tie lb, so 2L slots always suffice.
// ---------------------------------------------------------------------------
struct Queue {
    uint2* e;        // entries {vid word, dist bits}: one 8-byte access per entry
    uint32_t n;
    uint32_t L;
    uint32_t cap;
    uint32_t hint;   // no unexplored entry before this index
    float lb;        // d[L-1] once n >= L
};

__device__ __forceinline__ float ent_d(uint2 w) { return __uint_as_float(w.y); }
__device__ __forceinline__ uint2 make_ent(float d, uint32_t v) { return make_uint2(v, __float_as_uint(d)); }

__device__ __forceinline__ uint32_t queue_lower_bound(const Queue& q, float d, uint32_t v) {
    const int lane = lane_id();
    uint32_t lo = 0, hi = q.n;
    #pragma unroll 1
    while (hi - lo > 32) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t idx = lo + lane * step;
        bool less = false;
        if (idx < hi) {
            const uint2 w = q.e[idx];
            less = entry_less(ent_d(w), w.x, d, v);
        }
        const int c = __popc(__ballot_sync(kFull, less));
        const uint32_t new_lo = c == 0 ? lo : lo + (c - 1) * step + 1;
        const uint32_t new_hi = min(hi, lo + c * step);
        lo = new_lo;
        hi = new_hi;
    }
    const uint32_t idx = lo + lane;
    bool less = false;
    if (idx < hi) {
        const uint2 w = q.e[idx];
        less = entry_less(ent_d(w), w.x, d, v);
    }
    return lo + __popc(__ballot_sync(kFull, less));
}

// Insert (d, v); the caller has already applied try_push's rejection test.
__device__ __forceinline__ bool queue_insert(Queue& q, float d, uint32_t v, int* error) {
    const int lane = lane_id();
    if (q.n >= q.cap) {
        set_error(error, kErrQueue);
        return false;
    }
    const uint32_t pos = queue_lower_bound(q, d, v);
    #pragma unroll 1
    for (int end = static_cast<int>(q.n); end > static_cast<int>(pos); end -= 32) {
        const int s = max(static_cast<int>(pos), end - 32);
        const int idx = s + lane;
        const bool act = idx < end;
        uint2 ww = make_uint2(0u, 0u);
        if (act) ww = q.e[idx];
        __syncwarp();
        if (act) q.e[idx + 1] = ww;
        __syncwarp();
    }
    if (lane == 0) q.e[pos] = make_ent(d, v & kVidMask);
    __syncwarp();
    q.n++;
    if (pos < q.hint) q.hint = pos;
    if (q.n >= q.L) {
        q.lb = ent_d(q.e[q.L - 1]);
        if (q.n > q.L) {
            uint32_t newn = q.n;
            #pragma unroll 1
            for (uint32_t base = q.L; base < q.n; base += 32) {
                const uint32_t idx = base + lane;
                const bool dead = idx < q.n && ent_d(q.e[idx]) > q.lb;
                const uint32_t b = __ballot_sync(kFull, dead);
                if (b) { newn = base + __ffs(b) - 1; break; }
            }
            q.n = newn;
        }
    }
    return true;
}

// First unexplored entry at or after `from`, or -1.
__device__ __forceinline__ int queue_find_unexplored(const Queue& q, uint32_t from) {
    const int lane = lane_id();
    #pragma unroll 1
    for (uint32_t base = from; base < q.n; base += 32) {
        const uint32_t idx = base + lane;
        const bool un = idx < q.n && !(q.e[idx].x & kExplored);
        const uint32_t b = __ballot_sync(kFull, un);
        if (b) return static_cast<int>(base + __ffs(b) - 1);
    }
    return -1;
}

// pop_best_unexplored_entry + should_terminate (std_candidate_queue.hpp:398-406,
// 503-513): the first unexplored entry in order, or -1 when the reference's
// unexplored heap holds nothing at distance <= lb.
__device__ __forceinline__ int queue_pop(Queue& q) {
    const int p = queue_find_unexplored(q, q.hint);
    if (p < 0) {
        q.hint = q.n;
        return -1;
    }
    if (lane_id() == 0) q.e[p].x |= kExplored;
    __syncwarp();
    q.hint = static_cast<uint32_t>(p) + 1;
    return p;
}

// pop_best_unexplored_entry, plus a peek at the entry that would come next if
// nothing better is inserted meanwhile (-1 when none), in one scan.
__device__ __forceinline__ int queue_pop_peek(Queue& q, int* next) {
    const int lane = lane_id();
    int first = -1;
    *next = -1;
    uint32_t base = q.hint;
    #pragma unroll 1
    for (; base < q.n; base += 32) {
        const uint32_t idx = base + lane;
        const bool un = idx < q.n && !(q.e[idx].x & kExplored);
        uint32_t b = __ballot_sync(kFull, un);
        if (b) {
            if (first < 0) {
                first = static_cast<int>(base + __ffs(b) - 1);
                b &= b - 1;
            }
            if (b) {
                *next = static_cast<int>(base + __ffs(b) - 1);
                break;
            }
        }
    }
    if (first < 0) {
        q.hint = q.n;
        return -1;
    }
    if (lane == 0) q.e[first].x |= kExplored;
    __syncwarp();
    q.hint = static_cast<uint32_t>(first) + 1;
    return first;
}

// try_push for a whole batch at once (std_candidate_queue.hpp:358-388), in
// two steps: queue_accept decides which candidates the sequential pushes
// would accept, queue_merge applies them.
// Sequentially, candidate j is rejected iff T already holds L entries at
// distance <= d_j. A rejected candidate never enters T, and every later
// candidate at a distance >= a rejected one is rejected too, so candidate j
// is accepted iff
//     #{e in T : e.dist <= d_j} + #{i < j : d_i <= d_j}  <  L,
// which every lane evaluates independently. The accepted candidates are then
// merged into the sorted array in one pass; trimming the result at the new
// lb yields exactly the state the sequential pushes leave (entries trimmed
// in between are worse than every later lb).
//
// exact_pre: the second sum for candidate j < cnt, four candidates a step;
// the slots past cnt that the last step reads are not before j. (A walk over
// the earlier improving lanes by shuffles took a step per candidate.)
//
// queue_accept writes the accepted candidates (m <= cnt <= kCandBatch), in
// candidate order, to bd/bv and returns m.
__device__ __forceinline__ uint32_t exact_pre(const float* cdist, uint32_t cnt, uint32_t j, float d) {
    uint32_t pre = 0;
    #pragma unroll 1
    for (uint32_t i = 0; i < cnt; i += 4) {
        const float4 c = *reinterpret_cast<const float4*>(cdist + i);
        pre += (i < j) & (c.x <= d) ? 1u : 0u;
        pre += (i + 1u < j) & (c.y <= d) ? 1u : 0u;
        pre += (i + 2u < j) & (c.z <= d) ? 1u : 0u;
        pre += (i + 3u < j) & (c.w <= d) ? 1u : 0u;
    }
    return pre;
}

__device__ inline uint32_t queue_accept(const Queue& q, const uint32_t* cvid, const float* cdist, uint32_t cnt,
                                        float* bd, uint32_t* bv) {
    const int lane = lane_id();
    const uint32_t lt_mask = (1u << lane) - 1u;
    const uint32_t tn = min(q.n, q.L);
    // Only candidates closer than lb can enter a full T, and the earlier
    // candidates a closer one must be counted against are closer as well:
    // pre_j only involves "improving" candidates. Late in a search most
    // batches have none.
    const float lim = q.n >= q.L ? q.lb : INFINITY;
    uint32_t m = 0;
    uint32_t improving_before = 0;   // improving candidates in earlier chunks
    #pragma unroll 1
    for (uint32_t base = 0; base < cnt; base += 32) {
        const uint32_t j = base + lane;
        const bool valid = j < cnt;
        const float d = valid ? cdist[j] : INFINITY;
        const uint32_t v = valid ? cvid[j] : 0u;
        const bool improving = valid && d < lim;
        uint32_t imask = __ballot_sync(kFull, improving);
        if (imask == 0 && improving_before == 0) continue;
        // #{e in T : e.dist <= d} < L - pre  <=>  T[L-pre-1].dist > d (or T is
        // shorter than L-pre). pre = #{i < j : d_i <= d_j} is at most ub, the
        // number of earlier improving candidates, and the test is monotone in
        // pre: a lane accepted with ub is accepted, and only lanes it leaves
        // undecided need the exact count.
        const uint32_t ub = improving_before + __popc(imask & lt_mask);
        bool acc = false;
        if (improving && ub < q.L) {
            const uint32_t idx = q.L - ub - 1;
            acc = idx >= tn || ent_d(q.e[idx]) > d;
        }
        const bool undecided = improving && !acc && ub != 0;
        if (__any_sync(kFull, undecided)) {
            const uint32_t pre = exact_pre(cdist, cnt, j, d);
            if (undecided && pre < q.L) {
                const uint32_t idx = q.L - pre - 1;
                acc = idx >= tn || ent_d(q.e[idx]) > d;
            }
        }
        const uint32_t b = __ballot_sync(kFull, acc);
        if (acc) {
            const uint32_t k = m + __popc(b & lt_mask);
            bd[k] = d;
            bv[k] = v;
        }
        m += __popc(b);
        improving_before += __popc(imask);
    }
    __syncwarp();
    return m;
}

// Number of entries of the sorted array q[0, n) before (d, v) by (dist, vid).
__device__ __forceinline__ uint32_t old_lower_bound(const Queue& q, float d, uint32_t v) {
    uint32_t lo = 0, hi = q.n;
    #pragma unroll 1
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        const uint2 w = q.e[mid];
        if (entry_less(ent_d(w), w.x, d, v)) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// Places the m <= kFew sorted entries of bd/bv into the sorted array q[0, n), n
// >= 1: an old entry moves up by the number of batch entries before it; lane r
// finds batch entry r's rank among the old ones from a ballot a chunk and writes
// it last. Chunks of 32 entries go tail first; a chunk's outputs lie at or after
// its own first position, so the next chunk is read before they are written.
// Chunks before the first batch entry are not touched. Entries past the capacity
// are dropped. Returns the position of the smallest batch entry.
// Most merges have one to four entries: counting by comparison against that many
// registers replaces a binary search of 7-10 dependent shared-memory loads and
// two cross-lane reductions a chunk.
// (1M x 128, 10,000 queries: queue 100 4.25 -> 4.00 ms, queue 400 13.97 -> 13.20
// ms, with the ranking by four entries a step in queue_merge.)
template <int kFew>
__device__ __forceinline__ uint32_t queue_place_few(const Queue& q, const float* bd, const uint32_t* bv, uint32_t m) {
    const uint32_t lane = static_cast<uint32_t>(lane_id());
    const uint32_t n = q.n, cap = q.cap;
    float rd[kFew];
    uint32_t rv[kFew];
#pragma unroll
    for (int r = 0; r < kFew; ++r) {
        // Past m: after every entry (an entry at distance NaN, which compares
        // false with all, counts as after the whole batch).
        rd[r] = static_cast<uint32_t>(r) < m ? bd[r] : INFINITY;
        rv[r] = static_cast<uint32_t>(r) < m ? (bv[r] & kVidMask) : 0xffffffffu;
    }
    uint32_t rank = 0;        // lane r: old entries before batch entry r
    bool found = false;
    uint32_t cb = (n - 1u) & ~31u;
    uint2 w = make_uint2(0u, 0u);
    if (cb + lane < n) w = q.e[cb + lane];
    #pragma unroll 1
    for (;;) {
        const uint32_t idx = cb + lane;
        const bool in = idx < n;
        uint2 wn = make_uint2(0u, 0u);
        if (cb) wn = q.e[cb - 32u + lane];
        const float wd = ent_d(w);
        const uint32_t wv = w.x & kVidMask;
        uint32_t c = 0;       // batch entries before this one
        uint32_t before = 0;  // lane r: this chunk's entries before batch entry r
        bool any0 = false;
#pragma unroll
        for (int r = 0; r < kFew; ++r) {
            const bool less = (wd < rd[r]) | ((wd == rd[r]) & (wv < rv[r]));   // this entry is before batch entry r
            c += less ? 0u : 1u;
            const uint32_t b = __ballot_sync(kFull, in & less);
            if (lane == static_cast<uint32_t>(r)) before = b;
            if (r == 0) any0 = b != 0u;
        }
        c = min(c, m);
        if (!found && before) {
            rank = cb + __popc(before);
            found = true;
        }
        __syncwarp();   // the next chunk has been read
        if (in && c && idx + c < cap) q.e[idx + c] = w;
        if (any0 || cb == 0u) break;
        cb -= 32u;
        w = wn;
    }
    __syncwarp();
    if (lane < m && rank + lane < cap) q.e[rank + lane] = make_ent(bd[lane], bv[lane]);
    __syncwarp();
    return __shfl_sync(kFull, rank, 0);
}

// The same for any m <= kCandBatch: batch entries find their positions by binary
// search, every output gathers its source.
__device__ __forceinline__ int queue_place_many(const Queue& q, const float* bd, const uint32_t* bv, uint32_t m) {
    const int lane = lane_id();
    // Final positions of the batch entries: rank in the old array + rank in
    // the batch (sorted, distinct); lanes past m hold a sentinel above every
    // position.
    constexpr int kNoPos = 0x7fffffff;
    int posb0 = kNoPos, posb1 = kNoPos;
    if (static_cast<uint32_t>(lane) < m) posb0 = static_cast<int>(old_lower_bound(q, bd[lane], bv[lane]) + lane);
    const bool two = m > 32u;
    if (two && static_cast<uint32_t>(lane) + 32u < m)
        posb1 = static_cast<int>(old_lower_bound(q, bd[lane + 32], bv[lane + 32]) + lane + 32u);
    const int p0 = __shfl_sync(kFull, posb0, 0);   // position of the smallest batch entry
    // Output positions [p0, end) change. Output o holds batch entry r when
    // o = posb_r, else the old entry o - #{r : posb_r < o}, which lies at or
    // before o; within a chunk of 32 outputs every lane reads its source
    // before any lane writes. Chunks go tail first: a chunk's sources lie
    // before the outputs of every chunk written earlier.
    const int end = static_cast<int>(min(q.n + m, q.cap));
    const uint32_t lt = (1u << lane) - 1u;
    #pragma unroll 1
    for (int cb = end - 32; cb + 32 > p0; cb -= 32) {
        const uint32_t rel0 = static_cast<uint32_t>(posb0) - static_cast<uint32_t>(cb);
        const uint32_t rel1 = static_cast<uint32_t>(posb1) - static_cast<uint32_t>(cb);
        uint32_t mask = __reduce_or_sync(kFull, rel0 < 32u ? 1u << rel0 : 0u);   // batch outputs in the chunk
        uint32_t nb = __popc(__ballot_sync(kFull, posb0 < cb));                 // batch outputs before it
        if (two) {
            mask |= __reduce_or_sync(kFull, rel1 < 32u ? 1u << rel1 : 0u);
            nb += __popc(__ballot_sync(kFull, posb1 < cb));
        }
        const int before = static_cast<int>(nb + __popc(mask & lt));
        const int o = cb + lane;
        const bool act = o >= p0;
        const bool from_batch = (mask >> lane) & 1u;
        uint2 ww = make_uint2(0u, 0u);
        if (act) ww = from_batch ? make_ent(bd[before], bv[before]) : q.e[o - before];
        __syncwarp();
        if (act) q.e[o] = ww;
    }
    __syncwarp();
    return p0;
}

// Merges the m (<= kCandBatch) accepted entries of bd/bv into the sorted
// array and trims it at the new lb. The batch is first sorted by (dist, vid)
// in place (each lane holds at most two entries in registers). A vid word may
// carry the explored bit (an entry popped before it is merged); ordering
// ignores it.
// Returns true when an entry that may still be live was dropped: with a
// capacity below 2L (the compact layout), entries past the capacity are not
// kept; they are dead unless every kept entry past L ties lb, which is what
// is reported (the caller then hands the query to the full-capacity rerun).
__device__ inline bool queue_merge(Queue& q, float* bd, uint32_t* bv, uint32_t m) {
    const int lane = lane_id();
    if (m == 0) return false;
    const bool truncated = q.n + m > q.cap;
    if (m > 1u) {
        // Each lane ranks at most two of the entries, four at a time against
        // all (entries past m: a sentinel above every one).
        const uint32_t pad = m + static_cast<uint32_t>(lane);
        if (lane < 4 && pad < kCandBatch) {
            bd[pad] = INFINITY;
            bv[pad] = 0xffffffffu;
        }
        __syncwarp();
        const bool h0 = static_cast<uint32_t>(lane) < m, h1 = static_cast<uint32_t>(lane) + 32u < m;
        const float d0 = bd[lane], d1 = bd[lane + 32];
        const uint32_t w0 = bv[lane], w1 = bv[lane + 32];
        uint32_t r0 = 0, r1 = 0;
        #pragma unroll 1
        for (uint32_t i = 0; i < m; i += 4) {
            const float4 bd4 = *reinterpret_cast<const float4*>(bd + i);
            const uint4 bv4 = *reinterpret_cast<const uint4*>(bv + i);
            r0 += entry_less(bd4.x, bv4.x, d0, w0) + entry_less(bd4.y, bv4.y, d0, w0) +
                  entry_less(bd4.z, bv4.z, d0, w0) + entry_less(bd4.w, bv4.w, d0, w0);
            if (m > 32u)
                r1 += entry_less(bd4.x, bv4.x, d1, w1) + entry_less(bd4.y, bv4.y, d1, w1) +
                      entry_less(bd4.z, bv4.z, d1, w1) + entry_less(bd4.w, bv4.w, d1, w1);
        }
        __syncwarp();
        if (h0) {
            bd[r0] = d0;
            bv[r0] = w0;
        }
        if (h1) {
            bd[r1] = d1;
            bv[r1] = w1;
        }
        __syncwarp();
    }
    int p0;
    if (m == 1u && q.n) {
        p0 = static_cast<int>(queue_place_few<1>(q, bd, bv, m));
    } else if (m <= 4u && q.n) {
        p0 = static_cast<int>(queue_place_few<4>(q, bd, bv, m));
    } else {
        p0 = queue_place_many(q, bd, bv, m);
    }
    const uint32_t total = min(q.n + m, q.cap);
    q.n = total;
    if (static_cast<uint32_t>(p0) < q.hint) q.hint = static_cast<uint32_t>(p0);
    if (q.n >= q.L) {
        q.lb = ent_d(q.e[q.L - 1]);
        uint32_t newn = q.n;
        #pragma unroll 1
        for (uint32_t base = q.L; base < q.n; base += 32) {
            const uint32_t idx = base + lane;
            const bool dead = idx < q.n && ent_d(q.e[idx]) > q.lb;
            const uint32_t b = __ballot_sync(kFull, dead);
            if (b) { newn = base + __ffs(b) - 1; break; }
        }
        q.n = newn;
    }
    return truncated && q.n == q.cap;
}

// try_push of a whole batch (bd/bv: scratch for the accepted entries).
__device__ inline bool queue_push_batch(Queue& q, uint32_t* cvid, float* cdist, uint32_t cnt, float* bd, uint32_t* bv,
                                        int* error) {
    (void)error;
    return queue_merge(q, bd, bv, queue_accept(q, cvid, cdist, cnt, bd, bv));
}

// ---------------------------------------------------------------------------
// Row lookup: fetch_level_nbrs (index/compact_structure/hierarchical_graph.hpp:99-108).
// ---------------------------------------------------------------------------
__device__ __forceinline__ const uint32_t* level_row(const DeviceGraph& g, uint32_t vid, uint32_t level,
                                                     uint32_t* len) {
    const uint2 info = __ldg(g.vinfo + vid);
    const uint32_t hl = info.x;
    if (hl == kInvalidLevel || hl < level || hl >= kMaxGroups) {
        *len = 0;
        return g.nbrs;
    }
    const uint64_t row = static_cast<uint64_t>(info.y) * (hl + 1ull) + (hl - level);
    const uint64_t* off = g.offsets[hl];
    const uint64_t b = __ldg(reinterpret_cast<const unsigned long long*>(off + row));
    const uint64_t e = __ldg(reinterpret_cast<const unsigned long long*>(off + row + 1));
    *len = static_cast<uint32_t>(e - b);
    return g.nbrs + b;
}

struct Counters {
    uint32_t dist_evals, upper_rows, upper_row_ids, l0_rows, l0_row_ids, upper_dist_evals;
};

// Accumulates clock64() deltas per phase when enabled (warp-uniform flag);
// the accumulators live in the warp's shared memory, lane 0 updates them.
struct PhaseClock {
    bool on;
    long long t;
    unsigned long long* acc;
    __device__ __forceinline__ void start(bool enabled, unsigned long long* smem_acc) {
        on = enabled;
        acc = smem_acc;
        if (on) {
            if (lane_id() < kPhases) acc[lane_id()] = 0;
            __syncwarp();
            t = clock64();
        }
    }
    __device__ __forceinline__ void lap(int phase) {
        if (on) {
            const long long now = clock64();
            if (lane_id() == 0) acc[phase] += static_cast<unsigned long long>(now - t);
            t = now;
        }
    }
    __device__ __forceinline__ void count(int phase) {
        if (on && lane_id() == 0) acc[phase] += 1;
    }
};

// Shared memory words per warp for a launch.
constexpr uint32_t kPhaseWords = 2 * kPhases;   // kPhases uint64 accumulators

// Staged rows: a 4-word mbarrier slot, then kStageRows rows of dim + kStagePad words.
__host__ __device__ inline uint32_t stage_words(uint32_t dim, uint32_t stage_rows) {
    return stage_rows ? 4u + stage_rows * (dim + kStagePad) : 0u;
}

// The queue's entry array holds an even number of 8-byte entries
// (2 * queue_words(cap) words), so that the regions after it (the visited
// table, read 16 bytes at a time when cleared, the next warp's area) stay
// 16-byte aligned whatever the capacity (dim, the stage and the fixed parts
// are multiples of 4 words).
__host__ __device__ inline uint32_t queue_words(uint32_t cap) { return (cap + 1u) & ~1u; }

__host__ __device__ inline uint32_t warp_smem_words(uint32_t dim, uint32_t cap, uint32_t vh_bits,
                                                    uint32_t stage_rows = 0) {
    return dim + 2 * queue_words(cap) + 4 * kCandBatch + (vh_bits ? 4u * (1u << vh_bits) : 0u) + kPhaseWords +
           stage_words(dim, stage_rows);
}

struct WarpSmem {
    unsigned long long* phase;   // kPhases accumulators (8-byte aligned: first)
    unsigned long long* mbar;    // staging mbarrier (null without staging)
    float* stage;                // staged rows, 16-byte aligned (null without staging)
    float* q;
    uint2* qe;
    uint32_t* cvid;
    float* cdist;
    float* bd;
    uint32_t* bv;
    uint32_t* vh;
    CoopCtl* coop;               // cooperative search's control block (null otherwise)
};

__device__ __forceinline__ WarpSmem carve(float* base, uint32_t dim, uint32_t cap, uint32_t stage_rows = 0) {
    WarpSmem s;
    s.phase = reinterpret_cast<unsigned long long*>(base);
    s.mbar = stage_rows ? reinterpret_cast<unsigned long long*>(base + kPhaseWords) : nullptr;
    s.stage = stage_rows ? base + kPhaseWords + 4 : nullptr;
    s.q = base + kPhaseWords + stage_words(dim, stage_rows);
    s.qe = reinterpret_cast<uint2*>(s.q + dim);
    s.cvid = reinterpret_cast<uint32_t*>(s.q + dim + 2 * queue_words(cap));
    s.cdist = reinterpret_cast<float*>(s.cvid + kCandBatch);
    s.bd = s.cdist + kCandBatch;
    s.bv = reinterpret_cast<uint32_t*>(s.bd + kCandBatch);
    s.vh = s.bv + kCandBatch;
    s.coop = nullptr;
    return s;
}

// The visited set of search slot `slot` (as visited_clear leaves it).
__device__ __forceinline__ Visited visited_init(const SearchArgs& a, const WarpSmem& sm, uint32_t slot) {
    Visited vs;
    vs.tab = reinterpret_cast<uint2*>(sm.vh);
    vs.tbits = a.vh_bits ? a.vh_bits + 1 : 0u;   // a.vh_bits: log2 of the table's 16-byte units
    vs.kbits = a.vk_bits;
    vs.kmask = a.vk_bits >= 32 ? 0xFFFFFFFFu : ((1u << a.vk_bits) - 1u);
    vs.bits = a.vis_bits + static_cast<size_t>(slot) * a.words_per_slot;
    vs.list = a.vis_list + static_cast<size_t>(slot) * a.list_cap;
    vs.list_n = 0;
    vs.list_cap = a.list_cap;
    vs.words = a.words_per_slot;
    vs.global_used = false;
    vs.list_overflow = false;
    vs.spills = 0;
    return vs;
}

// collect_row64_unique for a fixed-stride row (ids0 = slot lane, ids1 = slot 32 +
// lane), counting the expansion.
__device__ __forceinline__ uint32_t collect_pad_row(const DeviceGraph& g, Visited& vs, uint32_t ids0, uint32_t ids1,
                                                    uint32_t* cvid, Counters& ct, int* error) {
    const uint32_t len = __popc(__ballot_sync(kFull, ids0 != 0xffffffffu)) +
                         __popc(__ballot_sync(kFull, ids1 != 0xffffffffu));
    ct.l0_rows++;
    ct.l0_row_ids += len;
    return collect_row64_unique(g, vs, ids0, ids1, len, cvid, error);
}

// Order-preserving unsigned key of a distance (-0 and +0 alike).
__device__ __forceinline__ uint32_t dist_key(float d) {
    const uint32_t u = __float_as_uint(d + 0.0f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ bool head_less(uint32_t ka, uint32_t va, uint32_t kb, uint32_t vb) {
    return ka < kb || (ka == kb && va < vb);
}

// queue_accept over slots [0, cnt) of cvid/cdist (two a lane), plus the smallest
// accepted candidate by (dist, vid), and with kTwo the second smallest: their
// distance keys and vids (~0u when absent). The candidates stay in registers:
// the decision is on the warp's own chain between a row's distances and the
// next row's collection, where a pass through shared memory and a shuffle tree
// for the smallest cost ~250 cycles more than two warp reductions. Before and
// after in the one-warp loop (fixed launches): 1M x 128, 10,000 queries, queue
// 100: 3.41 -> 3.23 ms; queue 400: 12.40 -> 11.81 ms; 96 elements, cosine,
// early stop: 5.56 -> 5.29 ms.
struct Batch {
    float d[2];
    uint32_t v[2];
    uint32_t acc[2];          // accepted lanes of each half
    uint32_t m;               // accepted candidates
    uint32_t k1, v1, k2, v2;
};

template <bool kTwo>
__device__ __forceinline__ void register_accept(const Queue& q, const uint32_t* cvid, const float* cdist, uint32_t cnt,
                                                Batch& s) {
    const uint32_t lane = static_cast<uint32_t>(lane_id());
    const uint32_t lt_mask = (1u << lane) - 1u;
    const uint32_t tn = min(q.n, q.L);
    const float lim = q.n >= q.L ? q.lb : INFINITY;
    s.k1 = s.v1 = s.k2 = s.v2 = 0xffffffffu;
    s.m = 0;
    s.d[0] = lane < cnt ? cdist[lane] : INFINITY;
    s.d[1] = lane + 32u < cnt ? cdist[lane + 32] : INFINITY;
    s.v[0] = cvid[lane];
    s.v[1] = cvid[lane + 32];
    s.acc[0] = s.acc[1] = 0u;
    const uint32_t imp0 = __ballot_sync(kFull, s.d[0] < lim), imp1 = __ballot_sync(kFull, s.d[1] < lim);
    if ((imp0 | imp1) == 0u) return;   // three of four rows improve nothing
    // See queue_accept: ub bounds pre, and only lanes it leaves undecided need
    // the exact count.
    bool open = false;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const bool improving = s.d[t] < lim;
        const uint32_t ub = (t ? __popc(imp0) : 0u) + __popc((t ? imp1 : imp0) & lt_mask);
        bool acc = false;
        if (improving && ub < q.L) {
            const uint32_t idx = q.L - ub - 1;
            acc = idx >= tn || ent_d(q.e[idx]) > s.d[t];
        }
        open |= improving && !acc && ub != 0u;
        s.acc[t] = __ballot_sync(kFull, acc);
    }
    if (__any_sync(kFull, open)) {
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const float d = s.d[t];
            const uint32_t pre = exact_pre(cdist, cnt, lane + 32u * t, d);
            bool acc = false;
            if (d < lim && pre < q.L) {
                const uint32_t idx = q.L - pre - 1u;
                acc = idx >= tn || ent_d(q.e[idx]) > d;
            }
            s.acc[t] = __ballot_sync(kFull, acc);
        }
    }
    s.m = __popc(s.acc[0]) + __popc(s.acc[1]);
    if (s.m == 0u) return;
    uint32_t key0 = (s.acc[0] >> lane) & 1u ? dist_key(s.d[0]) : 0xffffffffu;
    uint32_t key1 = (s.acc[1] >> lane) & 1u ? dist_key(s.d[1]) : 0xffffffffu;
    s.k1 = __reduce_min_sync(kFull, min(key0, key1));
    s.v1 = __reduce_min_sync(kFull, min(key0 == s.k1 ? s.v[0] : 0xffffffffu, key1 == s.k1 ? s.v[1] : 0xffffffffu));
    if (kTwo && s.m > 1u) {
        if (s.v[0] == s.v1) key0 = 0xffffffffu;
        if (s.v[1] == s.v1) key1 = 0xffffffffu;
        s.k2 = __reduce_min_sync(kFull, min(key0, key1));
        s.v2 = __reduce_min_sync(kFull, min(key0 == s.k2 ? s.v[0] : 0xffffffffu,
                                            key1 == s.k2 ? s.v[1] : 0xffffffffu));
    }
}

// The accepted candidates, in slot order, to bd/bv; the one popped already
// (`popped`) with the explored bit.
__device__ __forceinline__ void write_accepted(const Batch& s, uint32_t popped, float* bd, uint32_t* bv) {
    const uint32_t lane = static_cast<uint32_t>(lane_id());
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        if ((s.acc[t] >> lane) & 1u) {
            const uint32_t k = (t ? __popc(s.acc[0]) : 0u) + __popc(s.acc[t] & lt);
            bd[k] = s.d[t];
            bv[k] = s.v[t] | (s.v[t] == popped ? kExplored : 0u);
        }
    }
}

// The last warp of a CTA that still has a query: the CTA's flags, in the first
// warp's phase accumulators (a launch that measures phases has no helpers).
constexpr int kHelpers = 3;   // row warps of a helped search: a CTA of four warps
struct HelpFlags {
    uint32_t taken;   // row warp numbers given to warps without a query
    uint32_t host;    // the first of those warps: its candidate buffers hold the control block
    uint32_t idle;    // warps without a query, host known
    uint32_t quit;    // no warp of the CTA has a query
};
static_assert(sizeof(HelpFlags) <= 4 * kPhaseWords && sizeof(CoopCtl) <= 16 * kCandBatch, "both fit where they lie");

// ---------------------------------------------------------------------------
// Level-0 beam search, pipelined across expansions (single_layer_router.hpp:
// 145-163, beam_loop.hpp:90-119), for graphs whose level-0 rows hold at most 64
// distinct ids. On entry the queue holds the cursor and the cursor is visited.
//
// The reference pops the next entry only after pushing every candidate of the
// current row. That entry is known earlier: once the current batch's
// acceptance is decided, the next pop is the smaller (by dist, vid) of
//   * p2, the first unexplored entry after the one being expanded, and
//   * the smallest accepted candidate of the batch,
// because every other unexplored entry is larger than p2, rejected candidates
// never enter the unexplored heap, and the smallest accepted candidate always
// ends inside the top L (all entries before it are old entries, fewer than L
// by its acceptance). p2 cannot be trimmed by the merge either: if it is the
// smaller, it is at most the smallest accepted candidate, which stays within
// lb. With neither, should_terminate holds (std_candidate_queue.hpp:503-513).
// So the next expansion's row is collected (visited test_and_set; the merge
// does not touch the visited set) and its first rows' loads are issued before
// the current batch is merged, and the merge runs while they are in flight.
// The chosen entry is marked explored where it lies: p2 in the array, a new
// candidate in the batch before the merge places it.
// ---------------------------------------------------------------------------
// Returns true when the compact queue lost a live entry (see queue_merge). With
// kHelp and `help`, the loop ends early once the other warps of the CTA have no
// queries left: hand.first is then the next vertex to expand (marked explored,
// its row not read) and hand.m candidates in bd/bv are still to be merged.
struct Handover {
    uint32_t first;   // kVidMask: the search ran to its end
    uint32_t m;
};

template <int kMetric, bool kExact, bool kRegs, bool kHelp>
__device__ __forceinline__ bool l0_search_pipelined(const SearchArgs& a, Queue& q, Visited& vs, const WarpSmem& sm,
                                                    float qsq, uint32_t cur, Counters& ct, PhaseClock& pc,
                                                    Stage& st, bool help, Handover& hand) {
    extern __shared__ __align__(16) float smem[];
    hand.first = kVidMask;
    hand.m = 0;
    const int lane = lane_id();
    const DeviceGraph& g = a.g;
    const bool l2_next = a.pf_l2 != 0;
    uint32_t* cv = sm.cvid;
    float* cd = sm.cdist;
    // Pop the cursor: the queue's only entry.
    if (lane == 0) q.e[0].x |= kExplored;
    __syncwarp();
    q.hint = 1;
    const uint32_t* pad = g.l0pad + lane;
    uint32_t ids0 = __ldg(pad + static_cast<size_t>(cur) * kPadRow);
    uint32_t ids1 = __ldg(pad + static_cast<size_t>(cur) * kPadRow + 32);
    uint32_t cnt = collect_pad_row(g, vs, ids0, ids1, cv, ct, a.error);
    RowRegs pre;
    dist_preload<kRegs>(g, cv, cnt, pre, l2_next);
    pc.lap(kPhCollect);
    // The predicted entry after the one being expanded: its index (-1: none),
    // vid and ids.
    int p2 = -1;
    uint32_t pf_vid = kVidMask, pf_ids0 = 0u, pf_ids1 = 0u;
    uint32_t p2_key = 0xffffffffu;   // its distance key (~0u: none)
    for (uint32_t it = 0;; ++it) {
        if (it > g.n) { set_error(a.error, kErrBound); break; }
        bool helped = false;
        if (kHelp && help)
            helped = __all_sync(kFull, reinterpret_cast<const volatile HelpFlags*>(smem)->idle == kHelpers);
        if (cnt) batch_distances<kMetric, kExact, false, kRegs, false, true>(g, sm.q, qsq, cv, cd, cnt, st, a.error, &pre);
        ct.dist_evals += cnt;
        pc.lap(kPhDist);
        Batch s;
        register_accept<false>(q, cv, cd, cnt, s);
        const uint32_t m = s.m;
        // The next pop: min(p2, smallest accepted), or termination.
        const bool take_new = head_less(s.k1, s.v1, p2_key, pf_vid);
        uint32_t next = take_new ? s.v1 : kVidMask;
        if (m) write_accepted(s, next, sm.bd, sm.bv);
        if (!take_new && p2 >= 0) {
            next = pf_vid;
            if (lane == 0) q.e[p2].x |= kExplored;
            q.hint = static_cast<uint32_t>(p2) + 1;
        }
        __syncwarp();
        // CandidateEntry::is_invalid ends the loop as the reference's pop of an
        // invalid entry does (cannot occur on validated graphs).
        const bool go = (take_new || p2 >= 0) && next != kVidMask;
        if (kHelp && helped && go) {
            hand.first = next;
            hand.m = m;
            return false;
        }
        uint32_t ncnt = 0;
        if (go) {
            const bool hit = !take_new && next == pf_vid;
            if (hit) pc.count(kPhPrefetchHits);
            ids0 = hit ? pf_ids0 : __ldg(pad + static_cast<size_t>(next) * kPadRow);
            ids1 = hit ? pf_ids1 : __ldg(pad + static_cast<size_t>(next) * kPadRow + 32);
            pc.lap(kPhPop);
            // The current candidates are in bd/bv now: cv takes the next row's.
            ncnt = collect_pad_row(g, vs, ids0, ids1, cv, ct, a.error);
            dist_preload<kRegs>(g, cv, ncnt, pre, l2_next);
            pc.lap(kPhCollect);
        }
        // The current batch's merge runs while the next rows are loaded.
        const bool lost = queue_merge(q, sm.bd, sm.bv, m);
        __syncwarp();
        pc.lap(kPhMerge);
        if (lost && a.compact) return true;
        if (!go) break;
        // Predict the entry after `next`: the first unexplored entry now.
        p2 = queue_find_unexplored(q, q.hint);
        if (p2 >= 0) {
            q.hint = static_cast<uint32_t>(p2);
            const uint2 w = q.e[p2];
            pf_vid = w.x & kVidMask;
            p2_key = dist_key(ent_d(w));
            pf_ids0 = __ldg(pad + static_cast<size_t>(pf_vid) * kPadRow);
            pf_ids1 = __ldg(pad + static_cast<size_t>(pf_vid) * kPadRow + 32);
        } else {
            q.hint = q.n;
            pf_vid = kVidMask;
            p2_key = 0xffffffffu;
        }
        pc.lap(kPhPop);
        cnt = ncnt;
    }
    return false;
}

// ---------------------------------------------------------------------------
// Level-0 beam search by a team (graphs with fixed-stride rows). The pop order
// is the pipelined loop's: once the current row's distances are known, the
// next pop is the smaller of the first unexplored entry and the smallest
// accepted candidate. One expansion is two barriers: at A the row's distances
// are written, at B the leader has decided and published the next vertex.
// Between B and A the row warps expand it (visited test, row loads, distances)
// while the leader merges the previous row's accepted candidates.
//
// A row's 64 slots are divided over the row warps, contiguous slices for rows of at
// most kBlock chunks (8 rows a pass, and a slice's ids in one or two sectors); in
// turn for wide ones (2 rows a pass; near neighbours come first in a row and are
// mostly visited, so contiguous slices would leave the last warps most of the new
// ids: 1,000 queries of 200k x 960 25.3 against 18.2 ms). A warp tests its ids and
// writes the new ones and their distances at their slots (or at the front of its
// slice), which keeps row order, and +inf at the others (never accepted). Ids of a row are distinct, so the order in
// which warps mark them cannot change which are new.
//
// A search by one warp is one dependent chain of about 7,000 cycles an
// expansion on an idle GPU (row ids, visited set, two or three passes of eight
// rows, acceptance, merge). Here all rows of an expansion are in flight at
// once and the merge is off the chain; in addition the leader publishes the
// vertex expected after the next one (the second smallest head), whose ids the
// row warps load an expansion ahead and whose unvisited rows they start to
// load before the leader has decided, so on a correct guess (4 of 5) the chain
// is acceptance, visited test and the rest of the row latency.
// Against one warp a query: one query of 100k x 128 at queue 64 0.256 -> 0.127 ms,
// 16 of 200k x 96 cosine at queue 128 0.506 -> 0.262 ms, 256 at queue 100-400 2.20
// -> 1.16 ms, 1,000 of 100k x 128 at queue 200 1.60 -> 1.09 ms; 10,000 queries are
// faster with a warp each, which the autotuner finds.
// ---------------------------------------------------------------------------
template <int kMetric, bool kExact, int kG, bool kWide>
__device__ __forceinline__ void l0_team_rows(const SearchArgs& a, const WarpSmem& sm, Visited& vs, int gw, float qsq) {
    constexpr uint32_t kSlice = (kPadRow + kG - 1) / kG;
    static_assert(kSlice <= 32, "one id per lane");
    const DeviceGraph& g = a.g;
    const uint32_t lane = static_cast<uint32_t>(lane_id());
    const uint32_t lt = (1u << lane) - 1u;
    CoopCtl* ctl = sm.coop;
    uint32_t* ids = (kWide ? ctl->ids : sm.cvid) + gw * kSlice;
    uint32_t* slots = ctl->slots + gw * kSlice;
    uint32_t* spec = ctl->spec + gw * kSlice;
    const uint32_t slot = kWide ? lane * kG + gw : gw * kSlice + lane;   // of this lane's id
    const uint32_t* slice = g.l0pad + slot;
    const bool has = lane < kSlice && slot < kPadRow;
    constexpr uint32_t pass = kWide ? 2u : 8u;   // rows a pass
    uint32_t pf_vid = kVidMask, pf_id = 0xffffffffu, spec_mask = 0u;
    uint32_t evals = 0, row_ids = 0;
    std::conditional_t<kWide, WideRegs, RowRegs> x;
#pragma unroll
    for (int k = 0; k < (kWide ? 32 : 16); ++k) x[k] = 0;
    for (;;) {
        team_wait(kNextBarrier, kG + 1);   // B
        const uint32_t next = ctl->next;
        const uint32_t pf = ctl->pf;
        if (next == kVidMask) break;
        const bool hit = next == pf_vid;
        uint32_t id = pf_id;
        if (!hit) id = has ? __ldg(slice + static_cast<size_t>(next) * kPadRow) : 0xffffffffu;
        pf_vid = pf;
        pf_id = (has && pf != kVidMask) ? __ldg(slice + static_cast<size_t>(pf) * kPadRow) : 0xffffffffu;
        const bool is_new = team_test_and_set(vs, &ctl->list_n, id, id < g.n);
        const uint32_t b = __ballot_sync(kFull, is_new);
        const uint32_t cnt = __popc(b);
        if (kWide) {
            if (has) sm.cdist[slot] = INFINITY;
            if (is_new) {
                const uint32_t k = __popc(b & lt);
                ids[k] = id;
                slots[k] = slot;
                sm.cvid[slot] = id;
            }
        } else {   // compacted to the front of the slice: row order still
            if (is_new) ids[__popc(b & lt)] = id;
            if (has && lane >= cnt) sm.cdist[slot] = INFINITY;
        }
        __syncwarp();
        // The rows loaded ahead are the expansion's when the guess was right
        // and no id was marked in between.
        if (cnt && !(hit && b == spec_mask)) slice_load(g, ids, 0, cnt, x);
        #pragma unroll 1
        for (uint32_t p = 0; p < cnt; p += pass) {
            if (p) slice_load(g, ids, p, cnt, x);
            if constexpr (kWide) slice_distance<kMetric, kExact>(g, sm.q, qsq, ids, sm.cdist, slots, p, cnt, x);
            else slice_distance<kMetric, kExact>(g, sm.q, qsq, ids, sm.cdist + gw * kSlice, p, cnt, x);
        }
        __syncwarp();
        team_arrive(kRowsBarrier, kG + 1);   // A
        evals += cnt;
        row_ids += __popc(__ballot_sync(kFull, id != 0xffffffffu));
        if (has && id != 0xffffffffu && id >= g.n) set_error(a.error, kErrBadVid);
        // While the leader decides: the rows of the expected vertex's ids that
        // are unvisited now.
        spec_mask = __ballot_sync(kFull, pf_id < g.n && visited_open(vs, pf_id));
        if (spec_mask) {
            if ((spec_mask >> lane) & 1u) spec[__popc(spec_mask & lt)] = pf_id;
            __syncwarp();
            slice_load(g, spec, 0, __popc(spec_mask), x);
            if (kWide) {   // and all of them into L2
                const uint32_t sn = __popc(spec_mask), lines = g.dim >> 5;   // 128-byte lines of a row
                #pragma unroll 1
                for (uint32_t r = 0; r < sn; ++r) {
                    const float* row = g.vecs + static_cast<size_t>(spec[r]) * g.dim;
                    for (uint32_t i = lane; i < lines; i += 32) prefetch_l2(row + 32u * i);
                }
            }
        }
    }
    if (lane == 0) {
        atomicAdd(&ctl->evals, evals);
        atomicAdd(&ctl->row_ids, row_ids);
    }
    coop_barrier(kG + 1);   // end: counts are in
}

// An unexplored entry of the queue: distance key, vid, index (-1: absent).
struct Head {
    uint32_t k, v;
    int at;
};

__device__ __forceinline__ Head queue_head(const Queue& q, uint32_t from) {
    const int lane = lane_id();
    Head h;
    h.k = h.v = 0xffffffffu;
    h.at = -1;
    #pragma unroll 1
    for (uint32_t base = from; base < q.n; base += 32) {
        const uint32_t idx = base + lane;
        const uint2 w = idx < q.n ? q.e[idx] : make_uint2(kExplored, 0u);
        const uint32_t m = __ballot_sync(kFull, !(w.x & kExplored));
        if (m) {
            const int src = __ffs(m) - 1;
            h.v = __shfl_sync(kFull, w.x, src);
            h.k = dist_key(__uint_as_float(__shfl_sync(kFull, w.y, src)));
            h.at = static_cast<int>(base) + src;
            break;
        }
    }
    return h;
}

// The leader's side of the level-0 loop. `first` is the vertex to expand next,
// visited and marked explored; m accepted candidates in bd/bv are still to be
// merged. Returns true when the compact queue lost a live entry (see queue_merge).
template <int kG>
__device__ __forceinline__ bool l0_team_lead(const SearchArgs& a, Queue& q, Visited& vs, const WarpSmem& sm,
                                             uint32_t first, uint32_t m, Counters& ct, PhaseClock& pc) {
    const uint32_t lane = static_cast<uint32_t>(lane_id());
    CoopCtl* ctl = sm.coop;
    if (lane == 0) {
        ctl->next = first;
        ctl->pf = kVidMask;
        ctl->list_n = vs.list_overflow ? vs.list_cap + 1u : vs.list_n;
        ctl->evals = 0;
        ctl->row_ids = 0;
        ctl->cmd = kCmdLevel0;
    }
    coop_barrier(kG + 1);   // start: the row warps enter the loop
    team_arrive(kNextBarrier, kG + 1);   // B
    uint32_t guess = kVidMask;
    bool lost = false;
    Head h1, h2;   // the queue's first two unexplored entries (a merge finds both anew)
    h1 = queue_head(q, m ? q.n : q.hint);
    h2.k = h2.v = 0xffffffffu;
    h2.at = -1;
    for (uint32_t it = 0;; ++it) {
        ct.l0_rows++;
        // The previous row's merge runs while this row's distances are computed.
        if (m) {
            lost = queue_merge(q, sm.bd, sm.bv, m) && a.compact;
            h1 = queue_head(q, q.hint);
            q.hint = h1.at >= 0 ? static_cast<uint32_t>(h1.at) : q.n;
        }
        if (h1.at >= 0) h2 = queue_head(q, static_cast<uint32_t>(h1.at) + 1u);
        pc.lap(kPhMerge);
        team_wait(kRowsBarrier, kG + 1);   // A: the row's distances are written
        pc.lap(kPhDist);
        uint32_t next = kVidMask, pf = kVidMask;
        bool take_new = false;
        Batch s;
        s.m = 0;
        if (it > a.g.n) {
            set_error(a.error, kErrBound);
        } else if (!lost) {
            register_accept<true>(q, sm.cvid, sm.cdist, kPadRow, s);
            // Heads: queue (h1, h2) and batch (s.1, s.2), each ascending.
            take_new = head_less(s.k1, s.v1, h1.k, h1.v);
            next = take_new ? s.v1 : h1.v;
            pf = take_new ? (head_less(s.k2, s.v2, h1.k, h1.v) ? s.v2 : h1.v)
                          : (head_less(s.k1, s.v1, h2.k, h2.v) ? s.v1 : h2.v);
            next &= kVidMask;   // absent: kVidMask
            pf &= kVidMask;
        }
        if (lane == 0) {
            ctl->next = next;
            ctl->pf = pf;
        }
        __syncwarp();
        team_arrive(kNextBarrier, kG + 1);   // B
        if (next == kVidMask) break;
        // Off the row warps' chain: the accepted candidates, in slot order, to
        // bd/bv for the merge; the popped entry marked explored where it lies.
        m = s.m;
        if (m) write_accepted(s, take_new ? s.v1 : kVidMask, sm.bd, sm.bv);
        if (!take_new) {
            if (lane == 0) q.e[h1.at].x |= kExplored;
            q.hint = static_cast<uint32_t>(h1.at) + 1u;
            h1 = h2;
            h2.k = h2.v = 0xffffffffu;
            h2.at = -1;
        }
        __syncwarp();
        if (next == guess) pc.count(kPhPrefetchHits);
        guess = pf;
        pc.lap(kPhPop);
    }
    coop_barrier(kG + 1);   // end: counts are in
    const uint32_t list_n = ctl->list_n;
    vs.global_used = list_n != 0u;
    vs.list_overflow = list_n > vs.list_cap;
    vs.list_n = min(list_n, vs.list_cap);
    ct.dist_evals += ctl->evals;
    ct.l0_row_ids += ctl->row_ids;
    return lost;
}

// The row warps of a team: follow the leader's commands until it quits.
template <int kMetric, bool kExact, int kG, bool kPad>
__device__ void team_rows(const SearchArgs& a, const WarpSmem& sm, int warp) {
    CoopCtl* ctl = sm.coop;
    Stage st;
    st.buf = nullptr;
    st.mbar = 0u;
    st.phase = 0u;
    Visited vs = visited_init(a, sm, blockIdx.x);
    for (;;) {
        coop_barrier(kG + 1);   // start
        const uint32_t cmd = ctl->cmd;
        const float qsq = ctl->qsq;
        if (cmd == kCmdQuit) break;
        if constexpr (kPad) {
            if (cmd == kCmdLevel0) {
                if ((a.g.dim >> 4) <= kBlock) l0_team_rows<kMetric, kExact, kG, false>(a, sm, vs, warp - 1, qsq);
                else l0_team_rows<kMetric, kExact, kG, true>(a, sm, vs, warp - 1, qsq);
                continue;
            }
        }
        batch_distances<kMetric, kExact, false, false, true>(a.g, sm.q, qsq, ctl->cvid, ctl->cdist, ctl->cnt, st,
                                                            a.error, nullptr, static_cast<uint32_t>(warp), kG + 1);
        coop_barrier(kG + 1);   // done
    }
}

// ---------------------------------------------------------------------------
// Helped search: the end of a persistent launch of CTAs of four warps. Queries
// differ in length (1M x 128, queue 400: 400 to 1,122 expansions) and the long
// ones are not known beforehand, so the last quarter of a launch of 10,000
// queries had a few warps a CTA still searching, each alone at one warp's
// latency. A warp that finds no query left stays as a row warp; when three are
// there, the fourth goes on with its query as their leader (rows of at most
// kBlock chunks, graphs with fixed-stride rows). The functions below are
// not inlined: they run once or twice a warp, and the one-warp loop keeps its
// registers. Fixed launches, without -> with: 1M x 128, queue 100, 2,368
// queries 1.79 -> 1.46 ms, 10,000 3.31 -> 3.06 ms; queue 400, 2,368 queries 5.40
// -> 4.73 ms, 10,000 12.45 -> 11.9 ms; 1M x 96 cosine, queues 64-512, 10,000
// queries 5.32 -> 5.15 ms. (Two row warps, which are there earlier, gave less:
// 3.30, 12.8 and 5.18 ms.)
// ---------------------------------------------------------------------------
__device__ __forceinline__ CoopCtl* help_ctl(float* smem, uint32_t words, uint32_t dim, uint32_t cap) {
    const uint32_t host = reinterpret_cast<const volatile HelpFlags*>(smem)->host;
    return reinterpret_cast<CoopCtl*>(carve(smem + static_cast<size_t>(host) * words, dim, cap).cvid);
}

// A row warp, until the last query of the CTA is done.
template <int kMetric, bool kExact>
__device__ __noinline__ void help_rows(const SearchArgs& args, int gw) {
    extern __shared__ __align__(16) float smem[];
    const SearchArgs a = args;
    const uint32_t words = warp_smem_words(a.g.dim, a.cap, a.vh_bits);
    for (;;) {
        coop_barrier(kHelpers + 1);   // start
        if (reinterpret_cast<const volatile HelpFlags*>(smem)->quit) return;
        CoopCtl* ctl = help_ctl(smem, words, a.g.dim, a.cap);
        const uint32_t lead = ctl->lead;
        WarpSmem sm = carve(smem + static_cast<size_t>(lead) * words, a.g.dim, a.cap);
        sm.coop = ctl;
        Visited vs = visited_init(a, sm, blockIdx.x * (kHelpers + 1) + lead);
        l0_team_rows<kMetric, kExact, kHelpers, false>(a, sm, vs, gw, ctl->qsq);
    }
}

// The rest of a query at level 0, led by `warp`. The state is copied in and out,
// so that the one-warp loop's stays in registers.
struct HelpState {
    Queue q;
    Visited vs;
    Counters ct;
    Handover hand;
    float qsq;
};

template <int kG>
__device__ __noinline__ bool help_lead(const SearchArgs& args, uint32_t warp, HelpState& h) {
    extern __shared__ __align__(16) float smem[];
    const SearchArgs a = args;
    const uint32_t words = warp_smem_words(a.g.dim, a.cap, a.vh_bits);
    WarpSmem sm = carve(smem + static_cast<size_t>(warp) * words, a.g.dim, a.cap);
    sm.coop = help_ctl(smem, words, a.g.dim, a.cap);
    if (lane_id() == 0) {
        sm.coop->lead = warp;
        sm.coop->qsq = h.qsq;
    }
    Queue q = h.q;
    q.e = sm.qe;
    Visited vs = h.vs;
    vs.tab = reinterpret_cast<uint2*>(sm.vh);
    Counters ct = h.ct;
    PhaseClock pc;
    pc.start(false, nullptr);
    const bool lost = l0_team_lead<kG>(a, q, vs, sm, h.hand.first, h.hand.m, ct, pc);
    h.q = q;
    h.vs = vs;
    h.ct = ct;
    return lost;
}

// ---------------------------------------------------------------------------
// One query (hierarchical_graph_router.hpp:195-248; query_l0_only :258-286).
// ---------------------------------------------------------------------------
// stage_phase: with kStage, the parity of the next phase of the warp's staging
// mbarrier, which the caller initialised once (an mbarrier is not initialised
// again while it is valid) and which carries over from query to query.
// kPipe: level 0 by the pipelined loop, or the team's (fixed-stride rows), else
// one expansion at a time. kRegs: the
// pipelined loop holds the next expansion's first pass in registers (the
// 128-register budget) instead of prefetching it into L2. kG: row warps of a team
// whose leader runs this (0: one warp searches alone).
// kTrace: record the search in a.tr (the probes' trace kernel). kHelp: the
// pipelined loop may end as a helped search (`help`: this launch has helpers).
template <int kMetric, bool kExact, bool kStage = false, bool kRegs = false, int kG = 0, bool kPipe = false,
          bool kTrace = false, bool kHelp = false>
__device__ void search_one(const SearchArgs& a, uint32_t qi, uint32_t slot, const WarpSmem& sm,
                           uint32_t* stage_phase = nullptr, bool help = false) {
    const int lane = lane_id();
    const DeviceGraph& g = a.g;
    const uint32_t dim = g.dim;
    const uint32_t topk = a.topk ? (a.coherent ? __ldcg(a.topk + qi) : a.topk[qi]) : a.topk_default;
    const uint32_t L = a.queue ? (a.coherent ? __ldcg(a.queue + qi) : a.queue[qi]) : a.queue_default;
    uint64_t* out = a.out + static_cast<size_t>(qi) * a.k_stride;
    constexpr uint64_t kInvalidWord = (static_cast<uint64_t>(0x7f7fffffu) << 32) | kVidMask;

    if (topk > a.k_stride || L < topk || (a.compact ? L + 1ull : 2ull * L) > a.cap) {
        set_error(a.error, kErrArgs);
        #pragma unroll 1
        for (uint32_t i = lane; i < a.k_stride; i += 32) out[i] = kInvalidWord;
        return;
    }

    Counters ct = {};
    uint32_t nres = 0;
    bool overflowed = false;
    PhaseClock pc;
    pc.start(a.phase_cycles != nullptr, sm.phase);
    const long long t_begin = pc.on ? clock64() : 0;
    Visited vs = visited_init(a, sm, slot);
    uint32_t* cvid = sm.cvid;
    float* cdist = sm.cdist;
    Stage st;
    st.buf = sm.stage;
    st.mbar = kStage ? smem_addr(sm.mbar) : 0u;
    st.phase = kStage ? *stage_phase : 0u;

    if (g.n != 0 && g.top != kInvalidLevel && L > 0) {
        // Stage the query row in shared memory; reset the visited hash.
        const float4* src = reinterpret_cast<const float4*>(a.queries + static_cast<size_t>(qi) * dim);
        float4* dst = reinterpret_cast<float4*>(sm.q);
        #pragma unroll 1
        for (uint32_t i = lane; i < dim / 4; i += 32) dst[i] = a.coherent ? __ldcg(src + i) : __ldg(src + i);
        table_reset(vs);
        __syncwarp();
        const float qsq = (kMetric == ARTEA_GPU_COSINE) ? query_sqnorm<kExact>(sm.q, dim) : 0.f;

        // Entry point distance (hierarchical_graph_router.hpp:209-211), then the
        // greedy descent, levels top..1 (:228-236): one loop with one distance
        // call and one visited test for all of it, so that its code stays small.
        uint32_t cur = g.entry;
        float cur_d = 0.0f, best_d = 0.0f;
        uint32_t best_v = cur;
        uint32_t h = (a.l0_only ? 0u : g.top) + 1u;   // level walked (one above: the entry point is evaluated)
        const uint32_t h_top = h;
        const uint32_t* row = nullptr;
        uint32_t len = 0, pos = 0, hop = 0, cnt = 1;
        if (lane == 0) cvid[0] = cur;
        __syncwarp();
        #pragma unroll 1
        for (;;) {
            if (cnt) {
                dist_call<kMetric, kExact, kStage, kG>(g, sm.q, qsq, cvid, cdist, cnt, st, a.error, sm.coop);
                ct.dist_evals += cnt;
                if (h == h_top) {
                    cur_d = cdist[0];
                } else {
                    ct.upper_dist_evals += cnt;
                    // First strict improvement in row order (beam_loop.hpp:153-160).
                    float md = INFINITY;
                    uint32_t mi = 0xffffffffu;
                    #pragma unroll 1
                    for (uint32_t i = lane; i < cnt; i += 32) {
                        const float d = cdist[i];
                        if (d < md) { md = d; mi = i; }
                    }
                    #pragma unroll 1
                    for (int off = 16; off > 0; off >>= 1) {
                        const float od = __shfl_xor_sync(kFull, md, off);
                        const uint32_t oi = __shfl_xor_sync(kFull, mi, off);
                        if (od < md || (od == md && oi < mi)) { md = od; mi = oi; }
                    }
                    if (md < best_d) {
                        best_d = md;
                        best_v = cvid[mi];
                    }
                    __syncwarp();
                }
                cnt = 0;
            }
            if (pos < len) {
                uint32_t consumed;
                collect_unvisited(g, vs, row, len, pos, cvid, &cnt, &consumed, a.error, 0u, 0u, false);
                pos = consumed;
                continue;
            }
            // The row is done: walk on, or end the level.
            bool ends = h == h_top || best_v == cur;
            if (!ends) {
                cur = best_v;
                cur_d = best_d;
                if (++hop > g.n) { set_error(a.error, kErrBound); ends = true; }
            }
            // enable_early_stop: detail/beam_loop.hpp:147-150.
            if (!ends && a.early_stop && cur_d <= a.es_thr[h]) ends = true;
            if (ends) {
                if (h != h_top) visited_clear(vs);
                bool stop;
                do {
                    --h;
                    hop = 0;
                    visited_set(vs, cur);
                    stop = h != 0u && a.early_stop && cur_d <= a.es_thr[h];
                    if (stop) visited_clear(vs);
                } while (stop);
                if (h == 0u) break;
            }
            row = level_row(g, cur, h, &len);
            pos = 0;
            best_d = cur_d;
            best_v = cur;
            ct.upper_rows++;
            ct.upper_row_ids += len;
        }
        pc.lap(kPhUpper);

        // Level-0 beam search (single_layer_router.hpp:145-163, beam_loop.hpp:90-119).
        Queue q;
        q.e = sm.qe;
        q.n = 1;
        q.L = L;
        q.cap = a.cap;
        q.hint = 0;
        q.lb = L == 1u ? cur_d : FLT_MAX;
        if (lane == 0) q.e[0] = make_ent(cur_d, cur);
        __syncwarp();
        uint32_t tpos = 0, trows = 0;   // kTrace: candidates and rows recorded
        if (kTrace && lane == 0) a.tr.cur[qi] = make_uint2(cur, __float_as_uint(cur_d));
        if (kTrace && a.tr.upper_only) {
            // The greedy descent alone: level 0 is not searched.
        } else if (kG > 0 && kPipe) {
            if (lane == 0) q.e[0].x |= kExplored;   // pop the cursor: the queue's only entry
            q.hint = 1;
            overflowed = l0_team_lead<kG>(a, q, vs, sm, cur, 0u, ct, pc) && a.compact;
        } else if (kPipe) {
            Handover hand;
            overflowed = l0_search_pipelined<kMetric, kExact, kRegs, kHelp>(a, q, vs, sm, qsq, cur, ct, pc, st, help,
                                                                            hand) &&
                         a.compact;
            if (kHelp && hand.first != kVidMask) {
                HelpState h = {q, vs, ct, hand, qsq};
                overflowed = help_lead<kHelpers>(a, threadIdx.x >> 5, h) && a.compact;
                q.n = h.q.n;
                q.lb = h.q.lb;
                vs.global_used = h.vs.global_used;
                vs.list_overflow = h.vs.list_overflow;
                vs.list_n = h.vs.list_n;
                ct = h.ct;
            }
        } else {
            // Software pipeline: while one row is processed, the row descriptor and
            // then the neighbour ids of the entry that would be expanded next are
            // already being loaded (used if that entry is indeed popped next).
            uint32_t pf_vid = cur;
            unsigned long long pf_desc = __ldg(g.l0row + cur);
            uint32_t pf_ids0 = 0u, pf_ids1 = 0u;
            bool pf_have_ids = false;
            #pragma unroll 1
            for (uint32_t it = 0;; ++it) {
                if (it > g.n) { set_error(a.error, kErrBound); break; }
                int p2;
                const int p = queue_pop_peek(q, &p2);
                if (p < 0) break;
                const uint32_t v = q.e[p].x & kVidMask;
                if (v == kVidMask) break;   // CandidateEntry::is_invalid
                const bool hit = v == pf_vid;
                if (hit) pc.count(kPhPrefetchHits);
                const unsigned long long desc = hit ? pf_desc : __ldg(g.l0row + v);
                const uint32_t len = static_cast<uint32_t>(desc >> kRowLenShift);
                const uint32_t* row = g.nbrs + (desc & kRowStartMask);
                uint32_t ids0, ids1;
                if (hit && pf_have_ids) {
                    ids0 = pf_ids0;
                    ids1 = pf_ids1;
                } else {
                    ids0 = lane < len ? __ldg(row + lane) : 0xffffffffu;
                    ids1 = lane + 32 < len ? __ldg(row + lane + 32) : 0xffffffffu;
                }
                pf_have_ids = false;
                if (p2 >= 0) {
                    pf_vid = q.e[p2].x & kVidMask;
                    pf_desc = __ldg(g.l0row + pf_vid);
                } else {
                    pf_vid = kVidMask;
                }
                ct.l0_rows++;
                ct.l0_row_ids += len;
                pc.lap(kPhPop);
                uint32_t pos = 0;
                const bool one_pass = g.l0_unique && len <= 64u;
                #pragma unroll 1
                while (pos < len) {
                    uint32_t cnt, consumed;
                    if (one_pass) {
                        cnt = collect_row64_unique(g, vs, ids0, ids1, len, cvid, a.error);
                        consumed = len;
                    } else {
                        collect_unvisited(g, vs, row, len, pos, cvid, &cnt, &consumed, a.error, ids0, ids1, pos == 0);
                    }
                    pos = consumed;
                    pc.lap(kPhCollect);
                    if (kTrace) {
                        if (lane == 0 && trows < a.tr.rows_cap)
                            a.tr.rows[static_cast<size_t>(qi) * a.tr.rows_cap + trows] = make_uint2(v, cnt);
                        ++trows;
                    }
                    if (cnt == 0) continue;
                    if constexpr (kG == 0)
                        batch_distances<kMetric, kExact, kStage, false, false, true>(g, sm.q, qsq, cvid, cdist, cnt, st,
                                                                                    a.error);
                    else
                        dist_call<kMetric, kExact, kStage, kG>(g, sm.q, qsq, cvid, cdist, cnt, st, a.error, sm.coop);
                    ct.dist_evals += cnt;
                    if (kTrace) {
                        #pragma unroll 1
                        for (uint32_t i = lane; i < cnt; i += 32) {
                            if (tpos + i < a.tr.cap) {
                                a.tr.ids[static_cast<size_t>(qi) * a.tr.cap + tpos + i] = cvid[i];
                                a.tr.dists[static_cast<size_t>(qi) * a.tr.cap + tpos + i] = cdist[i];
                            }
                        }
                        tpos += cnt;
                    }
                    pc.lap(kPhDist);
                    if (p2 >= 0 && !pf_have_ids) {
                        // The next entry's descriptor has arrived by now: fetch its ids
                        // while the merge runs.
                        const uint32_t len2 = static_cast<uint32_t>(pf_desc >> kRowLenShift);
                        const uint32_t* row2 = g.nbrs + (pf_desc & kRowStartMask);
                        pf_ids0 = lane < len2 ? __ldg(row2 + lane) : 0xffffffffu;
                        pf_ids1 = lane + 32 < len2 ? __ldg(row2 + lane + 32) : 0xffffffffu;
                        pf_have_ids = true;
                    }
                    overflowed = queue_push_batch(q, cvid, cdist, cnt, sm.bd, sm.bv, a.error) && a.compact;
                    __syncwarp();
                    pc.lap(kPhMerge);
                    if (overflowed) break;
                }
                if (overflowed) break;
            }
        }
        if (kTrace && lane == 0 && !a.tr.upper_only)
            a.tr.len[qi] = make_uint2(min(tpos, a.tr.cap), min(trows, a.tr.rows_cap));
        visited_clear(vs);
        if (overflowed) {
            // The compact queue could have lost a live entry: the search is
            // redone by the full-capacity rerun, which writes this row.
            if (lane == 0) {
                const uint32_t pos = atomicAdd(a.overflow, 1u);
                a.overflow[2 + pos] = qi;
            }
            __syncwarp();
            if (kStage) *stage_phase = st.phase;
            return;
        }

        // extract_results(min(topk, |T|)) (std_candidate_queue.hpp:542-561).
        const uint32_t tsize = min(q.n, q.L);
        nres = min(topk, tsize);
        #pragma unroll 1
        for (uint32_t i = lane; i < a.k_stride; i += 32) {
            uint64_t w = kInvalidWord;
            if (i < nres) {
                const uint2 e = sm.qe[i];
                w = (static_cast<uint64_t>(e.y) << 32) | (e.x & kVidMask);
            }
            out[i] = w;
        }
    } else {
        #pragma unroll 1
        for (uint32_t i = lane; i < a.k_stride; i += 32) out[i] = kInvalidWord;
    }

    pc.lap(kPhTail);
    if (pc.on) {
        if (lane == 0) pc.acc[kPhTotal] = static_cast<unsigned long long>(clock64() - t_begin);
        __syncwarp();
        if (lane < kPhases) a.phase_cycles[static_cast<size_t>(qi) * kPhases + lane] = pc.acc[lane];
    }
    if (a.stats && lane == 0) {
        artea_gpu_query_stats s;
        s.dist_evals = ct.dist_evals;
        s.upper_rows = ct.upper_rows;
        s.upper_row_ids = ct.upper_row_ids;
        s.l0_rows = ct.l0_rows;
        s.l0_row_ids = ct.l0_row_ids;
        s.upper_dist_evals = ct.upper_dist_evals;
        s.results = nres;
        s.visited_spills = vs.spills;
        a.stats[qi] = s;
    }
    if (kStage) *stage_phase = st.phase;
    __syncwarp();
}

// Plain schedule: one CTA of one warp per query; slot = query index
// (24 resident CTAs per SM at the 85-register budget).
template <int kMetric, bool kExact, bool kPipe>
__global__ void __launch_bounds__(32, 24) search_plain_kernel(SearchArgs a) {
    extern __shared__ __align__(16) float smem[];
    const uint32_t qi = blockIdx.x;
    if (qi >= a.nq) return;
    const WarpSmem sm = carve(smem, a.g.dim, a.cap);
    search_one<kMetric, kExact, false, false, 0, kPipe>(a, qi, qi, sm);
}

// Persistent schedule: warps pull query indices from a shared counter (in
// the order a.order gives, if set). kBudget sets the register budget through
// the launch bounds: 64 (4 CTAs of 256 threads per SM, 32 resident warps), 85
// (3 x 256: 80 registers used, 24 warps), 96 (5 CTAs of at most 128 threads:
// 20 warps) or 128 (4 CTAs of at most 128 threads: 16 warps; the pipelined
// level-0 loop then holds the next expansion's first rows in registers).
// (__maxnreg__ with the same counts measured slower.) A warp that finds no query
// left helps the CTA's last one (help_rows).
constexpr int budget_threads(int budget) { return budget >= 96 ? 128 : 256; }
constexpr int budget_min_blocks(int budget) {
    return budget == 64 ? 4 : (budget == 96 ? 5 : (budget == 128 ? 4 : 3));
}

template <int kMetric, bool kExact, int kBudget, bool kStage = false, bool kPipe = false>
__global__ void __launch_bounds__(budget_threads(kBudget), budget_min_blocks(kBudget))
    search_persistent_kernel(const __grid_constant__ SearchArgs a) {
    extern __shared__ __align__(16) float smem[];
    const int warp = threadIdx.x >> 5;
    // Only the 96- and 128-register kernels take helpers, and only CTAs of four warps.
    constexpr bool kHelp = kPipe && !kStage;
    const bool help = kHelp && blockDim.x == 32u * (kHelpers + 1) && !a.phase_cycles && (a.g.dim >> 4) <= kBlock;
    HelpFlags* flags = reinterpret_cast<HelpFlags*>(smem);
    if (help) {
        if (threadIdx.x < 4) reinterpret_cast<uint32_t*>(smem)[threadIdx.x] = 0u;
        __syncthreads();
    }
    const uint32_t slot = blockIdx.x * (blockDim.x >> 5) + warp;
    const uint32_t stage_rows = kStage ? kStageRows : 0u;
    const WarpSmem sm = carve(smem + static_cast<size_t>(warp) * warp_smem_words(a.g.dim, a.cap, a.vh_bits,
                                                                                    stage_rows),
                              a.g.dim, a.cap, stage_rows);
    uint32_t stage_phase = 0u;
    if (kStage) {
        if (lane_id() == 0) mbar_init(smem_addr(sm.mbar));
        __syncwarp();
    }
    for (;;) {
        uint32_t qi = 0;
        if (lane_id() == 0) qi = atomicAdd(a.next_query, 1u);
        qi = __shfl_sync(kFull, qi, 0);
        if (qi >= a.nq) break;
        if (a.order) qi = __ldg(a.order + qi);
        search_one<kMetric, kExact, kStage, kBudget == 128, 0, kPipe, false, kHelp>(a, qi, slot, sm, &stage_phase,
                                                                                   help);
    }
    if (help) {
        uint32_t at = 0;
        if (lane_id() == 0) {
            at = atomicAdd(&flags->taken, 1u);
            if (at == 0) flags->host = warp;
            if (at == kHelpers) flags->quit = 1u;
            __threadfence_block();
            atomicAdd(&flags->idle, 1u);
        }
        at = __shfl_sync(kFull, at, 0);
        if (at < kHelpers) help_rows<kMetric, kExact>(a, static_cast<int>(at));
        else coop_barrier(kHelpers + 1);   // the last warp: the row warps leave
    }
    if (kStage) {
        __syncwarp();
        if (lane_id() == 0) asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_addr(sm.mbar)) : "memory");
    }
}

// Full-capacity rerun of the queries a compact-queue launch abandoned
// (a.overflow: count, work counter, indices). One warp per CTA, the queue at
// 2L, the HBM bitset as visited set; CTAs with nothing to do exit at once.
template <int kMetric, bool kExact>
__global__ void __launch_bounds__(32, 24) search_rerun_kernel(SearchArgs a) {
    extern __shared__ __align__(16) float smem[];
    const WarpSmem sm = carve(smem, a.g.dim, a.cap);
    for (;;) {
        uint32_t i = 0;
        if (lane_id() == 0) i = atomicAdd(a.overflow + 1, 1u);
        i = __shfl_sync(kFull, i, 0);
        if (i >= __ldcg(a.overflow)) break;
        const uint32_t qi = __ldcg(a.overflow + 2 + i);
        search_one<kMetric, kExact>(a, qi, blockIdx.x, sm);
    }
}

// Team schedule: a CTA of kG row warps and a leader searches one query at a
// time (queries from the shared counter, in a.order if set). Rows are read with
// vector loads. Launch bounds leave at least 96 registers a thread: the row
// warps hold the expected expansion's first rows in registers.
constexpr int team_min_blocks(int g) { return g == 1 ? 10 : (g == 2 ? 6 : (g == 3 ? 5 : (g == 4 ? 4 : 2))); }

// kPad: level 0 split over the team (fixed-stride rows); else one expansion at a
// time by the leader, its distance batches split over the warps.
template <int kMetric, bool kExact, int kG, bool kPad>
__global__ void __launch_bounds__((kG + 1) * 32, team_min_blocks(kG)) search_team_kernel(SearchArgs a) {
    extern __shared__ __align__(16) float smem[];
    const int warp = threadIdx.x >> 5;
    const uint32_t words = warp_smem_words(a.g.dim, a.cap, a.vh_bits);
    WarpSmem sm = carve(smem, a.g.dim, a.cap);
    sm.coop = reinterpret_cast<CoopCtl*>(smem + words);
    if (warp != 0) {
        team_rows<kMetric, kExact, kG, kPad>(a, sm, warp);
        return;
    }
    for (;;) {
        uint32_t qi = 0;
        if (lane_id() == 0) qi = atomicAdd(a.next_query, 1u);
        qi = __shfl_sync(kFull, qi, 0);
        if (qi >= a.nq) break;
        if (a.order) qi = __ldg(a.order + qi);
        search_one<kMetric, kExact, false, false, kG, kPad>(a, qi, blockIdx.x, sm);
    }
    if (lane_id() == 0) sm.coop->cmd = kCmdQuit;
    coop_barrier(kG + 1);   // the row warps see quit and leave
}

}  // namespace artea_gpu
