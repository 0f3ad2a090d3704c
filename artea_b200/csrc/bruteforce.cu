// Exact brute-force k-NN on the GPU: BruteforceRouter::query / batch_query and
// the subset overloads (router/bruteforce_router.hpp:74-160, 100-125, 164-190).
// This is the step after the query path (recall@k needs ground truth); the
// distances are the reference's, bit for bit: one thread evaluates a whole row,
// holding the 16 AVX-512 lane chains of utils/simd_distance.hpp:100-115 as
// eight packed FP32 pairs, then folds them with the _mm512_reduce_add_ps tree.
//
// Layout: a CTA takes kBfQueries queries (staged in shared memory) against a
// segment of the candidate rows; each thread loads one row chunk (16 floats)
// at a time and applies it to all the CTA's queries, so a row crosses HBM/L2
// once per CTA. Per query the CTA keeps a shared-memory list of (distance, vid)
// keys below the current k-th best; when a list fills, one warp sorts it and
// trims it to k. Several segments per query tile are merged by a second kernel.
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/artea_gpu.h"
#include "bruteforce.h"
#include "common.h"
#include "internal.h"

namespace artea_gpu {
namespace {

constexpr int kBfQueries = 8;        // queries per CTA
constexpr int kBfThreads = 128;      // rows per round (one per thread)
constexpr uint32_t kBfMaxTopk = 1024;
constexpr uint32_t kFilterRows = 8192;   // fewer rows: no filter
constexpr uint32_t kFewRows = 1024;      // fewer rows: the scan
constexpr uint32_t kFilterQueries = 4;   // fewer queries: bf_few, unless the index's rows are rounded already
// Dynamic shared memory that the kernels are allowed (the scan's own variables take
// less than 512 bytes of 227 KB, the merge sorts at most 16,384 keys). Fixed, since
// the limit belongs to the function and calls of other sizes run at the same time.
constexpr uint32_t kScanSmem = 227u * 1024u - 512u;
constexpr uint32_t kMergeKeys = 16384;
constexpr uint64_t kMaxKey = ~0ull;
// CandidateEntry() (router/data_structures/candidate_entry.hpp:72-74): vid =
// invalid_vertex_id (all ones), distance 0 -- the padding of batch rows whose
// query has fewer than topk candidates (bruteforce_router.hpp:142, 177).
constexpr uint64_t kDefaultEntryWord = 0x00000000FFFFFFFFull;

// (distance, vid) as one unsigned key whose order is the order by distance,
// then vid (negative distances included: DOT).
__device__ __forceinline__ uint64_t order_key(float d, uint32_t vid) {
    uint32_t u = __float_as_uint(d);
    u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    return (static_cast<uint64_t>(u) << 32) | vid;
}
__device__ __forceinline__ uint64_t key_word(uint64_t key) {
    uint32_t u = static_cast<uint32_t>(key >> 32);
    u = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
    return (static_cast<uint64_t>(u) << 32) | static_cast<uint32_t>(key);
}

// One sorted pass over n keys (n a power of two) by the calling warp.
__device__ void warp_bitonic_sort(uint64_t* a, uint32_t n) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t k2 = 2; k2 <= n; k2 <<= 1) {
        for (uint32_t j = k2 >> 1; j > 0; j >>= 1) {
            for (uint32_t i = lane; i < n; i += 32) {
                const uint32_t p = i ^ j;
                if (p > i) {
                    const uint64_t x = a[i], y = a[p];
                    const bool up = (i & k2) == 0;
                    if ((x > y) == up) {
                        a[i] = y;
                        a[p] = x;
                    }
                }
            }
            __syncwarp();
        }
    }
}

__host__ __device__ inline uint32_t next_pow2(uint32_t x) {
    uint32_t p = 1;
    while (p < x) p <<= 1;
    return p;
}

// Sort list q's first cnt keys (padding to a power of two) and keep the best k.
__device__ void trim_list(uint64_t* list, uint32_t cap, uint32_t* cnt, uint64_t* thr, uint32_t k) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t n = *cnt;
    const uint32_t p2 = next_pow2(max(n, 1u));
    for (uint32_t i = n + lane; i < p2; i += 32) list[i] = kMaxKey;
    __syncwarp();
    warp_bitonic_sort(list, p2);
    if (lane == 0) {
        const uint32_t kept = min(n, k);
        *cnt = kept;
        if (kept == k) *thr = list[k - 1];
    }
    __syncwarp();
    (void)cap;
}

struct BfArgs {
    const float* __restrict__ vecs;
    uint32_t dim;
    const uint32_t* __restrict__ subset;   // null: rows [0, n_rows)
    uint32_t n_rows;
    const float* __restrict__ queries;
    const uint32_t* __restrict__ which;    // nq queries' rows in queries and out (null: 0..nq-1)
    uint32_t nq;
    uint32_t k;
    uint32_t seg_len;                      // rows per segment (blockIdx.y)
    uint32_t segments;
    uint32_t list_cap;                     // power of two >= k + 2 * kBfThreads
    uint64_t* __restrict__ out;            // segments == 1: nq x k words
    uint64_t* __restrict__ part;           // segments > 1: nq x segments x k keys
    uint32_t* __restrict__ part_n;         // nq x segments counts
};

// CTAs an SM: three leave 168 registers a thread, which the L2 metrics use without
// spills; without the bound they took 180 and ran two (1,000 queries of 1M x 128:
// 34.7 -> 37.0 ms). Dot (188) and cosine (238) would spill.
constexpr int scan_min_blocks(int metric) {
    return metric == ARTEA_GPU_EUCLIDEAN_SQR || metric == ARTEA_GPU_EUCLIDEAN ? 3 : 2;
}

template <int kMetric>
__global__ void __launch_bounds__(kBfThreads, scan_min_blocks(kMetric)) bf_scan_kernel(BfArgs a) {
    extern __shared__ __align__(16) unsigned char bf_smem[];
    uint64_t* lists = reinterpret_cast<uint64_t*>(bf_smem);                       // kBfQueries x list_cap
    float* qs = reinterpret_cast<float*>(lists + static_cast<size_t>(kBfQueries) * a.list_cap);  // kBfQueries x dim
    __shared__ uint32_t cnt[kBfQueries];
    __shared__ uint64_t thr[kBfQueries];
    __shared__ float qsq[kBfQueries];
    __shared__ int need;

    const uint32_t tid = threadIdx.x;
    const uint32_t q0 = blockIdx.x * kBfQueries;
    const uint32_t nqt = min(static_cast<uint32_t>(kBfQueries), a.nq - q0);
    const uint32_t dim = a.dim;
    for (uint32_t i = tid; i < kBfQueries * dim; i += kBfThreads) {
        const uint32_t qi = i / dim;
        float v = 0.0f;
        if (qi < nqt) v = a.queries[static_cast<size_t>(a.which ? a.which[q0 + qi] : q0 + qi) * dim + (i - qi * dim)];
        qs[i] = v;
    }
    if (tid < kBfQueries) {
        cnt[tid] = 0;
        thr[tid] = kMaxKey;
    }
    __syncthreads();
    if (kMetric == ARTEA_GPU_COSINE && tid < kBfQueries) {
        // The query's own lane chains (nsq1, simd_distance.hpp:251-268).
        float l[16];
        for (int j = 0; j < 16; ++j) l[j] = 0.0f;
        for (uint32_t c = 0; c < dim; c += 16)
            for (int j = 0; j < 16; ++j) l[j] = fmaf(qs[tid * dim + c + j], qs[tid * dim + c + j], l[j]);
        float t8[8], t4[4];
        for (int i = 0; i < 8; ++i) t8[i] = __fadd_rn(l[i], l[i + 8]);
        for (int i = 0; i < 4; ++i) t4[i] = __fadd_rn(t8[i], t8[i + 4]);
        qsq[tid] = __fadd_rn(__fadd_rn(t4[0], t4[2]), __fadd_rn(t4[1], t4[3]));
    }
    __syncthreads();

    const uint32_t r0 = blockIdx.y * a.seg_len;
    const uint32_t r1 = min(a.n_rows, r0 + a.seg_len);
    for (uint32_t base = r0; base < r1; base += kBfThreads) {
        const uint32_t r = base + tid;
        const bool valid = r < r1;
        const uint32_t vid = valid ? (a.subset ? a.subset[r] : r) : 0u;
        const float* row = a.vecs + static_cast<size_t>(vid) * dim;
        f32x2 A[kBfQueries][8];
        f32x2 B[8];
#pragma unroll
        for (int qi = 0; qi < kBfQueries; ++qi)
#pragma unroll
            for (int p = 0; p < 8; ++p) A[qi][p] = 0ull;
#pragma unroll
        for (int p = 0; p < 8; ++p) B[p] = 0ull;
        if (valid) {
            for (uint32_t c = 0; c < dim; c += 16) {
                f32x2 x[8];
                const ulonglong2* xr = reinterpret_cast<const ulonglong2*>(row + c);
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const ulonglong2 v = __ldg(xr + h);
                    x[2 * h] = v.x;
                    x[2 * h + 1] = v.y;
                }
                if (kMetric == ARTEA_GPU_COSINE) {
#pragma unroll
                    for (int p = 0; p < 8; ++p) B[p] = fma2(x[p], x[p], B[p]);
                }
#pragma unroll
                for (int qi = 0; qi < kBfQueries; ++qi) {
                    const ulonglong2* yr = reinterpret_cast<const ulonglong2*>(qs + qi * dim + c);
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        const ulonglong2 y = yr[h];
                        if (kMetric == ARTEA_GPU_EUCLIDEAN_SQR || kMetric == ARTEA_GPU_EUCLIDEAN) {
                            const f32x2 d0 = sub2(y.x, x[2 * h]), d1 = sub2(y.y, x[2 * h + 1]);
                            A[qi][2 * h] = fma2(d0, d0, A[qi][2 * h]);
                            A[qi][2 * h + 1] = fma2(d1, d1, A[qi][2 * h + 1]);
                        } else {
                            A[qi][2 * h] = fma2(y.x, x[2 * h], A[qi][2 * h]);
                            A[qi][2 * h + 1] = fma2(y.y, x[2 * h + 1], A[qi][2 * h + 1]);
                        }
                    }
                }
            }
        }
        float xsq = 0.0f;
        if (kMetric == ARTEA_GPU_COSINE) {
            float l[16];
#pragma unroll
            for (int p = 0; p < 8; ++p) {
                l[2 * p] = lo32(B[p]);
                l[2 * p + 1] = hi32(B[p]);
            }
            float t8[8], t4[4];
#pragma unroll
            for (int i = 0; i < 8; ++i) t8[i] = __fadd_rn(l[i], l[i + 8]);
#pragma unroll
            for (int i = 0; i < 4; ++i) t4[i] = __fadd_rn(t8[i], t8[i + 4]);
            xsq = __fadd_rn(__fadd_rn(t4[0], t4[2]), __fadd_rn(t4[1], t4[3]));
        }
#pragma unroll
        for (int qi = 0; qi < kBfQueries; ++qi) {
            float l[16];
#pragma unroll
            for (int p = 0; p < 8; ++p) {
                l[2 * p] = lo32(A[qi][p]);
                l[2 * p + 1] = hi32(A[qi][p]);
            }
            float t8[8], t4[4];
#pragma unroll
            for (int i = 0; i < 8; ++i) t8[i] = __fadd_rn(l[i], l[i + 8]);
#pragma unroll
            for (int i = 0; i < 4; ++i) t4[i] = __fadd_rn(t8[i], t8[i + 4]);
            float d = __fadd_rn(__fadd_rn(t4[0], t4[2]), __fadd_rn(t4[1], t4[3]));
            if (kMetric == ARTEA_GPU_EUCLIDEAN) {
                d = __fsqrt_rn(d);
            } else if (kMetric == ARTEA_GPU_DOT) {
                d = -d;
            } else if (kMetric == ARTEA_GPU_COSINE) {
                // utils/simd_distance.hpp:263-274
                const float denom = __fsqrt_rn(__fmul_rn(qsq[qi], xsq));
                d = denom > 0.0f ? __fsub_rn(1.0f, __fdiv_rn(d, denom)) : 1.0f;
            }
            if (valid && static_cast<uint32_t>(qi) < nqt) {
                const uint64_t key = order_key(d, vid);
                if (key < thr[qi]) {
                    const uint32_t pos = atomicAdd(&cnt[qi], 1u);
                    lists[static_cast<size_t>(qi) * a.list_cap + pos] = key;   // pos < list_cap: see below
                }
            }
        }
        __syncthreads();
        // A round appends at most kBfThreads keys per list; trim any list that
        // could overflow in the next round (list_cap >= k + 2 * kBfThreads).
        if (tid == 0) {
            int any = 0;
            for (int qi = 0; qi < kBfQueries; ++qi) any |= cnt[qi] > a.list_cap - kBfThreads;
            need = any;
        }
        __syncthreads();
        if (need) {
            const uint32_t warp = tid >> 5;
            for (uint32_t qi = warp; qi < static_cast<uint32_t>(kBfQueries); qi += kBfThreads / 32) {
                if (cnt[qi] > a.list_cap - kBfThreads)
                    trim_list(lists + static_cast<size_t>(qi) * a.list_cap, a.list_cap, &cnt[qi], &thr[qi], a.k);
            }
            __syncthreads();
        }
    }
    // Final trim of every list, then write words (one segment) or keys (several).
    const uint32_t warp = tid >> 5;
    for (uint32_t qi = warp; qi < nqt; qi += kBfThreads / 32)
        trim_list(lists + static_cast<size_t>(qi) * a.list_cap, a.list_cap, &cnt[qi], &thr[qi], a.k);
    __syncthreads();
    for (uint32_t qi = 0; qi < nqt; ++qi) {
        const uint64_t* l = lists + static_cast<size_t>(qi) * a.list_cap;
        const uint32_t n = cnt[qi];
        if (a.segments == 1) {
            uint64_t* o = a.out + static_cast<size_t>(a.which ? a.which[q0 + qi] : q0 + qi) * a.k;
            for (uint32_t i = tid; i < a.k; i += kBfThreads) o[i] = i < n ? key_word(l[i]) : kDefaultEntryWord;
        } else {
            uint64_t* o = a.part + (static_cast<size_t>(q0 + qi) * a.segments + blockIdx.y) * a.k;
            for (uint32_t i = tid; i < n; i += kBfThreads) o[i] = l[i];
            if (tid == 0) a.part_n[static_cast<size_t>(q0 + qi) * a.segments + blockIdx.y] = n;
        }
    }
}

// One CTA per query: the best k of its segments' sorted key lists.
__global__ void __launch_bounds__(256) bf_merge_kernel(const uint64_t* __restrict__ part,
                                                       const uint32_t* __restrict__ part_n, uint32_t segments,
                                                       uint32_t k, uint32_t pow2, const uint32_t* __restrict__ which,
                                                       uint64_t* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char bf_smem[];
    uint64_t* keys = reinterpret_cast<uint64_t*>(bf_smem);   // pow2 >= segments * k
    const uint32_t q = blockIdx.x;
    // (Every key on its own: walking the segments one by one waited for each one's
    // count, 82 us at 390 segments.)
    const uint64_t* src = part + static_cast<size_t>(q) * segments * k;
    for (uint32_t i = threadIdx.x; i < pow2; i += blockDim.x) {
        const uint32_t s = i / k;
        const bool in = s < segments && i - s * k < part_n[static_cast<size_t>(q) * segments + s];
        keys[i] = in ? src[i] : kMaxKey;
    }
    __syncthreads();
    for (uint32_t k2 = 2; k2 <= pow2; k2 <<= 1) {
        for (uint32_t j = k2 >> 1; j > 0; j >>= 1) {
            for (uint32_t i = threadIdx.x; i < pow2; i += blockDim.x) {
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
    uint64_t* o = out + static_cast<size_t>(which ? which[q] : q) * k;
    for (uint32_t i = threadIdx.x; i < k; i += blockDim.x)
        o[i] = keys[i] != kMaxKey ? key_word(keys[i]) : kDefaultEntryWord;
}

using ScanFn = void (*)(BfArgs);

ScanFn scan_kernel(int metric) {
    switch (metric) {
        case ARTEA_GPU_EUCLIDEAN_SQR: return bf_scan_kernel<ARTEA_GPU_EUCLIDEAN_SQR>;
        case ARTEA_GPU_EUCLIDEAN: return bf_scan_kernel<ARTEA_GPU_EUCLIDEAN>;
        case ARTEA_GPU_COSINE: return bf_scan_kernel<ARTEA_GPU_COSINE>;
        case ARTEA_GPU_DOT: return bf_scan_kernel<ARTEA_GPU_DOT>;
        default: return nullptr;
    }
}

uint32_t scan_list_cap(uint32_t topk) { return next_pow2(topk + 2 * kBfThreads); }
size_t scan_smem(uint32_t dim, uint32_t topk) {
    return static_cast<size_t>(kBfQueries) * (scan_list_cap(topk) * sizeof(uint64_t) + dim * sizeof(float));
}

// The FP32 scan of rows [0, n_rows) (d_subset null) or d_subset's, for nq queries or
// those of `which` (in one launch: a query at a time cost a launch, a wait and a
// pass over the rows each, eight of which a CTA does at once); waits.
int scan(const artea_gpu_index* ix, int metric, const float* d_queries, uint32_t nq, uint32_t topk,
         const uint32_t* d_subset, uint32_t n_rows, uint64_t* d_out, BfWork& work, int dev_sms, cudaStream_t st,
         const std::vector<uint32_t>* which = nullptr) {
    if (which) nq = static_cast<uint32_t>(which->size());
    ScanFn fn = scan_kernel(metric);
    const uint32_t list_cap = scan_list_cap(topk);
    const size_t smem = scan_smem(ix->dim, topk);
    CUDA_TRY(cudaFuncSetAttribute(reinterpret_cast<const void*>(fn), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(kScanSmem)));
    int per_sm = 0;
    CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, reinterpret_cast<const void*>(fn), kBfThreads,
                                                           smem));
    const uint32_t tiles = (nq + kBfQueries - 1) / kBfQueries;
    // Rows are split into segments: one a CTA, whose lists are sorted at its end and
    // merged (about 100 us of its time at 384 keys, whatever the segment's length).
    // - Of 4,096 rows or more: until the grid covers the GPU twice over.
    // - Of 512 rows (4 rounds of a CTA) and 32 per result or more: until there are two
    //   CTAs an SM. (1,000 queries over 4,096 x 16 rows: 1, 2, 4 and 8 segments 222, 190,
    //   309 and 430 us; one query over 200k rows was left on 48 CTAs by 4,096 rows each.)
    // - With more CTAs than that: halves, where they save a quarter of the waves and are
    //   well longer than the sort (cosine, 2 CTAs an SM, 2,500 queries: over 8,191 x 400
    //   rows 2.79 -> 2.24 ms, over 4,096 x 96 rows 0.69 -> 0.75).
    const uint32_t sms = static_cast<uint32_t>(dev_sms), slots = static_cast<uint32_t>(std::max(per_sm, 1)) * sms;
    const uint32_t whole = std::min((2u * slots + tiles - 1) / tiles, n_rows / 4096u);
    const uint32_t fill = std::min(2u * sms / tiles, n_rows / std::min(4096u, std::max(512u, 32u * topk)));
    const bool halves = 2u * ((2u * tiles + slots - 1) / slots) <= 3u * ((tiles + slots - 1) / slots) &&
                        static_cast<uint64_t>(n_rows / 2u) * ix->dim >= 1000000u;
    uint32_t segments = std::max({1u, whole, fill, tiles > 2u * sms && halves ? 2u : 1u});
    segments = std::min(segments, std::max(4096u / topk, 2u * sms));
    segments = std::min(segments, std::max(1u, kMergeKeys / topk));
    const uint32_t seg_len = (n_rows + segments - 1) / segments;
    segments = (n_rows + seg_len - 1) / seg_len;

    BfArgs a;
    std::memset(&a, 0, sizeof(a));
    a.vecs = ix->d_vecs;
    a.dim = ix->dim;
    a.subset = d_subset;
    a.n_rows = n_rows;
    a.queries = d_queries;
    a.nq = nq;
    a.k = topk;
    a.seg_len = seg_len;
    a.segments = segments;
    a.list_cap = list_cap;
    a.out = d_out;
    if (segments > 1 || which) {
        const size_t keys = segments > 1 ? sizeof(uint64_t) * static_cast<size_t>(nq) * segments * topk : 0;
        const size_t counts = segments > 1 ? sizeof(uint32_t) * static_cast<size_t>(nq) * segments : 0;
        unsigned char* p = nullptr;
        if (int rc = work.get(1, keys + counts + (which ? sizeof(uint32_t) * nq : 0), &p)) return rc;
        a.part = reinterpret_cast<uint64_t*>(p);
        a.part_n = reinterpret_cast<uint32_t*>(p + keys);
        if (which) {
            a.which = reinterpret_cast<uint32_t*>(p + keys + counts);
            CUDA_TRY(cudaMemcpyAsync(p + keys + counts, which->data(), sizeof(uint32_t) * nq, cudaMemcpyHostToDevice, st));
        }
    }
    ix->bf->last_scanned += nq;
    ++ix->bf->last_scans;
    fn<<<dim3(tiles, segments), kBfThreads, smem, st>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && segments > 1) {
        const uint32_t pow2 = next_pow2(segments * topk);
        const size_t msmem = static_cast<size_t>(pow2) * sizeof(uint64_t);
        e = cudaFuncSetAttribute(reinterpret_cast<const void*>(bf_merge_kernel),
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(kMergeKeys * sizeof(uint64_t)));
        if (e == cudaSuccess) {
            bf_merge_kernel<<<nq, 256, msmem, st>>>(a.part, a.part_n, segments, topk, pow2, a.which, d_out);
            e = cudaGetLastError();
        }
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail(ARTEA_GPU_ECUDA, std::string("brute force: ") + cudaGetErrorString(e));
    return ARTEA_GPU_OK;
}

// use_subset: rows are d_subset[0, n_subset) (possibly empty), else all vectors.
int bruteforce_impl(const artea_gpu_index* ix, int metric, const float* d_queries, uint32_t nq, uint32_t topk,
                    bool use_subset, const uint32_t* d_subset, uint32_t n_subset, uint64_t* d_out, BfWork& work,
                    cudaStream_t st) {
    if (!ix || (nq && (!d_queries || !d_out))) return fail(ARTEA_GPU_EINVAL, "null argument");
    if (topk == 0 || topk > kBfMaxTopk)
        return fail(ARTEA_GPU_EINVAL, "brute-force topk must be in [1, " + std::to_string(kBfMaxTopk) + "]");
    if (!scan_kernel(metric)) return fail(ARTEA_GPU_EINVAL, "unknown metric");
    if (nq == 0) return ARTEA_GPU_OK;
    const uint32_t n_rows = use_subset ? n_subset : ix->nvecs;
    if (use_subset && n_subset && !d_subset) return fail(ARTEA_GPU_EINVAL, "null subset");
    DeviceGuard guard(ix->device);
    if (n_rows == 0) {
        // Every row is CandidateEntry() padding.
        std::vector<uint64_t> pad(static_cast<size_t>(nq) * topk, kDefaultEntryWord);
        CUDA_TRY(cudaMemcpyAsync(d_out, pad.data(), pad.size() * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
        CUDA_TRY(cudaStreamSynchronize(st));
        return ARTEA_GPU_OK;
    }
    // Sizes that the scan cannot take are refused whatever path the call would go
    // first: any of them may hand queries on to the scan.
    if (scan_smem(ix->dim, topk) > kScanSmem)
        return fail(ARTEA_GPU_EINVAL, "brute-force tile exceeds shared memory (topk or dim too large)");
    int dev_sms = 0;
    CUDA_TRY(cudaDeviceGetAttribute(&dev_sms, cudaDevAttrMultiProcessorCount, ix->device));
    work.start(st);
    ix->bf->last_scanned = 0;
    ix->bf->last_scans = 0;
    const uint32_t* subset = use_subset ? d_subset : nullptr;
    // The tensor-core filter reads every row twice in FP16 and pays a rounding pass
    // over the rows (once an index, or on every call for a subset); bf_few reads them
    // once in FP32 for every query; the scan once for every 8 queries, but with a
    // sorted list a CTA. (8 queries over 1M x 128, k 100: scan 1.7 ms; filter 0.16 ms,
    // 1.6 with the rounding.) With fewer rows the launches decide.
    const bool many = n_rows >= kFilterRows;
    const bool filter = many && (nq >= kFilterQueries || (!use_subset && bf_rows_ready(ix)));
    const bool few = nq < kFilterQueries && n_rows >= kFewRows;
    if ((filter || few) && 8ull * topk <= n_rows) {
        bool used = false;
        std::vector<uint32_t> redo;
        if (int rc = filter ? bf_tensor(ix, metric, d_queries, nq, topk, subset, n_rows, d_out, work, dev_sms, st, &used, &redo)
                            : bf_few(ix, metric, d_queries, nq, topk, subset, n_rows, d_out, work, dev_sms, st, &used, &redo))
            return rc;
        if (used && redo.size() < nq) {
            if (!redo.empty())
                if (int rc = scan(ix, metric, d_queries, nq, topk, subset, n_rows, d_out, work, dev_sms, st, &redo))
                    return rc;
            work.waited();
            return ARTEA_GPU_OK;
        }
    }
    if (int rc = scan(ix, metric, d_queries, nq, topk, subset, n_rows, d_out, work, dev_sms, st)) return rc;
    work.waited();
    return ARTEA_GPU_OK;
}

// Centroid of the bucket's rows (hierarchical_graph_compactor.hpp:261-300):
// block (x, y) sums rows [x * rows_per_block, ...) of dimensions [32 y, 32 y + 32) in
// double, in row order; the final pass adds the blocks' sums in block order. One
// warp a block and one chain of additions a lane: the order is part of the result,
// so what is left is to keep 64 rows in flight behind it.
constexpr int kCentroidRows = 64;

__global__ void __launch_bounds__(32) centroid_partial_kernel(const float* __restrict__ vecs, uint32_t dim,
                                                              const uint32_t* __restrict__ bucket, uint32_t n,
                                                              uint32_t rows_per_block, double* __restrict__ partial) {
    const uint32_t r0 = blockIdx.x * rows_per_block;
    const uint32_t r1 = min(n, r0 + rows_per_block);
    const uint32_t d = blockIdx.y * 32u + threadIdx.x;
    if (d >= dim) return;
    double s = 0.0;
    float next[kCentroidRows];
#pragma unroll
    for (int i = 0; i < kCentroidRows; ++i) {
        const uint32_t r = min(r0 + i, r1 - 1u);
        next[i] = __ldg(vecs + static_cast<size_t>(bucket ? bucket[r] : r) * dim + d);
    }
    for (uint32_t base = r0; base < r1; base += kCentroidRows) {
        float x[kCentroidRows];
#pragma unroll
        for (int i = 0; i < kCentroidRows; ++i) x[i] = next[i];
#pragma unroll
        for (int i = 0; i < kCentroidRows; ++i) {
            const uint32_t r = min(base + kCentroidRows + i, r1 - 1u);
            next[i] = __ldg(vecs + static_cast<size_t>(bucket ? bucket[r] : r) * dim + d);
        }
        if (base + kCentroidRows <= r1) {
#pragma unroll
            for (int i = 0; i < kCentroidRows; ++i) s += static_cast<double>(x[i]);
        } else {
#pragma unroll
            for (int i = 0; i < kCentroidRows; ++i)
                if (base + i < r1) s += static_cast<double>(x[i]);
        }
    }
    partial[static_cast<size_t>(blockIdx.x) * dim + d] = s;
}

__global__ void centroid_final_kernel(const double* __restrict__ partial, uint32_t blocks, uint32_t dim, uint32_t n,
                                      float* __restrict__ centroid) {
    const double inv_n = 1.0 / static_cast<double>(n);
    for (uint32_t d = blockIdx.x * blockDim.x + threadIdx.x; d < dim; d += gridDim.x * blockDim.x) {
        double s = 0.0;
#pragma unroll 16
        for (uint32_t b = 0; b < blocks; ++b) s += partial[static_cast<size_t>(b) * dim + d];
        centroid[d] = static_cast<float>(s * inv_n);
    }
}

}  // namespace
}  // namespace artea_gpu

using namespace artea_gpu;

extern "C" {

int artea_gpu_bruteforce_device(const artea_gpu_index* index, int metric, const float* d_queries, uint32_t nq,
                                uint32_t topk, const uint32_t* d_subset, uint32_t n_subset, uint64_t* d_out,
                                void* stream) {
    if (!index) return fail(ARTEA_GPU_EINVAL, "null argument");
    DeviceGuard guard(index->device);
    BfWork work(index);
    return bruteforce_impl(index, metric, d_queries, nq, topk, d_subset != nullptr, d_subset, n_subset, d_out, work,
                           static_cast<cudaStream_t>(stream));
}

int artea_gpu_bruteforce_last(const artea_gpu_index* index, uint32_t* scanned, uint32_t* scans) {
    if (!index || !scanned || !scans) return fail(ARTEA_GPU_EINVAL, "null argument");
    *scanned = index->bf->last_scanned;
    *scans = index->bf->last_scans;
    return ARTEA_GPU_OK;
}

int artea_gpu_bruteforce(const artea_gpu_index* index, int metric, const float* queries, uint32_t nq, uint32_t topk,
                         const uint32_t* subset, uint32_t n_subset, uint64_t* out) {
    if (!index || (nq && (!queries || !out))) return fail(ARTEA_GPU_EINVAL, "null argument");
    if (subset) {
        for (uint32_t i = 0; i < n_subset; ++i)
            if (subset[i] >= index->nvecs)
                return fail(ARTEA_GPU_EINVAL, "subset id " + std::to_string(subset[i]) + " out of range");
    }
    if (nq == 0) return ARTEA_GPU_OK;
    DeviceGuard guard(index->device);
    BfWork work(index);
    const size_t q_bytes = (sizeof(float) * nq * index->dim + 255) / 256 * 256;
    const size_t o_bytes = (sizeof(uint64_t) * nq * static_cast<size_t>(topk) + 255) / 256 * 256;
    unsigned char* p = nullptr;
    if (int rc = work.get(0, q_bytes + o_bytes + (subset ? sizeof(uint32_t) * n_subset : 0) + 1, &p)) return rc;
    float* d_q = reinterpret_cast<float*>(p);
    uint64_t* d_o = reinterpret_cast<uint64_t*>(p + q_bytes);
    uint32_t* d_s = subset && n_subset ? reinterpret_cast<uint32_t*>(p + q_bytes + o_bytes) : nullptr;
    if (cudaMemcpy(d_q, queries, sizeof(float) * nq * index->dim, cudaMemcpyHostToDevice) != cudaSuccess)
        return fail(ARTEA_GPU_ECUDA, "query upload failed");
    if (d_s && cudaMemcpy(d_s, subset, sizeof(uint32_t) * n_subset, cudaMemcpyHostToDevice) != cudaSuccess)
        return fail(ARTEA_GPU_ECUDA, "subset upload failed");
    if (int rc = bruteforce_impl(index, metric, d_q, nq, topk, subset != nullptr, d_s, subset ? n_subset : 0u, d_o, work,
                                 nullptr))
        return rc;
    if (cudaMemcpy(out, d_o, sizeof(uint64_t) * nq * topk, cudaMemcpyDeviceToHost) != cudaSuccess)
        return fail(ARTEA_GPU_ECUDA, "result download failed");
    return ARTEA_GPU_OK;
}

// _compute_entry_point_vid (hierarchical_graph_compactor.hpp:261-327): the
// bucket's centroid (double sums, rounded to float), then the bucket vid
// nearest to it under metric -- the brute force above with k = 1 over the
// bucket, the centroid as the query operand.
int artea_gpu_centroid_entry(const artea_gpu_index* index, int metric, const uint32_t* bucket, uint32_t n,
                             uint32_t* out_vid) {
    if (!index || !out_vid) return fail(ARTEA_GPU_EINVAL, "null argument");
    const uint32_t rows = bucket ? n : index->nvecs;
    *out_vid = 0xFFFFFFFFu;   // invalid_vertex_id: empty bucket
    if (rows == 0) return ARTEA_GPU_OK;
    if (bucket) {
        for (uint32_t i = 0; i < n; ++i)
            if (bucket[i] >= index->nvecs)
                return fail(ARTEA_GPU_EINVAL, "bucket id " + std::to_string(bucket[i]) + " out of range");
    }
    DeviceGuard guard(index->device);
    const uint32_t per_block = 4096;
    const uint32_t blocks = (rows + per_block - 1) / per_block;
    BfWork work(index);
    const size_t partial_bytes = sizeof(double) * static_cast<size_t>(blocks) * index->dim;
    const size_t centroid_bytes = (sizeof(float) * index->dim + 15) / 16 * 16;
    unsigned char* p = nullptr;
    if (int rc = work.get(0, partial_bytes + centroid_bytes + 16 + (bucket ? sizeof(uint32_t) * n : 0), &p)) return rc;
    double* d_partial = reinterpret_cast<double*>(p);
    float* d_centroid = reinterpret_cast<float*>(p + partial_bytes);
    uint64_t* d_word = reinterpret_cast<uint64_t*>(p + partial_bytes + centroid_bytes);
    uint32_t* d_bucket = bucket ? reinterpret_cast<uint32_t*>(p + partial_bytes + centroid_bytes + 16) : nullptr;
    if (bucket && cudaMemcpy(d_bucket, bucket, sizeof(uint32_t) * n, cudaMemcpyHostToDevice) != cudaSuccess)
        return fail(ARTEA_GPU_ECUDA, "bucket upload failed");
    work.start(nullptr);
    centroid_partial_kernel<<<dim3(blocks, (index->dim + 31) / 32), 32>>>(index->d_vecs, index->dim, d_bucket, rows,
                                                                         per_block, d_partial);
    centroid_final_kernel<<<(index->dim + 31) / 32, 32>>>(d_partial, blocks, index->dim, rows, d_centroid);
    if (cudaGetLastError() != cudaSuccess) return fail(ARTEA_GPU_ECUDA, "centroid kernels failed to launch");
    if (int rc = bruteforce_impl(index, metric, d_centroid, 1, 1, bucket != nullptr, d_bucket, rows, d_word, work,
                                 nullptr))
        return rc;
    uint64_t word = 0;
    if (cudaMemcpy(&word, d_word, sizeof(word), cudaMemcpyDeviceToHost) != cudaSuccess)
        return fail(ARTEA_GPU_ECUDA, "result download failed");
    *out_vid = static_cast<uint32_t>(word);
    return ARTEA_GPU_OK;
}

}  // extern "C"
