// Brute force through the tensor cores (bruteforce_tc.cu), used by bruteforce.cu.
#pragma once

#include <atomic>
#include <cstddef>
#include <cstdint>
#include <mutex>
#include <vector>

#include <cuda_fp16.h>
#include <cuda_runtime.h>

struct artea_gpu_index;

namespace artea_gpu {

struct BfPool;

// Norms of the whole index (one per index, on the device).
struct BfStats {
    uint32_t max_sq;     // largest x.x (float bits; sums of squares order as unsigned)
    uint32_t min_sq;     // smallest nonzero x.x
    uint32_t bad;        // some x.x is not finite
    uint32_t max_res;    // largest |x - fp16(x)| (float bits)
    uint32_t max_rel;    // largest |x - fp16(x)| / |x|
    uint32_t pad[3];
};

// The state an index keeps for brute force: norms, and the rounded rows once a call
// wanted them.
struct BfCache {
    int device = 0;
    std::mutex mu;                  // rows
    bool norms_ready = false, rows_ready = false;
    BfStats norms = {};             // host copy
    BfStats* d_norms = nullptr;
    __half* d_rows = nullptr;
    // The last call (artea_gpu_bruteforce_last): queries that the scan answered, its launches.
    std::atomic<uint32_t> last_scanned{0}, last_scans{0};
};
BfCache* bf_cache_create(int device, const float* d_xsq, uint32_t n, int sms);   // d_xsq: x.x of every row
void bf_cache_destroy(BfCache* c);

// A call's device workspace: the device's, unless another thread's call holds it.
// Slot 0: the host entry points' copies; slot 1: everything else. A call that ends
// early (an error) may leave kernels on its stream: they are waited for before the
// memory goes to another call.
constexpr size_t kBfKeepBytes = 256u << 20;   // no larger one is kept (per slot)
struct BfWork {
    explicit BfWork(const artea_gpu_index* ix);
    ~BfWork();
    BfWork(const BfWork&) = delete;
    BfWork& operator=(const BfWork&) = delete;
    void start(cudaStream_t st) { stream = st, running = true; }   // kernels may be in flight on st
    void waited() { running = false; }
    // At least bytes, valid until the slot's next get() or the end.
    int get(int slot, size_t bytes, unsigned char** p);

    BfPool* pool;
    bool held = false, running = false;
    cudaStream_t stream = nullptr;
    unsigned char* own[2] = {};
};

// Whether the index holds its rounded rows already.
bool bf_rows_ready(const artea_gpu_index* ix);
uint64_t bf_rows_bytes(const artea_gpu_index* ix);   // 0 without them
void bf_drop_rows(const artea_gpu_index* ix);        // no call is running on the index

// Ranks rows [0, n_rows) (or those of d_subset) for nq queries into d_out, and waits.
// *used false: nothing was written (the filter does not apply). redo: queries left
// to the scan.
int bf_tensor(const artea_gpu_index* ix, int metric, const float* d_queries, uint32_t nq, uint32_t topk,
              const uint32_t* d_subset, uint32_t n_rows, uint64_t* d_out, BfWork& work, int sms, cudaStream_t st,
              bool* used, std::vector<uint32_t>* redo);

// The same for a few queries, in FP32 throughout.
int bf_few(const artea_gpu_index* ix, int metric, const float* d_queries, uint32_t nq, uint32_t topk,
           const uint32_t* d_subset, uint32_t n_rows, uint64_t* d_out, BfWork& work, int sms, cudaStream_t st,
           bool* used, std::vector<uint32_t>* redo);

}  // namespace artea_gpu
