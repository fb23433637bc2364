// Shared host/device helpers of the inpc_b200 library (sm_100a only).
#pragma once

#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <cstdint>
#include <cstdio>
#include <cstdarg>
#include <mutex>
#include <utility>
#include "../../include/inpc_b200.h"

namespace inpc {

// ---- error reporting ---------------------------------------------------------------------
void set_error(const char* fmt, ...);
int cuda_fail(cudaError_t e, const char* what);

#define INPC_CUDA_TRY(expr)                                        \
    do {                                                           \
        cudaError_t _e = (expr);                                   \
        if (_e != cudaSuccess) return ::inpc::cuda_fail(_e, #expr); \
    } while (0)

// After every kernel launch: counts it (inpc_launch_count) and turns a launch error into a status.
#define INPC_LAUNCH_CHECK(name)                                       \
    do {                                                              \
        ::inpc::count_launch();                                       \
        cudaError_t _e = cudaGetLastError();                          \
        if (_e != cudaSuccess) return ::inpc::cuda_fail(_e, name);     \
    } while (0)

void count_launch();

// Optional per-stage device timing (inpc_profile_enable): a StageScope records a CUDA event pair
// around the launches of one pipeline stage on the stream they are issued to.
enum Stage : int {
    STAGE_SAMPLE = 0,        // leaf weights, CDF, draws
    STAGE_PREPROCESS = 1,    // project + SH
    STAGE_SORT_DEPTH = 2,
    STAGE_INSTANCES = 3,     // per-point tile counts, scan, emission
    STAGE_SORT_TILE = 4,     // tile sort + ranges
    STAGE_BLEND_FWD = 5,
    STAGE_BLEND_BWD = 6,
    STAGE_PREPROCESS_BWD = 7,
    STAGE_COUNT = 8,
};
struct StageScope {
    int slot;
    cudaStream_t stream;
    StageScope(Stage stage, cudaStream_t s);
    ~StageScope();
};

// Device-visible status words in mapped pinned host memory: a kernel stores 1 into its word when a
// bounded wait runs out (plain store, no atomics over PCIe); the host reads them without a device
// synchronisation.
enum : unsigned {
    STATUS_LOOKBACK_TIMEOUT = 0,   // a radix-sort tile gave up waiting for a predecessor tile
    STATUS_SAMPLER_EXHAUSTED = 1,  // informational: some sample slots ran out of rejection attempts
    STATUS_BULK_COPY_TIMEOUT = 2,  // a block gave up waiting for its bulk copy into shared memory
    STATUS_INDEX_OUT_OF_RANGE = 3, // checked build only: a gather index was outside its array (the access was skipped)
    STATUS_WORDS = 4,
};
// Takes the next status slot for a call of `entry` (a string literal): returns the device address of its
// STATUS_WORDS cleared words, or nullptr (error set).  *ticket_out names the slot for read_status.
unsigned* acquire_status(const char* entry, long long* ticket_out = nullptr);
int read_status(long long ticket, unsigned* words, const char** entry);
// INPC_E_DEVICE (with a message naming the entry point) if the last status-carrying call this host thread
// made has reported a failure since; every entry point that launches work calls it first, so a failure
// surfaces at the thread's next call at the latest -- or earlier through inpc_call_status.
int check_previous_calls();

// ---- small utilities ---------------------------------------------------------------------
template <typename T>
__host__ __device__ constexpr T ceil_div(T a, T b) { return (a + b - 1) / b; }

inline size_t align_up(size_t x, size_t a = 256) { return (x + a - 1) / a * a; }

// Carves consecutive 256-byte-aligned arrays out of one blob.
struct Carver {
    char* base;
    size_t off = 0;
    explicit Carver(void* p) : base(static_cast<char*>(p)) {}
    template <typename T>
    T* take(size_t count) {
        off = align_up(off);
        T* p = reinterpret_cast<T*>(base + off);
        off += sizeof(T) * count;
        return p;
    }
    size_t used() const { return align_up(off); }
};

inline int bit_length(uint32_t v) {
    int b = 0;
    while (v) { ++b; v >>= 1; }
    return b;
}

// ---- camera parameters passed by value to kernels -----------------------------------------
struct ViewParams {
    const float* w2c;   // device, 16 floats
    const float* cam;   // device, 3 floats
    int width, height;
    float fx, fy, cx, cy, near_plane, far_plane;
};

inline ViewParams to_params(const inpc_view* v) {
    ViewParams p;
    p.w2c = v->w2c; p.cam = v->cam_position;
    p.width = v->width; p.height = v->height;
    p.fx = v->fx; p.fy = v->fy; p.cx = v->cx; p.cy = v->cy;
    p.near_plane = v->near_plane; p.far_plane = v->far_plane;
    return p;
}

// ---- radix sort (radix_sort.cu) ------------------------------------------------------------
// The workspace for n pairs (an upper bound) of which n_likely are expected: the expectation picks the tile size, no more.
size_t sort_workspace_bytes(int64_t n, int64_t n_likely);
int sort_pass_count(int end_bit);   // passes a sort makes; the result is in the alternate buffers iff odd (sort_pairs: and n > 1)
// `status`: device address of the STATUS_WORDS words a tile that gives up its look-back reports to.
// `n_likely`: the one the workspace was sized with (for at least n pairs).  `zeroed`: the caller has cleared the first
// sort_zero_bytes(n, n_likely, end_bit) bytes of the workspace.
size_t sort_zero_bytes(int64_t n, int64_t n_likely, int end_bit);
int sort_pairs(uint32_t* keys, uint32_t* keys_alt, uint32_t* values, uint32_t* values_alt, int64_t n, int64_t n_likely,
               int end_bit, void* workspace, bool zeroed, unsigned* status, int* result_in_alt, cudaStream_t stream, bool position_values = false,
               bool counted = false);
// Digits of a sort, and where the histograms of its passes are collected and their exclusive scans (the digit bases) go.
constexpr int kRadixBits = 9;            // widest digit of a pass: 27 key bits sort in 3 passes, 32 in 4 x 8
constexpr int kRadix = 1 << kRadixBits;  // capacity of every per-digit array
constexpr int kMaxPasses = 4;
struct PassTable {
    int n_passes;
    int shift[kMaxPasses];
    int bits[kMaxPasses];
};
struct KeyHistogram {
    PassTable pt;
    unsigned *hist, *base;     // [kMaxPasses][kRadix]
    unsigned* blocks_done;
};
// A kernel that makes the keys of a sort can count their digits too (count_key, finish_histogram below) and spare the sort its pass over the
// keys: the histogram it fills, inside the workspace whose first sort_zero_bytes bytes have been cleared.  The sort is then called with `counted`.
KeyHistogram key_histogram(void* workspace, int64_t n, int64_t n_likely, int end_bit);
// Sorts the positions 0 .. n - 1 of the keys other than kNoKey: the first pass leaves the others out, so that whoever writes the keys need not compact them.  The
// keys have been counted (key_histogram(workspace, n, n, end_bit)), how many there are is in *count (device memory).  The workspace is sized for (n, n); the result is in the
// alternate buffers iff sort_pass_count(end_bit) is odd.  No key that takes part may equal kNoKey, also in bits above end_bit.
constexpr uint32_t kNoKey = 0xFFFFFFFFu;
int sort_marked_keys(uint32_t* keys, uint32_t* keys_alt, uint32_t* values, uint32_t* values_alt, int64_t n, unsigned long long* count, int end_bit, void* workspace,
                     unsigned* status, int* result_in_alt, cudaStream_t stream);
// The same, and every point carries a code with it: the first pass makes it from the point's footprint word (see Footprint in raster.cu), and code and position go
// through the other passes in one 64-bit word with the key bits that are still to be sorted by (the first pass's own are no longer needed), so that whoever
// reads the sorted positions need not gather the words.  Sorted positions and codes land in the values and in the keys of the result buffers (the
// keys themselves are gone).  A code is the word itself where bit 31 is clear, else `escape` + log2(tiles): the word is to be looked up then.
struct CarriedCodes {
    const uint32_t* quad = nullptr;   // per point; anything where the key is kNoKey
    int bits = 0;                     // of a code; 0: not carried
    uint32_t escape = 0;              // above every word with bit 31 clear
};
// The codes for n points with keys of end_bit bits and words below `words`; none (bits == 0) where key bits behind the first pass, code and position do
// not fit 64 bits.
CarriedCodes carried_codes(const uint32_t* quad, int64_t n, int end_bit, int64_t words);
int sort_marked_keys_with_codes(uint32_t* keys, uint32_t* keys_alt, uint32_t* values, uint32_t* values_alt, int64_t n, unsigned long long* count, int end_bit, const CarriedCodes& codes,
                                void* workspace, unsigned* status, int* result_in_alt, cudaStream_t stream);
// The number of pairs is *n_dev (device memory, <= n_max); the workspace is sized for (n_max, n_likely).  The result is in the
// alternate buffers iff sort_pass_count(end_bit) is odd, whatever the count turns out to be.
// Of this sort and of the marked ones: a tile that gives up its look-back leaves zero in the count.  Whatever reads the sorted lists has to take their length from there,
// in device memory: positions and keys that were not written are anything.
int sort_pairs_device_count(uint32_t* keys, uint32_t* keys_alt, uint32_t* values, uint32_t* values_alt, int64_t n_max, int64_t n_likely,
                            unsigned long long* n_dev, int end_bit, void* workspace, bool zeroed, unsigned* status, int* result_in_alt,
                            cudaStream_t stream, bool counted = false);

// More than 48 KB of dynamic shared memory is an opt-in per kernel AND per device: `done` is the
// caller's per-kernel table of devices already set up.
constexpr int kMaxDevices = 64;
// Number of multiprocessors of the current device (looked up once per device; 148 if the query fails).
int sm_count();

template <typename Kernel>
int opt_in_dynamic_smem(Kernel kernel, size_t bytes, bool (&done)[kMaxDevices]) {
    static std::mutex table_mutex;   // one per kernel: host threads may reach the same kernel's table together
    std::lock_guard<std::mutex> lock(table_mutex);
    int dev = 0;
    INPC_CUDA_TRY(cudaGetDevice(&dev));
    const bool tracked = dev >= 0 && dev < kMaxDevices;
    if (tracked && done[dev]) return INPC_OK;
    INPC_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    if (tracked) done[dev] = true;
    return INPC_OK;
}

// Blocks of `threads` threads and `bytes` of dynamic shared memory that fit a multiprocessor together, by what the runtime knows of the
// kernel's registers and shared memory (asked for once per kernel and device, with the opt-in above): the grid of a persistent kernel.
template <typename Kernel>
int resident_blocks(Kernel kernel, int threads, size_t bytes, int (&known)[kMaxDevices], int* blocks) {
    static std::mutex table_mutex;
    std::lock_guard<std::mutex> lock(table_mutex);
    int dev = 0;
    INPC_CUDA_TRY(cudaGetDevice(&dev));
    const bool tracked = dev >= 0 && dev < kMaxDevices;
    if (tracked && known[dev] > 0) { *blocks = known[dev]; return INPC_OK; }
    INPC_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    INPC_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, kernel, threads, bytes));
    if (*blocks < 1) *blocks = 1;
    if (tracked) known[dev] = *blocks;
    return INPC_OK;
}

// ---- device helpers ------------------------------------------------------------------------
#ifdef __CUDACC__
// ---- launches that overlap the end of the kernel before them ------------------------------------------
// Every kernel of the library is launched by `launch_chained` and starts with `await_previous_kernel()`.  The launch allows the
// grid to be set up, and its blocks to be placed, as soon as all blocks of the kernel before it in the stream have left, without
// waiting for that kernel's memory to be flushed and its completion to be reported; the wait returns when both are done.  A
// kernel that waits has also waited for everything before the one it waits for, so nothing but the gap between two
// launches changes.  No kernel may read or write global memory before the wait, and none may leave it out: a later one relies on it.
// Measured against plain launches, 36 kernels one after the other: training step of 10^6 samples at 801x533 485 -> 418 us, of 2^23 at
// 1237x822 1806 -> 1726, 2 * 10^6 gaussian splats 632 -> 580.  (With griddepcontrol.launch_dependents at the start of every kernel, so
// that the next one's blocks are placed while it still runs: 454, 1738 and 588, since waiting blocks take room from running
// ones; eight views on four streams 11318 -> 11464.)
template <typename... KernelArgs, typename... Args>
void launch_chained(void (*kernel)(KernelArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
    cudaLaunchAttribute attribute;
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = &attribute;
    config.numAttrs = 1;
    (void)cudaLaunchKernelEx(&config, kernel, static_cast<KernelArgs>(std::forward<Args>(args))...);   // the launch check behind it reads the error
}

__device__ __forceinline__ void await_previous_kernel() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31u; }

__device__ __forceinline__ unsigned warp_inclusive_scan(unsigned v) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane_id() >= (unsigned)o) v += t;
    }
    return v;
}

// ---- bulk asynchronous copies (the copy engine behind TMA, untiled form) ------------------------------
// global -> shared: one thread arms an mbarrier with the byte count and issues the copy; every thread
// that will read the data waits on the barrier's phase.  Source, destination and size must be
// multiples of 16 bytes.  The wait is bounded: a block that gives up reports it and the caller skips
// its work, the next entry point of the library then returns an error.
__device__ __forceinline__ unsigned shared_address(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbarrier_init(unsigned long long* bar, unsigned arrivals) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(shared_address(bar)), "r"(arrivals) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void bulk_load_to_shared(void* dst_shared, const void* src_global, unsigned bytes, unsigned long long* bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(shared_address(bar)), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(shared_address(dst_shared)),
                 "l"(src_global), "r"(bytes), "r"(shared_address(bar))
                 : "memory");
}

__device__ __forceinline__ bool mbarrier_wait_bounded(unsigned long long* bar, unsigned parity) {
    const unsigned addr = shared_address(bar);
    for (int spin = 0; spin < (1 << 20); ++spin) {
        unsigned done;
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n"
            "}\n"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// shared -> global: the writers of the shared data call `fence_shared_for_bulk()` before the block
// barrier, then one thread issues the store and waits until the source has been read.
__device__ __forceinline__ void fence_shared_for_bulk() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void bulk_store_from_shared(void* dst_global, const void* src_shared, unsigned bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst_global), "r"(shared_address(src_shared)), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

// ---- the block of a launch that finishes last goes on with what would be a one-block launch of its own ---------
// Every block calls this behind its last write; true in all threads of the last one.  `done` starts at zero.
__device__ __forceinline__ bool last_block(unsigned* done, unsigned n_blocks) {
    __shared__ bool s_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();   // covers the whole block's writes: they are ordered before it by the barrier
        s_last = atomicAdd(done, 1u) == n_blocks - 1u;
        __threadfence();
    }
    __syncthreads();
    return s_last;
}

// ---- digit histograms of the keys of a sort (see KeyHistogram) ------------------------------------------------
using BlockHistogram = unsigned[kMaxPasses][kRadix];   // in shared memory

__device__ __forceinline__ void clear_histogram(BlockHistogram& h) {
    for (unsigned i = threadIdx.x; i < kMaxPasses * kRadix; i += blockDim.x) (&h[0][0])[i] = 0u;
}

__device__ __forceinline__ void count_key(BlockHistogram& h, const PassTable& pt, uint32_t key) {
#pragma unroll
    for (int p = 0; p < kMaxPasses; ++p)
        if (p < pt.n_passes) atomicAdd(&h[p][(key >> pt.shift[p]) & ((1u << pt.bits[p]) - 1u)], 1u);
}

// Every block of the launch, behind its last count: adds the block's counts to the launch's; the block that finishes last turns those into
// digit bases (exclusive scans, all passes side by side: one round trip to memory and two barriers), which is a launch less.  *total, if
// asked for, receives the number of keys.  Blocks of at least kRadix / 2 threads.
__device__ __forceinline__ void finish_histogram(BlockHistogram& h, const KeyHistogram& out, unsigned n_blocks, unsigned long long* total) {
    constexpr unsigned kScanThreads = kRadix / 2, kScanWarps = kScanThreads / 32;   // two digits each
    __shared__ unsigned s_sum[kMaxPasses][kScanWarps];
    __syncthreads();
    for (unsigned i = threadIdx.x; i < kMaxPasses * kRadix; i += blockDim.x) {
        const unsigned c = (&h[0][0])[i];
        if (c) atomicAdd(out.hist + i, c);
    }
    if (!last_block(out.blocks_done, n_blocks)) return;
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    const bool scans = threadIdx.x < kScanThreads;
    uint2 own[kMaxPasses];
    unsigned inc[kMaxPasses];
    if (scans) {
#pragma unroll
        for (int p = 0; p < kMaxPasses; ++p) own[p] = p < out.pt.n_passes ? __ldcg(reinterpret_cast<const uint2*>(out.hist + p * kRadix) + threadIdx.x) : make_uint2(0u, 0u);
#pragma unroll
        for (int p = 0; p < kMaxPasses; ++p) {
            inc[p] = warp_inclusive_scan(own[p].x + own[p].y);
            if (lane == 31) s_sum[p][warp] = inc[p];
        }
    }
    __syncthreads();
    if (warp < (unsigned)kMaxPasses) {
        const unsigned sum = lane < kScanWarps ? s_sum[warp][lane] : 0u, before = warp_inclusive_scan(sum) - sum;
        if (lane < kScanWarps) s_sum[warp][lane] = before;
        if (total && warp == 0 && lane == kScanWarps - 1) *total = before + sum;
    }
    __syncthreads();
    if (scans) {
#pragma unroll
        for (int p = 0; p < kMaxPasses; ++p)
            if (p < out.pt.n_passes) {
                const unsigned second = s_sum[p][warp] + inc[p] - own[p].y;
                reinterpret_cast<uint2*>(out.base + p * kRadix)[threadIdx.x] = make_uint2(second - own[p].x, second);
            }
    }
}

// Block-wide exclusive scan of one unsigned per thread; `smem` needs (blockDim.x/32 + 1) words.
// Returns the exclusive prefix; *total receives the block sum (same value in every thread).
__device__ __forceinline__ unsigned block_exclusive_scan(unsigned v, unsigned* smem, unsigned* total) {
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
    const unsigned inc = warp_inclusive_scan(v);
    if (lane == 31) smem[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        unsigned w = lane < nwarps ? smem[lane] : 0u;
        unsigned winc = warp_inclusive_scan(w);
        if (lane < nwarps) smem[lane] = winc - w;
        if (lane == 31) smem[nwarps] = winc;
    }
    __syncthreads();
    const unsigned r = smem[warp] + inc - v;
    *total = smem[nwarps];
    __syncthreads();
    return r;
}
#endif

}  // namespace inpc
