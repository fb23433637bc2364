// Probability-field sampler of the inpc_b200 library.
//
// Per-view leaf weights -> normalised fp32 CDF (deterministic block scans) -> per-slot draws from a
// counter-based Philox4x32-10 stream: one Philox block yields the CDF uniform and the three jitter
// uniforms of a draw.  Every output slot owns its own sub-stream (seed, call, slot, attempt), so the
// training sampler needs no atomics and is reproducible; the reference's rejection sampler hands out
// slots with an atomic ticket and is not (sampling/src/sampling_kernels.cu:104-125).
// Citations are paths below INPCCudaBackend/INPCCudaBackend/sampling/ of the reference.
#include "common.cuh"
#include <type_traits>

namespace inpc {

namespace {

constexpr float kEps = 1e-8f;   // FLT_EPS of the reference's utils.h:8
constexpr int kThreads = 256;
constexpr int kMaxAttempts = 4096;

// ---- viewpoint weights: src/sampling_kernels.cu:9-64 ----------------------------------------
struct Rows {
    float r0[4], r1[4], r2[4];
};
__device__ __forceinline__ Rows load_rows(const float* __restrict__ w2c) {
    Rows m;
#pragma unroll
    for (int k = 0; k < 4; ++k) { m.r0[k] = __ldg(w2c + k); m.r1[k] = __ldg(w2c + 4 + k); m.r2[k] = __ldg(w2c + 8 + k); }
    return m;
}

// All sampler arithmetic spells out its fused multiply-adds, so that the CPU restatement used by the
// tests reproduces every value bit for bit.
__device__ __forceinline__ float affine(const float* r, float x, float y, float z) {
    return fmaf(r[2], z, fmaf(r[1], y, fmaf(r[0], x, r[3])));
}

__device__ __forceinline__ bool in_frustum(const Rows& m, const ViewParams& v, float px, float py, float pz, float* z_out) {
    const float vx = affine(m.r0, px, py, pz);
    const float vy = affine(m.r1, px, py, pz);
    const float z = affine(m.r2, px, py, pz);
    const float inv_z = 1.0f / (z + kEps);
    const float x = fmaf(vx * inv_z, v.fx, v.cx);
    const float y = fmaf(vy * inv_z, v.fy, v.cy);
    if (z_out) *z_out = z;
    return (z >= v.near_plane) & (z <= v.far_plane) & (x >= 0.0f) & (x < (float)v.width) & (y >= 0.0f) & (y < (float)v.height);
}

// weight of a leaf in a view: 0 outside the frustum
__device__ __forceinline__ float viewpoint_weight(const ViewParams& v, float cx, float cy, float cz, int level, float weight, float initial_size) {
    const Rows m = load_rows(v.w2c);
    float z;
    bool valid = in_frustum(m, v, cx, cy, cz, &z);
    if (!valid) {
        const float half_size = initial_size / scalbnf(1.0f, level + 1);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float ox = (k & 4) ? 1.0f : -1.0f, oy = (k & 2) ? 1.0f : -1.0f, oz = (k & 1) ? 1.0f : -1.0f;
            valid |= in_frustum(m, v, fmaf(half_size, ox, cx), fmaf(half_size, oy, cy), fmaf(half_size, oz, cz), nullptr);
        }
    }
    if (!valid) return 0.0f;
    const float depth_scale = fmaxf(fabsf(z - v.near_plane) / v.far_plane, kEps);
    // 2^(level/2), exact: the reference's exp2f(level * 0.5f) agrees to within the 2 ulp of exp2f
    const float size_scale = scalbnf((level & 1) ? 1.41421356237309504880f : 1.0f, level >> 1);
    return 1.0f / (depth_scale * size_scale) * weight;
}

// centre and edge length of a leaf in one 16-byte record: a draw then needs one load per leaf instead of four
__device__ __forceinline__ float4 leaf_record(float cx, float cy, float cz, int level, float initial_size) {
    return make_float4(cx, cy, cz, 1.0f / scalbnf(1.0f, level) * initial_size);
}

// The records alone, for the expected samples: they are drawn in the cells the filling call is given, which need not be those
// of the counting call.  (Reading the caller's four words per slot instead: 30 us more for 4 x 2^23 slots of 2^18 leaves.)
__global__ void __launch_bounds__(kThreads) leaf_records_kernel(int64_t n_cells, const float* __restrict__ centers, const int* __restrict__ levels,
                                                                float initial_size, float4* __restrict__ leaf_pack) {
    await_previous_kernel();
    const int64_t l = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (l < n_cells) leaf_pack[l] = leaf_record(__ldg(centers + 3 * l), __ldg(centers + 3 * l + 1), __ldg(centers + 3 * l + 2), __ldg(levels + l), initial_size);
}

// `max_bits` (optional, zero before): bit pattern of the largest weight, for the CDF behind it.
__global__ void __launch_bounds__(kThreads) viewpoint_weights_kernel(ViewParams v, int64_t n_cells,
                                                                     const float* __restrict__ centers,
                                                                     const int* __restrict__ levels,
                                                                     const float* __restrict__ weights,
                                                                     float initial_size, float* __restrict__ out,
                                                                     float4* __restrict__ leaf_pack, unsigned* max_bits) {
    await_previous_kernel();
    const int64_t l = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    const unsigned active = __ballot_sync(0xffffffffu, l < n_cells);
    if (l >= n_cells) return;
    const float cx = __ldg(centers + 3 * l), cy = __ldg(centers + 3 * l + 1), cz = __ldg(centers + 3 * l + 2);
    const int level = __ldg(levels + l);
    const float w = viewpoint_weight(v, cx, cy, cz, level, __ldg(weights + l), initial_size);
    out[l] = w;
    if (max_bits) {
        // NaN, infinite and non-positive weights do not take part (see to_fixed); the others order like their bit patterns
        const unsigned m = __reduce_max_sync(active, w > 0.0f && w <= 3.402823466e38f ? __float_as_uint(w) : 0u);
        if (lane_id() == 0 && m > 0u) atomicMax(max_bits, m);
    }
    if (leaf_pack) leaf_pack[l] = leaf_record(cx, cy, cz, level, initial_size);
}

// Largest weight of every leaf over up to kViewsPerPass views (and over *out, when earlier passes left something there).
// The leaf is read once for all views; one launch per view and a maximum after it were 32 launches for 16 views.
constexpr int kViewsPerPass = 32;
struct ViewSet {
    int count;
    ViewParams v[kViewsPerPass];
};
__global__ void __launch_bounds__(kThreads) max_viewpoint_weights_kernel(const __grid_constant__ ViewSet views, int64_t n_cells, const float* __restrict__ centers,
                                                                         const int* __restrict__ levels, const float* __restrict__ weights,
                                                                         float initial_size, bool first, float* __restrict__ out) {
    await_previous_kernel();
    const int64_t l = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (l >= n_cells) return;
    const float cx = __ldg(centers + 3 * l), cy = __ldg(centers + 3 * l + 1), cz = __ldg(centers + 3 * l + 2);
    const int level = __ldg(levels + l);
    const float weight = __ldg(weights + l);
    float best = first ? 0.0f : out[l];
    for (int j = 0; j < views.count; ++j) best = fmaxf(best, viewpoint_weight(views.v[j], cx, cy, cz, level, weight, initial_size));
    out[l] = best;
}

// ---- CDF: src/sampling.cu:97-125 (Sum, multiply by 1/sum, InclusiveSum) -------------------------
// The reference scans fp32 values with CUB, whose summation order is unspecified.  Here every weight
// is first expressed as a 39-bit fixed-point fraction of the largest weight; integer prefix sums are
// exact and associative, so the CDF is independent of how the scan is parallelised, monotone, and
// reproducible bit for bit anywhere (the CPU restatement is a plain loop):
//   q_i = trunc(w_i / w_max * 2^39),  P_i = q_0 + ... + q_i,  cdf_i = float(P_i / P_last),
//   sum = float(P_last * 2^-39 * w_max).
constexpr int kCdfThreads = 256;
constexpr int kCdfItems = 8;
constexpr int kCdfChunk = kCdfThreads * kCdfItems;
constexpr float kFixedOne = 549755813888.0f;   // 2^39
constexpr double kFixedInv = 1.0 / 549755813888.0;

// Non-finite and non-positive weights count as zero (an infinite one would make the quotient NaN, whose
// conversion to an integer is undefined).
__device__ __forceinline__ unsigned long long to_fixed(float w, float w_max) {
    return (w > 0.0f && w <= 3.402823466e38f) ? (unsigned long long)((w / w_max) * kFixedOne) : 0ull;
}

// largest weight via atomicMax on the bit pattern (valid for non-negative floats; order-free)
__global__ void __launch_bounds__(kCdfThreads) cdf_max_kernel(const float* __restrict__ w, int64_t n, unsigned* __restrict__ max_bits) {
    await_previous_kernel();
    const int64_t base = (int64_t)blockIdx.x * kCdfChunk + (int64_t)threadIdx.x * kCdfItems;
    float m = 0.0f;
#pragma unroll
    for (int k = 0; k < kCdfItems; ++k)
        if (base + k < n) {
            const float v = __ldg(w + base + k);
            if (v <= 3.402823466e38f) m = fmaxf(m, v);   // NaN and +inf do not take part
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
    if (lane_id() == 0 && m > 0.0f) atomicMax(max_bits, __float_as_uint(m));
}

__device__ __forceinline__ unsigned long long warp_inclusive_scan_u64(unsigned long long v) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane_id() >= (unsigned)o) v += t;
    }
    return v;
}

// exclusive scan of one u64 per thread over the block; smem needs blockDim/32 + 1 entries
__device__ __forceinline__ unsigned long long block_exclusive_scan_u64(unsigned long long v, unsigned long long* smem,
                                                                     unsigned long long* total) {
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
    const unsigned long long inc = warp_inclusive_scan_u64(v);
    if (lane == 31) smem[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const unsigned long long wv = lane < nwarps ? smem[lane] : 0ull;
        const unsigned long long winc = warp_inclusive_scan_u64(wv);
        if (lane < nwarps) smem[lane] = winc - wv;
        if (lane == 31) smem[nwarps] = winc;
    }
    __syncthreads();
    const unsigned long long r = smem[warp] + inc - v;
    *total = smem[nwarps];
    __syncthreads();
    return r;
}

__global__ void __launch_bounds__(kCdfThreads) cdf_chunk_sums_kernel(const float* __restrict__ w, int64_t n,
                                                                     const unsigned* __restrict__ max_bits, unsigned* done,
                                                                     unsigned long long* chunk_sums, unsigned long long* __restrict__ total_out,
                                                                     float* __restrict__ sum_out) {
    await_previous_kernel();
    __shared__ unsigned long long s[kCdfThreads / 32 + 1];
    const float w_max = __uint_as_float(__ldg(max_bits));
    const int64_t base = (int64_t)blockIdx.x * kCdfChunk + (int64_t)threadIdx.x * kCdfItems;
    unsigned long long acc = 0;
#pragma unroll
    for (int k = 0; k < kCdfItems; ++k)
        if (base + k < n) acc += to_fixed(__ldg(w + base + k), w_max);
    unsigned long long total;
    block_exclusive_scan_u64(acc, s, &total);
    if (threadIdx.x == 0) chunk_sums[blockIdx.x] = total;
    // the last block: exclusive scan of the chunk sums in place; total -> *total_out, fp32 sum -> *sum_out
    if (!last_block(done, gridDim.x)) return;
    unsigned long long running = 0;
    for (unsigned first = 0; first < gridDim.x; first += kCdfThreads) {
        const unsigned j = first + threadIdx.x;
        const unsigned long long c = j < gridDim.x ? __ldcg(chunk_sums + j) : 0ull;
        const unsigned long long ex = block_exclusive_scan_u64(c, s, &total);
        if (j < gridDim.x) chunk_sums[j] = running + ex;
        running += total;
    }
    if (threadIdx.x == 0) {
        *total_out = running;
        *sum_out = (float)((double)running * kFixedInv * (double)w_max);
    }
}

__global__ void __launch_bounds__(kCdfThreads) cdf_finalize_kernel(const float* __restrict__ w, int64_t n,
                                                                   const unsigned* __restrict__ max_bits,
                                                                   const unsigned long long* __restrict__ chunk_base,
                                                                   const unsigned long long* __restrict__ total_ptr,
                                                                   float* __restrict__ cdf) {
    await_previous_kernel();
    __shared__ unsigned long long s[kCdfThreads / 32 + 1];
    const float w_max = __uint_as_float(__ldg(max_bits));
    const double total = (double)__ldg(total_ptr);
    const int64_t base = (int64_t)blockIdx.x * kCdfChunk + (int64_t)threadIdx.x * kCdfItems;
    unsigned long long q[kCdfItems];
    unsigned long long acc = 0;
#pragma unroll
    for (int k = 0; k < kCdfItems; ++k) {
        acc += base + k < n ? to_fixed(__ldg(w + base + k), w_max) : 0ull;
        q[k] = acc;
    }
    unsigned long long block_total;
    const unsigned long long before = __ldg(chunk_base + blockIdx.x) + block_exclusive_scan_u64(acc, s, &block_total);
#pragma unroll
    for (int k = 0; k < kCdfItems; ++k)
        if (base + k < n) cdf[base + k] = (float)((double)(before + q[k]) / total);
}

// ---- Philox4x32-10 ----------------------------------------------------------------------------
// The ten round keys are the same for all threads of a launch: the host makes them, the kernels read them from the
// constant bank as operands of the xors.
struct PhiloxKeys {
    uint2 k[10];
    unsigned call_lo, call_hi;
};
PhiloxKeys philox_keys(unsigned long long seed, unsigned long long call) {
    PhiloxKeys p;
    unsigned x = (unsigned)seed, y = (unsigned)(seed >> 32);
    for (int r = 0; r < 10; ++r, x += 0x9E3779B9u, y += 0xBB67AE85u) p.k[r] = make_uint2(x, y);
    p.call_lo = (unsigned)call;
    p.call_hi = (unsigned)(call >> 32);
    return p;
}
__device__ __forceinline__ uint4 philox4x32_10(uint4 c, const PhiloxKeys& keys) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const unsigned long long p0 = (unsigned long long)0xD2511F53u * c.x, p1 = (unsigned long long)0xCD9E8D57u * c.z;
        c = make_uint4((unsigned)(p1 >> 32) ^ c.y ^ keys.k[r].x, (unsigned)p1, (unsigned)(p0 >> 32) ^ c.w ^ keys.k[r].y, (unsigned)p0);
    }
    return c;
}

// 23 random mantissa bits -> [0,1), the mapping of include/pcg32.h:105-114
__device__ __forceinline__ float unit_float(unsigned r) { return __uint_as_float((r >> 9) | 0x3f800000u) - 1.0f; }

struct Draw {
    float u, jx, jy, jz;
    unsigned raw_u;   // the 32 bits u was made of
};
// stream layout: counter = (slot, attempt, call lo, call hi), key = seed (lo, hi)
__device__ __forceinline__ Draw philox_draw(const PhiloxKeys& keys, unsigned slot, unsigned attempt) {
    const uint4 o = philox4x32_10(make_uint4(slot, attempt, keys.call_lo, keys.call_hi), keys);
    Draw d;
    d.u = unit_float(o.x); d.jx = unit_float(o.y); d.jy = unit_float(o.z); d.jz = unit_float(o.w);
    d.raw_u = o.x;
    return d;
}

// first index with cdf[idx] >= u, clamped to n-1: include/sampling_utils.h:49-69
__device__ __forceinline__ unsigned lower_bound_clamped(const float* __restrict__ cdf, float u, unsigned n) {
    unsigned first = 0, count = n;
    while (count > 0) {
        const unsigned step = count >> 1;
        if (__ldg(cdf + first + step) < u) { first += step + 1; count -= step + 1; }
        else count = step;
    }
    return min(first, n - 1);
}

// Guide table: one 16-byte record per bucket b of [0, 1), b = 0 .. 2^k - 1: {lower_bound(cdf, b / 2^k), the two CDF values from
// there on, lower_bound(cdf, (b + 1) / 2^k)}.  The CDF is monotone (integer prefix sums), so the look-up for a uniform in
// bucket b only has to search between the two bounds, with bit-identical results.  A draw is bound by the number of 32-byte
// sectors it gathers from L2 (all tables are larger than L1): the record settles the draws whose bucket holds at most two
// CDF steps, nine in ten with as many buckets as leaves, in one sector where separate guide and CDF arrays took three.
constexpr int kGuidePerBlock = kThreads - 1;   // the last thread of a block only finds the end of the last bucket
// With `leaf_pack` a record is 32 bytes, one sector: behind the four words lies the geometry of its first leaf, which is the leaf of
// most draws (a leaf of some weight covers whole buckets), and a draw that ends there makes one gather instead of two.
struct __align__(32) GuideRecord {
    uint4 steps;
    float4 leaf;
};
__global__ void __launch_bounds__(kThreads) guide_table_kernel(const float* __restrict__ cdf, unsigned n_cells, int k, uint4* __restrict__ guide,
                                                               const float4* __restrict__ leaf_pack) {
    await_previous_kernel();
    __shared__ unsigned s_first[kThreads];
    const unsigned b = blockIdx.x * kGuidePerBlock + threadIdx.x, n_buckets = 1u << k;
    unsigned first = 0, count = b <= n_buckets ? n_cells : 0u;
    // bucket edge as a float: (b << (23 - k)) * 2^-23, exact
    const float edge = (float)(b << (23 - k)) * 1.1920928955078125e-07f;
    while (count > 0) {
        const unsigned step = count >> 1;
        if (__ldg(cdf + first + step) < edge) { first += step + 1; count -= step + 1; }
        else count = step;
    }
    s_first[threadIdx.x] = first;
    __syncthreads();
    if (threadIdx.x == kGuidePerBlock || b >= n_buckets) return;
    const float c0 = first < n_cells ? __ldg(cdf + first) : 2.0f, c1 = first + 1u < n_cells ? __ldg(cdf + first + 1u) : 2.0f;
    const uint4 steps = make_uint4(first, __float_as_uint(c0), __float_as_uint(c1), s_first[threadIdx.x + 1]);
    if (leaf_pack) reinterpret_cast<GuideRecord*>(guide)[b] = GuideRecord{steps, __ldg(leaf_pack + min(first, n_cells - 1u))};
    else guide[b] = steps;
}

// The record of a uniform's bucket; r: the raw 32 random bits the uniform is made of (u = (r >> 9) * 2^-23)
__device__ __forceinline__ uint4 guide_record(const uint4* __restrict__ guide, int k, unsigned r) { return __ldg(guide + ((r >> 9) >> (23 - k))); }
// ... with its first leaf, in one 32-byte load.  That is of PTX ISA 8.8, CUDA 12.9; with an older toolkit that knows sm_100a two loads
// of 16 bytes take its place (2^23 training samples 128 -> 139 us, plain ones 113 -> 125, the weights and the CDF included).
#ifndef INPC_WIDE_LOADS
#define INPC_WIDE_LOADS (__CUDACC_VER_MAJOR__ > 12 || (__CUDACC_VER_MAJOR__ == 12 && __CUDACC_VER_MINOR__ >= 9))
#endif
__device__ __forceinline__ GuideRecord packed_guide_record(const uint4* __restrict__ guide, int k, unsigned r) {
    const GuideRecord* p = reinterpret_cast<const GuideRecord*>(guide) + ((r >> 9) >> (23 - k));
    GuideRecord g;
#if INPC_WIDE_LOADS
    asm volatile("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(g.steps.x), "=r"(g.steps.y), "=r"(g.steps.z), "=r"(g.steps.w), "=f"(g.leaf.x), "=f"(g.leaf.y), "=f"(g.leaf.z), "=f"(g.leaf.w)
                 : "l"(p));
#else
    g.steps = __ldg(&p->steps);
    g.leaf = __ldg(&p->leaf);
#endif
    return g;
}
__device__ __forceinline__ unsigned settle_lower_bound(const float* __restrict__ cdf, const uint4& g, float u, unsigned n) {
    unsigned first = g.x;
    if (__uint_as_float(g.y) < u) {
        first += 1u;
        if (__uint_as_float(g.z) < u) {
            first += 1u;
            unsigned count = g.w > first ? g.w - first : 0u;
            while (count > 0) {
                const unsigned step = count >> 1;
                if (__ldg(cdf + first + step) < u) { first += step + 1; count -= step + 1; }
                else count = step;
            }
        }
    }
    return min(first, n - 1);
}
__device__ __forceinline__ unsigned guided_lower_bound(const float* __restrict__ cdf, const uint4* __restrict__ guide, int k,
                                                       unsigned r, float u, unsigned n) {
    return settle_lower_bound(cdf, guide_record(guide, k, r), u, n);
}

// Positions of the kThreads consecutive samples of a block, first sample `first`, leave as 16-byte vectors through shared
// memory (three 4-byte stores with a stride of 12 bytes write every sector three times into L2).
__device__ __forceinline__ void store_positions(float* s_pos, float x, float y, float z, int64_t first, int64_t n, float* __restrict__ positions) {
    s_pos[3 * threadIdx.x] = x; s_pos[3 * threadIdx.x + 1] = y; s_pos[3 * threadIdx.x + 2] = z;
    __syncthreads();
    const int floats = 3 * (int)min((int64_t)kThreads, n - first);
    float* dst = positions + 3 * first;
    if (floats == 3 * kThreads && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
        if (threadIdx.x < 3 * kThreads / 4) reinterpret_cast<float4*>(dst)[threadIdx.x] = reinterpret_cast<const float4*>(s_pos)[threadIdx.x];
    } else {
        for (int k = threadIdx.x; k < floats; k += kThreads) dst[k] = s_pos[k];
    }
}

// ---- training samples: same acceptance test as src/sampling_kernels.cu:98-113 -------------------
// A block makes PER * kThreads consecutive samples.  The first attempts of a thread's PER slots go together, their gathers in
// flight at the same time; slots whose point lies outside the view go to a list in shared memory, which all threads of the block then
// work off, attempt by attempt.  What a slot draws at an attempt depends on nothing else, so the samples are those of a loop per slot.
// Bound by instruction issue (240 instructions per sample, a third of them Philox; 54 % of the issue slots) and by waiting for the
// gather.  2^23 samples of 2^18 leaves: one slot per thread looping until it succeeds (a warp then makes as many attempts as its
// unluckiest slot) 109 us; two slots per thread and the list 101, with the leaf's geometry in the guide record 97 (five blocks per
// multiprocessor; with six 101, four 107; four slots per thread 111).
template <int PER>
__global__ void __launch_bounds__(kThreads, PER == 1 ? 6 : 5) training_samples_kernel(
    ViewParams v, const __grid_constant__ PhiloxKeys keys, const float* __restrict__ cdf,
    const uint4* __restrict__ guide, int guide_bits, const float* __restrict__ sum_ptr, unsigned n_cells,
    const float4* __restrict__ leaf_pack, int64_t n_samples, float* __restrict__ positions, long long* __restrict__ indices,
    volatile unsigned* status) {
    await_previous_kernel();
    constexpr unsigned kBlock = PER * kThreads;
    __shared__ __align__(16) float s_pos[3 * kBlock];
    __shared__ unsigned s_leaf[kBlock];
    __shared__ unsigned short s_retry[2][kBlock];   // slots of the block that make another attempt: now, and after that
    __shared__ unsigned s_count[2];
    const unsigned tid = threadIdx.x;
    const int64_t block_first = (int64_t)blockIdx.x * kBlock;
    const unsigned in_block = (unsigned)min((int64_t)kBlock, n_samples - block_first);
    const bool any = __ldg(sum_ptr) > 0.0f;
    if (tid < 2u) s_count[tid] = 0u;
    __syncthreads();
    const Rows m = load_rows(v.w2c);
    // the point of slot `local` in the leaf a draw has found; false if it lies outside the view
    auto place = [&](unsigned local, const Draw& d, const GuideRecord& g) -> bool {
        const unsigned leaf = settle_lower_bound(cdf, g.steps, d.u, n_cells);
        float4 lp = g.leaf;
        if (leaf != min(g.steps.x, n_cells - 1u)) lp = __ldg(leaf_pack + leaf);
        const float x = fmaf(d.jx - 0.5f, lp.w, lp.x);
        const float y = fmaf(d.jy - 0.5f, lp.w, lp.y);
        const float z = fmaf(d.jz - 0.5f, lp.w, lp.z);
        s_pos[3 * local] = x; s_pos[3 * local + 1] = y; s_pos[3 * local + 2] = z;
        s_leaf[local] = leaf;
        const float vz = affine(m.r2, x, y, z);
        if (vz < v.near_plane || vz > v.far_plane) return false;
        const float inv_z = 1.0f / (vz + kEps);
        const float sx = fmaf(affine(m.r0, x, y, z) * inv_z, v.fx, v.cx);
        if (sx < 0.0f || sx >= (float)v.width) return false;
        const float sy = fmaf(affine(m.r1, x, y, z) * inv_z, v.fy, v.cy);
        return !(sy < 0.0f || sy >= (float)v.height);
    };
    auto retry = [&](unsigned list, unsigned local) { s_retry[list][atomicAdd(&s_count[list], 1u)] = (unsigned short)local; };
    if (any) {
        Draw d[PER];
        GuideRecord g[PER];
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            d[k] = philox_draw(keys, (unsigned)(block_first + k * kThreads + tid), 0u);
            g[k] = packed_guide_record(guide, guide_bits, d[k].raw_u);
        }
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const unsigned local = k * kThreads + tid;
            if (local < in_block && !place(local, d[k], g[k])) retry(0u, local);
        }
        unsigned cur = 0u;
        for (unsigned a = 1; a < (unsigned)kMaxAttempts; ++a, cur ^= 1u) {
            __syncthreads();
            const unsigned n = s_count[cur];
            if (n == 0u) break;
            for (unsigned i = tid; i < n; i += kThreads) {
                const unsigned local = s_retry[cur][i];
                const Draw e = philox_draw(keys, (unsigned)(block_first + local), a);
                const bool ok = place(local, e, packed_guide_record(guide, guide_bits, e.raw_u));
                if (!ok) {
                    if (a + 1u < (unsigned)kMaxAttempts) retry(cur ^ 1u, local);
                    else status[STATUS_SAMPLER_EXHAUSTED] = 1u;   // the last attempt's point stays
                }
            }
            __syncthreads();
            if (tid == 0u) s_count[cur] = 0u;
        }
    } else {
        // src/sampling.cu:107-111: zero positions, indices of -1
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const unsigned local = k * kThreads + tid;
            s_pos[3 * local] = s_pos[3 * local + 1] = s_pos[3 * local + 2] = 0.0f;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const unsigned local = k * kThreads + tid;
        if (local < in_block) indices[block_first + local] = any ? (long long)s_leaf[local] : -1;
    }
    const unsigned floats = 3u * in_block;
    float* dst = positions + 3 * block_first;
    if (in_block == kBlock && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
        for (unsigned k = tid; k < 3u * kBlock / 4u; k += kThreads) reinterpret_cast<float4*>(dst)[k] = reinterpret_cast<const float4*>(s_pos)[k];
    } else {
        for (unsigned k = tid; k < floats; k += kThreads) dst[k] = s_pos[k];
    }
}

// ---- unconditional samples: src/sampling_kernels.cu:128-150 with the Philox stream ----------------
__global__ void __launch_bounds__(kThreads) samples_kernel(const __grid_constant__ PhiloxKeys keys,
                                                           const float* __restrict__ cdf, const uint4* __restrict__ guide,
                                                           int guide_bits, unsigned n_cells,
                                                           const float4* __restrict__ leaf_pack, int64_t n_samples,
                                                           float* __restrict__ positions) {
    await_previous_kernel();
    __shared__ __align__(16) float s_pos[3 * kThreads];
    const int64_t block_first = (int64_t)blockIdx.x * kThreads;
    const Draw d = philox_draw(keys, (unsigned)(block_first + threadIdx.x), 0u);
    const GuideRecord g = packed_guide_record(guide, guide_bits, d.raw_u);
    const unsigned leaf = settle_lower_bound(cdf, g.steps, d.u, n_cells);
    float4 lp = g.leaf;
    if (leaf != min(g.steps.x, n_cells - 1u)) lp = __ldg(leaf_pack + leaf);
    store_positions(s_pos, fmaf(d.jx - 0.5f, lp.w, lp.x), fmaf(d.jy - 0.5f, lp.w, lp.y), fmaf(d.jz - 0.5f, lp.w, lp.z), block_first, n_samples, positions);
}

__global__ void __launch_bounds__(kThreads) draw_leaves_kernel(const float* __restrict__ cdf, unsigned n_cells,
                                                               const float* __restrict__ u, int64_t n,
                                                               long long* __restrict__ out) {
    await_previous_kernel();
    const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (i >= n) return;
    out[i] = (long long)lower_bound_clamped(cdf, __ldg(u + i), n_cells);
}

// ---- expected samples: src/sampling_kernels.cu:152-205 ----------------------------------------
// Sums of the counts of kThreads leaves, exclusively scanned in place by the block that finishes last; the total -> *total_out.
// `weights` (optional): the counts are made here, max(1, round(w / sum * n_samples)) for every leaf with a positive weight.
__global__ void __launch_bounds__(kThreads) count_chunk_sums_kernel(const float* __restrict__ weights, const float* __restrict__ sum_ptr, unsigned n_samples,
                                                                    unsigned* __restrict__ counts, int64_t n, unsigned* done, unsigned* chunk_sums,
                                                                    unsigned long long* __restrict__ total_out) {
    await_previous_kernel();
    __shared__ unsigned s_scan[kThreads / 32 + 1];
    const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    unsigned c = 0;
    if (i < n) {
        if (weights) {
            const float w = __ldg(weights + i);
            const float sum = __ldg(sum_ptr);
            if (w > 0.0f && sum > 0.0f) {
                const float norm = 1.0f / sum;
                c = (unsigned)max(__float2int_rn(w * norm * static_cast<float>(n_samples)), 1);
            }
            counts[i] = c;
        } else {
            c = counts[i];
        }
    }
    unsigned total;
    block_exclusive_scan(c, s_scan, &total);
    if (threadIdx.x == 0) chunk_sums[blockIdx.x] = total;
    if (!last_block(done, gridDim.x)) return;
    unsigned long long running = 0;
    for (unsigned first = 0; first < gridDim.x; first += kThreads * 8) {
        const unsigned j0 = first + threadIdx.x * 8;
        unsigned v[8], sum = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) { v[k] = j0 + k < gridDim.x ? __ldcg(chunk_sums + j0 + k) : 0u; sum += v[k]; }
        unsigned ex = (unsigned)running + block_exclusive_scan(sum, s_scan, &total);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (j0 + k < gridDim.x) chunk_sums[j0 + k] = ex;
            ex += v[k];
        }
        running += total;
    }
    if (threadIdx.x == 0) *total_out = running;
}

// offsets[l] = inclusive prefix of counts (the reference's sample_offsets)
__global__ void __launch_bounds__(kThreads) count_offsets_kernel(const unsigned* __restrict__ counts, int64_t n,
                                                                 const unsigned* __restrict__ chunk_base,
                                                                 unsigned* __restrict__ offsets) {
    await_previous_kernel();
    __shared__ unsigned s_scan[kThreads / 32 + 1];
    const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    const unsigned c = i < n ? counts[i] : 0u;
    unsigned total;
    const unsigned ex = block_exclusive_scan(c, s_scan, &total);
    if (i < n) offsets[i] = chunk_base[blockIdx.x] + ex + c;
}

// Slots whose leaves are given by inclusive offsets: slot r lies in leaf upper_bound(offsets, r).  A block takes
// kRunSlots consecutive slots, so its leaves are consecutive too: one warp finds the first and last of them (a 32-way
// search, four dependent trips to L2 for 2^20 leaves), their offsets are copied to shared memory and every slot searches
// those few.  (A search of all leaves per slot was 18 dependent gathers: 561 us for 2^25 slots over 2^18 leaves.)
constexpr int kRunPerThread = 8;
constexpr int kRunSlots = kThreads * kRunPerThread;
constexpr unsigned kRunLeaves = 2048;   // offsets kept in shared memory; a run over more leaves (empty ones between) reads L2

struct LeafRun {
    unsigned offsets[kRunLeaves];
    unsigned first, count;   // leaves first .. first + count - 1 hold the block's slots
};

// first index with offsets[idx] > r, by all lanes of one warp; n if there is none
__device__ __forceinline__ unsigned warp_upper_bound(const unsigned* __restrict__ offsets, unsigned n, unsigned r) {
    unsigned lo = 0, hi = n;   // the answer lies in [lo, hi]
    while (hi - lo > 0) {
        const unsigned step = (hi - lo + 31u) / 32u;
        const unsigned probe = lo + lane_id() * step + step - 1u;   // last element of this lane's piece
        const bool above = probe >= hi || __ldg(offsets + probe) > r;
        const unsigned b = __ballot_sync(0xffffffffu, above);
        if (b == 0u) return hi;
        lo += (unsigned)(__ffs(b) - 1) * step;
        hi = min(hi, lo + step - 1u);
    }
    return lo;
}

// Finds the run of leaves that holds slots [r0, r1]; ends with a block barrier.
__device__ __forceinline__ void find_leaf_run(LeafRun& run, const unsigned* __restrict__ offsets, unsigned n_cells, unsigned r0, unsigned r1) {
    const unsigned warp = threadIdx.x >> 5;
    if (warp < 2) {
        const unsigned l = min(warp_upper_bound(offsets, n_cells, warp == 0 ? r0 : r1), n_cells - 1u);
        if (lane_id() == 0) { if (warp == 0) run.first = l; else run.count = l; }
    }
    __syncthreads();
    const unsigned first = run.first, count = run.count - first + 1u;
    __syncthreads();
    if (threadIdx.x == 0) run.count = count;
    for (unsigned k = threadIdx.x; k < min(count, kRunLeaves); k += kThreads) run.offsets[k] = __ldg(offsets + first + k);
    __syncthreads();
}

// The leaf (index within the run) of slot r, r ascending over the lanes of a warp and from row to row; `k`: where the last row ended, all lanes
// the same.  Most rows lie in one leaf, which one comparison shows; the others search from there.
__device__ __forceinline__ unsigned leaf_of_row(const LeafRun& run, const unsigned* __restrict__ offsets, unsigned r, unsigned& k) {
    const unsigned m = run.count;
    const bool local = m <= kRunLeaves;
    auto end_of = [&](unsigned l) { return local ? run.offsets[l] : __ldg(offsets + run.first + l); };
    unsigned l = k;
    if (__any_sync(0xffffffffu, l + 1u < m && end_of(l) <= r)) {
        unsigned count = m - l;
        while (count > 0) {
            const unsigned step = count >> 1;
            if (end_of(l + step) <= r) { l += step + 1; count -= step + 1; }
            else count = step;
        }
        l = min(l, m - 1u);
    }
    k = __shfl_sync(0xffffffffu, l, 31);
    return l;
}

// The positions of a warp's row of `here` consecutive slots leave as 16-byte vectors where they are aligned, in whole 128-byte lines otherwise.
__device__ __forceinline__ void store_row(float* s_row, float x, float y, float z, unsigned here, float* __restrict__ dst) {
    const unsigned lane = lane_id();
    __syncwarp();   // the row before has been read
    s_row[3 * lane] = x; s_row[3 * lane + 1] = y; s_row[3 * lane + 2] = z;
    __syncwarp();
    if (here == 32u && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
        if (lane < 24u) reinterpret_cast<float4*>(dst)[lane] = reinterpret_cast<const float4*>(s_row)[lane];
    } else {
#pragma unroll
        for (unsigned k = 0; k < 3; ++k)
            if (32u * k + lane < 3u * here) dst[32u * k + lane] = s_row[32u * k + lane];
    }
}

// slot i jitters inside leaf upper_bound(offsets, i % n_created): the load-balanced form of the reference's per-leaf fill
// loop + gather.  blockIdx.y counts the copies i / n_created, whose slots a run never leaves; a warp takes kRunPerThread rows of 32 consecutive
// slots, finds their leaves once for all copies (before: a search in every slot and copy, the run found once per copy, and a barrier per store: 4 x 2^23 slots 242 -> 156 us).
__global__ void __launch_bounds__(kThreads) expected_samples_kernel(const __grid_constant__ PhiloxKeys keys,
                                                                    const unsigned* __restrict__ offsets, unsigned n_cells,
                                                                    const float4* __restrict__ leaf_pack, unsigned n_created,
                                                                    unsigned n_copies, float* __restrict__ positions) {
    await_previous_kernel();
    __shared__ LeafRun run;
    __shared__ __align__(16) float s_pos[kThreads / 32][96];
    const unsigned r0 = blockIdx.x * (unsigned)kRunSlots;
    const unsigned in_block = min((unsigned)kRunSlots, n_created - r0);
    find_leaf_run(run, offsets, n_cells, r0, r0 + in_block - 1u);
    const unsigned warp = threadIdx.x >> 5, lane = lane_id();
    unsigned k = 0;
    for (unsigned row = 0; row < (unsigned)kRunPerThread; ++row) {
        const unsigned first = (warp * kRunPerThread + row) * 32u;
        if (first >= in_block) break;
        const unsigned here = min(32u, in_block - first), r = r0 + first + min(lane, here - 1u);
        const float4 lp = __ldg(leaf_pack + run.first + leaf_of_row(run, offsets, r, k));
        for (unsigned copy = blockIdx.y; copy < n_copies; copy += gridDim.y) {
            const int64_t copy_first = (int64_t)copy * n_created;
            const Draw d = philox_draw(keys, (unsigned)(copy_first + r), 0u);
            store_row(s_pos[warp], fmaf(d.jx - 0.5f, lp.w, lp.x), fmaf(d.jy - 0.5f, lp.w, lp.y), fmaf(d.jz - 0.5f, lp.w, lp.z), here, positions + 3 * (copy_first + r0 + first));
        }
    }
}

// ---- global point cloud: Modules/ProbabilityField.py:121-144 + utils.py:36-64 -----------------------
// counts[leaf] = number of the n multinomial draws that fell into the leaf (torch.multinomial +
// bincount in the reference; here the library's own Philox stream, one draw per slot)
constexpr int kDrawsPerThread = 4;
// One counter takes an addition every 2.7 ns, and the heaviest of 2.3 * 10^5 leaves of a trained field is drawn every two hundredth time: with
// one array of counts that leaf alone set the time: 2^25 draws 355 us, with 4 / 8 / 16 arrays 294 / 270 / 264.  The blocks share kCountParts, the caller's
// and the rest in the workspace, added up afterwards.
constexpr unsigned kCountParts = 8;
// Where they pay.  A call with one array / eight, us: equal weights, 64 draws a leaf and more: 2.3 * 10^5 leaves and 2^24 draws 189 / 180, 4096 and
// 2^20 85 / 76; fewer: 2.3 * 10^5 leaves and 2^22 draws 92 / 97, 2^20 leaves and 2^25 draws 320 / 333.  Normal deviates of two in the exponent, the
// heaviest leaf drawn some 5000 times 79 / 69, 10^4 times 155 / 127, 1.6 * 10^5 times 582 / 386; 2400 times 98 / 98.  The arrays of 2^22 leaves no longer stay in
// L2: 2^25 draws of them 475 / 830, of 2^24 941 / 1998.
constexpr int64_t kManyDraws = 1 << 20;
constexpr int64_t kManyDrawsOfLeaf = 4096, kManyDrawsPerLeaf = 64;
constexpr int64_t kCountPartLeaves = 1 << 20;
bool use_count_parts(int64_t n_samples, int64_t n_cells, float largest, float sum) {
    return n_samples >= kManyDraws && n_cells <= kCountPartLeaves &&
           ((double)n_samples * largest >= (double)kManyDrawsOfLeaf * sum || n_samples >= kManyDrawsPerLeaf * n_cells);
}
__global__ void __launch_bounds__(kThreads) add_count_parts_kernel(const unsigned* __restrict__ parts, int64_t n, unsigned* __restrict__ counts) {
    await_previous_kernel();
    const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (i >= n) return;
    unsigned sum = counts[i];
#pragma unroll
    for (unsigned k = 0; k + 1u < kCountParts; ++k) sum += __ldg(parts + k * n + i);
    counts[i] = sum;
}
__global__ void __launch_bounds__(kThreads) leaf_histogram_kernel(const __grid_constant__ PhiloxKeys keys,
                                                                  const float* __restrict__ cdf, const uint4* __restrict__ guide,
                                                                  int guide_bits, unsigned n_cells, int64_t n_samples,
                                                                  unsigned* counts, unsigned* parts, unsigned n_parts) {
    await_previous_kernel();
    const unsigned part = blockIdx.x % n_parts;
    if (part > 0u) counts = parts + (size_t)(part - 1u) * n_cells;
    // the table gathers of a thread's draws are in flight together
    const int64_t first = (int64_t)blockIdx.x * (kThreads * kDrawsPerThread) + threadIdx.x;
    unsigned leaf[kDrawsPerThread];
#pragma unroll
    for (int k = 0; k < kDrawsPerThread; ++k) {
        const Draw d = philox_draw(keys, (unsigned)(first + k * kThreads), 0u);
        leaf[k] = guided_lower_bound(cdf, guide, guide_bits, d.raw_u, d.u, n_cells);
    }
#pragma unroll
    for (int k = 0; k < kDrawsPerThread; ++k)
        if (first + k * kThreads < n_samples) atomicAdd(counts + leaf[k], 1u);
}

// Element `index` (1-based) of the Halton sequence in base B, with the reference's arithmetic (utils.py:36-46): double
// precision, one rounding per product, sum and division f = f / B; the value is then stored as float32 (utils.py:52-55).
// The scale factors f do not depend on the index: they are divided out at compile time, with the same roundings.
// They, and the sums over every value of the first kHead digits (in the same order), are tables: most indices are settled by
// one look-up, the others add one table entry per further digit.
// DIGITS: digits of 2^32 - 1.
template <unsigned B, int HEAD, int DIGITS>
struct HaltonTable {
    static constexpr unsigned kBase = B;
    static constexpr int kHead = HEAD;         // digits summed up in advance
    static constexpr unsigned kHeads = B == 3u ? 729u : 625u;   // B^HEAD
    double head[kHeads];
    double term[DIGITS][B];                    // digit value * f
    constexpr HaltonTable() : head(), term() {
        double v = 1.0;
        for (int k = 0; k < DIGITS; ++k) {
            v = v / (double)B;
            for (unsigned d = 0; d < B; ++d) term[k][d] = v * (double)d;
        }
        for (unsigned h = 0; h < kHeads; ++h) {
            double r = 0.0;
            unsigned i = h;
            for (int k = 0; k < HEAD; ++k) { r = r + term[k][i % B]; i /= B; }
            head[h] = r;
        }
    }
};
struct HaltonTables {
    HaltonTable<3u, 6, 21> b3;
    HaltonTable<5u, 4, 14> b5;
};
__device__ const HaltonTables g_halton{};

__device__ __forceinline__ float halton_base2(unsigned index) {
    // in base 2 every term is a power of two and every sum exact: the value is the reversed index, rounded once
    return __uint2float_rn(__brev(index)) * 2.3283064365386962890625e-10f;
}
template <typename Table>
__device__ __forceinline__ float halton_element(const Table& t, unsigned index) {
    double result = t.head[index % Table::kHeads];
    unsigned i = index / Table::kHeads;
    for (int k = Table::kHead; i > 0u; ++k) {
        result = __dadd_rn(result, t.term[k][i % Table::kBase]);
        i /= Table::kBase;
    }
    return __double2float_rn(result);
}

// Minimum and maximum that are NaN when an operand is, as a tensor's amin and amax are.
__device__ __forceinline__ float min_nan(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// Corners of the cloud's bounding box, one partial result {min x, y, z, max x, y, z} per block: one pass over the positions,
// four of them per thread and round in three 16-byte loads where the array allows.
constexpr int kMaxBoxBlocks = 1024;   // room for the partial boxes; four blocks per multiprocessor are launched
template <int WARPS>
__device__ __forceinline__ void block_box(float* box, float (&s_box)[WARPS][6]) {
    // box[0..2] minima, box[3..5] maxima of a thread -> of the block, in every thread
#pragma unroll
    for (int c = 0; c < 6; ++c)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float t = __shfl_xor_sync(0xffffffffu, box[c], o);
            box[c] = c < 3 ? min_nan(box[c], t) : max_nan(box[c], t);
        }
    if (lane_id() == 0) {
#pragma unroll
        for (int c = 0; c < 6; ++c) s_box[threadIdx.x >> 5][c] = box[c];
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        box[c] = s_box[0][c];
#pragma unroll
        for (int w = 1; w < WARPS; ++w) box[c] = c < 3 ? min_nan(box[c], s_box[w][c]) : max_nan(box[c], s_box[w][c]);
    }
}

// A bounding box collected by many blocks: words that start at zero and only grow, the maxima as keys that order
// like the values, the minima as the complements of such keys; all ones where a coordinate is no number.  Several copies, so that the blocks do not queue
// for six words.
constexpr int kBoxCopies = 64;
__device__ __forceinline__ unsigned box_word(float v, bool minimum) {
    const unsigned bits = __float_as_uint(v), key = bits & 0x80000000u ? ~bits : bits | 0x80000000u;
    return v != v ? 0xFFFFFFFFu : minimum ? ~key : key;
}
__device__ __forceinline__ float box_value(unsigned word, bool minimum) {
    if (word == 0u) return minimum ? INFINITY : -INFINITY;   // of no position
    if (word == 0xFFFFFFFFu) return __uint_as_float(0x7FFFFFFFu);
    const unsigned key = minimum ? ~word : word;
    return __uint_as_float(key & 0x80000000u ? key & 0x7FFFFFFFu : ~key);
}

// 30-bit Morton code (10 bits per axis, x lowest) of a position inside the box [lo, lo + extent]^3: the bits of an axis two apart, by table (through L1, where neighbouring
// samples meet few entries; eight operations per axis otherwise)
struct SpreadTable {
    unsigned spread[1024];
    constexpr SpreadTable() : spread() {
        for (unsigned v = 0; v < 1024u; ++v)
            for (unsigned bit = 0; bit < 10u; ++bit) spread[v] |= (v >> bit & 1u) << (3u * bit);
    }
};
__device__ const SpreadTable g_spread{};
// The cube the codes refer to: lower corner and reciprocal edge.
struct MortonCube {
    float lo[3];
    float inv_extent;
};
__device__ __forceinline__ unsigned morton_code(const MortonCube& cube, float px, float py, float pz) {
    // trunc(1024 t) of t in [0, 1], 1023 at most, without a conversion (a quarter of the rate of an addition and less): a sum rounded down, whose unit is one.  No number counts as 0
    auto cell = [&](float p, float lo) -> unsigned {
        return __ldg(g_spread.spread + (min(__float_as_uint(__fmaf_rz(__saturatef(__fmul_rn(p - lo, cube.inv_extent)), 1024.0f, 8388608.0f)), 0x4B0003FFu) & 0x3FFu));
    };
    return cell(px, cube.lo[0]) | (cell(py, cube.lo[1]) << 1) | (cell(pz, cube.lo[2]) << 2);
}
// A bounding box {min x, y, z, max x, y, z} -> its cube, the edge widened by a millionth so that the largest coordinate stays inside.  Same roundings as float32
// corners and a double product.  An axis with a NaN in it has no corner and takes no part in the codes, and the edge is then 1.
__device__ __forceinline__ MortonCube cube_of_box(const float* box) {
    const float extent = max_nan(max_nan(__fsub_rn(box[3], box[0]), __fsub_rn(box[4], box[1])), __fsub_rn(box[5], box[2]));
    return {{box[0], box[1], box[2]}, extent > 0.0f ? __fdiv_rn(1.0f, __double2float_rn(__dmul_rn((double)extent, 1.0 + 1e-6))) : 1.0f};
}

// Sample i lies in leaf upper_bound(offsets, i) and is that leaf's h-th sample, h = i - first sample
// of the leaf: Halton point h+1 in bases (2, 3, 5) scaled into the cell; a leaf with a single sample
// puts it at its centre (ProbabilityField.py:131-140).
// Bound by instruction issue.  Of a run's leaves the corner and the edge lie in shared memory, a warp finds the leaves of 32 consecutive samples
// at a time, and heads of 729 and 625 values, read through L1, settle most digits: 2^25 samples of 2.3 * 10^5 leaves 234 -> 197 us (before: a
// search, six gathers and a division per sample, heads of 81 and 125 values in shared memory; with those and the rest as here 212, with the long heads in shared
// memory 201, with persistent blocks 229 to 254).
// CODES: also the Morton codes, whose cube is known from the leaves (halton_box_kernel), so that nothing reads the positions for them: 2^25 samples 191 -> 243 us, and 53 for the
// histogram of the codes, where a kernel that read the positions and counted took 134 (with conversions and spread by shifts 267).
constexpr unsigned kRunRecords = 256;   // leaves of a run whose records are staged; a run over more makes them per sample
struct HaltonLeaf {
    float x, y, z, cell;   // lower corner and edge, or the centre where there is a single sample
};
__device__ __forceinline__ HaltonLeaf halton_leaf(const float* __restrict__ centers, const int* __restrict__ levels, float initial_size, unsigned leaf, unsigned count) {
    HaltonLeaf l;
    l.x = __ldg(centers + 3 * (int64_t)leaf); l.y = __ldg(centers + 3 * (int64_t)leaf + 1); l.z = __ldg(centers + 3 * (int64_t)leaf + 2);
    l.cell = 0.0f;
    if (count != 1u) {
        // cell edge = initial_size / 2^level, exact in fp32 for the levels an octree has; every further
        // operation rounds on its own like the torch expression  centre - cell/2 + halton * cell
        l.cell = __fdiv_rn(initial_size, (float)(1u << __ldg(levels + leaf)));
        const float half = __fmul_rn(l.cell, 0.5f);
        l.x = __fsub_rn(l.x, half); l.y = __fsub_rn(l.y, half); l.z = __fsub_rn(l.z, half);
    }
    return l;
}
template <bool CODES>
__global__ void __launch_bounds__(kThreads) halton_samples_kernel(const unsigned* __restrict__ counts, const unsigned* __restrict__ offsets,
                                                                  unsigned n_cells, const float* __restrict__ centers,
                                                                  const int* __restrict__ levels, float initial_size, unsigned n_total,
                                                                  float* __restrict__ positions, const MortonCube* __restrict__ cube_at, unsigned* __restrict__ codes) {
    await_previous_kernel();
    __shared__ LeafRun run;
    __shared__ unsigned s_start;   // first sample of the run's first leaf
    __shared__ HaltonLeaf s_leaf[kRunRecords];
    __shared__ __align__(16) float s_pos[kThreads / 32][96];
    const HaltonTables& tables = g_halton;
    const unsigned warp = threadIdx.x >> 5, lane = lane_id();
    const unsigned r0 = blockIdx.x * (unsigned)kRunSlots;
    const unsigned in_block = min((unsigned)kRunSlots, n_total - r0);
    find_leaf_run(run, offsets, n_cells, r0, r0 + in_block - 1u);
    const unsigned m = run.count, leaf0 = run.first;
    const bool staged = m <= kRunRecords;
    if (threadIdx.x == 0) s_start = __ldg(offsets + leaf0) - __ldg(counts + leaf0);
    if (staged)
        for (unsigned k = threadIdx.x; k < m; k += kThreads) s_leaf[k] = halton_leaf(centers, levels, initial_size, leaf0 + k, __ldg(counts + leaf0 + k));
    __syncthreads();
    MortonCube cube;
    if (CODES) {
        const float4 q = __ldg(reinterpret_cast<const float4*>(cube_at));
        cube = {{q.x, q.y, q.z}, q.w};
    }
    unsigned k = 0;
    for (unsigned row = 0; row < (unsigned)kRunPerThread; ++row) {
        const unsigned first = (warp * kRunPerThread + row) * 32u;
        if (first >= in_block) break;
        const unsigned here = min(32u, in_block - first), i = r0 + first + min(lane, here - 1u);
        const unsigned l = leaf_of_row(run, offsets, i, k);
        const unsigned c = __ldg(counts + leaf0 + l);
        const unsigned h = i - (l == 0u ? s_start : m <= kRunLeaves ? run.offsets[l - 1u] : __ldg(offsets + leaf0 + l - 1u));
        const HaltonLeaf at = staged ? s_leaf[l] : halton_leaf(centers, levels, initial_size, leaf0 + l, c);
        float x = at.x, y = at.y, z = at.z;
        if (c != 1u) {
            x = __fadd_rn(x, __fmul_rn(halton_base2(h + 1u), at.cell));
            y = __fadd_rn(y, __fmul_rn(halton_element(tables.b3, h + 1u), at.cell));
            z = __fadd_rn(z, __fmul_rn(halton_element(tables.b5, h + 1u), at.cell));
        }
        if (CODES && lane < here) codes[i] = morton_code(cube, x, y, z);
        store_row(s_pos[warp], x, y, z, here, positions + 3 * (int64_t)(r0 + first));
    }
}

// Of the indices 1 .. c the one whose radical inverse is largest: digit by digit from the least significant, which weighs most, the largest there is an index for.
template <unsigned BASE>
__device__ __forceinline__ unsigned largest_halton_index(unsigned c) {
    unsigned h = 0u;
    for (unsigned long long m = 1u; m <= c - h; m *= BASE) h += (unsigned)m * min(BASE - 1u, (unsigned)((c - h) / (unsigned)m));
    return h;
}
// ... and smallest: the largest power of the base.
template <unsigned BASE>
__device__ __forceinline__ unsigned smallest_halton_index(unsigned c) {
    unsigned long long m = 1u;
    while (m * BASE <= c) m *= BASE;
    return (unsigned)m;
}

// Bounding box of the cloud that halton_samples_kernel makes, from the leaves: along an axis the extreme samples of a leaf are those of its extreme Halton elements
// (placing one rounds, but monotonically).  Spares the Morton order a pass over the positions: 2^25 samples of 2.3 * 10^5 leaves 78 us -> 11 (in the placement itself,
// six comparisons per sample, 39).  The block that finishes last leaves the cube of the codes.  box_words: kBoxCopies boxes, and a word for the finished blocks.
__global__ void __launch_bounds__(kThreads) halton_box_kernel(const unsigned* __restrict__ counts, unsigned n_cells, const float* __restrict__ centers, const int* __restrict__ levels,
                                                              float initial_size, unsigned* box_words, MortonCube* __restrict__ cube) {
    await_previous_kernel();
    __shared__ float s_box[kThreads / 32][6];
    float box[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
    auto add = [&](int axis, float v) {
        box[axis] = min_nan(box[axis], v);
        box[3 + axis] = max_nan(box[3 + axis], v);
    };
    for (unsigned leaf = blockIdx.x * kThreads + threadIdx.x; leaf < n_cells; leaf += gridDim.x * kThreads) {
        const unsigned c = __ldg(counts + leaf);
        if (c == 0u) continue;
        const HaltonLeaf at = halton_leaf(centers, levels, initial_size, leaf, c);
        if (c == 1u) {
            add(0, at.x); add(1, at.y); add(2, at.z);
            continue;
        }
        add(0, __fadd_rn(at.x, __fmul_rn(halton_base2(smallest_halton_index<2u>(c)), at.cell)));
        add(0, __fadd_rn(at.x, __fmul_rn(halton_base2(largest_halton_index<2u>(c)), at.cell)));
        add(1, __fadd_rn(at.y, __fmul_rn(halton_element(g_halton.b3, smallest_halton_index<3u>(c)), at.cell)));
        add(1, __fadd_rn(at.y, __fmul_rn(halton_element(g_halton.b3, largest_halton_index<3u>(c)), at.cell)));
        add(2, __fadd_rn(at.z, __fmul_rn(halton_element(g_halton.b5, smallest_halton_index<5u>(c)), at.cell)));
        add(2, __fadd_rn(at.z, __fmul_rn(halton_element(g_halton.b5, largest_halton_index<5u>(c)), at.cell)));
    }
    block_box(box, s_box);
#pragma unroll
    for (int c = 0; c < 6; ++c)
        if (threadIdx.x == c) atomicMax(box_words + (blockIdx.x % kBoxCopies) * 6 + c, box_word(box[c], c < 3));
    if (!last_block(box_words + 6 * kBoxCopies, gridDim.x)) return;
    static_assert(kBoxCopies <= kThreads, "a thread per copy");
#pragma unroll
    for (int c = 0; c < 6; ++c) box[c] = box_value(threadIdx.x < kBoxCopies ? __ldcg(box_words + 6 * threadIdx.x + c) : 0u, c < 3);
    block_box(box, s_box);
    if (threadIdx.x == 0) *cube = cube_of_box(box);
}

__global__ void __launch_bounds__(kThreads) bounding_box_kernel(const float* __restrict__ positions, int64_t n, bool vec_ok, float* __restrict__ partial) {
    await_previous_kernel();
    __shared__ float s_box[kThreads / 32][6];
    float box[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
    auto add = [&](float x, float y, float z) {
        box[0] = min_nan(box[0], x); box[1] = min_nan(box[1], y); box[2] = min_nan(box[2], z);
        box[3] = max_nan(box[3], x); box[4] = max_nan(box[4], y); box[5] = max_nan(box[5], z);
    };
    const int64_t stride = (int64_t)gridDim.x * kThreads, tid = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    const int64_t n4 = vec_ok ? n / 4 : 0;
    const float4* src = reinterpret_cast<const float4*>(positions);
    for (int64_t v = tid; v < n4; v += stride) {
        const float4 a = __ldg(src + 3 * v), b = __ldg(src + 3 * v + 1), c = __ldg(src + 3 * v + 2);
        add(a.x, a.y, a.z); add(a.w, b.x, b.y); add(b.z, b.w, c.x); add(c.y, c.z, c.w);
    }
    for (int64_t i = 4 * n4 + tid; i < n; i += stride) add(__ldg(positions + 3 * i), __ldg(positions + 3 * i + 1), __ldg(positions + 3 * i + 2));
    block_box(box, s_box);
    if (threadIdx.x < 6) partial[6 * blockIdx.x + threadIdx.x] = threadIdx.x == 0 ? box[0] : threadIdx.x == 1 ? box[1] : threadIdx.x == 2 ? box[2] : threadIdx.x == 3 ? box[3] : threadIdx.x == 4 ? box[4] : box[5];
}

// The cube of a cloud that lies there already: the caller's, or (box_parts > 0) from the partial boxes.
struct MortonBox {
    MortonCube cube;
    const float* parts;
    int box_parts;
};
// Also counts the digits of the codes for their sort, which spares it a pass over them: 2^25 codes and their histogram 90 + 53 -> 132 us.
constexpr int kCodeThreads = kRadix;
__global__ void __launch_bounds__(kCodeThreads) morton_codes_kernel(const float* __restrict__ positions, int64_t n, bool vec_ok, MortonBox mb, KeyHistogram digits,
                                                                unsigned* __restrict__ codes) {
    await_previous_kernel();
    __shared__ BlockHistogram s_digits;
    clear_histogram(s_digits);
    __syncthreads();
    if (mb.box_parts > 0) {
        __shared__ float s_box[kCodeThreads / 32][6];
        float box[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
        for (int k = threadIdx.x; k < mb.box_parts; k += kCodeThreads)
#pragma unroll
            for (int c = 0; c < 6; ++c) {
                const float t = __ldg(mb.parts + 6 * k + c);
                box[c] = c < 3 ? min_nan(box[c], t) : max_nan(box[c], t);
            }
        block_box(box, s_box);
        mb.cube = cube_of_box(box);
    }
    auto code = [&](float px, float py, float pz) -> unsigned {
        const unsigned key = morton_code(mb.cube, px, py, pz);
        count_key(s_digits, digits.pt, key);
        return key;
    };
    // four points per thread: three 16-byte loads where the positions are aligned, one 16-byte store (without counting, 2^25 points 91 us, bound by DRAM;
    // one point per thread, and the point numbers written for the sort, which now makes them itself: 131; with the four shared-memory atomics per code 132)
    const int64_t stride = (int64_t)gridDim.x * kCodeThreads * 4;
    for (int64_t i = ((int64_t)blockIdx.x * kCodeThreads + threadIdx.x) * 4; i < n; i += stride) {
        if (vec_ok && i + 4 <= n) {
            const float4* src = reinterpret_cast<const float4*>(positions + 3 * i);
            const float4 a = __ldg(src), b = __ldg(src + 1), c = __ldg(src + 2);
            *reinterpret_cast<uint4*>(codes + i) = make_uint4(code(a.x, a.y, a.z), code(a.w, b.x, b.y), code(b.z, b.w, c.x), code(c.y, c.z, c.w));
        } else {
            for (int64_t k = i; k < n && k < i + 4; ++k) codes[k] = code(__ldg(positions + 3 * k), __ldg(positions + 3 * k + 1), __ldg(positions + 3 * k + 2));
        }
    }
    finish_histogram(s_digits, digits, gridDim.x, nullptr);
}

// Four points per thread, their gathers in flight together, two loads of 8 bytes each, and three 16-byte stores (2^25 points 142 us; three loads of 4 bytes 166; one
// point per thread with three 4-byte stores 201, the same with the stores staged through shared memory 211).
__global__ void __launch_bounds__(kThreads) gather_positions_kernel(const float* __restrict__ positions, const unsigned* __restrict__ order,
                                                                    int64_t n, bool pairs_ok, bool vec_ok, float* __restrict__ out) {
    await_previous_kernel();
    const int64_t i = ((int64_t)blockIdx.x * kThreads + threadIdx.x) * 4;
    if (i >= n) return;
    const unsigned last = (unsigned)(n - 1);   // behind a sort that has given up (and reported it) the order has holes, which may hold anything
    if (vec_ok && i + 4 <= n) {
        const uint4 o = __ldg(reinterpret_cast<const uint4*>(order + i));
        const unsigned j[4] = {min(o.x, last), min(o.y, last), min(o.z, last), min(o.w, last)};
        float v[12];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (!pairs_ok) {
#pragma unroll
                for (int c = 0; c < 3; ++c) v[3 * k + c] = __ldg(positions + 3 * (int64_t)j[k] + c);
                continue;
            }
            // around the 12 bytes (behind the last point there may be nothing)
            const float2* src = reinterpret_cast<const float2*>(positions) + ((3 * (int64_t)j[k]) >> 1);
            const float2 a = __ldg(src);
            float2 b = make_float2(0.0f, 0.0f);
            if (j[k] < last || (j[k] & 1u)) b = __ldg(src + 1);
            else b.x = __ldg(reinterpret_cast<const float*>(src + 1));
            const bool odd = j[k] & 1u;
            v[3 * k] = odd ? a.y : a.x; v[3 * k + 1] = odd ? b.x : a.y; v[3 * k + 2] = odd ? b.y : b.x;
        }
        float4* dst = reinterpret_cast<float4*>(out + 3 * i);
#pragma unroll
        for (int k = 0; k < 3; ++k) dst[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
        return;
    }
    for (int64_t k = i; k < n && k < i + 4; ++k) {
        const int64_t j = min(__ldg(order + k), last);
#pragma unroll
        for (int c = 0; c < 3; ++c) out[3 * k + c] = __ldg(positions + 3 * j + c);
    }
}

constexpr int kSumWord = 4;
struct SamplerWs {
    float* vw;          // viewpoint weights (n_cells)
    float* cdf;         // (n_cells)
    unsigned long long* chunk_sums64;   // fixed-point chunk sums / bases
    unsigned long long* total64;        // fixed-point total
    unsigned* max_bits;                 // [0] bit pattern of the largest weight, [1] finished blocks of the CDF's sums, [2] of the counts': zero before
    float* sum;         // 1 float, kSumWord words behind max_bits: one copy fetches both
    unsigned* counts;   // expected-sample counts (n_cells)
    unsigned* offsets;  // inclusive offsets (n_cells)
    unsigned* chunk_sums;
    unsigned long long* total;
    uint4* guide;       // 2^guide_bits bucket records, of 32 bytes (GuideRecord); of 16 for draw counts.  Shares its place with `counts` and `offsets`
    unsigned* count_parts;   // kCountParts - 1 arrays of draw counts (the caller's is the first), over the end of the guide, `leaf_pack` and `vw`
    int guide_bits;
    float4* leaf_pack;  // (n_cells) centre + edge length
    size_t bytes;
};

int guide_bits_for(int64_t n_cells) {
    int k = 8;
    while (k < 20 && ((int64_t)1 << k) < n_cells) ++k;
    return k;
}

SamplerWs carve_sampler_ws(void* p, int64_t n_cells) {
    SamplerWs w;
    Carver c(p);
    const int64_t n = n_cells > 0 ? n_cells : 1;
    w.cdf = c.take<float>(n);
    w.chunk_sums64 = c.take<unsigned long long>(ceil_div<int64_t>(n, kCdfChunk));
    w.total64 = c.take<unsigned long long>(2);
    w.max_bits = c.take<unsigned>(2 * kSumWord);
    w.sum = reinterpret_cast<float*>(w.max_bits + kSumWord);
    w.chunk_sums = c.take<unsigned>(ceil_div<int64_t>(n, kThreads));
    w.total = c.take<unsigned long long>(2);
    // No call uses all of what follows, and a training view takes a workspace of its own on every step and stream, so it lies in one place:
    //   training and plain samples    [ guide, 32 bytes a record  ] [leaf_pack] [vw]
    //   expected and Halton samples   [ counts, offsets           ] [leaf_pack] [vw]
    //   draw counts                   [ guide, 16 bytes ] [ count_parts ............ ]
    // One record more than there are buckets: 32-byte loads need an alignment the caller's workspace need not have.
    w.guide_bits = guide_bits_for(n);
    const size_t records = ((size_t)1 << w.guide_bits) + 1;
    Carver samples = c, counts = c, draws = c;
    const uintptr_t guide = reinterpret_cast<uintptr_t>(samples.take<GuideRecord>(records));
    w.guide = reinterpret_cast<uint4*>((guide + sizeof(GuideRecord) - 1) / sizeof(GuideRecord) * sizeof(GuideRecord));
    w.counts = counts.take<unsigned>(n);
    w.offsets = counts.take<unsigned>(n);
    (void)draws.take<uint4>(records + 1);
    w.count_parts = draws.take<unsigned>((size_t)n * (kCountParts - 1));
    // leaf_pack and vw, 20 bytes per leaf, are the end of the 28 that the arrays of draw counts take
    const size_t overlap = (size_t)n * (sizeof(float4) + sizeof(float)), draws_before = draws.off > overlap ? draws.off - overlap : 0;
    c.off = samples.off > counts.off ? samples.off : counts.off;
    if (c.off < draws_before) c.off = draws_before;
    w.leaf_pack = c.take<float4>(n);
    w.vw = c.take<float>(n);
    w.bytes = c.used();
    return w;
}

// weight sum only (expected-sample mode) or sum + CDF.  `max_known`: the largest weight is in w.max_bits already.
int build_cdf(const float* weights, int64_t n_cells, float* cdf, float* sum_out, const SamplerWs& w, bool max_known, cudaStream_t stream, const float4* leaf_pack = nullptr) {
    const int64_t chunks = ceil_div<int64_t>(n_cells, kCdfChunk);
    if (!max_known) {
        INPC_CUDA_TRY(cudaMemsetAsync(w.max_bits, 0, 4 * sizeof(unsigned), stream));
        launch_chained(cdf_max_kernel, (unsigned)chunks, kCdfThreads, 0, stream, weights, n_cells, w.max_bits);
        INPC_LAUNCH_CHECK("cdf_max_kernel");
    }
    launch_chained(cdf_chunk_sums_kernel, (unsigned)chunks, kCdfThreads, 0, stream, weights, n_cells, w.max_bits, w.max_bits + 1, w.chunk_sums64, w.total64, sum_out);
    INPC_LAUNCH_CHECK("cdf_chunk_sums_kernel");
    if (cdf) {
        launch_chained(cdf_finalize_kernel, (unsigned)chunks, kCdfThreads, 0, stream, weights, n_cells, w.max_bits, w.chunk_sums64, w.total64, cdf);
        INPC_LAUNCH_CHECK("cdf_finalize_kernel");
        if (cdf == w.cdf) {
            launch_chained(guide_table_kernel, (unsigned)ceil_div<int64_t>((int64_t)1 << w.guide_bits, kGuidePerBlock), kThreads, 0, stream,
                cdf, (unsigned)n_cells, w.guide_bits, w.guide, leaf_pack);
            INPC_LAUNCH_CHECK("guide_table_kernel");
        }
    }
    return INPC_OK;
}

// viewpoint weights into w.vw, the largest weight, and the leaf records of the draws behind them (`leaf_pack`, optional)
int view_weights(const ViewParams& v, int64_t n_cells, const float* centers, const int32_t* levels, const float* weights, float initial_size,
                 const SamplerWs& w, float4* leaf_pack, cudaStream_t stream) {
    INPC_CUDA_TRY(cudaMemsetAsync(w.max_bits, 0, 4 * sizeof(unsigned), stream));
    launch_chained(viewpoint_weights_kernel, (unsigned)ceil_div<int64_t>(n_cells, kThreads), kThreads, 0, stream, v, n_cells, centers, levels, weights, initial_size, w.vw,
                                                                                                   leaf_pack, w.max_bits);
    INPC_LAUNCH_CHECK("viewpoint_weights_kernel");
    return INPC_OK;
}

int check_cells(const inpc_view* view, int64_t n_cells, const void* a, const void* b, const void* c) {
    if (!view || !view->w2c) { set_error("sampler: view and view.w2c must be non-null"); return INPC_E_INVALID; }
    // 2^24 leaves is the reference octree's own cap (Modules/ProbabilityField.py:217-257); the 39-bit
    // fixed-point fractions of the CDF add up in 64 bits without wrapping for up to 2^25 of them
    if (n_cells <= 0 || n_cells > ((int64_t)1 << 24)) { set_error("sampler: n_cells=%lld out of range [1, 2^24]", (long long)n_cells); return INPC_E_INVALID; }
    if (!a || !b || !c) { set_error("sampler: null leaf array"); return INPC_E_INVALID; }
    return INPC_OK;
}

float* pinned_float() {
    static thread_local float* p = nullptr;
    if (!p && cudaHostAlloc(reinterpret_cast<void**>(&p), 64, cudaHostAllocDefault) != cudaSuccess) p = nullptr;
    return p;
}

}  // namespace

}  // namespace inpc

using namespace inpc;

struct inpc_sampler {
    unsigned long long seed;
    unsigned long long counter;
    long long training_ticket;   // status slot of the last inpc_generate_training_samples call (0: none)
};

extern "C" inpc_sampler* inpc_sampler_create(int64_t seed) {
    inpc_sampler* s = new inpc_sampler;
    s->seed = (unsigned long long)seed;
    s->counter = 0;
    s->training_ticket = 0;
    return s;
}
extern "C" void inpc_sampler_destroy(inpc_sampler* s) { delete s; }
// 1 if some slots of the sampler's last inpc_generate_training_samples call ran out of rejection attempts
// (they hold their last candidate, a position outside the view frustum), 0 if none did, -1 if that is no longer
// known (the status slot has been reused).  Meaningful once the call's stream has been synchronised.
extern "C" int inpc_sampler_exhausted(const inpc_sampler* s) {
    if (!s || s->training_ticket == 0) return 0;
    unsigned w[inpc::STATUS_WORDS];
    if (inpc::read_status(s->training_ticket, w, nullptr) != INPC_OK) return -1;
    return w[inpc::STATUS_SAMPLER_EXHAUSTED] ? 1 : 0;
}
extern "C" uint64_t inpc_sampler_get_counter(const inpc_sampler* s) { return s ? s->counter : 0; }
extern "C" void inpc_sampler_set_counter(inpc_sampler* s, uint64_t counter) { if (s) s->counter = counter; }

extern "C" size_t inpc_sampler_workspace_bytes(int64_t n_cells) { return carve_sampler_ws(nullptr, n_cells).bytes; }

extern "C" int inpc_compute_viewpoint_weights(const inpc_view* view, int64_t n_cells, const float* centers,
                                              const int32_t* levels, const float* weights, float initial_size,
                                              float* out, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (n_cells == 0) return INPC_OK;
    int rc = check_cells(view, n_cells, centers, levels, weights);
    if (rc != INPC_OK) return rc;
    if (!out) { set_error("inpc_compute_viewpoint_weights: null output"); return INPC_E_INVALID; }
    launch_chained(viewpoint_weights_kernel, (unsigned)ceil_div<int64_t>(n_cells, kThreads), kThreads, 0, stream,
        to_params(view), n_cells, centers, levels, weights, initial_size, out, nullptr, nullptr);
    INPC_LAUNCH_CHECK("viewpoint_weights_kernel");
    return INPC_OK;
}

extern "C" int inpc_max_viewpoint_weights(const inpc_view* views, int n_views, int64_t n_cells, const float* centers, const int32_t* levels,
                                          const float* weights, float initial_size, float* out, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (n_cells == 0) return INPC_OK;
    if (n_views < 1 || !out) { set_error("inpc_max_viewpoint_weights: bad argument"); return INPC_E_INVALID; }
    for (int j = 0; j < n_views; ++j) {
        const int rc = check_cells(views ? views + j : nullptr, n_cells, centers, levels, weights);
        if (rc != INPC_OK) return rc;
    }
    for (int j = 0; j < n_views; j += kViewsPerPass) {
        ViewSet set;
        set.count = n_views - j < kViewsPerPass ? n_views - j : kViewsPerPass;
        for (int k = 0; k < set.count; ++k) set.v[k] = to_params(views + j + k);
        launch_chained(max_viewpoint_weights_kernel, (unsigned)ceil_div<int64_t>(n_cells, kThreads), kThreads, 0, stream, set, n_cells, centers, levels, weights,
                                                                                                           initial_size, j == 0, out);
        INPC_LAUNCH_CHECK("max_viewpoint_weights_kernel");
    }
    return INPC_OK;
}

extern "C" int inpc_build_cdf(const float* weights, int64_t n_cells, float* cdf, float* sum_out, void* workspace,
                              void* stream_) {
    if (n_cells <= 0 || !weights || !cdf || !sum_out || !workspace) { set_error("inpc_build_cdf: bad argument"); return INPC_E_INVALID; }
    SamplerWs w = carve_sampler_ws(workspace, n_cells);
    return build_cdf(weights, n_cells, cdf, sum_out, w, false, static_cast<cudaStream_t>(stream_));
}

extern "C" int inpc_draw_leaves(const float* cdf, int64_t n_cells, const float* u, int64_t n, int64_t* out, void* stream_) {
    if (n == 0) return INPC_OK;
    if (n_cells <= 0 || n_cells >= ((int64_t)1 << 31) || !cdf || !u || !out || n < 0) { set_error("inpc_draw_leaves: bad argument"); return INPC_E_INVALID; }
    launch_chained(draw_leaves_kernel, (unsigned)ceil_div<int64_t>(n, kThreads), kThreads, 0, static_cast<cudaStream_t>(stream_),
        cdf, (unsigned)n_cells, u, n, reinterpret_cast<long long*>(out));
    INPC_LAUNCH_CHECK("draw_leaves_kernel");
    return INPC_OK;
}

extern "C" int inpc_generate_training_samples(inpc_sampler* s, const inpc_view* view, int64_t n_cells, const float* centers,
                                              const int32_t* levels, const float* weights, float initial_size,
                                              int64_t n_samples, float* positions, int64_t* indices, void* workspace,
                                              void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (!s) { set_error("null sampler"); return INPC_E_INVALID; }
    if (n_samples == 0) return INPC_OK;
    int rc = check_cells(view, n_cells, centers, levels, weights);
    if (rc != INPC_OK) return rc;
    if (n_samples < 0 || n_samples >= ((int64_t)1 << 32) || !positions || !indices || !workspace) { set_error("inpc_generate_training_samples: bad argument"); return INPC_E_INVALID; }
    SamplerWs w = carve_sampler_ws(workspace, n_cells);
    const ViewParams v = to_params(view);
    StageScope scope(STAGE_SAMPLE, stream);
    rc = view_weights(v, n_cells, centers, levels, weights, initial_size, w, w.leaf_pack, stream);
    if (rc != INPC_OK) return rc;
    rc = build_cdf(w.vw, n_cells, w.cdf, w.sum, w, true, stream, w.leaf_pack);
    if (rc != INPC_OK) return rc;
    unsigned* status = acquire_status("inpc_generate_training_samples", &s->training_ticket);
    if (!status) return INPC_E_CUDA;
    constexpr int kPer = 2;   // small calls need the blocks
    auto launch = [&](auto per) {
        launch_chained(training_samples_kernel<decltype(per)::value>, (unsigned)ceil_div<int64_t>(n_samples, kThreads * decltype(per)::value), kThreads, 0, stream,
            v, philox_keys(s->seed, s->counter), w.cdf, w.guide, w.guide_bits, w.sum, (unsigned)n_cells, w.leaf_pack, n_samples, positions,
            reinterpret_cast<long long*>(indices), status);
    };
    if (n_samples >= (int64_t)kThreads * kPer * sm_count() * 4) launch(std::integral_constant<int, kPer>());
    else launch(std::integral_constant<int, 1>());
    INPC_LAUNCH_CHECK("training_samples_kernel");
    s->counter += 1;
    return INPC_OK;
}

extern "C" int inpc_generate_samples(inpc_sampler* s, const inpc_view* view, int64_t n_cells, const float* centers,
                                     const int32_t* levels, const float* weights, float initial_size, int64_t n_samples,
                                     float* positions, int64_t* n_written, void* workspace, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (!s || !n_written) { set_error("null sampler or n_written"); return INPC_E_INVALID; }
    *n_written = 0;
    int rc = check_cells(view, n_cells, centers, levels, weights);
    if (rc != INPC_OK) return rc;
    if (n_samples < 0 || n_samples >= ((int64_t)1 << 32) || !workspace || (n_samples > 0 && !positions)) { set_error("inpc_generate_samples: bad argument"); return INPC_E_INVALID; }
    SamplerWs w = carve_sampler_ws(workspace, n_cells);
    const ViewParams v = to_params(view);
    rc = view_weights(v, n_cells, centers, levels, weights, initial_size, w, w.leaf_pack, stream);
    if (rc != INPC_OK) return rc;
    rc = build_cdf(w.vw, n_cells, w.cdf, w.sum, w, true, stream, w.leaf_pack);
    if (rc != INPC_OK) return rc;
    float* host = pinned_float();
    if (!host) return cuda_fail(cudaGetLastError(), "cudaHostAlloc");
    INPC_CUDA_TRY(cudaMemcpyAsync(host, w.sum, sizeof(float), cudaMemcpyDeviceToHost, stream));
    INPC_CUDA_TRY(cudaStreamSynchronize(stream));
    if (!(host[0] > 0.0f)) return INPC_OK;   // src/sampling_api.cu:154: empty result
    if (n_samples > 0) {
        launch_chained(samples_kernel, (unsigned)ceil_div<int64_t>(n_samples, kThreads), kThreads, 0, stream,
            philox_keys(s->seed, s->counter), w.cdf, w.guide, w.guide_bits, (unsigned)n_cells, w.leaf_pack, n_samples, positions);
        INPC_LAUNCH_CHECK("samples_kernel");
    }
    s->counter += 1;
    *n_written = n_samples;
    return INPC_OK;
}

extern "C" int inpc_generate_expected_samples_count(inpc_sampler* s, const inpc_view* view, int64_t n_cells,
                                                    const float* centers, const int32_t* levels, const float* weights,
                                                    float initial_size, int64_t n_samples, int64_t* n_created,
                                                    void* workspace, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (!s || !n_created) { set_error("null sampler or n_created"); return INPC_E_INVALID; }
    *n_created = 0;
    int rc = check_cells(view, n_cells, centers, levels, weights);
    if (rc != INPC_OK) return rc;
    if (n_samples < 0 || n_samples >= ((int64_t)1 << 32) || !workspace) { set_error("inpc_generate_expected_samples_count: bad argument"); return INPC_E_INVALID; }
    SamplerWs w = carve_sampler_ws(workspace, n_cells);
    const ViewParams v = to_params(view);
    const unsigned blocks = (unsigned)ceil_div<int64_t>(n_cells, kThreads);
    rc = view_weights(v, n_cells, centers, levels, weights, initial_size, w, nullptr, stream);
    if (rc != INPC_OK) return rc;
    rc = build_cdf(w.vw, n_cells, nullptr, w.sum, w, true, stream);
    if (rc != INPC_OK) return rc;
    launch_chained(count_chunk_sums_kernel, blocks, kThreads, 0, stream, w.vw, w.sum, (unsigned)n_samples, w.counts, n_cells, w.max_bits + 2, w.chunk_sums, w.total);
    INPC_LAUNCH_CHECK("count_chunk_sums_kernel");
    launch_chained(count_offsets_kernel, blocks, kThreads, 0, stream, w.counts, n_cells, w.chunk_sums, w.offsets);
    INPC_LAUNCH_CHECK("count_offsets_kernel");
    unsigned long long* host = reinterpret_cast<unsigned long long*>(pinned_float());
    if (!host) return cuda_fail(cudaGetLastError(), "cudaHostAlloc");
    INPC_CUDA_TRY(cudaMemcpyAsync(host, w.total, sizeof(unsigned long long), cudaMemcpyDeviceToHost, stream));
    INPC_CUDA_TRY(cudaStreamSynchronize(stream));
    if (host[0] >= (1ull << 32)) { set_error("expected sample count %llu exceeds 2^32", host[0]); return INPC_E_CAPACITY; }
    *n_created = (int64_t)host[0];
    return INPC_OK;
}

extern "C" int inpc_generate_expected_samples_fill(inpc_sampler* s, int64_t n_cells, const float* centers,
                                                   const int32_t* levels, float initial_size, int64_t n_created,
                                                   int64_t n_multi, float* positions, void* workspace, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (!s) { set_error("null sampler"); return INPC_E_INVALID; }
    const int64_t total = n_created * n_multi;
    if (n_cells <= 0 || n_created <= 0 || n_multi <= 0 || total >= ((int64_t)1 << 32) || !centers || !levels || !positions || !workspace) {
        set_error("inpc_generate_expected_samples_fill: bad argument");
        return INPC_E_INVALID;
    }
    SamplerWs w = carve_sampler_ws(workspace, n_cells);
    launch_chained(leaf_records_kernel, (unsigned)ceil_div<int64_t>(n_cells, kThreads), kThreads, 0, stream, n_cells, centers, levels, initial_size, w.leaf_pack);
    INPC_LAUNCH_CHECK("leaf_records_kernel");
    // all copies in one block where there are blocks enough without
    const int64_t runs = ceil_div<int64_t>(n_created, kRunSlots), copies = runs >= (int64_t)sm_count() * 8 ? 1 : n_multi < 65535 ? n_multi : 65535;
    const dim3 grid((unsigned)runs, (unsigned)copies);
    launch_chained(expected_samples_kernel, grid, kThreads, 0, stream, philox_keys(s->seed, s->counter), w.offsets, (unsigned)n_cells, w.leaf_pack, (unsigned)n_created,
                                                           (unsigned)n_multi, positions);
    INPC_LAUNCH_CHECK("expected_samples_kernel");
    s->counter += 1;
    return INPC_OK;
}

namespace {
// inclusive offsets of w.counts into w.offsets
int scan_counts(const SamplerWs& w, int64_t n_cells, cudaStream_t stream) {
    const unsigned blocks = (unsigned)ceil_div<int64_t>(n_cells, kThreads);
    INPC_CUDA_TRY(cudaMemsetAsync(w.max_bits, 0, 4 * sizeof(unsigned), stream));
    launch_chained(count_chunk_sums_kernel, blocks, kThreads, 0, stream, nullptr, nullptr, 0u, w.counts, n_cells, w.max_bits + 2, w.chunk_sums, w.total);
    INPC_LAUNCH_CHECK("count_chunk_sums_kernel");
    launch_chained(count_offsets_kernel, blocks, kThreads, 0, stream, w.counts, n_cells, w.chunk_sums, w.offsets);
    INPC_LAUNCH_CHECK("count_offsets_kernel");
    return INPC_OK;
}
}  // namespace

extern "C" int inpc_draw_leaf_counts(inpc_sampler* s, int64_t n_cells, const float* weights, int64_t n_samples, uint32_t* counts,
                                     void* workspace, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (!s || n_cells <= 0 || n_cells >= ((int64_t)1 << 31) || n_samples < 0 || n_samples >= ((int64_t)1 << 32) || !weights || !counts || !workspace) {
        set_error("inpc_draw_leaf_counts: bad argument");
        return INPC_E_INVALID;
    }
    SamplerWs w = carve_sampler_ws(workspace, n_cells);
    int rc = build_cdf(weights, n_cells, w.cdf, w.sum, w, false, stream);
    if (rc != INPC_OK) return rc;
    INPC_CUDA_TRY(cudaMemsetAsync(counts, 0, sizeof(uint32_t) * (size_t)n_cells, stream));   // also what a call leaves that fails below
    float* host = pinned_float();
    if (!host) return cuda_fail(cudaGetLastError(), "cudaHostAlloc");
    INPC_CUDA_TRY(cudaMemcpyAsync(host, w.max_bits, (kSumWord + 1) * sizeof(float), cudaMemcpyDeviceToHost, stream));
    INPC_CUDA_TRY(cudaStreamSynchronize(stream));
    const float largest = host[0], sum = host[kSumWord];
    if (!(sum > 0.0f)) { set_error("inpc_draw_leaf_counts: the weights sum to zero"); return INPC_E_INVALID; }
    if (n_samples > 0) {
        const unsigned n_parts = use_count_parts(n_samples, n_cells, largest, sum) ? kCountParts : 1u;
        if (n_parts > 1u) INPC_CUDA_TRY(cudaMemsetAsync(w.count_parts, 0, sizeof(uint32_t) * (size_t)n_cells * (kCountParts - 1), stream));
        launch_chained(leaf_histogram_kernel, (unsigned)ceil_div<int64_t>(n_samples, kThreads * kDrawsPerThread), kThreads, 0, stream,
            philox_keys(s->seed, s->counter), w.cdf, w.guide, w.guide_bits, (unsigned)n_cells, n_samples, counts, w.count_parts, n_parts);
        INPC_LAUNCH_CHECK("leaf_histogram_kernel");
        if (n_parts > 1u) {
            launch_chained(add_count_parts_kernel, (unsigned)ceil_div<int64_t>(n_cells, kThreads), kThreads, 0, stream, w.count_parts, n_cells, counts);
            INPC_LAUNCH_CHECK("add_count_parts_kernel");
        }
    }
    s->counter += 1;
    return INPC_OK;
}

// `box_words` (optional): 6 kBoxCopies words, see box_word, and the count of finished blocks behind them; all start at zero.
static int launch_halton(const char* who, const uint32_t* counts, int64_t n_cells, const float* centers, const int32_t* levels, float initial_size, int64_t n_total,
                         float* positions, void* workspace, unsigned* box_words, MortonCube* cube, unsigned* codes, cudaStream_t stream) {
    if (n_cells <= 0 || n_cells >= ((int64_t)1 << 31) || n_total < 0 || n_total >= ((int64_t)1 << 32) || !counts || !centers || !levels || !positions || !workspace) {
        set_error("%s: bad argument", who);
        return INPC_E_INVALID;
    }
    SamplerWs w = carve_sampler_ws(workspace, n_cells);
    INPC_CUDA_TRY(cudaMemcpyAsync(w.counts, counts, sizeof(uint32_t) * (size_t)n_cells, cudaMemcpyDeviceToDevice, stream));
    const int rc = scan_counts(w, n_cells, stream);
    if (rc != INPC_OK) return rc;
    if (box_words) {
        const int64_t box_blocks = ceil_div<int64_t>(n_cells, kThreads), box_cap = (int64_t)sm_count() * 8;
        launch_chained(halton_box_kernel, (unsigned)(box_blocks < box_cap ? box_blocks : box_cap), kThreads, 0, stream, w.counts, (unsigned)n_cells, centers, levels, initial_size, box_words, cube);
        INPC_LAUNCH_CHECK("halton_box_kernel");
    }
    launch_chained(codes ? halton_samples_kernel<true> : halton_samples_kernel<false>, (unsigned)ceil_div<int64_t>(n_total, kRunSlots), kThreads, 0, stream, w.counts, w.offsets,
                   (unsigned)n_cells, centers, levels, initial_size, (unsigned)n_total, positions, cube, codes);
    INPC_LAUNCH_CHECK("halton_samples_kernel");
    return INPC_OK;
}

extern "C" int inpc_halton_samples(const uint32_t* counts, int64_t n_cells, const float* centers, const int32_t* levels, float initial_size,
                                   int64_t n_total, float* positions, void* workspace, void* stream) {
    if (n_total == 0) return INPC_OK;
    return launch_halton("inpc_halton_samples", counts, n_cells, centers, levels, initial_size, n_total, positions, workspace, nullptr, nullptr, nullptr, static_cast<cudaStream_t>(stream));
}

extern "C" size_t inpc_morton_workspace_bytes(int64_t n) {
    const size_t arr = align_up(sizeof(uint32_t) * (size_t)(n > 0 ? n : 1));
    return 4 * arr + align_up(6 * sizeof(float) * kMaxBoxBlocks) + sort_workspace_bytes(n, n) + 256;
}

namespace {
struct MortonWs {
    uint32_t *codes[2], *order[2];
    float* parts;             // partial boxes
    void* sort_ws;
};
MortonWs carve_morton_ws(void* workspace, int64_t n) {
    Carver c(workspace);
    MortonWs w;
    for (int k = 0; k < 2; ++k) w.codes[k] = c.take<uint32_t>(n);
    for (int k = 0; k < 2; ++k) w.order[k] = c.take<uint32_t>(n);
    w.parts = c.take<float>(6 * kMaxBoxBlocks);
    c.off = align_up(c.off);
    w.sort_ws = c.base + c.off;
    return w;
}

constexpr int kCodeBits = 30;

// The codes' sort and the positions in that order.  `counted`: see sort_pairs; the front of the sort's workspace has been cleared.
int order_along_curve(const char* who, const float* positions, int64_t n, const MortonWs& w, bool counted, float* out, cudaStream_t stream) {
    int in_alt = 0;
    {
        const int rc_prev = check_previous_calls();
        if (rc_prev != INPC_OK) return rc_prev;
    }
    unsigned* status = acquire_status(who);
    if (!status) return INPC_E_CUDA;
    if (n == 1) INPC_CUDA_TRY(cudaMemsetAsync(w.order[0], 0, sizeof(uint32_t), stream));   // a single pair is not sorted
    const int rc = sort_pairs(w.codes[0], w.codes[1], w.order[0], w.order[1], n, n, kCodeBits, w.sort_ws, true, status, &in_alt, stream, true, counted);
    if (rc != INPC_OK) return rc;
    launch_chained(gather_positions_kernel, (unsigned)ceil_div<int64_t>(n, 4 * kThreads), kThreads, 0, stream, positions, w.order[in_alt], n,
                   (reinterpret_cast<uintptr_t>(positions) & 7u) == 0, (reinterpret_cast<uintptr_t>(out) & 15u) == 0, out);
    INPC_LAUNCH_CHECK("gather_positions_kernel");
    return INPC_OK;
}
}  // namespace

extern "C" int inpc_morton_order(const float* positions, int64_t n, const float* box_lo, float box_extent, float* out, void* workspace,
                                 void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (n == 0) return INPC_OK;
    if (n < 0 || n >= ((int64_t)1 << 30) || !positions || (box_lo && !(box_extent > 0.0f)) || !out || !workspace || out == positions) {
        set_error("inpc_morton_order: bad argument");
        return INPC_E_INVALID;
    }
    const MortonWs w = carve_morton_ws(workspace, n);
    MortonBox mb{{{0.0f, 0.0f, 0.0f}, 1.0f}, w.parts, 0};
    if (box_lo) {
        for (int k = 0; k < 3; ++k) mb.cube.lo[k] = box_lo[k];
        mb.cube.inv_extent = 1.0f / box_extent;
    } else {
        const int64_t blocks = ceil_div<int64_t>(n, 4 * kThreads), cap = 4 * sm_count() < kMaxBoxBlocks ? 4 * sm_count() : kMaxBoxBlocks;
        mb.box_parts = (int)(blocks < cap ? blocks : cap);
        launch_chained(bounding_box_kernel, mb.box_parts, kThreads, 0, stream, positions, n, (reinterpret_cast<uintptr_t>(positions) & 15u) == 0, w.parts);
        INPC_LAUNCH_CHECK("bounding_box_kernel");
    }
    INPC_CUDA_TRY(cudaMemsetAsync(w.sort_ws, 0, sort_zero_bytes(n, n, kCodeBits), stream));
    const int64_t code_blocks = ceil_div<int64_t>(n, 4 * kCodeThreads), code_cap = (int64_t)sm_count() * 4;
    launch_chained(morton_codes_kernel, (unsigned)(code_blocks < code_cap ? code_blocks : code_cap), kCodeThreads, 0, stream, positions, n, (reinterpret_cast<uintptr_t>(positions) & 15u) == 0,
                   mb, key_histogram(w.sort_ws, n, n, kCodeBits), w.codes[0]);
    INPC_LAUNCH_CHECK("morton_codes_kernel");
    return order_along_curve("inpc_morton_order", positions, n, w, true, out, stream);
}

extern "C" int inpc_halton_morton_order(const uint32_t* counts, int64_t n_cells, const float* centers, const int32_t* levels, float initial_size, int64_t n_total,
                                        float* positions, float* out, void* sampler_workspace, void* morton_workspace, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (n_total == 0) return INPC_OK;
    if (n_total < 0 || n_total >= ((int64_t)1 << 30) || !out || !morton_workspace || out == positions) {
        set_error("inpc_halton_morton_order: bad argument");
        return INPC_E_INVALID;
    }
    const MortonWs w = carve_morton_ws(morton_workspace, n_total);
    static_assert(kBoxCopies + 2 <= kMaxBoxBlocks, "words and cube lie where partial boxes would");
    unsigned* words = reinterpret_cast<unsigned*>(w.parts);
    MortonCube* cube = reinterpret_cast<MortonCube*>(words + 6 * kBoxCopies + 4);   // 16-byte aligned
    INPC_CUDA_TRY(cudaMemsetAsync(words, 0, sizeof(unsigned) * (6 * kBoxCopies + 1), stream));
    INPC_CUDA_TRY(cudaMemsetAsync(w.sort_ws, 0, sort_zero_bytes(n_total, n_total, kCodeBits), stream));
    const int rc = launch_halton("inpc_halton_morton_order", counts, n_cells, centers, levels, initial_size, n_total, positions, sampler_workspace, words, cube, w.codes[0], stream);
    if (rc != INPC_OK) return rc;
    return order_along_curve("inpc_halton_morton_order", positions, n_total, w, false, out, stream);
}
