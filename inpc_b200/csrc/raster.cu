// Rasterizer of the inpc_b200 library: cull/project/SH-evaluate -> order by (tile, depth) ->
// front-to-back blend, forward, backward and inference, bilinear and gaussian splats.
//
// Data layout in HBM (all carved from two caller-allocated blobs):
//   per point   : PointRec 32 B {screen x, screen y, opacity, depth | 4 view-space feature channels}
//                 (one 32-byte sector per gather in the blend), tile bounds 8 B or, bilinear on 8x8 tiles, a packed
//                 footprint of 4 B that they follow from, conic 16 B (gaussian)
//                 depth key + point id, ping-pong pair for the depth sort: the key of every point where it lies, culled ones marked
//   per instance: tile key + point id, ping-pong pair for the tile sort
//   per tile    : [first, last+1) instance range
//
// The arithmetic follows the reference kernels expression by expression (cited per function, paths
// below INPCCudaBackend/INPCCudaBackend/rasterization/ of the reference); the organisation of the
// work does not: culled points are left out by the first pass of the depth sort instead of compacted by atomics, the sorts are the library's own onesweep, and the bilinear blend walks per-pixel bit masks of the staged batch
// instead of testing every staged point against every pixel.
#include "common.cuh"

#include <type_traits>

namespace inpc {

namespace {

constexpr float kTransmittanceEps = 1e-4f;      // include/bilinear/config.h:16
// Alpha of a fragment, rounded: the passes that walk a list (products of segments, forward, backward) must form the same 1 - alpha, or
// they do not agree where a pixel stops.  From the exact product, in one multiply-add, it is another by up to 2^-25, of an almost opaque fragment 10^-4.
__device__ __forceinline__ float rounded_alpha(float opacity, float weight) { return __fmul_rn(opacity, weight); }
constexpr float kOneMinusAlphaEps = 1e-8f;      // include/bilinear/config.h:17
// 1 / (1 - alpha) of the backward passes: the approximate reciprocal (an ulp) and one step of Newton's method, which leaves the rounding of the last operation.  Without
// the branch a division has for operands at the ends of the range; those that are met here, from 10^-8 up, lie far inside, and what is infinite stays as it is.
__device__ __forceinline__ float one_minus_alpha_reciprocal(float one_minus_alpha) {
    const float x = fmaxf(one_minus_alpha, kOneMinusAlphaEps);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    const float off = __fmaf_rn(-x, r, 1.0f);
    return __fmaf_rn(r, x < 3.0e38f ? off : 0.0f, r);
}
constexpr float kDilation = 0.16f;              // include/gaussian/config.h:19
constexpr float kTrainGaussThreshold = 0.01110899653f;   // src/gaussian/kernels.cu:452


// Checked build (-DINPC_CHECK_INDICES, `python -m inpc_b200._build --checked`): every point index read
// from a sorted list is range-checked before it is used for a gather; a bad one is counted, reported
// through a status word and replaced by 0, so the access itself never leaves its array.  The limit
// lives in a device variable the entry points set before they launch anything.
#ifdef INPC_CHECK_INDICES
__device__ unsigned long long g_check_n_points;
__device__ unsigned g_check_failures;
__device__ __forceinline__ uint32_t checked_point(uint32_t id) {
    if ((unsigned long long)id >= g_check_n_points) {
        atomicAdd(&g_check_failures, 1u);
        return 0u;
    }
    return id;
}
#else
__device__ __forceinline__ uint32_t checked_point(uint32_t id) { return id; }
#endif

enum { VAR_TRAIN = 0, VAR_RAW37 = 1, VAR_PREEXTRACTED = 2, VAR_ROWS = 3 };   // VAR_ROWS: features stay in the caller's (n, C) fp32 array

struct __align__(16) PointRec {
    float sx, sy, opacity, depth;
    float f[4];
};

struct RasterParams {
    ViewParams v;
    int tile;       // tile edge in pixels (8 or 16)
    float inv_tile; // its reciprocal: the edge is a power of two, so x * inv_tile == x / tile bit for bit
    int gw, gh;     // tile grid of one image
    int n_sets;     // images drawn by the call (1 except for batched multi-set inference): the grid has n_sets * gh rows
    float sigma_world, sigma_cutoff;
    const float* scales;   // optional per-point sigma (gaussian, pre-extracted)
    float reach;           // gaussian: -2 log(threshold), the squared Mahalanobis distance at which a splat is cut off
};

// Input points of a call: one array triple, or (batched multi-set inference) up to kMaxSets of them laid end to end in
// a virtual index space in which every set starts at a multiple of 1024, so that a block of the two input passes never
// straddles two sets.  Set j is drawn into its own image: its tiles are rows [j * gh, (j + 1) * gh) of a stacked grid.
constexpr int kMaxSets = 8;
constexpr int64_t kSetAlign = 1024;
struct PointSets {
    int count;
    int64_t start[kMaxSets + 1];      // virtual index of every set's first point; start[count] = virtual total
    int64_t size[kMaxSets];
    const float* positions[kMaxSets];
    const void* features[kMaxSets];
    const float* opacities[kMaxSets];
};
__device__ __forceinline__ int set_of_block(const PointSets& ps, int64_t block_first) {
    int j = 0;
    while (j + 1 < ps.count && block_first >= ps.start[j + 1]) ++j;
    return j;
}

struct Projection {
    bool visible;
    float depth, sx, sy;
    unsigned x0, x1, y0, y1;
    float cx, cy, cz;   // conic
};

struct W2C {
    float r0[4], r1[4], r2[4];
};

__device__ __forceinline__ W2C load_w2c(const float* w2c) {
    W2C m;
#pragma unroll
    for (int k = 0; k < 4; ++k) { m.r0[k] = w2c[k]; m.r1[k] = w2c[4 + k]; m.r2[k] = w2c[8 + k]; }
    return m;
}

// One row of the world-to-camera transform applied to a point: r.x p.x + r.y p.y + r.z p.z + r.w with the
// roundings of the reference binary (src/bilinear/kernels.cu:43-49 as nvcc contracts it): the second
// product is rounded, the first and the third are fused onto it, the translation is added last.  Written
// with intrinsics so that depth keys and screen positions, which are compared bit for bit, do not depend
// on the compiler's choice of contraction.
__device__ __forceinline__ float affine_row(const float* r, float px, float py, float pz) {
    float t = __fmul_rn(r[1], py);
    t = __fmaf_rn(r[0], px, t);
    t = __fmaf_rn(r[2], pz, t);
    return __fadd_rn(t, r[3]);
}

// src/bilinear/kernels.cu:41-65 and src/gaussian/kernels.cu:41-90 (training), :145-186 (inference),
// :243-292 (pre-extracted): depth cull, perspective divide, pixel coordinates, tile bounds.
// `scales_index`: index into rp.scales; `set`: which image of the stacked tile grid the point is drawn into.
template <int MODE, int VARIANT>
__device__ __forceinline__ Projection project_point(const float px, const float py, const float pz, const W2C& m,
                                                    const RasterParams& rp, const int64_t i, const int set = 0) {
    Projection o;
    o.visible = false;
    o.x0 = o.x1 = o.y0 = o.y1 = 0;
    o.cx = o.cy = o.cz = 0.0f;
    const float depth = affine_row(m.r2, px, py, pz);
    o.depth = depth;
    o.sx = o.sy = 0.0f;
    if (depth < rp.v.near_plane || depth > rp.v.far_plane) return o;
    const float x = __fdiv_rn(affine_row(m.r0, px, py, pz), depth);
    const float y = __fdiv_rn(affine_row(m.r1, px, py, pz), depth);
    const float sx = __fmaf_rn(x, rp.v.fx, rp.v.cx);
    const float sy = __fmaf_rn(y, rp.v.fy, rp.v.cy);
    float ex = 0.5f, ey = 0.5f;
    if (MODE == INPC_MODE_GAUSSIAN) {
        float variance_world;
        float k = 3.0f;
        if (VARIANT == VAR_TRAIN) {
            constexpr float numerator = 0.3f * 0.3f * 0.5f * 0.5f;
            variance_world = numerator / (rp.v.fx * rp.v.fy);
        } else {
            k = rp.sigma_cutoff;
            if (VARIANT == VAR_PREEXTRACTED && rp.scales != nullptr) {
                const float s = __ldg(rp.scales + i);
                variance_world = s * s;
            } else {
                variance_world = rp.sigma_world * rp.sigma_world;
            }
        }
        const float fx = rp.v.fx, fy = rp.v.fy, cx = rp.v.cx, cy = rp.v.cy;
        const float J_00 = fx / depth;
        const float J_02 = -J_00 * fminf(fmaxf(x, -1.3f * cx / fx), 1.3f * cx / fx);
        const float J_11 = fy / depth;
        const float J_12 = -J_11 * fminf(fmaxf(y, -1.3f * cy / fy), 1.3f * cy / fy);
        float cov_x = variance_world * (J_00 * J_00 + J_02 * J_02);
        const float cov_y = variance_world * (J_02 * J_12);
        float cov_z = variance_world * (J_11 * J_11 + J_12 * J_12);
        cov_x += kDilation;
        cov_z += kDilation;
        const float det = cov_x * cov_z - cov_y * cov_y;
        if (det == 0.0f) return o;
        const float det_rcp = 1.0f / det;
        o.cx = cov_z * det_rcp;
        o.cy = -cov_y * det_rcp;
        o.cz = cov_x * det_rcp;
        ex = k * sqrtf(cov_x) - 0.5f;
        ey = k * sqrtf(cov_z) - 0.5f;
    }
    const float itf = rp.inv_tile;
    const unsigned gw = (unsigned)rp.gw, gh = (unsigned)rp.gh;
    o.x0 = min(gw, (unsigned)max(0, __float2int_rd((sx - ex) * itf)));
    o.x1 = min(gw, (unsigned)max(0, __float2int_ru((sx + ex) * itf)));
    o.y0 = min(gh, (unsigned)max(0, __float2int_rd((sy - ey) * itf)));
    o.y1 = min(gh, (unsigned)max(0, __float2int_ru((sy + ey) * itf)));
    o.sx = sx;
    o.sy = sy;
    o.visible = (o.x1 - o.x0) * (o.y1 - o.y0) != 0u;
    o.y0 += (unsigned)set * gh;   // rows of this set's image in the stacked grid (screen coordinates stay the set's own)
    o.y1 += (unsigned)set * gh;
    return o;
}

// ---- one launch for everything a call needs zeroed (images, weights, sort state, counters) ---------
// Nine separate memsets were a fifth of the launches of a small training step.
constexpr int kMaxClear = 8;
struct ClearList {
    int count = 0;
    void* ptr[kMaxClear];
    size_t bytes[kMaxClear];   // multiples of 4
    void add(void* p, size_t n) {
        if (p && n) { ptr[count] = p; bytes[count] = n; ++count; }
    }
};
__global__ void __launch_bounds__(256) clear_kernel(const __grid_constant__ ClearList list) {
    await_previous_kernel();
    const size_t tid = (size_t)blockIdx.x * 256 + threadIdx.x, stride = (size_t)gridDim.x * 256;
    for (int r = 0; r < list.count; ++r) {
        char* p = static_cast<char*>(list.ptr[r]);
        const size_t lead = min(list.bytes[r], (size_t)((16u - (unsigned)(reinterpret_cast<uintptr_t>(p) & 15u)) & 15u));
        const size_t n16 = (list.bytes[r] - lead) / 16, tail = lead + n16 * 16;
        for (size_t k = tid; k < n16; k += stride) reinterpret_cast<uint4*>(p + lead)[k] = make_uint4(0u, 0u, 0u, 0u);
        if (4 * tid < lead) *reinterpret_cast<unsigned*>(p + 4 * tid) = 0u;
        if (tail + 4 * tid < list.bytes[r]) *reinterpret_cast<unsigned*>(p + tail + 4 * tid) = 0u;
    }
}

// Exclusive scan of n words in place by one block of THREADS threads (16 words per thread and round, read past L1: other
// blocks have just written them).  Returns the total; smem: THREADS / 32 + 1 words.
template <int THREADS>
__device__ __forceinline__ unsigned scan_words(unsigned* data, int64_t n, unsigned* smem) {
    constexpr int kPer = 16;
    unsigned running = 0;
    for (int64_t base = 0; base < n; base += THREADS * kPer) {
        const int64_t j0 = base + (int64_t)threadIdx.x * kPer;
        unsigned v[kPer], sum = 0;
        if (j0 + kPer <= n) {
#pragma unroll
            for (int k = 0; k < kPer; k += 4) {
                const uint4 q = __ldcg(reinterpret_cast<const uint4*>(data + j0 + k));
                v[k] = q.x; v[k + 1] = q.y; v[k + 2] = q.z; v[k + 3] = q.w;
            }
        } else {
#pragma unroll
            for (int k = 0; k < kPer; ++k) v[k] = j0 + k < n ? __ldcg(data + j0 + k) : 0u;
        }
#pragma unroll
        for (int k = 0; k < kPer; ++k) sum += v[k];
        unsigned total;
        unsigned ex = running + block_exclusive_scan(sum, smem, &total);
        if (j0 + kPer <= n) {
#pragma unroll
            for (int k = 0; k < kPer; k += 4) {
                uint4 q;
                q.x = ex; q.y = q.x + v[k]; q.z = q.y + v[k + 1]; q.w = q.z + v[k + 2];
                ex = q.w + v[k + 3];
                *reinterpret_cast<uint4*>(data + j0 + k) = q;
            }
        } else {
#pragma unroll
            for (int k = 0; k < kPer; ++k) {
                if (j0 + k < n) data[j0 + k] = ex;
                ex += v[k];
            }
        }
        running += total;
    }
    return running;
}

constexpr int kPreThreads = 256;
constexpr int projection_blocks(int mode) { return mode == INPC_MODE_GAUSSIAN ? 5 : 6; }   // per multiprocessor, see preprocess_kernel
// The number of tiles a splat touches rides in the key bits above the depth offsets where these leave room (the sort ignores bits above its range and carries
// them along), which saves the instance count a gather: bilinear 1, 2 or 4, less one, in bits 30..31; gaussian 1..30 in bits 27..31, 0 for more, which are looked up.
constexpr unsigned kCountShift = 30, kGaussCountShift = 27, kMostKeyTiles = 30;

constexpr int kScanThreads = 1024;

// SH degree 2 along the view ray -> 4 channels: include/sh_utils.cuh:6-23.  `h` points at 36 halves
// (coefficient-major, channel-minor) in shared memory.
__device__ __forceinline__ void sh_basis(const float px, const float py, const float pz, const float* __restrict__ cam,
                                         float* b) {
    const float vx = px - __ldg(cam), vy = py - __ldg(cam + 1), vz = pz - __ldg(cam + 2);
    const float inv = rsqrtf(vx * vx + vy * vy + vz * vz);
    const float x = vx * inv, y = vy * inv, z = vz * inv;
    const float xx = x * x, yy = y * y, zz = z * z;
    const float xy = x * y, yz = y * z, xz = x * z;
    b[0] = 0.28209479177387814f;
    b[1] = 0.48860251190291987f * y;
    b[2] = 0.48860251190291987f * z;
    b[3] = 0.48860251190291987f * x;
    b[4] = 1.0925484305920792f * xy;
    b[5] = 1.0925484305920792f * yz;
    b[6] = 0.94617469575755997f * zz - 0.31539156525251999f;
    b[7] = 1.0925484305920792f * xz;
    b[8] = 0.54627421529603959f * xx - 0.54627421529603959f * yy;
}

// One point's 36 coefficients from the shared slab, four channels of a coefficient at a time.  ODD (rows of 37 halves, the first of which is the raw opacity): the
// coefficients begin at a multiple of four bytes in every second row only, so whole words are read and shifted by half a word in the others.  (Rows of 36: nine 8-byte
// loads that meet every bank once, where 36 loads of a half took four times the wavefronts.)
template <bool ODD>
__device__ __forceinline__ void sh_eval(const float* b, const unsigned char* slab, unsigned row, float* f, float* raw_opacity) {
    unsigned carry = 0u;
    const unsigned char* p = slab + row * (ODD ? 74u : 72u);
    const bool half_word = ODD && (row & 1u) == 0u;   // the coefficients begin in the middle of a word
    if (ODD) {
        const unsigned first = *reinterpret_cast<const unsigned*>(p - (half_word ? 0u : 2u));
        *raw_opacity = __half2float(__ushort_as_half((unsigned short)(half_word ? first : first >> 16)));
        carry = first;
        p += half_word ? 4u : 2u;
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        uint2 w;
        if (ODD) {
            const unsigned* q = reinterpret_cast<const unsigned*>(p) + 2 * k;
            const unsigned w0 = q[0], w1 = q[1];
            w = half_word ? make_uint2(__funnelshift_r(carry, w0, 16), __funnelshift_r(w0, w1, 16)) : make_uint2(w0, w1);
            carry = w1;
        } else {
            w = reinterpret_cast<const uint2*>(p)[k];
        }
        const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&w.x)), hi = __half22float2(*reinterpret_cast<const __half2*>(&w.y));
        const float h[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (k == 0) f[c] = b[0] * h[c];
            else if (k & 1) f[c] = f[c] - b[k] * h[c];
            else f[c] = f[c] + b[k] * h[c];
        }
    }
}

// What the instance emission of the warp blend needs of a bilinear splat, in one word: 4 bytes per point keep the array (33 MB for 2^23 points) resident
// in L2 where the emission gathers from it in depth order, and in most calls the depth sort has room to carry the word along (CarriedCodes).
//   bit 31 clear: first tile it touches in the (stacked) grid * 64 + row * 8 + column of the upper left pixel of its 2x2 footprint in that tile; it touches a
//                 second tile column or row if and only if that is the last pixel column or row of the tile.
//   bit 31 set:   the splats of which this is not so -- the footprint begins in front of the image, or ends at its border, or the splat lies exactly between two
//                 pixels at a tile's edge: first tile column in bits 4..15, row in bits 20..30, and in front of them the column and row of that pixel in
//                 the tile plus one (0..8), 9 for 8 and a second tile.  (8 it is whenever there is a second tile: with sx - 0.5 rounded below the last
//                 pixel of a tile, sx + 0.5 rounds to the tile's end at most.)
constexpr int kMaxCodedSide = 32760;       // widest image of this path, in pixels
constexpr int kMaxCodedTileRows = 2047;    // most tile rows of the (stacked) grid
constexpr uint32_t kNoQuad = 0xFFFFFFFFu;  // of a culled point
struct Footprint {
    unsigned tile;          // first tile
    unsigned column, row;   // of the upper left pixel in that tile, plus one: 0 .. 8
    bool two_columns, two_rows;
};
__device__ __forceinline__ uint32_t pack_quad(const Projection& pr, int tile_rows_before, int gw) {
    // rows are relative to the tile: the first row of an image other than the first is not row 0 of the grid
    const unsigned column = (unsigned)(__float2int_rd(pr.sx - 0.5f) - (int)pr.x0 * 8 + 1);
    const unsigned row = (unsigned)(__float2int_rd(pr.sy - 0.5f) - ((int)pr.y0 - tile_rows_before) * 8 + 1);
    const unsigned two_columns = pr.x1 - pr.x0 - 1u, two_rows = pr.y1 - pr.y0 - 1u;
    if (column - 1u < 8u && row - 1u < 8u && two_columns == (column == 8u ? 1u : 0u) && two_rows == (row == 8u ? 1u : 0u))
        return (pr.y0 * (unsigned)gw + pr.x0) << 6 | (row - 1u) << 3 | (column - 1u);
    return 0x80000000u | pr.y0 << 20 | (min(row, 8u) + two_rows) << 16 | pr.x0 << 4 | (min(column, 8u) + two_columns);
}
__device__ __forceinline__ Footprint footprint_of_quad(uint32_t q, int gw) {
    if (!(q >> 31)) {
        const unsigned column = (q & 7u) + 1u, row = (q >> 3 & 7u) + 1u;
        return {q >> 6, column, row, column == 8u, row == 8u};
    }
    const unsigned column = q & 0xFu, row = q >> 16 & 0xFu;
    return {(q >> 20 & 0x7FFu) * (unsigned)gw + (q >> 4 & 0xFFFu), min(column, 8u), min(row, 8u), column == 9u, row == 9u};
}
__device__ __forceinline__ unsigned tiles_of_footprint(bool two_columns, bool two_rows) { return (two_columns ? 2u : 1u) << (two_rows ? 1 : 0); }

// Tile bounds of a splat in the form of the `bounds` array.
__device__ __forceinline__ uint2 quad_bounds(uint32_t q, int gw) {
    if (q == kNoQuad) return make_uint2(0u, 0u);
    const Footprint f = footprint_of_quad(q, gw);
    const unsigned y0 = f.tile / (unsigned)gw, x0 = f.tile - y0 * (unsigned)gw;
    return make_uint2(x0 | ((x0 + 1u + f.two_columns) << 16), y0 | ((y0 + 1u + f.two_rows) << 16));
}

// What the instance emission needs of a gaussian splat on 8x8 tiles: its tile bounds, and how far its ellipse stays away from
// their sides in cells of 2x2 pixels, four bits each (left, right, top, bottom; rounded down, so the cells between are a superset).
__device__ __forceinline__ uint4 pack_footprint(const Projection& pr, float reach) {
    const float det = pr.cx * pr.cz - pr.cy * pr.cy;
    unsigned inset = 0u;
    if (det > 0.0f) {
        const float s = reach / det;
        const float rx = sqrtf(fmaxf(s * pr.cz, 0.0f)) * 1.001f + 0.01f;
        const float ry = sqrtf(fmaxf(s * pr.cx, 0.0f)) * 1.001f + 0.01f;
        const int left = (__float2int_ru(pr.sx - rx - 0.5f) >> 1) - 4 * (int)pr.x0, right = 4 * (int)pr.x1 - 1 - (__float2int_rd(pr.sx + rx - 0.5f) >> 1);
        const int top = (__float2int_ru(pr.sy - ry - 0.5f) >> 1) - 4 * (int)pr.y0, bottom = 4 * (int)pr.y1 - 1 - (__float2int_rd(pr.sy + ry - 0.5f) >> 1);
        inset = (unsigned)min(max(left, 0), 15) | ((unsigned)min(max(right, 0), 15) << 4) | ((unsigned)min(max(top, 0), 15) << 8) |
                ((unsigned)min(max(bottom, 0), 15) << 12);
    }
    return make_uint4(pr.x0 | (pr.x1 << 16), pr.y0 | (pr.y1 << 16), inset, 0u);
}

// Project, evaluate SH, write the point record, what the instance passes need of the splat, and the depth key, all of it where the point lies: the key of a culled
// point is kNoKey, and the depth sort leaves it out, so that nothing is compacted.
// src/bilinear/kernels.cu:11-84, :106-184; src/gaussian/kernels.cu:11-111, :113-217, :219-324.
//
// Persistent blocks take chunks of kPreThreads points; they count the digits of the keys for the depth sort (and so the visible points: *n_visible), and, where the host
// wants to know, the (point, tile) instances (*n_instances, which starts at zero).  The pass is bound by DRAM (128 bytes per point) as long as enough copies are in
// flight: six blocks of 40 registers (five of 48 where ellipses are formed), the matrix in shared memory, or they spill.  Against one block per chunk, a histogram of the keys of its
// own and, where the host sizes the instance arrays, a pass that projected and counted first: 2^23 bilinear 156 + 19 -> 167 us, 2^25 of a cloud 598 + 51 -> 630, 2^22 gaussian
// 119 + 36 + 13 -> 115, 2^23 feature rows 97 + 40 + 17 -> 91.  Four blocks of 63 registers with positions loaded and the next slab asked for ahead: 168 / 635 / 130; five blocks of the same with 80 bytes
// spilled 200 / 760; eight of 32 registers, 44 bytes spilled, 178 / 653.
template <int MODE, int VARIANT>
__global__ void __launch_bounds__(kPreThreads, projection_blocks(MODE)) preprocess_kernel(
    const __grid_constant__ PointSets ps, const __grid_constant__ RasterParams rp, unsigned n_chunks, unsigned key_base, PointRec* __restrict__ rec, uint2* __restrict__ bounds,
    uint32_t* __restrict__ quad, float4* __restrict__ conic, uint4* __restrict__ foot, uint32_t* __restrict__ depth_keys, int pack_count, int rec_stride,
    KeyHistogram digits, unsigned long long* n_visible, unsigned long long* n_instances, volatile unsigned* status) {
    await_previous_kernel();
    constexpr int kHalves = VARIANT == VAR_RAW37 ? 37 : 36;
    constexpr int kSlabBytes = VARIANT == VAR_ROWS ? 16 : kPreThreads * kHalves * 2;   // multiple of 16 for both layouts
    __shared__ __align__(16) unsigned char s_feat[kSlabBytes];
    __shared__ BlockHistogram s_digits;
    __shared__ __align__(8) unsigned long long s_bar;
    __shared__ float s_w2c[12];
    clear_histogram(s_digits);
    if (threadIdx.x < 12u) s_w2c[threadIdx.x] = __ldg(rp.v.w2c + threadIdx.x);
    if (VARIANT != VAR_ROWS && threadIdx.x == 0) mbarrier_init(&s_bar, 1);
    __syncthreads();
    unsigned phase = 0u;
    unsigned long long instances = 0ull;
    bool slab_ready = true;
    for (unsigned chunk = blockIdx.x; chunk < n_chunks; chunk += gridDim.x) {
        // this chunk's set: the input arrays are indexed by the point's position in its set (i), everything this pass
        // writes by its position in the virtual index space of the call (iv); the two coincide for a single set
        const int64_t block_first_v = (int64_t)chunk * kPreThreads;
        const int set = set_of_block(ps, block_first_v);
        const float* __restrict__ positions = ps.positions[set];
        const __half* __restrict__ features = static_cast<const __half*>(ps.features[set]);
        const int64_t n = ps.size[set];
        const int64_t block_first = block_first_v - ps.start[set];
        const int in_block = (int)max((int64_t)0, min((int64_t)kPreThreads, n - block_first));
        // The chunk's feature slab is contiguous in global memory.  When base and size allow (multiples of
        // 16 bytes) one bulk asynchronous copy brings it in while the threads project their points;
        // otherwise loads through registers do, of 16 bytes (odd last chunk) or 2 (caller view that is not aligned).
        const bool aligned = (reinterpret_cast<uintptr_t>(features) & 15u) == 0;
        const bool bulk = VARIANT != VAR_ROWS && slab_ready && aligned && in_block > 0 && ((in_block * kHalves * 2) & 15) == 0;
        if (bulk) {
            if (threadIdx.x == 0)
                bulk_load_to_shared(s_feat, reinterpret_cast<const unsigned char*>(features) + block_first * (kHalves * 2), (unsigned)(in_block * kHalves * 2), &s_bar);
        } else if (VARIANT != VAR_ROWS) {
            const unsigned char* src = reinterpret_cast<const unsigned char*>(features) + block_first * (kHalves * 2);
            const int bytes = in_block * kHalves * 2;
            const int n16 = aligned ? bytes / 16 : 0;
            const uint4* src16 = reinterpret_cast<const uint4*>(src);
            uint4* dst16 = reinterpret_cast<uint4*>(s_feat);
            for (int k = threadIdx.x; k < n16; k += kPreThreads) dst16[k] = __ldg(src16 + k);
            for (int k = n16 * 16 + 2 * threadIdx.x; k < bytes; k += 2 * kPreThreads)
                *reinterpret_cast<unsigned short*>(s_feat + k) = __ldg(reinterpret_cast<const unsigned short*>(src + k));
            fence_shared_for_bulk();   // a bulk copy may overwrite the slab in the next round
        }
        const int64_t i = block_first + threadIdx.x;
        const int64_t iv = block_first_v + threadIdx.x;
        Projection pr;
        pr.visible = false;
        float px = 0, py = 0, pz = 0;
        if (i < n) {
            px = __ldg(positions + 3 * i); py = __ldg(positions + 3 * i + 1); pz = __ldg(positions + 3 * i + 2);
            pr = project_point<MODE, VARIANT>(px, py, pz, load_w2c(s_w2c), rp, i, set);
        }
        if (bulk) {
            slab_ready = mbarrier_wait_bounded(&s_bar, phase);
            phase ^= 1u;
            if (!slab_ready && status) status[STATUS_BULK_COPY_TIMEOUT] = 1u;
        } else if (VARIANT != VAR_ROWS) {
            __syncthreads();
        }
        if (!slab_ready) pr.visible = false;   // the results are invalid, and reported so, but everything behind this pass finds keys and words that it can read
        if (pr.visible) {
            float4* const dst = reinterpret_cast<float4*>(rec) + (VARIANT == VAR_ROWS ? (size_t)iv * rec_stride : 2 * (size_t)iv);
            if (VARIANT == VAR_ROWS) {
                // feature rows are gathered by the blend itself: the record carries the geometry only.  The warp blend reads such
                // records 16 bytes apart (rec_stride 1): half-written 32-byte sectors cost as much DRAM traffic as whole ones
                dst[0] = make_float4(pr.sx, pr.sy, __ldg(ps.opacities[set] + i), pr.depth);
            } else {
                float b[9];
                sh_basis(px, py, pz, rp.v.cam, b);
                float opacity, f[4];
                sh_eval<VARIANT == VAR_RAW37>(b, s_feat, threadIdx.x, f, &opacity);
                // opacity = 1 - exp(-exp(raw)) with the fast exponential: src/bilinear/kernels.cu:144
                if (VARIANT == VAR_RAW37) opacity = 1.0f - __expf(-__expf(opacity));
                else opacity = __ldg(ps.opacities[set] + i);
                dst[0] = make_float4(pr.sx, pr.sy, opacity, pr.depth);
                dst[1] = make_float4(f[0], f[1], f[2], f[3]);
            }
            if (MODE == INPC_MODE_GAUSSIAN) {
                conic[iv] = make_float4(pr.cx, pr.cy, pr.cz, 0.0f);
                if (foot) foot[iv] = pack_footprint(pr, rp.reach);
            }
            if (n_instances) instances += (pr.x1 - pr.x0) * (pr.y1 - pr.y0);
        }
        if (iv < ps.start[ps.count]) {   // (also the padding behind a set)
            // what the instance passes need of a point: its packed footprint where splats are bilinear on 8x8 tiles, else its tile bounds
            if (MODE == INPC_MODE_BILINEAR && quad) quad[iv] = pr.visible ? pack_quad(pr, set * rp.gh, rp.gw) : kNoQuad;
            else bounds[iv] = pr.visible ? make_uint2(pr.x0 | (pr.x1 << 16), pr.y0 | (pr.y1 << 16)) : make_uint2(0u, 0u);
            // sort key: offset of the depth's bit pattern from the smallest there can be (fewer radix passes), and the number of tiles
            uint32_t key = kNoKey;
            if (pr.visible) {
                key = __float_as_uint(pr.depth) - key_base;
                count_key(s_digits, digits.pt, key);
                const unsigned tiles = (pr.x1 - pr.x0) * (pr.y1 - pr.y0);
                if (pack_count) key |= MODE == INPC_MODE_BILINEAR ? (tiles - 1u) << kCountShift : (tiles <= kMostKeyTiles ? tiles : 0u) << kGaussCountShift;
            }
            depth_keys[iv] = key;
        }
        if (VARIANT != VAR_ROWS) slab_ready = !__syncthreads_or(!slab_ready);   // everybody has read the slab
    }
    if (n_instances) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) instances += __shfl_down_sync(0xffffffffu, instances, o);
        if (lane_id() == 0 && instances) atomicAdd(n_instances, instances);
    }
    finish_histogram(s_digits, digits, gridDim.x, n_visible);
}

__device__ __forceinline__ unsigned tiles_of(const uint2 b) {
    return ((b.x >> 16) - (b.x & 0xffffu)) * ((b.y >> 16) - (b.y & 0xffffu));
}

// Instances per depth-sorted point, reduced per block (src/bilinear/kernels.cu:186-196 + the
// cub::DeviceScan::ExclusiveSum of src/bilinear/forward.cu:109-115, first half).
constexpr int kInstThreads = 1024;   // block sums over 1024 points keep the one-block scan short
__device__ __forceinline__ unsigned tiles_of_code(uint32_t code, uint32_t escape) {
    return code >= escape ? 1u << (code - escape) : tiles_of_footprint((code & 7u) == 7u, (code >> 3 & 7u) == 7u);
}

// COUNTS_IN_KEYS, COUNTS_IN_CODES (see CarriedCodes): a warp sums one block's worth of points, all its loads in flight together, no barrier before the last
// block's scan (a barrier per group of a block and one load per thread: 2^23 / 2^25 points 16 / 61 -> 11 / 39 us).
enum { COUNTS_GATHERED = 0, COUNTS_IN_KEYS = 1, COUNTS_IN_CODES = 2, COUNTS_IN_GAUSS_KEYS = 3 };
template <int SOURCE>
__global__ void __launch_bounds__(kInstThreads / 4) instance_count_kernel(const uint32_t* __restrict__ sorted_keys,
                                                                          const uint32_t* __restrict__ sorted_ids,
                                                                          const uint2* __restrict__ bounds, const uint32_t* __restrict__ quad, const unsigned long long* __restrict__ n_visible_dev,
                                                                          unsigned* block_sums, unsigned n_groups, unsigned* done, unsigned long long* n_instances, uint32_t escape) {
    await_previous_kernel();
    const int64_t n_visible = (int64_t)*n_visible_dev;
    constexpr unsigned kWarps = kInstThreads / 4 / 32;
    if (SOURCE != COUNTS_GATHERED) {
        auto count_of = [&](uint32_t word) -> unsigned {
            if (SOURCE == COUNTS_IN_KEYS) return (word >> kCountShift) + 1u;
            if (SOURCE == COUNTS_IN_GAUSS_KEYS) return word >> kGaussCountShift;
            return tiles_of_code(word, escape);
        };
        constexpr int kLoads = kInstThreads / 128;   // 16-byte loads per lane and group
        for (unsigned group = blockIdx.x * kWarps + (threadIdx.x >> 5); group < n_groups; group += gridDim.x * kWarps) {
            const int64_t first = (int64_t)group * kInstThreads + 4 * (int64_t)lane_id();
            unsigned c = 0;
            if ((int64_t)(group + 1) * kInstThreads <= n_visible) {
                uint4 k[kLoads];
#pragma unroll
                for (int q = 0; q < kLoads; ++q) k[q] = __ldg(reinterpret_cast<const uint4*>(sorted_keys + first + 128 * q));   // the key buffers are 16-byte aligned
#pragma unroll
                for (int q = 0; q < kLoads; ++q) {
                    const unsigned t[4] = {count_of(k[q].x), count_of(k[q].y), count_of(k[q].z), count_of(k[q].w)};
                    if (SOURCE == COUNTS_IN_GAUSS_KEYS && (t[0] == 0u || t[1] == 0u || t[2] == 0u || t[3] == 0u)) {
                        // more tiles than the field holds
                        const uint4 id = __ldg(reinterpret_cast<const uint4*>(sorted_ids + first + 128 * q));
                        const uint2 none = make_uint2(0u, 0u);
                        const uint2 b0 = t[0] ? none : __ldg(bounds + checked_point(id.x)), b1 = t[1] ? none : __ldg(bounds + checked_point(id.y));
                        const uint2 b2 = t[2] ? none : __ldg(bounds + checked_point(id.z)), b3 = t[3] ? none : __ldg(bounds + checked_point(id.w));
                        c += tiles_of(b0) + tiles_of(b1) + tiles_of(b2) + tiles_of(b3);
                    }
                    c += t[0] + t[1] + t[2] + t[3];
                }
            } else {
                for (int64_t s = (int64_t)group * kInstThreads + lane_id(); s < n_visible; s += 32) {
                    const unsigned t = count_of(__ldg(sorted_keys + s));
                    c += SOURCE == COUNTS_IN_GAUSS_KEYS && t == 0u ? tiles_of(__ldg(bounds + checked_point(__ldg(sorted_ids + s)))) : t;
                }
            }
            c = __reduce_add_sync(0xffffffffu, c);
            if (lane_id() == 0) block_sums[group] = c;
        }
    } else {
        // two dependent gathers per point: a block per group, so that more of them are in flight (a warp per group: 16 -> 27 us for 2 * 10^6 points)
        __shared__ unsigned s_w[2][kWarps];
        int flip = 0;
        for (unsigned group = blockIdx.x; group < n_groups; group += gridDim.x, flip ^= 1) {
            const int64_t first = (int64_t)group * kInstThreads + 4 * (int64_t)threadIdx.x;
            unsigned c = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int64_t s = first + q;
                if (s >= n_visible) continue;
                const uint32_t id = checked_point(__ldg(sorted_ids + s));
                if (quad) {
                    const Footprint f = footprint_of_quad(__ldg(quad + id), 0);
                    c += tiles_of_footprint(f.two_columns, f.two_rows);
                } else {
                    c += tiles_of(__ldg(bounds + id));
                }
            }
            c = __reduce_add_sync(0xffffffffu, c);
            if (lane_id() == 0) s_w[flip][threadIdx.x >> 5] = c;
            __syncthreads();
            if (threadIdx.x == 0) {
                unsigned t = 0;
#pragma unroll
                for (unsigned w = 0; w < kWarps; ++w) t += s_w[flip][w];
                block_sums[group] = t;
            }
        }
    }
    __shared__ unsigned s_scan[kInstThreads / 4 / 32 + 1];
    if (!last_block(done, gridDim.x)) return;
    const unsigned total = scan_words<kInstThreads / 4>(block_sums, n_groups, s_scan);   // sums -> first instance of every block
    if (threadIdx.x == 0 && n_instances) n_instances[0] = n_instances[1] = total;   // the second: see emit_quads_kernel
}

// Instance key: the tile index in the low 24 bits, the only bits the tile sort looks at (it carries the
// bits above its range along).  For bilinear splats on 8x8 tiles the 8 bits above hold where the 2x2
// pixel footprint sits in the tile: column of its left pixel relative to the tile plus one (0..8) in
// bits 24..27, row of its upper pixel plus one in bits 28..31.  The blend then knows which pixels an
// instance can reach from the key alone, without fetching the point record.
constexpr unsigned kTileKeyBits = 24;
constexpr uint32_t kTileKeyMask = (1u << kTileKeyBits) - 1u;

// For gaussian splats on 8x8 tiles the 8 bits above the tile index name the 2x2-pixel cells of the tile that the ellipse can
// reach: columns [left, right] and rows [top, bottom] of the 4x4 cells, clipped to the tile, ten times ten ranges.
constexpr unsigned kNoCells = 255u;
__device__ __forceinline__ unsigned cell_range_index(unsigned lo, unsigned hi) { return lo * 4u - lo * (lo - 1u) / 2u + (hi - lo); }
__device__ __forceinline__ void cell_range(unsigned index, unsigned* lo, unsigned* hi) {
    unsigned l = 0;
    while (l < 3u && index >= 4u - l) { index -= 4u - l; ++l; }
    *lo = l;
    *hi = l + index;
}
__device__ __forceinline__ unsigned cell_code(int left, int right, int top, int bottom) {
    left = max(left, 0); top = max(top, 0);
    right = min(right, 3); bottom = min(bottom, 3);
    if (left > right || top > bottom) return kNoCells;
    return cell_range_index((unsigned)left, (unsigned)right) + 10u * cell_range_index((unsigned)top, (unsigned)bottom);
}

// One (tile key, point id) pair per touched tile, row-major over the point's bounds, points in depth
// order (src/bilinear/kernels.cu:198-220).
//
// Bilinear splats on 8x8 tiles: bounds and footprint origin come from the packed word the projection pass left per point (see pack_quad), a 4-byte
// gather.  Bound by these random gathers, one 32-byte sector each, and by instruction issue.  What is read or written once bypasses
// the caches' replacement, so that more of the gathered array stays in L2.  A splat has one, two or four instances: the sums over a warp
// come from three ballots, those over a block from one barrier and a warp reduction, and the keys are put together without a loop.  A block takes
// groups of 1024 points one after the other and counts the digits of the keys it writes (and so the keys: *n_emitted, which inpc_raster_resolve compares with the
// count made from the sorted keys; not where there is one tile, or nothing is visible), which spares the tile sort its pass over them: emission and
// histogram of 2^20 / 2^23 / 2^24 / 2^25 points 21 / 104 / 207 / 496 -> 16 / 95 / 192 / 412 us (half of the last by fewer blocks).
// (Four consecutive points per thread with their gathers in flight together and the instances staged in shared memory: the emission alone 116 us for
// 2^23 points, 396 for 2^24, 952 for 2^25.)
__global__ void __launch_bounds__(kInstThreads, 2) emit_quads_kernel(const uint32_t* __restrict__ sorted_ids, const uint32_t* __restrict__ quad, const unsigned long long* __restrict__ n_visible_dev, const unsigned* __restrict__ block_base, int gw,
                                                                     KeyHistogram digits, unsigned long long* __restrict__ n_emitted, uint32_t* __restrict__ inst_keys,
                                                                     uint32_t* __restrict__ inst_ids) {
    await_previous_kernel();
    __shared__ unsigned s_total[2][kInstThreads / 32];   // of two groups in turn, so that one barrier does
    __shared__ BlockHistogram s_digits;
    const int64_t n_visible = (int64_t)*n_visible_dev;
    const int64_t n_groups = ceil_div<int64_t>(n_visible, kInstThreads);
    if ((int64_t)blockIdx.x >= n_groups) return;
    clear_histogram(s_digits);
    __syncthreads();
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5, lt_mask = (1u << lane) - 1u;
    auto emit = [&](unsigned at, uint32_t key, uint32_t id) {
        __stcs(inst_keys + at, key);
        __stcs(inst_ids + at, id);
        count_key(s_digits, digits.pt, key);
    };
    unsigned flip = 0;
    for (int64_t group = blockIdx.x; group < n_groups; group += gridDim.x, flip ^= 1u) {
        const int64_t s = group * kInstThreads + threadIdx.x;
        const bool there = s < n_visible;
        const uint32_t id = there ? checked_point(__ldcs(sorted_ids + s)) : 0u;
        const uint32_t q = there ? __ldg(quad + id) : 0u;
        const Footprint f = footprint_of_quad(q, gw);
        const bool two_columns = there && f.two_columns, two_rows = there && f.two_rows;
        // one, two or four instances per point: the sum over the lanes before this one from three ballots
        const unsigned bt = __ballot_sync(0xffffffffu, there), bc = __ballot_sync(0xffffffffu, two_columns), br = __ballot_sync(0xffffffffu, two_rows);
        if (lane == 0) s_total[flip][warp] = __popc(bt) + __popc(bc) + __popc(br) + __popc(bc & br);
        __syncthreads();
        unsigned off = __ldg(block_base + group) + __reduce_add_sync(0xffffffffu, lane < warp ? s_total[flip][lane] : 0u) + __popc(bt & lt_mask) + __popc(bc & lt_mask) +
                       __popc(br & lt_mask) + __popc(bc & br & lt_mask);
        if (!there) continue;
        // in a second column or row of tiles the footprint starts one pixel before the tile: its code there is zero
        const uint32_t column = f.column << kTileKeyBits, row = f.row << (kTileKeyBits + 4), tile = f.tile;
        emit(off, tile | column | row, id);
        if (two_columns) emit(off + 1u, (tile + 1u) | row, id);
        if (two_rows) {
            off += two_columns ? 2u : 1u;
            emit(off, (tile + (unsigned)gw) | column, id);
            if (two_columns) emit(off + 1u, tile + (unsigned)gw + 1u, id);
        }
    }
    finish_histogram(s_digits, digits, (unsigned)min(n_groups, (int64_t)gridDim.x), n_emitted);
}

// Bilinear splats whose codes the depth sort has carried along: no gather, but where a code does not say it all (one splat in 500 at 1237x822).  A thread takes four
// consecutive points, the loads of the next group under way while this one's instances are written; a warp stages its instances in shared memory and writes them side
// by side.  Bound by instruction issue: 2^20 / 2^23 / 2^25 points 11.5 / 44 / 160 us (16 / 95 / 412 with the kernel above; 43 million instances in 160 us are 3.8 TB/s read and
// written).  What the sort pays for it: 0.2 us of 66 for 2^23 points, 13 of 220 for 2^25, where the words it reads come from DRAM.
// With three blocks (47 / 166 us): two points per thread 54 / 216 us for 2^23 / 2^25; 256 staged pairs per warp and four blocks 58 / 201; no loads ahead 52 / 188; codes of a grid that is one pixel
// larger, which name the splats at the border too but take a division, 59 / 207.  With the gathers of the kernel above this form is the slower one: 2^24 points 193 -> 408 us,
// fewer and busier warps miss L2 more often.
// Two blocks per multiprocessor, which stage 128 of its 228 KB: three take 47 / 163 us alone and leave no room for blocks of other streams' kernels until they end (64 views of 2^23
// samples, four in flight: 1.388 ms per view with three, 1.251 with two, 1.246 with one, which takes longer alone: a view at a time 1.475 / 1.472 / 1.488).
constexpr int kCodedThreads = 512, kCodedPoints = 4, kCodedBlocks = 2;
struct EmitCodedSmem {
    uint2 pairs[kCodedThreads / 32][32 * kCodedPoints * 4];   // the most a warp's points can make
};
__global__ void __launch_bounds__(kCodedThreads, kCodedBlocks) emit_coded_kernel(const uint32_t* __restrict__ sorted_ids, const uint32_t* __restrict__ sorted_codes, const CarriedCodes codes,
                                                                      const unsigned long long* __restrict__ n_visible_dev, const unsigned* __restrict__ block_base, int gw,
                                                                      KeyHistogram digits, unsigned long long* __restrict__ n_emitted, uint32_t* __restrict__ inst_keys,
                                                                      uint32_t* __restrict__ inst_ids) {
    await_previous_kernel();
    constexpr unsigned kGroup = kCodedThreads * kCodedPoints, kWarps = kCodedThreads / 32, kSums = kInstThreads / (32 * kCodedPoints);   // kSums: warps per sum
    static_assert(kGroup % kInstThreads == 0 && kCodedPoints == 4, "groups begin where sums do; 16-byte loads");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    EmitCodedSmem& s_stage = *reinterpret_cast<EmitCodedSmem*>(smem_raw);
    __shared__ unsigned s_total[2][kWarps];   // of two groups in turn, so that one barrier does
    __shared__ BlockHistogram s_digits;
    const unsigned n_visible = (unsigned)*n_visible_dev, n_groups = (n_visible + kGroup - 1u) / kGroup;   // < 2^30
    if (blockIdx.x >= n_groups) return;
    clear_histogram(s_digits);
    __syncthreads();
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    uint2* const stage = s_stage.pairs[warp];
    constexpr uint32_t kNone = 0xFFFFFFFFu;
    uint32_t next_id[kCodedPoints], next_code[kCodedPoints];
    auto load = [&](unsigned group) {
        const unsigned first = group * kGroup + threadIdx.x * kCodedPoints;
        if (group < n_groups && first + kCodedPoints <= n_visible) {
            const uint4 a = __ldcs(reinterpret_cast<const uint4*>(sorted_ids + first)), b = __ldcs(reinterpret_cast<const uint4*>(sorted_codes + first));
            next_id[0] = a.x; next_id[1] = a.y; next_id[2] = a.z; next_id[3] = a.w;
            next_code[0] = b.x; next_code[1] = b.y; next_code[2] = b.z; next_code[3] = b.w;
        } else {
#pragma unroll
            for (int k = 0; k < kCodedPoints; ++k) {
                const bool there = group < n_groups && first + k < n_visible;
                next_id[k] = there ? __ldg(sorted_ids + first + k) : 0u;
                next_code[k] = there ? __ldg(sorted_codes + first + k) : kNone;
            }
        }
    };
    load(blockIdx.x);
    unsigned flip = 0;
    for (unsigned group = blockIdx.x; group < n_groups; group += gridDim.x, flip ^= 1u) {
        uint32_t id[kCodedPoints], code[kCodedPoints];
#pragma unroll
        for (int k = 0; k < kCodedPoints; ++k) { id[k] = next_id[k]; code[k] = next_code[k]; }
        load(group + gridDim.x);
        unsigned own = 0u;
#pragma unroll
        for (int k = 0; k < kCodedPoints; ++k) own += code[k] == kNone ? 0u : tiles_of_code(code[k], codes.escape);
        const unsigned inc = warp_inclusive_scan(own), warp_total = __shfl_sync(0xffffffffu, inc, 31);
        if (lane == 0) s_total[flip][warp] = warp_total;
        unsigned at = inc - own;
#pragma unroll
        for (int k = 0; k < kCodedPoints; ++k) {
            if (code[k] == kNone) continue;
            const Footprint f = footprint_of_quad(code[k] >= codes.escape ? __ldg(codes.quad + checked_point(id[k])) : code[k], gw);
            // in a second column or row of tiles the footprint starts one pixel before the tile: its code there is zero
            const uint32_t column = f.column << kTileKeyBits, row = f.row << (kTileKeyBits + 4);
            stage[at++] = make_uint2(f.tile | column | row, id[k]);
            if (f.two_columns) stage[at++] = make_uint2((f.tile + 1u) | row, id[k]);
            if (f.two_rows) {
                stage[at++] = make_uint2((f.tile + (unsigned)gw) | column, id[k]);
                if (f.two_columns) stage[at++] = make_uint2(f.tile + (unsigned)gw + 1u, id[k]);
            }
        }
        __syncthreads();
        // behind the sums of kInstThreads points each, those of the warps between them and this one
        const unsigned sum_first = warp / kSums * kSums;
        const unsigned base = __ldg(block_base + (group * kGroup + warp * 32u * kCodedPoints) / kInstThreads) +
                              __reduce_add_sync(0xffffffffu, lane >= sum_first && lane < warp ? s_total[flip][lane] : 0u);
        for (unsigned i = lane; i < warp_total; i += 32u) {
            const uint2 pair = stage[i];
            __stcs(inst_keys + base + i, pair.x);
            __stcs(inst_ids + base + i, pair.y);
            count_key(s_digits, digits.pt, pair.x);
        }
        __syncwarp();
    }
    finish_histogram(s_digits, digits, min(n_groups, gridDim.x), n_emitted);
}

// Other splats.  CELLS (gaussian, 8x8 tiles): the key also says which cells of the tile the ellipse can reach (see cell_code).  The keys are counted by the
// sort: a gaussian splat has many instances, whose atomics would go one after the other (2^22 of them, emission and histogram 61 + 13 -> 90 us).
template <bool CELLS>
__device__ __forceinline__ uint32_t instance_key(unsigned tx, unsigned ty, unsigned x0, unsigned x1, unsigned y0, unsigned y1, unsigned inset, int gw) {
    const uint32_t tile = ty * (unsigned)gw + tx;
    if (!CELLS) return tile;
    const int left = (int)(inset & 15u) - 4 * (int)(tx - x0), right = 4 * (int)(x1 - tx) - 1 - (int)((inset >> 4) & 15u);
    const int top = (int)((inset >> 8) & 15u) - 4 * (int)(ty - y0), bottom = 4 * (int)(y1 - ty) - 1 - (int)(inset >> 12);
    return tile | cell_code(left, right, top, bottom) << kTileKeyBits;
}
// Up to how many instances of a warp's points every lane writes those of its own; of more the lanes take equal shares and write side by side.  2^22 splats of 1.4
// tiles on average 62 us with own ones, 69 shared (68 staged in shared memory); 2 * 10^6 splats of about a pixel and more 59 and 45 (47).
constexpr unsigned kFewInstances = 64;
template <bool CELLS>
__global__ void __launch_bounds__(kInstThreads) emit_instances_kernel(const uint32_t* __restrict__ sorted_ids,
                                                                      const uint2* __restrict__ bounds,
                                                                      const uint4* __restrict__ foot, const unsigned long long* __restrict__ n_visible_dev,
                                                                      const unsigned* __restrict__ block_base, int gw,
                                                                      uint32_t* __restrict__ inst_keys,
                                                                      uint32_t* __restrict__ inst_ids) {
    await_previous_kernel();
    __shared__ unsigned s_total[kInstThreads / 32];
    const int64_t n_visible = (int64_t)*n_visible_dev;
    if ((int64_t)blockIdx.x * kInstThreads >= n_visible) return;
    const int64_t s = (int64_t)blockIdx.x * kInstThreads + threadIdx.x;
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    const bool there = s < n_visible;
    const uint32_t id = there ? checked_point(__ldcs(sorted_ids + s)) : 0u;
    // instances of the warps of this block before this one; one barrier
    auto before_warp = [&](unsigned total) -> unsigned {
        if (lane == 0) s_total[warp] = total;
        __syncthreads();
        return __ldg(block_base + blockIdx.x) + __reduce_add_sync(0xffffffffu, lane < warp ? s_total[lane] : 0u);
    };
    unsigned x0 = 0, x1 = 0, y0 = 0, y1 = 0, inset = 0;
    if (there) {
        uint2 b;
        if (CELLS) {
            const uint4 f = __ldg(foot + id);
            b = make_uint2(f.x, f.y);
            inset = f.z;
        } else {
            b = __ldg(bounds + id);
        }
        x0 = b.x & 0xffffu; x1 = b.x >> 16; y0 = b.y & 0xffffu; y1 = b.y >> 16;
    }
    const unsigned c = (x1 - x0) * (y1 - y0), inc = warp_inclusive_scan(c), before = inc - c, total = __shfl_sync(0xffffffffu, inc, 31);
    const unsigned base = before_warp(total);
    if (total <= kFewInstances) {
        unsigned at = base + before;
        for (unsigned ty = y0; ty < y1; ++ty)
            for (unsigned tx = x0; tx < x1; ++tx) {
                __stcs(inst_keys + at, instance_key<CELLS>(tx, ty, x0, x1, y0, y1, inset, gw));
                __stcs(inst_ids + at, id);
                ++at;
            }
        return;
    }
    // the lanes share them: lane l takes every 32nd and finds the point it belongs to among the sums
    const unsigned columns = x0 | (x1 << 16), rows = y0 | (y1 << 16);
    for (unsigned first = 0; first < total; first += 32u) {
        const unsigned i = first + lane;
        unsigned point = 0u;   // the last lane whose instances begin at i at the latest (lanes without a point lie behind all others)
#pragma unroll
        for (unsigned step = 16u; step > 0u; step >>= 1) {
            const unsigned begins = __shfl_sync(0xffffffffu, before, point + step);
            point += begins <= i ? step : 0u;
        }
        const unsigned at = i - __shfl_sync(0xffffffffu, before, point), cols = __shfl_sync(0xffffffffu, columns, point), rws = __shfl_sync(0xffffffffu, rows, point);
        const uint32_t who = __shfl_sync(0xffffffffu, id, point);
        const unsigned in = CELLS ? __shfl_sync(0xffffffffu, inset, point) : 0u;
        if (i >= total) continue;
        const unsigned px0 = cols & 0xffffu, px1 = cols >> 16, py0 = rws & 0xffffu, py1 = rws >> 16, width = px1 - px0;
        const unsigned dy = at / width, dx = at - dy * width;
        __stcs(inst_keys + base + i, instance_key<CELLS>(px0 + dx, py0 + dy, px0, px1, py0, py1, in, gw));
        __stcs(inst_ids + base + i, who);
    }
}

// Run boundaries of the sorted tile keys -> [first, last+1) per tile (src/bilinear/kernels.cu:222-239).  A thread compares the first of its 16 or
// 64 keys and of the next thread's, and reads those between only if a run ends there: of long lists an eighth of the sectors.  (64 keys take
// longer to look through, and only pay where there is more to skip than a wave of warps covers.)  10^6 / 10.6 / 17 / 43 million instances, all keys read / 16 / 64 keys:
// 4 / 12 / 21 / 36 us, 3 / 8 / 16 / 32, 8 / 8 / 16 / 24.
constexpr unsigned kRangeKeysFew = 16, kRangeKeysMany = 64, kRangeMany = 1 << 23;
__host__ __device__ constexpr unsigned range_keys(int64_t n_instances) { return n_instances < kRangeMany ? kRangeKeysFew : kRangeKeysMany; }
__global__ void __launch_bounds__(256) tile_ranges_kernel(const uint32_t* __restrict__ keys, const unsigned long long* __restrict__ n_instances_dev,
                                                          uint2* __restrict__ ranges) {
    await_previous_kernel();
    const unsigned n = (unsigned)*n_instances_dev;   // < 2^30
    const unsigned per = range_keys(n), n_steps = (n + per * 32u - 1u) / (per * 32u), lane = lane_id();   // of a warp
    // the grid fits the chip: sized for the bound on the instance count it was three quarters empty blocks
    for (unsigned step = blockIdx.x * 8u + (threadIdx.x >> 5); step < n_steps; step += gridDim.x * 8u) {
        const unsigned first = (step * 32u + lane) * per, end = min(n, first + per);
        const bool there = first < n;
        const uint32_t head = there ? __ldg(keys + first) & kTileKeyMask : 0u;
        uint32_t next = __shfl_down_sync(0xffffffffu, head, 1);   // of the first key behind this thread's
        if (lane == 31u && end < n) next = __ldg(keys + end) & kTileKeyMask;
        if (!there) continue;
        if (first == 0u) ranges[head].x = 0u;
        if (end < n && next == head) continue;
        uint32_t prev = head;
        auto look = [&](unsigned i, uint32_t key) {
            if (key != prev) { ranges[prev].y = i; ranges[key].x = i; }
            prev = key;
        };
        if (end - first == per) {
#pragma unroll 2
            for (unsigned i = first; i < end; i += 4u) {
                const uint4 k = __ldg(reinterpret_cast<const uint4*>(keys + i));   // the key buffers are 16-byte aligned
                look(i, k.x & kTileKeyMask); look(i + 1u, k.y & kTileKeyMask); look(i + 2u, k.z & kTileKeyMask); look(i + 3u, k.w & kTileKeyMask);
            }
        } else {
            for (unsigned i = first; i < end; ++i) look(i, __ldg(keys + i) & kTileKeyMask);
        }
        if (end < n) look(end, next);   // (the thread behind has no run to begin with its first key)
        else ranges[prev].y = n;
    }
}

// ------------------------------------------------------------------------------------------------
// Bilinear blend.
//
// (1) Per-pixel bit masks.  A point reaches only the 2x2 pixels whose centres lie within distance
// < 1 of it, so a block stages T*T instances at a time, every instance thread sets its bit in the
// masks of the (up to four) pixels it reaches, and every pixel thread then walks only its own set
// bits, in staged (= depth) order.  Per-fragment results that belong to the point (blending weight,
// gradients) go to a private shared-memory slot per (instance, footprint corner) and are reduced by
// the instance thread in a fixed order (the only shared-memory atomics are the ORs that build the masks),
// one global (vector) atomic per instance.  Two block barriers per batch.
//
// (2) Segments.  Front-to-back compositing is associative: (C, T) o (C', T') = (C + T C', T T').  A
// tile's instance list is cut into segments of at least 16 batches (at most 64 segments per tile) and
// every (tile, segment) pair is one block, so a tile that carries 100x the average load no longer
// sets the kernel's critical path.  For tiles with more than one segment a first pass computes each
// segment's per-pixel transmittance product, a per-tile prefix turns these into the transmittance at
// the start of every segment, and the main pass starts from that value (keeping the reference's
// early-termination rule); partial colours are added up per tile in segment order.  The backward
// pass starts every segment from the stored transmittance and colour prefix.
//
// Arithmetic per fragment: src/bilinear/kernels.cu:283-303 (forward), :361-415 (backward),
// :462-475 (inference).
// ------------------------------------------------------------------------------------------------
enum { BLEND_TRAIN = 0, BLEND_INFER = 1 };

struct __align__(16) Segment {
    uint32_t tile;
    uint32_t begin, end;   // instance range of this segment
    uint32_t info;         // index of the segment within its tile | number of segments of the tile << 16
};
constexpr int kMaxSegmentsPerTile = 64;
constexpr int kMinBatchesPerSegment = 16;

__device__ __forceinline__ unsigned segment_length(unsigned len, unsigned batch) {
    const unsigned s_min = batch * (unsigned)kMinBatchesPerSegment;
    const unsigned want = ceil_div(len, (unsigned)kMaxSegmentsPerTile);
    return max(s_min, ceil_div(want, batch) * batch);
}

// One block: number of segments per tile and their exclusive scan (tile_first), total in *n_segments.
__global__ void __launch_bounds__(kScanThreads) count_segments_kernel(const uint2* __restrict__ ranges, int n_tiles, int batch,
                                                                      uint32_t* __restrict__ tile_first,
                                                                      uint32_t* __restrict__ n_segments) {
    await_previous_kernel();
    // four consecutive tiles per thread: short serial chains, two 16-byte loads
    constexpr int kItems = 4;
    __shared__ unsigned s_scan[kScanThreads / 32 + 1];
    unsigned running = 0;
    for (int base = 0; base < n_tiles; base += kScanThreads * kItems) {
        const int t0 = base + threadIdx.x * kItems;
        unsigned v[kItems];
        unsigned sum = 0;
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            v[k] = 0u;
            if (t0 + k < n_tiles) {
                const uint2 r = __ldg(ranges + t0 + k);
                const unsigned len = r.y - r.x;
                v[k] = max(1u, ceil_div(len, segment_length(len, (unsigned)batch)));
            }
            sum += v[k];
        }
        unsigned total;
        unsigned ex = running + block_exclusive_scan(sum, s_scan, &total);
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            if (t0 + k < n_tiles) tile_first[t0 + k] = ex;
            ex += v[k];
        }
        running += total;
    }
    if (threadIdx.x == 0) *n_segments = running;
}

// One thread per tile writes the tile's segment records.
__global__ void __launch_bounds__(256) emit_segments_kernel(const uint2* __restrict__ ranges, int n_tiles, int batch,
                                                            const uint32_t* __restrict__ tile_first, Segment* __restrict__ segs) {
    await_previous_kernel();
    const int t = blockIdx.x * 256 + threadIdx.x;
    if (t >= n_tiles) return;
    const uint2 r = ranges[t];
    const unsigned len = r.y - r.x;
    const unsigned seg_len = segment_length(len, (unsigned)batch);
    const unsigned n = max(1u, ceil_div(len, seg_len));
    const unsigned first = tile_first[t];
    for (unsigned s = 0; s < n; ++s) {
        Segment g;
        g.tile = (uint32_t)t;
        g.begin = r.x + s * seg_len;
        g.end = min(r.y, g.begin + seg_len);
        g.info = s | (n << 16);
        segs[first + s] = g;
    }
}

// Stages instance `j` of the batch starting at `base`: record into shared memory, bit into the masks of
// the pixels it reaches.  Returns the point id.
template <int T, int B, bool NEED_F>
__device__ __forceinline__ uint32_t stage_instance(int j, int cnt, unsigned base, const uint32_t* __restrict__ inst_ids,
                                                   const PointRec* __restrict__ rec, int tile_x, int tile_y, float4* s_a,
                                                   float4* s_f, unsigned (*s_mask)[T * T]) {
    uint32_t id = 0;
    if (j < cnt) {
        id = checked_point(__ldg(inst_ids + base + j));
        const float4* r = reinterpret_cast<const float4*>(rec + id);
        const float4 a = __ldg(r);
        s_a[j] = a;
        if (NEED_F) s_f[j] = __ldg(r + 1);
        // first pixel column / row whose centre is within reach; the second is the next one
        const int qx = __float2int_rd(a.x - 0.5f) - tile_x * T;
        const int qy = __float2int_rd(a.y - 0.5f) - tile_y * T;
        const unsigned bit = 1u << (j & 31);
        unsigned* mrow = s_mask[j >> 5];
#pragma unroll
        for (int dy = 0; dy < 2; ++dy)
#pragma unroll
            for (int dx = 0; dx < 2; ++dx) {
                const int cx = qx + dx, cy = qy + dy;
                if (cx >= 0 && cx < T && cy >= 0 && cy < T) atomicOr(mrow + cy * T + cx, bit);
            }
    }
    return id;
}

// The same staging split in two, so that a batch's loads can be in flight while the batch before it is
// walked: `fetch` only issues the loads (instance id, then the record it names: two dependent trips to
// memory), `commit` writes the values to shared memory and sets the mask bits.
template <bool NEED_F>
struct Fetched {
    uint32_t id;
    float4 a, f;
};

template <bool NEED_F>
__device__ __forceinline__ Fetched<NEED_F> fetch_instance(int j, int cnt, unsigned base, const uint32_t* __restrict__ inst_ids,
                                                          const PointRec* __restrict__ rec) {
    Fetched<NEED_F> r;
    r.id = 0;
    r.a = make_float4(0.f, 0.f, 0.f, 0.f);
    r.f = make_float4(0.f, 0.f, 0.f, 0.f);
    if (j < cnt) {
        r.id = checked_point(__ldg(inst_ids + base + j));
        const float4* p = reinterpret_cast<const float4*>(rec + r.id);
        r.a = __ldg(p);
        if (NEED_F) r.f = __ldg(p + 1);
    }
    return r;
}

template <int T, bool NEED_F>
__device__ __forceinline__ void commit_instance(int j, int cnt, const Fetched<NEED_F>& r, int tile_x, int tile_y, float4* s_a, float4* s_f,
                                                unsigned (*s_mask)[T * T]) {
    if (j < cnt) {
        s_a[j] = r.a;
        if (NEED_F) s_f[j] = r.f;
        const int qx = __float2int_rd(r.a.x - 0.5f) - tile_x * T;
        const int qy = __float2int_rd(r.a.y - 0.5f) - tile_y * T;
        const unsigned bit = 1u << (j & 31);
        unsigned* mrow = s_mask[j >> 5];
#pragma unroll
        for (int dy = 0; dy < 2; ++dy)
#pragma unroll
            for (int dx = 0; dx < 2; ++dx) {
                const int cx = qx + dx, cy = qy + dy;
                if (cx >= 0 && cx < T && cy >= 0 && cy < T) atomicOr(mrow + cy * T + cx, bit);
            }
    }
}

// Pass 1 (tiles with several segments only): per-pixel product of (1 - alpha) over one segment.
// A block is one (tile, segment): T*T threads = pixels, batches of B = T*T*IPT instances.
template <int T, int IPT>
__global__ void __launch_bounds__(T * T) blend_bilinear_transmittance_kernel(
    const Segment* __restrict__ segs, const uint32_t* __restrict__ n_segments, const uint32_t* __restrict__ inst_ids,
    const PointRec* __restrict__ rec, float* __restrict__ seg_T, int width, int height, int gw) {
    await_previous_kernel();
    constexpr int P = T * T;
    constexpr int B = P * IPT;
    constexpr int WORDS = B / 32;
    if (blockIdx.x >= *n_segments) return;
    const Segment sg = segs[blockIdx.x];
    const unsigned seg_idx = sg.info & 0xffffu, n_seg = sg.info >> 16;
    if (n_seg == 1u || seg_idx == n_seg - 1u) return;   // the last segment's product is never needed

    __shared__ float4 s_a[B];
    __shared__ unsigned s_mask[WORDS][P];
    const int t = threadIdx.x;
    const int tx = (int)(sg.tile % (unsigned)gw), ty = (int)(sg.tile / (unsigned)gw);
    const int px = tx * T + t % T, py = ty * T + t / T;
    const bool inside = px < width && py < height;
    const float pcx = (float)px + 0.5f, pcy = (float)py + 0.5f;
#pragma unroll
    for (int w = 0; w < WORDS; ++w) s_mask[w][t] = 0u;
    __syncthreads();
    float Tr = 1.0f;
    bool done = !inside;
    // (fetching the next batch before the current one is walked costs more registers than the overlap gains)
    Fetched<false> next[IPT];
    for (unsigned base = sg.begin; base < sg.end; base += B) {
        const int cnt = (int)min((unsigned)B, sg.end - base);
#pragma unroll
        for (int k = 0; k < IPT; ++k) next[k] = fetch_instance<false>(t + k * P, cnt, base, inst_ids, rec);
#pragma unroll
        for (int k = 0; k < IPT; ++k) commit_instance<T, false>(t + k * P, cnt, next[k], tx, ty, s_a, nullptr, s_mask);
        __syncthreads();
#pragma unroll 1
        for (int w = 0; w < WORDS; ++w) {
            unsigned mbits = s_mask[w][t];
            if (mbits) s_mask[w][t] = 0u;
            while (mbits && !done) {
                const int j = w * 32 + __ffs(mbits) - 1;
                mbits &= mbits - 1u;
                const float4 a = s_a[j];
                const float dx = fabsf(a.x - pcx), dy = fabsf(a.y - pcy);
                if (dx >= 1.0f || dy >= 1.0f) continue;
                const float wgt = __saturatef(1.0f - dx) * __saturatef(1.0f - dy);
                Tr *= 1.0f - rounded_alpha(a.z, wgt);
                if (Tr < kTransmittanceEps) done = true;
            }
        }
        if (__syncthreads_count(done) == P) break;
    }
    seg_T[(size_t)blockIdx.x * P + t] = Tr;
}

// Per tile with several segments: products of the segments before -> transmittance at segment start.
template <int T>
__global__ void __launch_bounds__(T * T) blend_prefix_kernel(const Segment* __restrict__ segs, const uint32_t* __restrict__ tile_first,
                                                             float* __restrict__ seg_T) {
    await_previous_kernel();
    constexpr int P = T * T;
    const unsigned first = tile_first[blockIdx.x];
    const unsigned n_seg = segs[first].info >> 16;
    if (n_seg == 1u) return;
    const int t = threadIdx.x;
    float run = 1.0f;
    for (unsigned s0 = 0; s0 < n_seg; s0 += 8) {
        float loc[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const unsigned s = s0 + k;
            loc[k] = s + 1u < n_seg ? seg_T[(size_t)(first + s) * P + t] : 1.0f;
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const unsigned s = s0 + k;
            if (s < n_seg) seg_T[(size_t)(first + s) * P + t] = run;
            run *= loc[k];
        }
    }
}

template <int T, int IPT, int KIND>
__global__ void __launch_bounds__(T * T) blend_bilinear_forward_kernel(
    const Segment* __restrict__ segs, const uint32_t* __restrict__ n_segments, const uint32_t* __restrict__ inst_ids,
    const PointRec* __restrict__ rec, float* __restrict__ seg_T, float4* __restrict__ seg_C, float* __restrict__ seg_Z,
    float* __restrict__ image, float* __restrict__ depth_image, float* __restrict__ alpha_image,
    float* __restrict__ blending_weights, int width, int height, int gw) {
    await_previous_kernel();
    constexpr int P = T * T;
    constexpr int B = P * IPT;
    constexpr int WORDS = B / 32;
    if (blockIdx.x >= *n_segments) return;
    const Segment sg = segs[blockIdx.x];
    const unsigned seg_idx = sg.info & 0xffffu, n_seg = sg.info >> 16;

    __shared__ float4 s_a[B];
    __shared__ float4 s_f[B];
    __shared__ unsigned s_mask[WORDS][P];
    __shared__ float s_slot[KIND == BLEND_TRAIN ? 4 : 1][KIND == BLEND_TRAIN ? B : 1];

    const int t = threadIdx.x;
    const int tx = (int)(sg.tile % (unsigned)gw), ty = (int)(sg.tile / (unsigned)gw);
    const int px = tx * T + t % T, py = ty * T + t / T;
    const bool inside = px < width && py < height;
    const float pcx = (float)px + 0.5f, pcy = (float)py + 0.5f;
    const size_t state_idx = (size_t)blockIdx.x * P + t;

#pragma unroll
    for (int w = 0; w < WORDS; ++w) s_mask[w][t] = 0u;
    if (KIND == BLEND_TRAIN) {
#pragma unroll
        for (int k = 0; k < IPT; ++k)
#pragma unroll
            for (int q = 0; q < 4; ++q) s_slot[q][t + k * P] = 0.0f;
    }
    float C0 = 0.0f, C1 = 0.0f, C2 = 0.0f, C3 = 0.0f, Z = 0.0f;
    float Tr = 1.0f;
    if (seg_idx > 0u && inside) Tr = seg_T[state_idx];
    bool done = !inside || Tr < kTransmittanceEps;
    __syncthreads();

    uint32_t id[IPT];
    int cnt = 0;
    auto flush_weights = [&]() {
        // blending weights of the instances this thread staged last: the (up to) four fragments of each
        // in fixed order; the slots are cleared for the next batch
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            const int j = t + k * P;
            if (j < cnt) {
                const float sum = ((s_slot[0][j] + s_slot[1][j]) + s_slot[2][j]) + s_slot[3][j];
                if (sum > 0.0f) atomicAdd(blending_weights + id[k], sum);
                s_slot[0][j] = 0.0f; s_slot[1][j] = 0.0f; s_slot[2][j] = 0.0f; s_slot[3][j] = 0.0f;
            }
        }
    };
    // (fetching the next batch before the current one is walked costs more registers than the overlap gains)
    Fetched<true> next[IPT];
    for (unsigned base = sg.begin; base < sg.end; base += B) {
        if (KIND == BLEND_TRAIN) flush_weights();
        cnt = (int)min((unsigned)B, sg.end - base);
#pragma unroll
        for (int k = 0; k < IPT; ++k) next[k] = fetch_instance<true>(t + k * P, cnt, base, inst_ids, rec);
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            id[k] = next[k].id;
            commit_instance<T, true>(t + k * P, cnt, next[k], tx, ty, s_a, s_f, s_mask);
        }
        __syncthreads();
#pragma unroll 1
        for (int w = 0; w < WORDS; ++w) {
            unsigned mbits = s_mask[w][t];
            if (mbits) s_mask[w][t] = 0u;
            while (mbits && !done) {
                const int j = w * 32 + __ffs(mbits) - 1;
                mbits &= mbits - 1u;
                const float4 a = s_a[j];
                const float dx = fabsf(a.x - pcx), dy = fabsf(a.y - pcy);
                if (dx >= 1.0f || dy >= 1.0f) continue;
                const float wgt = __saturatef(1.0f - dx) * __saturatef(1.0f - dy);
                const float al = rounded_alpha(a.z, wgt);
                const float bw = Tr * al;
                if (KIND == BLEND_TRAIN) {
                    // corner of the point's 2x2 footprint this pixel is: exactly one writer per slot
                    if (bw > 0.0f) s_slot[(pcx > a.x ? 1 : 0) + (pcy > a.y ? 2 : 0)][j] = bw * wgt;
                }
                const float4 f = s_f[j];
                C0 += bw * f.x; C1 += bw * f.y; C2 += bw * f.z; C3 += bw * f.w;
                if (KIND == BLEND_INFER) Z += bw * a.w;
                Tr *= 1.0f - al;
                if (Tr < kTransmittanceEps) done = true;
            }
        }
        if (__syncthreads_count(done) == P) break;
    }
    if (KIND == BLEND_TRAIN) flush_weights();

    if (n_seg == 1u) {
        if (inside) {
            const int64_t n_px = (int64_t)width * height;
            const int64_t pi = (int64_t)py * width + px;
            image[pi] = C0;
            image[n_px + pi] = C1;
            image[2 * n_px + pi] = C2;
            image[3 * n_px + pi] = C3;
            if (KIND == BLEND_INFER) {
                const float A = 1.0f - Tr;
                depth_image[pi] = A > 0.0f ? Z / A : 0.0f;
                alpha_image[pi] = Tr < kTransmittanceEps ? 1.0f : A;
            } else {
                alpha_image[pi] = Tr < kTransmittanceEps ? 1.0f : 1.0f - Tr;
            }
        }
    } else {
        // partial colour of this segment; the per-tile combine adds the segments up in order
        seg_C[state_idx] = make_float4(C0, C1, C2, C3);
        if (KIND == BLEND_INFER) {
            seg_Z[state_idx] = Z;
            seg_T[state_idx] = Tr;
        } else if (seg_idx == n_seg - 1u && inside) {
            alpha_image[(int64_t)py * width + px] = Tr < kTransmittanceEps ? 1.0f : 1.0f - Tr;
        }
    }
}

// Per tile with several segments: image = sum of the segment colours in order.  For training the
// running sum before each segment is written back (the backward pass starts from it).
template <int T, int KIND>
__global__ void __launch_bounds__(T * T) blend_combine_kernel(const Segment* __restrict__ segs, const uint32_t* __restrict__ tile_first,
                                                              float4* __restrict__ seg_C, const float* __restrict__ seg_Z,
                                                              const float* __restrict__ seg_T, float* __restrict__ image,
                                                              float* __restrict__ depth_image, float* __restrict__ alpha_image,
                                                              int width, int height, int gw) {
    await_previous_kernel();
    constexpr int P = T * T;
    const unsigned first = tile_first[blockIdx.x];
    const unsigned n_seg = segs[first].info >> 16;
    if (n_seg == 1u) return;
    const int t = threadIdx.x;
    const int tx = (int)(blockIdx.x % (unsigned)gw), ty = (int)(blockIdx.x / (unsigned)gw);
    const int px = tx * T + t % T, py = ty * T + t / T;
    float4 run = make_float4(0.f, 0.f, 0.f, 0.f);
    float z = 0.0f;
    // transmittance where the pixel stopped: the end value of the first segment that fell below the
    // threshold (later segments start below it and only carry the product of everything skipped)
    float t_final = 1.0f;
    bool stopped = false;
    for (unsigned s0 = 0; s0 < n_seg; s0 += 4) {
        float4 c[4];
        float zz[4], tt[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const unsigned s = s0 + k;
            c[k] = s < n_seg ? seg_C[(size_t)(first + s) * P + t] : make_float4(0.f, 0.f, 0.f, 0.f);
            zz[k] = (KIND == BLEND_INFER && s < n_seg) ? seg_Z[(size_t)(first + s) * P + t] : 0.0f;
            tt[k] = (KIND == BLEND_INFER && s < n_seg) ? seg_T[(size_t)(first + s) * P + t] : 1.0f;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const unsigned s = s0 + k;
            if (KIND == BLEND_TRAIN && s < n_seg) seg_C[(size_t)(first + s) * P + t] = run;
            run.x += c[k].x; run.y += c[k].y; run.z += c[k].z; run.w += c[k].w;
            z += zz[k];
            if (KIND == BLEND_INFER && s < n_seg && !stopped) {
                t_final = tt[k];
                stopped = t_final < kTransmittanceEps;
            }
        }
    }
    if (px < width && py < height) {
        const int64_t n_px = (int64_t)width * height;
        const int64_t pi = (int64_t)py * width + px;
        image[pi] = run.x;
        image[n_px + pi] = run.y;
        image[2 * n_px + pi] = run.z;
        image[3 * n_px + pi] = run.w;
        if (KIND == BLEND_INFER) {
            const float Tr = t_final;
            const float A = 1.0f - Tr;
            depth_image[pi] = A > 0.0f ? z / A : 0.0f;
            alpha_image[pi] = Tr < kTransmittanceEps ? 1.0f : A;
        }
    }
}

template <int T, int IPT>
__global__ void __launch_bounds__(T * T) blend_bilinear_backward_kernel(
    const Segment* __restrict__ segs, const uint32_t* __restrict__ n_segments, const uint32_t* __restrict__ inst_ids,
    const PointRec* __restrict__ rec, const float* __restrict__ seg_T, const float4* __restrict__ seg_C,
    const float* __restrict__ grad_image, const float* __restrict__ grad_alpha, const float* __restrict__ image,
    const float* __restrict__ alpha_image, float4* __restrict__ grad_feat_view, float* __restrict__ grad_opacity,
    int width, int height, int gw) {
    await_previous_kernel();
    constexpr int P = T * T;
    constexpr int B = P * IPT;
    constexpr int WORDS = B / 32;
    if (blockIdx.x >= *n_segments) return;
    const Segment sg = segs[blockIdx.x];
    const unsigned seg_idx = sg.info & 0xffffu;
    if (sg.begin == sg.end) return;

    extern __shared__ __align__(16) unsigned char blend_smem[];
    float4* s_a = reinterpret_cast<float4*>(blend_smem);            // [B]
    float4* s_f = s_a + B;                                          // [B]
    float4* s_gf = s_f + B;                                         // [4][B] per footprint corner: feature gradient
    float* s_go = reinterpret_cast<float*>(s_gf + 4 * B);           // [4][B] per footprint corner: opacity gradient
    unsigned (*s_mask)[P] = reinterpret_cast<unsigned (*)[P]>(s_go + 4 * B);   // [WORDS][P]

    const int t = threadIdx.x;
    const int tx = (int)(sg.tile % (unsigned)gw), ty = (int)(sg.tile / (unsigned)gw);
    const int px = tx * T + t % T, py = ty * T + t / T;
    const bool inside = px < width && py < height;
    const float pcx = (float)px + 0.5f, pcy = (float)py + 0.5f;
    const size_t state_idx = (size_t)blockIdx.x * P + t;

#pragma unroll
    for (int w = 0; w < WORDS; ++w) s_mask[w][t] = 0u;
#pragma unroll
    for (int k = 0; k < IPT; ++k)
#pragma unroll
        for (int q = 0; q < 4; ++q) { s_gf[q * B + t + k * P] = make_float4(0.f, 0.f, 0.f, 0.f); s_go[q * B + t + k * P] = 0.0f; }

    float4 g = make_float4(0.f, 0.f, 0.f, 0.f), Cfin = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 Crun = make_float4(0.f, 0.f, 0.f, 0.f);
    float K = 0.0f, Tr = 1.0f;
    if (inside) {
        const int64_t n_px = (int64_t)width * height;
        const int64_t pi = (int64_t)py * width + px;
        g = make_float4(__ldg(grad_image + pi), __ldg(grad_image + n_px + pi), __ldg(grad_image + 2 * n_px + pi),
                        __ldg(grad_image + 3 * n_px + pi));
        Cfin = make_float4(__ldg(image + pi), __ldg(image + n_px + pi), __ldg(image + 2 * n_px + pi),
                           __ldg(image + 3 * n_px + pi));
        K = __ldg(grad_alpha + pi) * (1.0f - __ldg(alpha_image + pi));
        if (seg_idx > 0u) { Tr = seg_T[state_idx]; Crun = seg_C[state_idx]; }
    }
    bool done = !inside || Tr < kTransmittanceEps;
    __syncthreads();

    uint32_t id[IPT];
    int cnt = 0;
    auto flush_gradients = [&]() {
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            const int j = t + k * P;
            if (j < cnt) {
                float4 sf = s_gf[j];
                float so = s_go[j];
#pragma unroll
                for (int q = 1; q < 4; ++q) {
                    const float4 v = s_gf[q * B + j];
                    sf.x += v.x; sf.y += v.y; sf.z += v.z; sf.w += v.w;
                    so += s_go[q * B + j];
                }
                if (sf.x != 0.0f || sf.y != 0.0f || sf.z != 0.0f || sf.w != 0.0f) atomicAdd(grad_feat_view + id[k], sf);
                if (so != 0.0f) atomicAdd(grad_opacity + id[k], so);
#pragma unroll
                for (int q = 0; q < 4; ++q) { s_gf[q * B + j] = make_float4(0.f, 0.f, 0.f, 0.f); s_go[q * B + j] = 0.0f; }
            }
        }
    };
    // (fetching the next batch before the current one is walked costs more registers than the overlap gains)
    Fetched<true> next[IPT];
    for (unsigned base = sg.begin; base < sg.end; base += B) {
        flush_gradients();
        cnt = (int)min((unsigned)B, sg.end - base);
#pragma unroll
        for (int k = 0; k < IPT; ++k) next[k] = fetch_instance<true>(t + k * P, cnt, base, inst_ids, rec);
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            id[k] = next[k].id;
            commit_instance<T, true>(t + k * P, cnt, next[k], tx, ty, s_a, s_f, s_mask);
        }
        __syncthreads();
#pragma unroll 1
        for (int w = 0; w < WORDS; ++w) {
            unsigned mbits = s_mask[w][t];
            if (mbits) s_mask[w][t] = 0u;
            while (mbits && !done) {
                const int j = w * 32 + __ffs(mbits) - 1;
                mbits &= mbits - 1u;
                const float4 a = s_a[j];
                const float dx = fabsf(a.x - pcx), dy = fabsf(a.y - pcy);
                if (dx >= 1.0f || dy >= 1.0f) continue;
                const float wgt = __saturatef(1.0f - dx) * __saturatef(1.0f - dy);
                const float al = rounded_alpha(a.z, wgt);
                const float bw = Tr * al;
                const int q = (pcx > a.x ? 1 : 0) + (pcy > a.y ? 2 : 0);
                if (bw > 0.0f) s_gf[q * B + j] = make_float4(bw * g.x, bw * g.y, bw * g.z, bw * g.w);
                const float4 f = s_f[j];
                Crun.x += bw * f.x; Crun.y += bw * f.y; Crun.z += bw * f.z; Crun.w += bw * f.w;
                const float oma = 1.0f - al;
                const float rcp = 1.0f / fmaxf(oma, kOneMinusAlphaEps);
                const float from_features = (Tr * f.x + (Crun.x - Cfin.x) * rcp) * g.x +
                                            (Tr * f.y + (Crun.y - Cfin.y) * rcp) * g.y +
                                            (Tr * f.z + (Crun.z - Cfin.z) * rcp) * g.z +
                                            (Tr * f.w + (Crun.w - Cfin.w) * rcp) * g.w;
                const float dalpha = from_features + K * rcp;
                const float dop = dalpha * wgt;
                if (dop != 0.0f) s_go[q * B + j] = dop;
                Tr *= oma;
                if (Tr < kTransmittanceEps) done = true;
            }
        }
        if (__syncthreads_count(done) == P) break;
    }
    flush_gradients();
}

template <int T, int IPT>
constexpr size_t backward_smem_bytes() {
    return (size_t)T * T * IPT * (16 + 16 + 4 * 16 + 4 * 4) + (size_t)(T * T * IPT / 32) * T * T * 4;
}

// ------------------------------------------------------------------------------------------------
// Bilinear blend on 8x8 tiles, one warp per work item (the default path).
//
// (1) Dead instances.  A pixel stops taking fragments once its transmittance has fallen below the
// threshold, and in a dense scene most instances of a tile's list lie behind pixels that have already
// stopped.  Such an instance has no effect whatsoever, so it is discarded from its sort key alone --
// the key says which pixels of the tile it reaches (see kTileKeyBits), a mask of stopped pixels lives
// in registers -- and its 32-byte record is never fetched.  A warp streams the keys of its item (128
// per step, loaded one step ahead), pushes the point ids of the instances that may still contribute
// into a ring in shared memory and blends them in batches of 32, the records of the next batch being
// in flight while the current one is blended.  The mask used by the filter lags the blend by a batch;
// that only lets a few extra instances through, whose fragments are then dropped.
//
// (2) A batch is 32 staged instances.  Lane j finds the pixels of the half that the 2x2 footprint of instance j covers and that
// have not stopped; a 32x32 bit transposition over the warp turns these masks into one word per pixel, and every lane walks the
// set bits of its own pixel front to back: it reads the record, forms weight and alpha, accumulates and updates the transmittance.
// What a fragment adds to its point (blending weight, gradient) goes to a slot per instance and parity of the pixel's column
// and row -- the four pixels of a footprint have four different parities, so the slot is a constant of the lane -- and lane j adds
// up the slots of instance j in a fixed order.  Against forming weight and alpha per instance and sorting the fragments by pixel in
// shared memory (masks by atomics, a scan, a slot per fragment): forward passes of 16-channel rows 614 -> 496 us (2^23
// samples at 1237x822), first pass of a 2^25-point cloud at 1920x1080 411 -> 343, all passes of the 4-channel
// training step 342 -> 332.  In the backward passes lane j also forms weight, alpha and <g, f> of its instance in the (up to) four pixels beforehand, so that
// a step of the walk is left with the transmittance and a running sum (see FragmentSlots): against sorting the fragments by pixel (four
// channels) and forming everything in the walk (rows), 10^6 samples at 801x533 50 -> 44 us, 2^24 points at 3840x2160 466 -> 453, 2^23 samples of 16 channels
// at 1237x822 373 -> 332; of four channels 236 -> 233, which its longest list takes whatever a step costs less.
//
// (3) Segments.  Front-to-back compositing is associative: (C, T) o (C', T') = (C + T C', T T').  A
// tile's list is cut into a first segment and later ones (see segment_lengths), and every (tile half, segment) is one
// item, so a tile with 100x the average load does not set the critical path.  Pass FIRST blends
// segment 0 of every tile exactly; the pixels that dense clusters hit stop there.  Pass PRODUCT
// computes, for the later segments, the per-pixel product of (1 - alpha) over the segment, starting
// from (and filtering by) the state segment 0 left, so the work it repeats is small, and turns the products into the
// transmittance at the start of every segment; pass REST blends the later segments from there; a per-tile combine adds the segment colours in order (and leaves the
// colour prefix for the backward pass, whose items are then independent).
//
// An item covers the upper or lower 8x4 half of a tile, one pixel per lane; both halves stream the same
// list and each keeps what reaches its own pixels.
//
// The forward passes write the compacted lists they blended (point ids in depth order, per item) for
// the backward pass, which therefore neither filters nor reads keys.
//
// Arithmetic per fragment: src/bilinear/kernels.cu:283-303 (forward), :361-415 (backward),
// :462-475 (inference).
// ------------------------------------------------------------------------------------------------
constexpr int kWarpBlendWarps = 8;        // warps per block; every warp works on items of its own
constexpr int kQueueCap = 256;            // ring of candidate point ids per warp: >= 31 left over + 128 of one filter step
// Segment lengths.  Measured on B200 (2^23 clustered samples, 1237x822; forward / backward stage in microseconds), first + later
// segment: 1024 + 4096: 422 / 276, 1024 + 2048: 439 / 268, 512 + 4096: 437 / 297, 512 + 2048: 458 / 274, 1024 + 1024: 488 / 291,
// 512 + 1024: 518 / 283, 256 + 2048: 469 / 283 (before the forward walk over pixel masks, as the figures below): with this many instances the
// warps are busy (2800 of the 3552 that fit) for a third of a pass and more, and shorter segments add more work (more lists to filter, more states to carry) than they
// save.  With fewer instances the passes are as long as their longest items, at 1.3 - 2.4 us per batch of 32, while most
// warps have none: the segments then get shorter, so that the later ones of all tiles number about kSegmentTarget (two items
// each, one and a half times the resident warps, twice to three times the pairs of warps where two take an item).  10^6 samples, 801x533: forward / backward 283 / 153 us with 1024 + 4096,
// 120 / 56 with the lengths below (149 / 70 with half the target); 2 * 10^5 samples, 600x400: 190 / 86 -> 85 / 35; first segments
// of a quarter or of all of a later one measured the same or worse.
constexpr unsigned kSegmentMin = 256;
constexpr unsigned kFirstSegmentMax = 1024;
constexpr unsigned kLaterSegmentMax = 4096;
constexpr unsigned kSegmentTarget = 2560;
constexpr int kManyTiles = 1 << 15;   // from here on the first segments alone keep the chip busy: half as many later ones are aimed at
struct SegmentLengths {
    unsigned first, later;   // instances in a tile's first segment, and in every later one
};
// Whether the training passes that have such a form (first and later segments, and backward of four channels) take an item by two warps, see blend_bilinear_pair_forward_kernel.  It makes the
// longest lists faster, by a third, and leaves room for half to two thirds as many items: a gain where the passes are as long as their longest items, nothing where all lists are long, a loss where
// all are short.  How the points are spread over the tiles is not known here, how many there are for each is.  Whole step, one warp / two, with samples of an octree (part of the image, lists of any
// length) and points spread evenly over the image:
//   points per tile            16          32          64         128         256         512
//   560x420    octree      140 / 133   168 / 158   196 / 185   246 / 239   312 / 306   455 / 434
//              even        112 / 119   126 / 132   148 / 155   206 / 210   306 / 318   485 / 503
//   1237x822   octree      188 / 184   248 / 248   332 / 333   505 / 502   796 / 770  1280 / 1244
//              even        181 / 214   230 / 265   324 / 358   521 / 550   933 / 943  1868 / 1862
//   1920x1080  octree      249 / 254   342 / 351   524 / 532   837 / 828  1389 / 1369 2380 / 2346
//              even        282 / 342   355 / 416   550 / 612   960 / 991  2122 / 2106 4100 / 4076
//   3840x2160  octree      602 / 634  1016 / 1022 1777 / 1758 3132 / 3098 5332 / 5290
//              even        844 / 1080 1203 / 1412 2192 / 2248 4704 / 4391 9896 / 9782
//              a corner    614 / 732   854 / 992  1290 / 1442 2236 / 2341 4074 / 4086
// so two warps up to kFewTiles tiles, where the items are few, and with 128 points per tile up to kManyTiles.  Rows, whose longer lists weigh more, forward only: 16 channels at 1920x1080, 16 / 64 points
// per tile, even 500 / 534 and 906 / 912, octree 328 / 327 and 676 / 672.  Gaussian splats, forward only: at 1237x822 octree 224 / 209 and 506 / 493 with 8 / 64 per tile, even 196 / 218 and 442 / 433;
// 1920x1080 octree 267 / 257 and 848 / 811, even 315 / 363 and 930 / 900; 3840x2160, 16 / 32, octree 932 / 908 and 1585 / 1491, even 1109 / 1286 and 1693 / 1735.
constexpr int kFewTiles = 1 << 12, kFewTilesGaussian = 1 << 14;
bool by_two_warps(int mode, bool rows, int64_t tiles, int64_t n_points) {
    if (mode == INPC_MODE_GAUSSIAN) return tiles <= kFewTilesGaussian || n_points >= 64 * tiles;
    return tiles <= kFewTiles || (tiles <= kManyTiles && n_points >= (rows ? 32 : 128) * tiles);
}
// The largest lengths, and how many later segments are aimed at.  A batch of gaussian splats takes a training pass two to three
// times as long (more fragments, their sums), so its long items weigh more than the states of more segments; inference has little of
// that work.  Blend passes of a training step at 1237x822, forward and backward, first + later segment 1024 + 4096 / 512 + 2048 /
// 512 + 1024 / 256 + 512: 2^22 samples 1086 / 999 / 991 / 1035 us, 2^20 (which twice the number of segments gives 256 + 512)
// - / 472 / 462 / 350; inference, 2 * 10^6 splats at 1297x840: 200 / 216 / - / 251 (256 + 1024).
struct SegmentLimits {
    unsigned first_max, later_max, target;
};
constexpr SegmentLimits segment_limits(int mode, bool training) {
    return mode == INPC_MODE_GAUSSIAN && training ? SegmentLimits{512u, 1024u, 2u * kSegmentTarget} : SegmentLimits{kFirstSegmentMax, kLaterSegmentMax, kSegmentTarget};
}
__device__ __forceinline__ SegmentLengths segment_lengths(unsigned long long n_instances, int n_tiles, const SegmentLimits limits) {
    const unsigned target = n_tiles > kManyTiles ? limits.target / 2u : limits.target;
    SegmentLengths s;
    s.later = kSegmentMin;
    while (s.later < limits.later_max && (unsigned long long)s.later * target < n_instances) s.later *= 2u;
    s.first = max(kSegmentMin, min(limits.first_max, s.later / 2u));
    return s;
}
// How far past its stop a pixel must be before pass PRODUCT closes it, relative (or in units of log2, where the same number
// is wider).  REST multiplies up to `len` factors into a transmittance of its own, each product rounded by at most 2^-24 and, for
// faint splats, mostly in one direction; PRODUCT's chain of products does the same from another start (gaussian), its sum of
// logarithms is off by at most 2^-27 a term and 2^-23 of the 13.3 it can reach (bilinear): together less than len 2^-23.  (Both
// from the same 1 - alpha: with alpha rounded in one only, up to 2^-25 / (1 - alpha) would lie between them.)  A
// pixel closed too early loses the fragments behind it, a ten-thousandth of the image's range.
__device__ __forceinline__ float stop_margin(unsigned len) { return fmaxf(1e-4f, (float)(len + 8u) * 1.1920928955078125e-07f); }

enum { PASS_FIRST = 0, PASS_PRODUCT = 1, PASS_REST = 2 };
// Launch bounds of the passes: blocks per multiprocessor that the registers must leave room for.
__host__ __device__ constexpr int forward_blocks(int pass, int c4) { return pass == PASS_PRODUCT ? 4 : c4 == 8 ? 2 : 3; }
__host__ __device__ constexpr int rows_backward_blocks(int c4) { return c4 == 8 ? 1 : c4 == 4 ? 2 : 3; }   // 16 and 32 channels: one more takes L1 from the rows and registers from their sums (321 -> 360, 543 -> 586 us)
constexpr int kBackwardBlocks = 3, kGaussForwardBlocks = 3, kGaussBackwardBlocks = 2;
constexpr float kLogScale = 67108864.0f;   // 2^26, see the product of pass PRODUCT
constexpr float kLogNaN = 1048576.0f;      // far above what 32 factors add up to

// Pixels of the tile (bit = row * 8 + column) that the instance with this key reaches.
__device__ __forceinline__ unsigned long long key_pixels(unsigned code) {
    const unsigned cx = code & 15u, cy = code >> 4;
    const unsigned m = ((3u << cx) >> 1) & 0xFFu;                        // columns cx - 1 and cx, clipped to the tile
    const unsigned long long two = (unsigned long long)(m | (m << 8));   // the same columns in two consecutive rows
    if (cx > 8u || cy > 8u) return 0ull;
    return cy == 0u ? two >> 8 : two << (8u * (cy - 1u));                // rows cy - 1 and cy, clipped likewise
}

__device__ __forceinline__ unsigned warp_segments(unsigned len, const SegmentLengths& sl) {
    return len <= sl.first ? 1u : 1u + ceil_div(len - sl.first, sl.later);
}

// Work lists of the warp blend.  The first segments lie in the order of three classes of length, so that the longest are taken first and a
// pass does not end with one that was found late (with the tiles in order within a class, since neighbours share records in L1): 2^24 points
// of which nine tenths crowd one corner of a 3840x2160 image, first pass and backward 397 + 455 -> 345 + 442 us, 2^22 gaussian splats at 1237x822 backward
// 309 -> 289, 2 * 10^6 with sizes at 1297x840 171 -> 167, 2^25 points at 1920x1080 the same.  Not for feature rows: their backward pass, whose points' rows several
// tiles add to, took 331 -> 344 with 2^23 samples of 16 channels.
// Step 1 (one block per 1024 tiles): segments and non-empty tiles of each class of the block's tiles.
// Its last block scans those block sums; counts[0] = non-empty tiles, counts[1] = segments behind a tile's first, counts[kLongTiles] and counts[kLongTiles + 1] =
// tiles of the first class and of the first two.  Step 2 (same blocks as step 1): every tile's position from its block's base and a scan inside the
// block, and its items.  (One block scanning all tiles took 177 us for the 129,600 tiles of a 3840x2160 image.)
constexpr int kLongTiles = 8;
__device__ __forceinline__ unsigned length_class(unsigned len, const SegmentLengths& sl, bool by_length) {
    return !by_length ? 2u : len >= sl.first ? 0u : len >= sl.first / 4u ? 1u : 2u;
}

constexpr int kItemThreads = 256;
constexpr int kItemTilesPerThread = 4;
constexpr int kItemTilesPerBlock = kItemThreads * kItemTilesPerThread;

__device__ __forceinline__ void load_tile_segments(const uint2* __restrict__ ranges, int n_tiles, int t0, const SegmentLengths& sl, unsigned (&ns)[kItemTilesPerThread],
                                                   uint2 (&rg)[kItemTilesPerThread]) {
#pragma unroll
    for (int k = 0; k < kItemTilesPerThread; k += 2) {
        // two ranges per 16-byte load (t0 is even, the array 256-byte aligned)
        uint4 r = make_uint4(0u, 0u, 0u, 0u);
        if (t0 + k + 1 < n_tiles) r = __ldg(reinterpret_cast<const uint4*>(ranges + t0 + k));
        else if (t0 + k < n_tiles) { const uint2 r0 = __ldg(ranges + t0 + k); r.x = r0.x; r.y = r0.y; }
        rg[k] = make_uint2(r.x, r.y);
        rg[k + 1] = make_uint2(r.z, r.w);
        ns[k] = r.y > r.x ? warp_segments(r.y - r.x, sl) : 0u;
        ns[k + 1] = r.w > r.z ? warp_segments(r.w - r.z, sl) : 0u;
    }
}

// {segments, non-empty tiles of class 0, 1, 2} of a thread's tiles
__device__ __forceinline__ uint4 count_tile_segments(const unsigned (&ns)[kItemTilesPerThread], const uint2 (&rg)[kItemTilesPerThread], const SegmentLengths& sl,
                                                     bool by_length) {
    uint4 c = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int k = 0; k < kItemTilesPerThread; ++k) {
        if (ns[k] == 0u) continue;
        const unsigned cls = length_class(rg[k].y - rg[k].x, sl, by_length);
        c.x += ns[k];
        c.y += cls == 0u ? 1u : 0u;
        c.z += cls == 1u ? 1u : 0u;
        c.w += cls == 2u ? 1u : 0u;
    }
    return c;
}

__global__ void __launch_bounds__(kItemThreads) warp_items_count_kernel(const uint2* __restrict__ ranges, int n_tiles, const SegmentLimits limits, bool by_length, unsigned long long n_instances_arg,
                                                                        const unsigned long long* __restrict__ n_instances_dev, uint4* block_sums, unsigned* done,
                                                                        uint32_t* __restrict__ counts) {
    await_previous_kernel();
    __shared__ uint4 s_sums[kItemThreads / 32];
    unsigned ns[kItemTilesPerThread];
    uint2 rg[kItemTilesPerThread];
    const SegmentLengths sl = segment_lengths(n_instances_dev ? *n_instances_dev : n_instances_arg, n_tiles, limits);
    load_tile_segments(ranges, n_tiles, blockIdx.x * kItemTilesPerBlock + threadIdx.x * kItemTilesPerThread, sl, ns, rg);
    uint4 c = count_tile_segments(ns, rg, sl, by_length);
    c.x = __reduce_add_sync(0xffffffffu, c.x);
    c.y = __reduce_add_sync(0xffffffffu, c.y);
    c.z = __reduce_add_sync(0xffffffffu, c.z);
    c.w = __reduce_add_sync(0xffffffffu, c.w);
    if (lane_id() == 0) s_sums[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint4 t = s_sums[0];
#pragma unroll
        for (int w = 1; w < kItemThreads / 32; ++w) { t.x += s_sums[w].x; t.y += s_sums[w].y; t.z += s_sums[w].z; t.w += s_sums[w].w; }
        block_sums[blockIdx.x] = t;
    }
    if (!last_block(done, gridDim.x)) return;
    __shared__ unsigned s_scan[kItemThreads / 32 + 1];
    uint4 run = make_uint4(0u, 0u, 0u, 0u);
    for (unsigned base = 0; base < gridDim.x; base += kItemThreads) {
        const unsigned j = base + threadIdx.x;
        const uint4 v = j < gridDim.x ? __ldcg(block_sums + j) : make_uint4(0u, 0u, 0u, 0u);
        uint4 total, ex;
        ex.x = run.x + block_exclusive_scan(v.x, s_scan, &total.x);
        ex.y = run.y + block_exclusive_scan(v.y, s_scan, &total.y);
        ex.z = run.z + block_exclusive_scan(v.z, s_scan, &total.z);
        ex.w = run.w + block_exclusive_scan(v.w, s_scan, &total.w);
        if (j < gridDim.x) block_sums[j] = ex;
        run.x += total.x; run.y += total.y; run.z += total.z; run.w += total.w;
    }
    if (threadIdx.x == 0) {
        const unsigned tiles = run.y + run.z + run.w;
        counts[0] = tiles;
        counts[1] = run.x - tiles;
        counts[kLongTiles] = run.y;
        counts[kLongTiles + 1] = run.y + run.z;
    }
}

// Everything a warp needs to know about a (tile, segment), in one 32-byte record: the blend kernels read it with
// loads of 16 and 8 bytes, one item ahead of the one they work on, instead of chasing tile -> range -> first segment.
struct __align__(16) WarpItem {
    uint32_t tile, seg;       // which tile, which of its segments
    uint32_t begin, end;      // instance range of the segment
    uint32_t first, n_seg;    // slot of the tile's segment 0 in the per-segment arrays; segments of the tile
    uint32_t finished[2];     // of the tile's first later segment: how many of the later ones pass PRODUCT is through with, per half
};

__device__ __forceinline__ WarpItem load_item(const WarpItem* p) {
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(p));
    const uint2 b = __ldg(reinterpret_cast<const uint2*>(p) + 2);
    WarpItem w;
    w.tile = a.x; w.seg = a.y; w.begin = a.z; w.end = a.w; w.first = b.x; w.n_seg = b.y; w.finished[0] = 0; w.finished[1] = 0;
    return w;
}

// Step 2: items0 = segment 0 of the non-empty tiles by class, and from its end backwards the empty tiles (their number alone); items1 = every later segment, tile by tile.
__global__ void __launch_bounds__(kItemThreads) warp_items_fill_kernel(const uint2* __restrict__ ranges, int n_tiles, const SegmentLimits limits, bool by_length, unsigned long long n_instances_arg,
                                                                      const unsigned long long* __restrict__ n_instances_dev,
                                                                      const uint4* __restrict__ block_base, const uint32_t* __restrict__ counts, WarpItem* __restrict__ items0,
                                                                      WarpItem* __restrict__ items1) {
    await_previous_kernel();
    __shared__ unsigned s_scan[kItemThreads / 32 + 1];
    unsigned ns[kItemTilesPerThread];
    uint2 rg[kItemTilesPerThread];
    const int t0 = blockIdx.x * kItemTilesPerBlock + threadIdx.x * kItemTilesPerThread;
    const SegmentLengths sl = segment_lengths(n_instances_dev ? *n_instances_dev : n_instances_arg, n_tiles, limits);
    load_tile_segments(ranges, n_tiles, t0, sl, ns, rg);
    const uint4 c = count_tile_segments(ns, rg, sl, by_length), base = __ldg(block_base + blockIdx.x);
    // a block has at most 1024 tiles: the counts of two classes share a word
    unsigned total;
    const unsigned seg_before = block_exclusive_scan(c.x, s_scan, &total);
    const unsigned first_two = block_exclusive_scan(c.y | (c.z << 16), s_scan, &total);
    const unsigned third = block_exclusive_scan(c.w, s_scan, &total);
    unsigned before[3] = {base.y + (first_two & 0xFFFFu), base.z + (first_two >> 16), base.w + third};   // non-empty tiles of a class before this one
    const unsigned class_base[3] = {0u, __ldg(counts + kLongTiles), __ldg(counts + kLongTiles + 1)};
    unsigned first = base.x + seg_before;                      // segments of the tiles before this one
    unsigned rank = before[0] + before[1] + before[2];         // non-empty tiles before this one
#pragma unroll
    for (int k = 0; k < kItemTilesPerThread; ++k) {
        if (ns[k] == 0u) {
            if (t0 + k < n_tiles) items0[n_tiles - 1 - (t0 + k - (int)rank)].tile = (uint32_t)(t0 + k);
            continue;
        }
        const uint2 r = rg[k];
        const unsigned cls = length_class(r.y - r.x, sl, by_length);
        const unsigned place = cls == 0u ? class_base[0] + before[0]++ : cls == 1u ? class_base[1] + before[1]++ : class_base[2] + before[2]++;
        for (unsigned sg = 0; sg < ns[k]; ++sg) {
            const unsigned begin = sg == 0 ? r.x : r.x + sl.first + (sg - 1u) * sl.later;
            const unsigned end = min(r.y, begin + (sg == 0 ? sl.first : sl.later));
            // later segments: position = segments before this tile minus tiles before it
            WarpItem* dst = sg == 0 ? items0 + place : items1 + (first - rank + sg - 1u);
            reinterpret_cast<uint4*>(dst)[0] = make_uint4((uint32_t)(t0 + k), sg, begin, end);
            reinterpret_cast<uint4*>(dst)[1] = make_uint4(first, ns[k], 0u, 0u);
        }
        first += ns[k];
        rank += 1u;
    }
}

// The items of a pass as a warp takes them, through a ticket counter: consecutive items cost about the same (neighbouring
// tiles, or consecutive segments of one tile), so a warp that reserved items ahead would sit on work that idle warps
// could take (measured: holding two tickets ahead to prefetch the records made every pass 10-70 % slower).
// ... unless there are very many of them: a single counter hands out one ticket every 2.7 ns at best (measured:
// 259,200 items of a 3840x2160 image took 700 us whatever the occupancy), so with many small items a warp takes
// several consecutive ones per visit, behind the first n_single, which are long.
// How many items a visit takes is measured, with 8 / 4 / 2 visits per resident warp (8 / 16 / 32 items per visit at most):
// bilinear, 3840x2160, points crowding one part of the image: first pass 295 / 255 / 259 us, backward 391 / 373 / 415;
// the same at 2560x1440, first pass 91 / 75 / 89, backward 98 / 100 / 127.  Gaussian splats, 1920x1080: first pass
// 238 / 248 / 271, rows: step 1827 / 1829 / 1834, so these keep 8 items at most, and 8 visits for each of 32 warps of a multiprocessor, resident or not:
// with 8 for each resident one (24, 16, 8) the items come in larger shares and a pass ends later, step of rows of 32 / 16 channels, 2^24 points crowding
// one part of 3840x2160, 4050 -> 4210 / 3028 -> 3113 us (first pass 675 -> 808 / 570 -> 587, backward 1400 -> 1447 / 813 -> 873), 2^23 gaussian splats evenly over
// 3840x2160 3522 -> 3572.  Of later segments, which are long or find every pixel stopped, larger shares do no harm: 8 visits for each of 24 warps (2^20 opaque
// gaussian splats of 8 pixels at 1920x1080, products and later segments 49 + 51 -> 27 + 29).
// The long ones go out one by one however many there are.  Evenly filled images of 3840x2160, where nearly all are long, one by one / the first four
// of every warp one by one, the others 8 or 16 per visit / before there were classes, 6 per visit: training step of 2^25 bilinear splats 9955 / 10620 /
// 10425 us (first pass 2733 / 2590 / 2488, backward 3658 / 4450 / 4100), 2^26 almost opaque ones 19300 / 21870 / 21460, 2^25 gaussian splats 13630 / 15940 /
// 15960; inference, 2^22 splats of 3 pixels, faint 4648 / 4778 / 4760, opaque, where most of a list is behind stopped pixels, 2800 / 2856 / 2840.
// Where two warps take an item the visits are those of a pair (counted as if each warp took items, shares were half as large): step of 512 points per tile, nine tenths in a corner, 1237x822
// 1066 -> 1001 us, 1920x1080 1865 -> 1819; points spread evenly, 128 per tile, 998 -> 1015 with 6 visits of a pair backward (4: 1028); rows of 16 channels evenly 1428 -> 1325, 2^22 gaussian splats,
// nine tenths in a corner, 1048 -> 1015, samples of an octree all the same.
constexpr unsigned kMostItems = 8, kMostItemsBilinear = 16;
struct ItemQueue {
    unsigned n_items, n_single, per_visit;
    unsigned next = 0, end = 0;
    // `n_visits` at least, as far as there are items; `most` items per visit at most
    __device__ __forceinline__ ItemQueue(unsigned n_items_, unsigned n_single_, unsigned n_visits, unsigned most)
        : n_items(n_items_), n_single(min(n_single_, n_items_)), per_visit(max(1u, min(most, (n_items_ - n_single) / n_visits))) {}
    __device__ __forceinline__ bool take(unsigned* ticket, unsigned lane, unsigned* item) {
        if (next == end) {
            unsigned visit = 0;
            if (lane == 0) visit = atomicAdd(ticket, 1u);
            visit = __shfl_sync(0xffffffffu, visit, 0);
            const bool single = visit < n_single;
            next = single ? visit : n_single + (visit - n_single) * per_visit;
            if (next >= n_items) return false;
            end = single ? next + 1u : min(next + per_visit, n_items);
        }
        *item = next++;
        return true;
    }
};

// Asynchronous copies (global -> shared, 16 bytes, not through registers) and their completion groups.
__device__ __forceinline__ void async_copy_16(void* smem_dst, const void* gmem_src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void async_copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void async_copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A warp walks its list one batch of 32 instances at a time, and a batch cannot start before its 32 records have
// arrived (gathers from DRAM or, for the other half of the tile and for neighbouring tiles, from L1: hence the
// L1-caching form of the copy -- the form that bypasses L1 made the blend of a dense 2^25-point scene 30 % slower).
// The records of the next batch travel while the current one is blended, copied asynchronously into a two-stage ring
// in shared memory rather than through registers, and the per-pixel loops read a fragment's features from that
// ring instead of from a copy per fragment.  Measured with four stages (three batches in flight): the same
// single-view time, but 6 % less throughput with four views in flight on four streams (4985 against 5315
// Mpoints/s), since the larger rings leave room for fewer blocks of other views' kernels on an SM.
constexpr int kGatherDepthFilter = 2;     // stages of the ring, a power of two: first segments and products,
constexpr int kGatherDepthRest = 2;       // later segments,
constexpr int kGatherDepthBackward = 2;   // backward pass
constexpr int kIdsAhead = 3;      // later segments: batches whose point ids are loaded ahead of their gather

// Where the features of a splat come from: the second half of its record (four view-space channels), or, for feature rows,
// the caller's (n, 4 C4) array.  A staged row of more than four channels is padded by one float4, so that the lanes of a
// warp, which read the same channels of different rows, meet different shared-memory banks.
__host__ __device__ constexpr int feature_stride(int c4) { return c4 == 1 ? 1 : c4 + 1; }

// Starts the copies of the feature rows of a batch (`id` of lane j: the point of staged instance j) into `ring`:
// C4 neighbouring lanes copy the C4 16-byte pieces of one row.
template <int C4>
__device__ __forceinline__ void gather_rows(float4* ring, const float4* __restrict__ features, uint32_t id, unsigned lane) {
#pragma unroll
    for (int k = 0; k < C4; ++k) {
        const int piece = k * 32 + (int)lane, row = piece / C4, c = piece % C4;
        const uint32_t rid = __shfl_sync(0xffffffffu, id, row);
        if (rid != 0xffffffffu) async_copy_16(ring + row * feature_stride(C4) + c, features + (size_t)rid * C4 + c);
    }
}

// Bit l of lane k's word becomes bit k of lane l's word.
__device__ __forceinline__ unsigned warp_transpose_bits(unsigned x, unsigned lane) {
    unsigned m = 0x0000FFFFu;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        const unsigned y = __shfl_xor_sync(0xffffffffu, x, s);
        x = (lane & (unsigned)s) ? (x & ~m) | ((y >> s) & m) : (x & m) | ((y & m) << s);
        m ^= m << (s >> 1);
    }
    return x;
}

// Pixels (bit = row * 8 + column) of the 8x4 half at (px0, py0) that the 2x2 footprint of a bilinear splat at (x, y) covers.  A
// pixel at a distance of exactly one is among them; its weight is zero, by which it is told apart where the weight is formed.
__device__ __forceinline__ unsigned footprint_pixels(float x, float y, int px0, int py0) {
    const int qx = __float2int_rd(x - 0.5f) - px0, qy = __float2int_rd(y - 0.5f) - py0;   // left column, upper row
    if ((unsigned)(qx + 1) > 8u || (unsigned)(qy + 1) > 4u) return 0u;
    const unsigned two_by_two = qx < 0 ? 0x202u : qx == 7 ? 0x101u : 0x303u;              // clipped to the eight columns
    return (unsigned)(((unsigned long long)two_by_two << (8 * qy + qx + 9)) >> 9);        // rows outside the half fall off either end
}

// The same for the backward passes: `weights` receives the bilinear weights in the four pixels, by the parity of a pixel's column
// and row (the halves start at even ones), and pixels with a weight of zero are not named.
__device__ __forceinline__ unsigned footprint_weights(float x, float y, int px0, int py0, float4& weights) {
    const int qx = __float2int_rd(x - 0.5f) - px0, qy = __float2int_rd(y - 0.5f) - py0;   // left column, upper row
    const float wx0 = __saturatef(1.0f - fabsf(x - ((float)(px0 + qx) + 0.5f))), wx1 = __saturatef(1.0f - fabsf(x - ((float)(px0 + qx + 1) + 0.5f)));
    const float wy0 = __saturatef(1.0f - fabsf(y - ((float)(py0 + qy) + 0.5f))), wy1 = __saturatef(1.0f - fabsf(y - ((float)(py0 + qy + 1) + 0.5f)));
    const bool odd_x = qx & 1, odd_y = qy & 1;
    const float even_column = odd_x ? wx1 : wx0, odd_column = odd_x ? wx0 : wx1, even_row = odd_y ? wy1 : wy0, odd_row = odd_y ? wy0 : wy1;
    weights = make_float4(even_column * even_row, odd_column * even_row, even_column * odd_row, odd_column * odd_row);
    if ((unsigned)(qx + 1) > 8u || (unsigned)(qy + 1) > 4u) return 0u;
    const unsigned columns = (qx >= 0 && wx0 > 0.0f ? 0x101u : 0u) | (qx < 7 && wx1 > 0.0f ? 0x202u : 0u);
    const unsigned two_by_two = columns & ((wy0 > 0.0f ? 0x003u : 0u) | (wy1 > 0.0f ? 0x300u : 0u));
    return (unsigned)(((unsigned long long)two_by_two << (8 * qy + qx + 9)) >> 9);        // rows outside the half fall off either end
}

// The instances of a work item that can still have an effect, in list order: streams the item's keys and point ids, keeps those whose
// pixels (`reach`, by key code, of this half) have not all stopped, and queues their ids.  A step is 128 keys, four consecutive
// ones per lane in one 16-byte load, asked for a step ahead; the list need not start or end at such a boundary.
struct CandidateStream {
    const uint32_t *keys, *ids;
    unsigned begin, end;    // the item's range
    unsigned pos;           // next step to load, a multiple of 4 (the arrays are 256-byte aligned)
    unsigned head, tail;    // candidates [head, tail) wait for their gather
    bool loaded;
    uint4 key, id;          // the step that is loaded; behind `end` and before `begin` keys whose code reaches nothing

    __device__ __forceinline__ void load(unsigned lane) {
        const unsigned first = pos + 4u * lane;
        key = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
        id = make_uint4(0u, 0u, 0u, 0u);
        if (first < end) {
            key = __ldg(reinterpret_cast<const uint4*>(keys + first));
            id = __ldg(reinterpret_cast<const uint4*>(ids + first));
        }
        if (pos < begin || pos + 128u > end) {   // the first or the last step of the list
            const unsigned n = end - begin;
            if (first - begin >= n) key.x = 0xFFFFFFFFu;
            if (first + 1u - begin >= n) key.y = 0xFFFFFFFFu;
            if (first + 2u - begin >= n) key.z = 0xFFFFFFFFu;
            if (first + 3u - begin >= n) key.w = 0xFFFFFFFFu;
        }
        pos += 128u;
        loaded = true;
    }
    __device__ __forceinline__ void start(const uint32_t* keys_, const uint32_t* ids_, unsigned begin_, unsigned end_, unsigned lane) {
        keys = keys_; ids = ids_;
        begin = begin_; end = end_;
        pos = begin_ & ~3u;
        head = tail = 0u;
        loaded = false;
        if (begin < end) load(lane);
    }
    // until 32 candidates wait or the list ends
    __device__ __forceinline__ void fill(const unsigned* reach, unsigned done_w, uint32_t* queue, unsigned lane, unsigned lt_mask) {
        while (tail - head < 32u && loaded) {
            const uint4 k4 = key, i4 = id;
            loaded = false;
            if (pos < end) load(lane);
            const bool k0 = (reach[k4.x >> kTileKeyBits] & ~done_w) != 0u, k1 = (reach[k4.y >> kTileKeyBits] & ~done_w) != 0u;
            const bool k2 = (reach[k4.z >> kTileKeyBits] & ~done_w) != 0u, k3 = (reach[k4.w >> kTileKeyBits] & ~done_w) != 0u;
            const unsigned b0 = __ballot_sync(0xffffffffu, k0), b1 = __ballot_sync(0xffffffffu, k1);
            const unsigned b2 = __ballot_sync(0xffffffffu, k2), b3 = __ballot_sync(0xffffffffu, k3);
            unsigned at = tail + __popc(b0 & lt_mask) + __popc(b1 & lt_mask) + __popc(b2 & lt_mask) + __popc(b3 & lt_mask);
            if (k0) queue[at++ & (kQueueCap - 1)] = i4.x;
            if (k1) queue[at++ & (kQueueCap - 1)] = i4.y;
            if (k2) queue[at++ & (kQueueCap - 1)] = i4.z;
            if (k3) queue[at & (kQueueCap - 1)] = i4.w;
            tail += __popc(b0) + __popc(b1) + __popc(b2) + __popc(b3);
        }
    }
};

// Pass PRODUCT, a warp that has left an item's products in seg_T (a pixel per lane): where it is the last of the tile half to do so, seg_T of every later segment becomes the transmittance at its
// start = the state behind segment 0 times the products of the segments between.  `item`: of the list of later segments, where those of a tile lie in a row.
// A kernel of its own between the passes took 4 to 8 us and a launch.  Where every item formed its start itself, in the later segments and again backward, lists of many segments were read in the
// square of their number: training step of 2^24 almost opaque splats in one tile (4096 segments) 2660 us, 2520 so (backward 132 -> 35), of 2^26 rows of four channels 10760 -> 9040
// (511 -> 54); of 2^24 faint ones 5360 -> 5230.  Products 1 to 3 us longer for it, with a fence on either side of a relaxed addition 2 to 4: 2^23 samples at 1237x822 122.6 -> 125.3 (127.0), of
// which the backward pass gains 1.5; 10^6 at 801x533 32.8 -> 34.8.  More loads at once than 16 spill.
__device__ __forceinline__ void finish_products(const WarpItem* items, unsigned item, unsigned half, unsigned seg, unsigned n_seg, float* seg_T, unsigned first, bool inside, unsigned lane) {
    if (n_seg > 2u) {
        __syncwarp();   // every lane's product, before it counts as finished
        unsigned before = 0u;
        if (lane == 0u) asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(&items[item - (seg - 1u)].finished[half]) : "memory");
        if (__shfl_sync(0xffffffffu, before, 0) != n_seg - 2u) return;
        __syncwarp();   // what the first lane has acquired, the others see too
    }
    float* base = seg_T + ((size_t)first * 2u + half) * 32 + lane;   // segment g of this half: base[g * 64]
    constexpr int kAtOnce = 16;   // loads that do not wait for one another
    float run = base[0];
    for (unsigned g0 = 1; g0 < n_seg; g0 += kAtOnce) {
        if (__all_sync(0xffffffffu, !inside || run < kTransmittanceEps)) {
            // every pixel has stopped: nothing behind has an effect, and any state below the threshold says so
            for (unsigned g = g0; g < n_seg; ++g) base[(size_t)g * 64] = run;
            break;
        }
        float product[kAtOnce];
#pragma unroll
        for (int k = 0; k < kAtOnce; ++k) product[k] = g0 + k + 1u < n_seg ? __ldcg(base + (size_t)(g0 + k) * 64) : 1.0f;   // (of other warps: not through L1)
#pragma unroll
        for (int k = 0; k < kAtOnce; ++k) {
            if (g0 + k < n_seg) base[(size_t)(g0 + k) * 64] = run;
            run *= product[k];
        }
    }
}

// Shared memory of one warp of the forward passes.
template <bool BLEND, bool WEIGHTS, int DEPTH, int C4>
struct __align__(16) WarpForwardSmem {
    float4 ring_a[DEPTH][32];                        // records of the batches in flight: position, alpha, depth ...
    float4 ring_f[BLEND ? DEPTH : 1][BLEND ? 32 * feature_stride(C4) : 1];   // ... and features
    float4 weight[WEIGHTS ? 32 : 1];                 // per staged instance: what its pixels add to its blending weight, by parity
    uint32_t ring_id[DEPTH][32];                     // point ids of the batches in flight (0xFFFFFFFF: no instance)
    unsigned sum[BLEND ? 1 : 2][BLEND ? 1 : 32];     // PRODUCT: per pixel, the two words of a batch's sum of logarithms
    uint32_t queue[kQueueCap];
};

template <int PASS, int KIND, int C4>
constexpr size_t warp_forward_smem_bytes() {
    return 2 * 256 * sizeof(unsigned) +
           kWarpBlendWarps * sizeof(WarpForwardSmem<PASS != PASS_PRODUCT, PASS != PASS_PRODUCT && KIND == BLEND_TRAIN,
                                                    PASS == PASS_REST ? kGatherDepthRest : kGatherDepthFilter, C4>);
}

// ROWS: features are rows of 4 C4 channels in `rows` (a (4 C4, H, W) image); otherwise C4 is 1 and they are in the record.
template <int PASS, int KIND, int C4, bool ROWS>
__global__ void __launch_bounds__(kWarpBlendWarps * 32, forward_blocks(PASS, C4)) blend_bilinear_warp_forward_kernel(
    const WarpItem* __restrict__ items, const uint32_t* __restrict__ counts, unsigned* __restrict__ ticket, unsigned n_visits, const uint32_t* __restrict__ inst_keys,
    const uint32_t* __restrict__ inst_ids, const PointRec* __restrict__ rec, const float4* __restrict__ rows, float* __restrict__ seg_T, float4* __restrict__ seg_C,
    float* __restrict__ seg_Z, float* __restrict__ seg_E, float* __restrict__ image, float* __restrict__ depth_image,
    float* __restrict__ alpha_image, float* __restrict__ blending_weights, uint32_t* kept0, uint32_t* kept1,
    uint32_t* __restrict__ n_kept, int width, int height, int gw, int gh) {
    await_previous_kernel();
    constexpr unsigned kFull = 0xffffffffu;
    constexpr unsigned kNoInstance = 0xffffffffu;
    constexpr bool kBlend = PASS != PASS_PRODUCT;               // colours and weights; PRODUCT only multiplies
    constexpr bool kWeights = kBlend && KIND == BLEND_TRAIN;
    constexpr bool kDepth = kBlend && KIND == BLEND_INFER;
    constexpr int kGatherDepth = PASS == PASS_REST ? kGatherDepthRest : kGatherDepthFilter;
    constexpr int kStride = feature_stride(C4);
    static_assert(ROWS || C4 == 1, "a record holds four channels");
    using Smem = WarpForwardSmem<kBlend, kWeights, kGatherDepth, C4>;
    extern __shared__ __align__(16) unsigned char blend_smem[];
    unsigned* s_reach = reinterpret_cast<unsigned*>(blend_smem);     // [half][key code] -> pixels of the half reached
    Smem& sm = reinterpret_cast<Smem*>(blend_smem + 2 * 256 * sizeof(unsigned))[threadIdx.x >> 5];
    const unsigned lane = lane_id();
    const unsigned lt_mask = (1u << lane) - 1u;
    const unsigned parity = (lane & 1u) | ((lane >> 2) & 2u);        // of this lane's pixel: a footprint has each of the four once
    {
        const unsigned long long m = key_pixels(threadIdx.x);
        s_reach[threadIdx.x] = (unsigned)m;
        s_reach[256 + threadIdx.x] = (unsigned)(m >> 32);
    }
    if (PASS == PASS_PRODUCT) { sm.sum[0][lane] = 0u; sm.sum[1][lane] = 0u; }   // every batch leaves the sums at zero again
    __syncthreads();
    const unsigned n_items = __ldg(counts + (PASS == PASS_FIRST ? 0 : 1)) * 2u;
    ItemQueue queue(n_items, PASS == PASS_FIRST ? __ldg(counts + kLongTiles + 1) * 2u : 0u, n_visits, ROWS ? kMostItems : kMostItemsBilinear);
    unsigned item;
    while (queue.take(ticket, lane, &item)) {
        const WarpItem it = load_item(items + (item >> 1));
        const unsigned tile = it.tile, seg = it.seg, n_seg = it.n_seg, first = it.first;
        const int half = (int)(item & 1u);
        const size_t sidx = (size_t)(first + seg) * 2u + half;      // this item's slot in the per-segment arrays
        const size_t sidx0 = (size_t)first * 2u + half;             // segment 0 of the same tile half
        const uint2 rg = make_uint2(it.begin, it.end);
        // rows [j gh, (j + 1) gh) of the tile grid are image j of the call (one image except for batched inference)
        const int tx = (int)(tile % (unsigned)gw), ty_all = (int)(tile / (unsigned)gw);
        const int set = ty_all / gh, ty = ty_all - set * gh;
        const int px0 = tx * 8, py0 = ty * 8 + 4 * half;            // first pixel of this half
        const int px = px0 + (int)(lane & 7u), py = py0 + (int)(lane >> 3);
        const bool inside = px < width && py < height;
        const float pcx = (float)px + 0.5f, pcy = (float)py + 0.5f;

        float Tr = 1.0f, Z = 0.0f;
        float4 C[C4];
#pragma unroll
        for (int c = 0; c < C4; ++c) C[c] = make_float4(0.f, 0.f, 0.f, 0.f);
        double log_sum = 0.0, log_stop = 0.0;   // PRODUCT: -log2 of the product so far, and where the pixel counts as stopped
        bool done = !inside;
        if (PASS == PASS_PRODUCT) {
            // the state segment 0 left: a pixel that has stopped there stays stopped; for the others the
            // product is taken until T0 * product falls below the threshold (the true transmittance at
            // that point is smaller still, so everything behind is dead whatever the product says).  The margin
            // keeps a pixel open when rounding, of this sum or of the products REST forms, could be what carries it over.
            const float T0 = seg_T[sidx0 * 32 + lane];
            done = done || T0 < kTransmittanceEps;
            log_stop = done ? 0.0 : log2((double)T0 / (double)kTransmittanceEps) + (double)stop_margin(rg.y - rg.x);
        } else if (PASS == PASS_REST) {
            Tr = seg_T[sidx * 32 + lane];
            done = done || Tr < kTransmittanceEps;
        }
        unsigned done_w = __ballot_sync(kFull, done);   // bit l = pixel of lane l has stopped (warp-uniform)

        uint32_t* kept = half ? kept1 : kept0;
        unsigned n_out = 0;
        if (done_w != kFull) {   // else: nothing in this list can have an effect, and it is not even read
            // ---- where the instances come from.  FIRST and PRODUCT filter the item's keys; REST blends the list PRODUCT
            // compacted for this item (a superset of what is still alive at the true transmittance, see above), its ids
            // loaded kIdsAhead batches ahead of their gather.
            CandidateStream in;
            const unsigned* reach = s_reach + 256 * half;
            auto fill = [&]() {
                if (PASS != PASS_REST) in.fill(reach, done_w, sm.queue, lane, lt_mask);
                __syncwarp();
            };
            uint32_t idf[kIdsAhead];
            if (PASS == PASS_REST) {
                in.head = 0u;
                in.tail = n_kept[sidx];     // length of PRODUCT's list; the list itself starts at kept[rg.x]
#pragma unroll
                for (int k = 0; k < kIdsAhead; ++k) idf[k] = 32u * k + lane < in.tail ? kept[rg.x + 32u * k + lane] : 0u;
            } else {
                in.start(inst_keys, inst_ids, rg.x, rg.y, lane);
            }
            // the next (up to) 32 candidates become a batch: their records start to travel into `stage` of the ring
            auto gather = [&](unsigned stage) {
                const unsigned n = min(32u, in.tail - in.head);
                uint32_t id = kNoInstance;
                if (lane < n) {
                    id = checked_point(PASS == PASS_REST ? idf[0] : sm.queue[(in.head + lane) & (kQueueCap - 1)]);
                    const float4* p = reinterpret_cast<const float4*>(rec) + (size_t)id * (ROWS ? 1 : 2);
                    async_copy_16(&sm.ring_a[stage][lane], p);
                    if (kBlend && !ROWS) async_copy_16(&sm.ring_f[stage][lane], p + 1);
                }
                if (kBlend && ROWS) gather_rows<C4>(sm.ring_f[stage], rows, id, lane);
                sm.ring_id[stage][lane] = id;
                async_copy_commit();   // one group per batch, empty or not: the waits below count groups
                if (PASS == PASS_REST) {
#pragma unroll
                    for (int k = 0; k + 1 < kIdsAhead; ++k) idf[k] = idf[k + 1];
                    const unsigned nxt = in.head + 32u * kIdsAhead + lane;
                    idf[kIdsAhead - 1] = nxt < in.tail ? kept[rg.x + nxt] : 0u;
                }
                in.head += n;
            };
            fill();
#pragma unroll
            for (int st = 0; st + 1 < kGatherDepth; ++st) {
                gather((unsigned)st);
                fill();
            }
            for (unsigned batch = 0;; ++batch) {
                gather((batch + kGatherDepth - 1) & (kGatherDepth - 1));
                async_copy_wait<kGatherDepth - 1>();   // all but the newest kGatherDepth - 1 groups: this batch has arrived
                const unsigned stage = batch & (kGatherDepth - 1);
                const uint32_t id_cur = sm.ring_id[stage][lane];
                const bool staged = id_cur != kNoInstance;
                if (__ballot_sync(kFull, staged) == 0u) break;   // batches are filled in order: nothing is left
                // ---- lane j: the pixels of staged instance j that have not stopped
                const float4 own = sm.ring_a[stage][lane];
                const unsigned pixels = staged ? footprint_pixels(own.x, own.y, px0, py0) & ~done_w : 0u;
                if (kWeights) sm.weight[lane] = make_float4(0.f, 0.f, 0.f, 0.f);
                fill();   // (its __syncwarp also shows every lane what the others have copied)
                if (PASS == PASS_PRODUCT) {
                    // A product does not care about order.  Its factors are added up as -log2(1 - alpha) in fixed
                    // point (integer part and 26 fractional bits in two words per pixel, 32 of which fit a word): integer
                    // atomics commute, so the sum is the same on every run, and none of the per-pixel ordering below is
                    // needed.  (24 bits round a factor as coarsely as an fp32 product; on top of the rounding of 1 - alpha
                    // that made the alpha of 200,000 splats of opacity 10^-6 twice as far off as a chain of products.)
                    // An opacity below zero makes a factor above one: the integer part is signed.  A factor that is not a number
                    // counts more than 32 others can, by which the pixel's product is known to be none either.
                    const int qx = __float2int_rd(own.x - 0.5f) - px0, qy = __float2int_rd(own.y - 0.5f) - py0;
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const int cx = qx + (c & 1), cy = qy + (c >> 1), p = cy * 8 + cx;
                        const float dx = fabsf(own.x - ((float)(px0 + cx) + 0.5f)), dy = fabsf(own.y - ((float)(py0 + cy) + 0.5f));
                        const float wg = __saturatef(1.0f - dx) * __saturatef(1.0f - dy);
                        if ((unsigned)p < 32u && ((pixels >> (p & 31)) & 1u) && wg > 0.0f) {
                            const float x = 1.0f - rounded_alpha(own.z, wg);
                            const float t = x > 0.0f ? fminf(-log2f(x), 64.0f) : x <= 0.0f ? 64.0f : kLogNaN;   // 2^-64: far below the threshold
                            const float ti = floorf(t);
                            atomicAdd(&sm.sum[0][p], __float2uint_rn((t - ti) * kLogScale));
                            if (ti != 0.0f) atomicAdd(&sm.sum[1][p], (unsigned)(int)ti);
                        }
                    }
                }
                if (PASS == PASS_PRODUCT || kWeights) {   // inference keeps no lists for a backward pass
                    // What reaches a pixel that has not stopped goes into the list of this item: FIRST's list is the
                    // backward pass's, PRODUCT's is blended by REST, REST's (what is still alive at the true
                    // transmittance; written in place, behind the part of PRODUCT's list already read) the backward
                    // pass's again.  The filter runs several batches ahead of the blend, so some of what it let
                    // through is dead by now and is dropped here.
                    const unsigned b = __ballot_sync(kFull, pixels != 0u);
                    if (pixels) kept[rg.x + n_out + __popc(b & lt_mask)] = id_cur;
                    n_out += __popc(b);
                }
                if (PASS == PASS_PRODUCT) {
                    __syncwarp();
                    const unsigned frac = sm.sum[0][lane], whole = sm.sum[1][lane];
                    if (frac | whole) {
                        sm.sum[0][lane] = 0u;
                        sm.sum[1][lane] = 0u;
                        log_sum += (int)whole < (int)(kLogNaN / 2.0f) ? (double)(int)whole + (double)frac * (1.0 / (double)kLogScale) : (double)NAN;
                    }
                    done = done || log_sum > log_stop;
                    done_w = __ballot_sync(kFull, done);
                    __syncwarp();
                    if (done_w == kFull) break;   // every pixel has stopped: the rest of the list has no effect
                    continue;
                }
                // ---- every lane runs down the instances of its own pixel, front to back
                unsigned todo = warp_transpose_bits(pixels, lane);
                while (todo) {
                    // A few at a time: what they load and the weights they form do not wait for one another, and the chain from one
                    // fragment to the next is one multiply (the transmittance), everything else of a step hanging off it.  The steps
                    // are written without branches: a stopped pixel selects its old values.
                    constexpr int kChunk = C4 == 1 ? 3 : 2;
                    int j[kChunk];
                    float wg[kChunk], al[kChunk], zd[kChunk];
                    float4 f[kChunk];
                    bool ok[kChunk];
#pragma unroll
                    for (int u = 0; u < kChunk; ++u) {
                        ok[u] = todo != 0u;
                        j[u] = ok[u] ? __ffs(todo) - 1 : j[0];
                        todo &= todo - 1u;
                        const float4 a = sm.ring_a[stage][j[u]];
                        if (C4 == 1) f[u] = sm.ring_f[stage][j[u]];
                        wg[u] = __saturatef(1.0f - fabsf(a.x - pcx)) * __saturatef(1.0f - fabsf(a.y - pcy));
                        al[u] = rounded_alpha(a.z, wg[u]);
                        zd[u] = a.w;
                        ok[u] = ok[u] && wg[u] > 0.0f;
                    }
#pragma unroll
                    for (int u = 0; u < kChunk; ++u) {
                        const bool live = ok[u] && !done;
                        const float bw = Tr * al[u];
                        if (kWeights && live && bw > 0.0f) reinterpret_cast<float*>(sm.weight + j[u])[parity] = bw * wg[u];
                        if (C4 == 1) {
                            C[0].x = live ? C[0].x + bw * f[u].x : C[0].x;
                            C[0].y = live ? C[0].y + bw * f[u].y : C[0].y;
                            C[0].z = live ? C[0].z + bw * f[u].z : C[0].z;
                            C[0].w = live ? C[0].w + bw * f[u].w : C[0].w;
                        } else if (live) {
                            // wide rows are read where they are used: a chunk of them would not fit the registers
                            const float4* row = sm.ring_f[stage] + j[u] * kStride;
#pragma unroll
                            for (int c = 0; c < C4; ++c) {
                                const float4 v = row[c];
                                C[c].x += bw * v.x; C[c].y += bw * v.y; C[c].z += bw * v.z; C[c].w += bw * v.w;
                            }
                        }
                        if (kDepth) Z = live ? Z + bw * zd[u] : Z;
                        Tr = live ? Tr * (1.0f - al[u]) : Tr;
                        done = done || Tr < kTransmittanceEps;
                    }
                    if (done) todo = 0u;
                }
                __syncwarp();
                if (kWeights) {
                    // blending weight of every staged instance: its (up to) four pixels in a fixed order
                    const float4 v = sm.weight[lane];
                    const float sum = ((v.x + v.y) + v.z) + v.w;
                    if (sum > 0.0f) atomicAdd(blending_weights + id_cur, sum);
                }
                done_w = __ballot_sync(kFull, done);
                __syncwarp();
                if (done_w == kFull) break;   // every pixel has stopped: the rest of the list has no effect
            }
            async_copy_wait<0>();   // whatever is still travelling lands before the next item reuses the ring
            __syncwarp();
        }
        if ((PASS == PASS_PRODUCT || kWeights) && lane == 0) n_kept[sidx] = n_out;

        if (PASS == PASS_PRODUCT) {
            seg_T[sidx * 32 + lane] = (float)exp2(-log_sum);   // this segment's product
            finish_products(items, item >> 1, (unsigned)half, seg, n_seg, seg_T, first, inside, lane);
            continue;
        }
        const int64_t n_px = (int64_t)width * height;
        const int64_t pi = (int64_t)py * width + px;
        float* image_s = image + (int64_t)set * 4 * n_px;
        float* alpha_s = alpha_image + (int64_t)set * n_px;
        if (n_seg == 1u) {
            if (inside) {
#pragma unroll
                for (int c = 0; c < C4; ++c) {
                    float* plane = image_s + (int64_t)(4 * c) * n_px + pi;
                    plane[0] = C[c].x;
                    plane[n_px] = C[c].y;
                    plane[2 * n_px] = C[c].z;
                    plane[3 * n_px] = C[c].w;
                }
                if (KIND == BLEND_INFER) {
                    const float A = 1.0f - Tr;
                    depth_image[(int64_t)set * n_px + pi] = A > 0.0f ? Z / A : 0.0f;
                    alpha_s[pi] = Tr < kTransmittanceEps ? 1.0f : A;
                } else {
                    alpha_s[pi] = Tr < kTransmittanceEps ? 1.0f : 1.0f - Tr;
                }
            }
        } else {
            // partial colour of this segment; the per-tile combine adds the segments up in order
            const size_t si = sidx * 32 + lane;
#pragma unroll
            for (int c = 0; c < C4; ++c) seg_C[(sidx * C4 + c) * 32 + lane] = C[c];
            if (PASS == PASS_FIRST) seg_T[si] = Tr;   // the exact state behind segment 0
            if (KIND == BLEND_INFER) {
                seg_Z[si] = Z;
                seg_E[si] = Tr;
            } else if (seg + 1u == n_seg && inside) {
                alpha_s[pi] = Tr < kTransmittanceEps ? 1.0f : 1.0f - Tr;
            }
        }
    }
}

// ---- first and later segments of a training pass: two warps per item ---------------------------------------------
// What bounds these passes is the chain of instructions of one batch after the other of the longest lists.  Half of it does not depend on the pixels' state: finding the
// candidates, their records, the pixels they reach and the transposition of those masks.  One warp of a pair does that for the next batch while the other runs down the pixels'
// lists of this one; they meet at one barrier per batch.
// Batch b lies in stage b % 3 of the ring (b is walked, b + 1 made ready, b + 2 under way); its words, and whether there is such a batch, in place b % 2, where the state of the pixels before
// it lies too.  Both warps leave the loop at the same barrier: what they decide by is written before it and not again before the next but one.
// Step of 2^23 samples at 1237x822, first / later segments 96 / 112 -> 84 / 106 us, 16 channels 156 / 231 -> 156 / 189, 10^6 samples 24 / 34 -> 21 / 34.  Half as many items are under way, so
// where there are many short ones (see by_two_warps) or the passes wait for memory (inference) one warp per item is the faster form: 2^24 points crowding a corner of
// 3840x2160, first segments 255 against 290 us, 2^25 points of a cloud 347 + 109 against 367 + 118.  Four blocks per multiprocessor of 64 registers (of wide rows three): with three
// 333 us in place of 290, with five (48 registers) 333; four stages the same.
constexpr int kPairs = kWarpBlendWarps / 2;
template <int C4>
struct __align__(16) PairForwardSmem {
    float4 ring_a[3][32];                        // records of the batches in flight: position, alpha, depth ...
    float4 ring_f[3][32 * feature_stride(C4)];   // ... and features
    float4 weight[32];                           // per staged instance: what its pixels add to its blending weight, by parity
    uint32_t ring_id[3][32];                     // point ids of the batches in flight (0xFFFFFFFF: no instance)
    unsigned words[2][32];                       // per pixel, the instances of a batch that reach it
    unsigned stopped[2];                         // pixels that have stopped before a batch
    unsigned end[2];                             // there is no such batch
    unsigned item;                               // 0xFFFFFFFF: no more
    uint32_t queue[kQueueCap];
};
template <int C4>
constexpr size_t pair_forward_smem_bytes() { return 2 * 256 * sizeof(unsigned) + kPairs * sizeof(PairForwardSmem<C4>); }
__host__ __device__ constexpr int pair_forward_blocks(int c4) { return c4 == 1 ? 4 : c4 == 8 ? 2 : 3; }

__device__ __forceinline__ void pair_barrier(unsigned pair) {
    __syncwarp();
    asm volatile("bar.sync %0, 64;" ::"r"(1u + pair) : "memory");
}

// ROWS: features are rows of 4 C4 channels in `rows` (a (4 C4, H, W) image); otherwise C4 is 1 and they are in the record.
template <int PASS, int C4, bool ROWS>
__global__ void __launch_bounds__(kWarpBlendWarps * 32, pair_forward_blocks(C4)) blend_bilinear_pair_forward_kernel(
    const WarpItem* __restrict__ items, const uint32_t* __restrict__ counts, unsigned* __restrict__ ticket, unsigned n_visits, const uint32_t* __restrict__ inst_keys,
    const uint32_t* __restrict__ inst_ids, const PointRec* __restrict__ rec, const float4* __restrict__ rows, float* __restrict__ seg_T, float4* __restrict__ seg_C,
    float* __restrict__ image, float* __restrict__ alpha_image, float* __restrict__ blending_weights, uint32_t* kept0, uint32_t* kept1,
    uint32_t* __restrict__ n_kept, int width, int height, int gw) {
    await_previous_kernel();
    static_assert(PASS != PASS_PRODUCT && (ROWS || C4 == 1), "blends; a record holds four channels");
    constexpr unsigned kFull = 0xffffffffu, kNoInstance = 0xffffffffu, kNoItem = 0xffffffffu;
    constexpr int kStride = feature_stride(C4);
    using Smem = PairForwardSmem<C4>;
    extern __shared__ __align__(16) unsigned char blend_smem[];
    unsigned* s_reach = reinterpret_cast<unsigned*>(blend_smem);     // [half][key code] -> pixels of the half reached
    const unsigned lane = lane_id(), pair = threadIdx.x >> 6;
    const bool prepares = ((threadIdx.x >> 5) & 1u) == 0u;
    Smem& sm = reinterpret_cast<Smem*>(blend_smem + 2 * 256 * sizeof(unsigned))[pair];
    const unsigned lt_mask = (1u << lane) - 1u;
    const unsigned parity = (lane & 1u) | ((lane >> 2) & 2u);        // of this lane's pixel: a footprint has each of the four once
    {
        const unsigned long long m = key_pixels(threadIdx.x);
        s_reach[threadIdx.x] = (unsigned)m;
        s_reach[256 + threadIdx.x] = (unsigned)(m >> 32);
    }
    if (!prepares) sm.weight[lane] = make_float4(0.f, 0.f, 0.f, 0.f);   // every batch leaves them at zero again
    __syncthreads();
    const unsigned n_items = __ldg(counts + (PASS == PASS_FIRST ? 0 : 1)) * 2u;
    ItemQueue queue(n_items, PASS == PASS_FIRST ? __ldg(counts + kLongTiles + 1) * 2u : 0u, n_visits, ROWS ? kMostItems : kMostItemsBilinear);
    for (;;) {
        if (prepares) {
            unsigned taken;
            if (!queue.take(ticket, lane, &taken)) taken = kNoItem;
            if (lane == 0) sm.item = taken;
        }
        pair_barrier(pair);
        const unsigned item = sm.item;
        if (item == kNoItem) break;
        const WarpItem it = load_item(items + (item >> 1));
        const unsigned tile = it.tile, seg = it.seg, n_seg = it.n_seg, first = it.first;
        const int half = (int)(item & 1u);
        const size_t sidx = (size_t)(first + seg) * 2u + half;      // this item's slot in the per-segment arrays
        const uint2 rg = make_uint2(it.begin, it.end);
        const int tx = (int)(tile % (unsigned)gw), ty = (int)(tile / (unsigned)gw);
        const int px0 = tx * 8, py0 = ty * 8 + 4 * half;            // first pixel of this half
        const int px = px0 + (int)(lane & 7u), py = py0 + (int)(lane >> 3);
        const bool inside = px < width && py < height;

        if (prepares) {
            // ---- where the instances come from.  FIRST filters the item's keys; REST blends the list PRODUCT
            // compacted for this item (a superset of what is still alive at the true transmittance, see above), its ids
            // loaded kIdsAhead batches ahead of their gather.
            uint32_t* kept = half ? kept1 : kept0;
            const unsigned* reach = s_reach + 256 * half;
            CandidateStream in;
            uint32_t idf[kIdsAhead];
            if (PASS == PASS_REST) {
                in.head = 0u;
                in.tail = n_kept[sidx];     // length of PRODUCT's list; the list itself starts at kept[rg.x]
#pragma unroll
                for (int k = 0; k < kIdsAhead; ++k) idf[k] = 32u * k + lane < in.tail ? kept[rg.x + 32u * k + lane] : 0u;
            } else {
                in.start(inst_keys, inst_ids, rg.x, rg.y, lane);
            }
            pair_barrier(pair);
            unsigned done_w = sm.stopped[0], n_out = 0;
            if (done_w != kFull) {   // else: nothing in this list can have an effect
                auto fill = [&]() {
                    if (PASS != PASS_REST) in.fill(reach, done_w, sm.queue, lane, lt_mask);
                    __syncwarp();
                };
                // the next (up to) 32 candidates become a batch: their records start to travel into `stage` of the ring
                auto gather = [&](unsigned stage) {
                    const unsigned n = min(32u, in.tail - in.head);
                    uint32_t id = kNoInstance;
                    if (lane < n) {
                        id = checked_point(PASS == PASS_REST ? idf[0] : sm.queue[(in.head + lane) & (kQueueCap - 1)]);
                        const float4* p = reinterpret_cast<const float4*>(rec) + (size_t)id * (ROWS ? 1 : 2);
                        async_copy_16(&sm.ring_a[stage][lane], p);
                        if (!ROWS) async_copy_16(&sm.ring_f[stage][lane], p + 1);
                    }
                    if (ROWS) gather_rows<C4>(sm.ring_f[stage], rows, id, lane);
                    sm.ring_id[stage][lane] = id;
                    async_copy_commit();   // one group per batch, empty or not: the waits below count groups
                    if (PASS == PASS_REST) {
#pragma unroll
                        for (int k = 0; k + 1 < kIdsAhead; ++k) idf[k] = idf[k + 1];
                        const unsigned nxt = in.head + 32u * kIdsAhead + lane;
                        idf[kIdsAhead - 1] = nxt < in.tail ? kept[rg.x + nxt] : 0u;
                    }
                    in.head += n;
                };
                fill();
                gather(0u);
                fill();
                gather(1u);
                unsigned stage = 0u;   // of batch b
                for (unsigned b = 0;; ++b) {
                    fill();
                    async_copy_wait<1>();   // all but the newest group: batch b has arrived
                    const uint32_t id_cur = sm.ring_id[stage][lane];
                    const bool staged = id_cur != kNoInstance;
                    const bool end = __ballot_sync(kFull, staged) == 0u;   // batches are filled in order: nothing is left
                    if (!end) {
                        // ---- lane j: the pixels of staged instance j that have not stopped
                        const float4 own = sm.ring_a[stage][lane];
                        const unsigned pixels = staged ? footprint_pixels(own.x, own.y, px0, py0) & ~done_w : 0u;
                        // what reaches a pixel that has not stopped goes into the list of this item, as in blend_bilinear_warp_forward_kernel
                        const unsigned alive = __ballot_sync(kFull, pixels != 0u);
                        if (pixels) kept[rg.x + n_out + __popc(alive & lt_mask)] = id_cur;
                        n_out += __popc(alive);
                        sm.words[b & 1u][lane] = warp_transpose_bits(pixels, lane);
                    }
                    if (lane == 0) sm.end[b & 1u] = end ? 1u : 0u;
                    pair_barrier(pair);
                    if (end) break;
                    done_w = sm.stopped[b & 1u];
                    if (done_w == kFull) break;   // every pixel has stopped: the rest of the list has no effect
                    stage = stage == 2u ? 0u : stage + 1u;
                    gather(stage == 2u ? 0u : stage + 1u);   // batch b + 2, where batch b - 1 lay
                }
                async_copy_wait<0>();   // whatever is still travelling lands before the next item reuses the ring
                __syncwarp();
            }
            if (lane == 0) n_kept[sidx] = n_out;
            continue;
        }

        const float pcx = (float)px + 0.5f, pcy = (float)py + 0.5f;
        float Tr = 1.0f;
        float4 C[C4];
#pragma unroll
        for (int c = 0; c < C4; ++c) C[c] = make_float4(0.f, 0.f, 0.f, 0.f);
        bool done = !inside;
        if (PASS == PASS_REST) {
            Tr = seg_T[sidx * 32 + lane];
            done = done || Tr < kTransmittanceEps;
        }
        unsigned done_w = __ballot_sync(kFull, done);   // bit l = pixel of lane l has stopped (warp-uniform)
        if (lane == 0) sm.stopped[0] = done_w;
        pair_barrier(pair);
        if (done_w != kFull) {
            unsigned stage = 0u;
            for (unsigned b = 0;; ++b, stage = stage == 2u ? 0u : stage + 1u) {
                pair_barrier(pair);
                if (sm.end[b & 1u] || done_w == kFull) break;
                // ---- every lane runs down the instances of its own pixel, front to back
                unsigned todo = done ? 0u : sm.words[b & 1u][lane];   // (made before the pixels that stopped in the batch in front of it were known)
                while (todo) {
                    // a few at a time, without branches: see blend_bilinear_warp_forward_kernel
                    constexpr int kChunk = C4 == 1 ? 3 : 2;
                    int j[kChunk];
                    float wg[kChunk], al[kChunk];
                    float4 f[kChunk];
                    bool ok[kChunk];
#pragma unroll
                    for (int u = 0; u < kChunk; ++u) {
                        ok[u] = todo != 0u;
                        j[u] = ok[u] ? __ffs(todo) - 1 : j[0];
                        todo &= todo - 1u;
                        const float4 a = sm.ring_a[stage][j[u]];
                        if (C4 == 1) f[u] = sm.ring_f[stage][j[u]];
                        wg[u] = __saturatef(1.0f - fabsf(a.x - pcx)) * __saturatef(1.0f - fabsf(a.y - pcy));
                        al[u] = rounded_alpha(a.z, wg[u]);
                        ok[u] = ok[u] && wg[u] > 0.0f;
                    }
#pragma unroll
                    for (int u = 0; u < kChunk; ++u) {
                        const bool live = ok[u] && !done;
                        const float bw = Tr * al[u];
                        if (live && bw > 0.0f) reinterpret_cast<float*>(sm.weight + j[u])[parity] = bw * wg[u];
                        if (C4 == 1) {
                            C[0].x = live ? C[0].x + bw * f[u].x : C[0].x;
                            C[0].y = live ? C[0].y + bw * f[u].y : C[0].y;
                            C[0].z = live ? C[0].z + bw * f[u].z : C[0].z;
                            C[0].w = live ? C[0].w + bw * f[u].w : C[0].w;
                        } else if (live) {
                            // wide rows are read where they are used: a chunk of them would not fit the registers
                            const float4* row = sm.ring_f[stage] + j[u] * kStride;
#pragma unroll
                            for (int c = 0; c < C4; ++c) {
                                const float4 v = row[c];
                                C[c].x += bw * v.x; C[c].y += bw * v.y; C[c].z += bw * v.z; C[c].w += bw * v.w;
                            }
                        }
                        Tr = live ? Tr * (1.0f - al[u]) : Tr;
                        done = done || Tr < kTransmittanceEps;
                    }
                    if (done) todo = 0u;
                }
                __syncwarp();
                // blending weight of every staged instance: its (up to) four pixels in a fixed order
                const float4 v = sm.weight[lane];
                const float sum = ((v.x + v.y) + v.z) + v.w;
                if (sum > 0.0f) {
                    sm.weight[lane] = make_float4(0.f, 0.f, 0.f, 0.f);
                    atomicAdd(blending_weights + sm.ring_id[stage][lane], sum);
                }
                done_w = __ballot_sync(kFull, done);
                if (lane == 0) sm.stopped[(b + 1u) & 1u] = done_w;
            }
        }
        const int64_t n_px = (int64_t)width * height, pi = (int64_t)py * width + px;
        const float alpha = Tr < kTransmittanceEps ? 1.0f : 1.0f - Tr;
        if (n_seg == 1u) {
            if (inside) {
#pragma unroll
                for (int c = 0; c < C4; ++c) {
                    float* plane = image + (int64_t)(4 * c) * n_px + pi;
                    plane[0] = C[c].x;
                    plane[n_px] = C[c].y;
                    plane[2 * n_px] = C[c].z;
                    plane[3 * n_px] = C[c].w;
                }
                alpha_image[pi] = alpha;
            }
        } else {
            // partial colour of this segment; the per-tile combine adds the segments up in order
#pragma unroll
            for (int c = 0; c < C4; ++c) seg_C[(sidx * C4 + c) * 32 + lane] = C[c];
            if (PASS == PASS_FIRST) seg_T[sidx * 32 + lane] = Tr;   // the exact state behind segment 0
            if (seg + 1u == n_seg && inside) alpha_image[pi] = alpha;
        }
    }
}

// Last kernel of the forward passes.  Empty tiles, up to n_tiles (feature rows: none, their images are cleared beforehand): zeros; the passes write every pixel of the others.
// Per tile half with several segments: image = sum of the segment colours in order.
// For training the sum of a segment's colour and those behind it replaces the segment's own: what the backward pass takes the
// segment's running colour from.  Where a pixel stops in a segment nothing is behind it, and the two agree to the bit at the last
// fragment, as in an undivided list; the image less the colours before the segment would leave their rounding there, which an
// opacity close to one multiplies by 1 / (1 - alpha).
// Inference: expected depth, and the transmittance where the pixel stopped = the end value
// of the first segment that fell below the threshold.
template <int KIND, int C4>
__global__ void __launch_bounds__(kWarpBlendWarps * 32) warp_blend_combine_kernel(
    const WarpItem* __restrict__ items0, const uint32_t* __restrict__ counts, int n_tiles_at, float4* __restrict__ seg_C, const float* __restrict__ seg_Z,
    const float* __restrict__ seg_E,
    float* __restrict__ image, float* __restrict__ depth_image, float* __restrict__ alpha_image, int width, int height, int gw, int gh, int n_tiles) {
    await_previous_kernel();
    const unsigned lane = lane_id();
    const unsigned n_parts = __ldg(counts + n_tiles_at) * 2u;
    // four empty tiles at a time, a row of eight pixels of each: they mostly lie side by side
    for (int t = (int)(__ldg(counts) + 4u * (blockIdx.x * kWarpBlendWarps + (threadIdx.x >> 5))); t < n_tiles; t += (int)(gridDim.x * kWarpBlendWarps * 4u)) {
        if (t + (int)(lane >> 3) >= n_tiles) continue;
        const int tile = (int)__ldg(&items0[t + (lane >> 3)].tile), tx = tile % gw, ty_all = tile / gw, set = ty_all / gh;
        const int px = tx * 8 + (int)(lane & 7u), py = (ty_all - set * gh) * 8, rows = px < width ? min(8, height - py) : 0;
        const int64_t n_px = (int64_t)width * height, pi = (int64_t)py * width + px;
#pragma unroll 1
        for (int c = 0; c < 4 * C4 + (KIND == BLEND_INFER ? 2 : 1); ++c) {
            float* plane = (c < 4 * C4 ? image + ((int64_t)set * 4 * C4 + c) * n_px : (c == 4 * C4 ? alpha_image : depth_image) + (int64_t)set * n_px) + pi;
#pragma unroll
            for (int y = 0; y < 8; ++y)
                if (y < rows) plane[(int64_t)y * width] = 0.0f;
        }
    }
    // a warp takes one group of four channels of a tile half
    for (unsigned wc = blockIdx.x * kWarpBlendWarps + (threadIdx.x >> 5); wc < n_parts * C4; wc += gridDim.x * kWarpBlendWarps) {
        const unsigned w = wc / C4, ch = wc % C4;
        const WarpItem it = load_item(items0 + (w >> 1));
        const unsigned half = w & 1u;
        const unsigned tile = it.tile, n_seg = it.n_seg, first = it.first;
        if (n_seg == 1u) continue;
        const int tx = (int)(tile % (unsigned)gw), ty_all = (int)(tile / (unsigned)gw);
        const int set = ty_all / gh, ty = ty_all - set * gh;
        const int px = tx * 8 + (int)(lane & 7u);
        const int py = ty * 8 + 4 * (int)half + (int)(lane >> 3);
        const size_t base = ((size_t)first * 2u + half) * 32 + lane;   // segment g of this half: base + g * 64
        const bool inside = px < width && py < height;
        const int64_t n_px = (int64_t)width * height;
        const int64_t pi = (int64_t)py * width + px;
        float* image_s = image + (int64_t)set * 4 * n_px;
        {
            float4 run = make_float4(0.f, 0.f, 0.f, 0.f);
            float4* part = seg_C + (((size_t)first * 2u + half) * C4 + ch) * 32 + lane;   // segment g: part + g * 64 C4
            for (unsigned g0 = 0; g0 < n_seg; g0 += 4) {
                float4 c[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) c[k] = g0 + k < n_seg ? part[(size_t)(g0 + k) * (64 * C4)] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int k = 0; k < 4; ++k) { run.x += c[k].x; run.y += c[k].y; run.z += c[k].z; run.w += c[k].w; }
            }
            if (KIND == BLEND_TRAIN) {
                float4 rest = make_float4(0.f, 0.f, 0.f, 0.f);
                for (int g0 = (int)((n_seg - 1u) & ~3u); g0 >= 0; g0 -= 4) {
                    float4 c[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) c[k] = g0 + k < (int)n_seg ? part[(size_t)(g0 + k) * (64 * C4)] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int k = 3; k >= 0; --k) {
                        rest.x += c[k].x; rest.y += c[k].y; rest.z += c[k].z; rest.w += c[k].w;
                        if (g0 + k < (int)n_seg) part[(size_t)(g0 + k) * (64 * C4)] = rest;
                    }
                }
            }
            if (inside) {
                float* plane = image_s + (int64_t)(4 * ch) * n_px + pi;
                plane[0] = run.x;
                plane[n_px] = run.y;
                plane[2 * n_px] = run.z;
                plane[3 * n_px] = run.w;
            }
        }
        if (KIND == BLEND_INFER && ch == 0) {
            float z = 0.0f, t_final = 1.0f;
            bool stopped = false;
            for (unsigned g0 = 0; g0 < n_seg; g0 += 4) {
                float zz[4], ee[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const bool ok = g0 + k < n_seg;
                    zz[k] = ok ? seg_Z[base + (size_t)(g0 + k) * 64] : 0.0f;
                    ee[k] = ok ? seg_E[base + (size_t)(g0 + k) * 64] : 1.0f;
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    z += zz[k];
                    if (g0 + k < n_seg && !stopped) { t_final = ee[k]; stopped = t_final < kTransmittanceEps; }
                }
            }
            if (inside) {
                const float A = 1.0f - t_final;
                depth_image[(int64_t)set * n_px + pi] = A > 0.0f ? z / A : 0.0f;
                alpha_image[(int64_t)set * n_px + pi] = t_final < kTransmittanceEps ? 1.0f : A;
            }
        }
    }
}

// What the passes backward through a list share.  Per staged instance and pixel of its footprint (by the parity of the pixel's column
// and row, see footprint_weights) lane j leaves {alpha, G} with G = <g, f>, the upstream gradient of the pixel times the features of
// the instance; the lanes of the pixels run down their lists and leave {T, S}: the transmittance the fragment met and
// S = K - <g, what lies behind it>, K = grad_alpha * (1 - alpha of the pixel).  With these dL/dalpha = T G + S / (1 - alpha), formed per instance again.
struct __align__(16) FragmentSlots {
    float4 in[32][2];     // {alpha, G} of the parities 0 and 1 | 2 and 3
    float4 out[32][2];    // {T, S}; T = 0: the pixel had stopped, or does not belong to the footprint
};

// Stores without a branch around it.  (What it writes is read behind a __syncwarp only, across which volatile assembly does not move.)
__device__ __forceinline__ void store_shared_if(bool p, float2* dst, float2 v) {
    asm volatile("{\n.reg .pred q;\nsetp.ne.u32 q, %0, 0;\n@q st.shared.v2.f32 [%1], {%2, %3};\n}" ::"r"((unsigned)p), "r"(shared_address(dst)), "f"(v.x), "f"(v.y));
}

// Every lane runs down the instances `todo` of its pixel, front to back, a few at a time: what they load does not wait for one another,
// the chain from one transmittance to the next is one multiply, and the steps are written without branches.
//
// What lies behind a fragment is the final sum less the running one, but nothing lies behind the fragment at which a pixel stops: there
// the difference of the two, zero but for their roundings, would be multiplied by 1 / (1 - alpha), up to 10^8.  (At any other fragment
// T' = T (1 - alpha) >= 10^-4 bounds the factor by 10^4 T.)
__device__ __forceinline__ void walk_backward(unsigned todo, FragmentSlots& slots, unsigned parity, float G_final, float K, float& Tr, float& G_run, bool& done) {
    const float2* in = reinterpret_cast<const float2*>(slots.in) + parity;
    float2* out = reinterpret_cast<float2*>(slots.out) + parity;
    constexpr int kChunk = 4;
    while (todo) {
        int j[kChunk];
        float al[kChunk], G[kChunk], met[kChunk];
        bool ok[kChunk], live[kChunk];
#pragma unroll
        for (int u = 0; u < kChunk; ++u) {
            ok[u] = todo != 0u;
            j[u] = ok[u] ? __ffs(todo) - 1 : 0;
            todo &= todo - 1u;
            const float2 e = in[4 * j[u]];
            al[u] = e.x;
            G[u] = e.y;
        }
        float next = Tr;
        bool open = true;   // no fragment so far has stopped the pixel (it is not called with pixels that had stopped before)
#pragma unroll
        for (int u = 0; u < kChunk; ++u) {
            met[u] = next;
            live[u] = open && ok[u];
            const float behind = next * (1.0f - al[u]);
            next = live[u] ? behind : next;
            open = open && !(next < kTransmittanceEps);
        }
        Tr = next;
#pragma unroll
        for (int u = 0; u < kChunk; ++u) {
            G_run = live[u] ? G_run + met[u] * al[u] * G[u] : G_run;
            const float rest = met[u] * (1.0f - al[u]) < kTransmittanceEps ? 0.0f : G_run - G_final;
            store_shared_if(live[u], out + 4 * j[u], make_float2(met[u], rest + K));
        }
        if (!open) { done = true; todo = 0u; }
    }
}

// The same for four channels, whose running colours are kept one by one: at the last fragment of a list their sum is the final colour to the bit, and what
// lies behind it exactly zero.  (With the running sum <g, C> alone the opacity gradient is 1.35 to 1.5 times as far from 64 bits.)
__device__ __forceinline__ void walk_backward(unsigned todo, FragmentSlots& slots, const float4* features, unsigned parity, const float4& g, const float4& C_final, float K,
                                              float& Tr, float4& C_run, bool& done) {
    const float2* in = reinterpret_cast<const float2*>(slots.in) + parity;
    float2* out = reinterpret_cast<float2*>(slots.out) + parity;
    constexpr int kChunk = 4;
    while (todo) {
        int j[kChunk];
        float al[kChunk], met[kChunk];
        float4 f[kChunk];
        bool live[kChunk];
#pragma unroll
        for (int u = 0; u < kChunk; ++u) {
            live[u] = todo != 0u;
            j[u] = live[u] ? __ffs(todo) - 1 : 0;
            todo &= todo - 1u;
            al[u] = in[4 * j[u]].x;
            f[u] = features[j[u]];
        }
        bool open = true;
#pragma unroll
        for (int u = 0; u < kChunk; ++u) {
            met[u] = Tr;
            live[u] = open && live[u];
            Tr = live[u] ? Tr * (1.0f - al[u]) : Tr;
            open = open && !(Tr < kTransmittanceEps);
        }
#pragma unroll
        for (int u = 0; u < kChunk; ++u) {
            const float bw = met[u] * al[u];
            C_run.x = live[u] ? C_run.x + bw * f[u].x : C_run.x;
            C_run.y = live[u] ? C_run.y + bw * f[u].y : C_run.y;
            C_run.z = live[u] ? C_run.z + bw * f[u].z : C_run.z;
            C_run.w = live[u] ? C_run.w + bw * f[u].w : C_run.w;
            const float S = (C_run.x - C_final.x) * g.x + (C_run.y - C_final.y) * g.y + (C_run.z - C_final.z) * g.z + (C_run.w - C_final.w) * g.w;
            store_shared_if(live[u], out + 4 * j[u], make_float2(met[u], S + K));
        }
        if (!open) { done = true; todo = 0u; }
    }
}

// Pixels of a footprint (index row * 8 + column in the half) by parity; one that lies outside the half has an index (modulo 32) whose bit is not
// among the pixels footprint_weights names.
__device__ __forceinline__ void footprint_indices(float x, float y, int px0, int py0, unsigned (&pix)[4]) {
    const int qx = __float2int_rd(x - 0.5f) - px0, qy = __float2int_rd(y - 0.5f) - py0;
    const int even_column = qx + (qx & 1), odd_column = qx | 1, even_row = qy + (qy & 1), odd_row = qy | 1;
    pix[0] = (unsigned)(even_row * 8 + even_column) & 31u;
    pix[1] = (unsigned)(even_row * 8 + odd_column) & 31u;
    pix[2] = (unsigned)(odd_row * 8 + even_column) & 31u;
    pix[3] = (unsigned)(odd_row * 8 + odd_column) & 31u;
}

// Which of the four places for a point's gradients this half writes.  A splat's 2x2 pixels lie in at most two tile columns and two (tile row, half) groups, and which of
// them this item is follows from where the footprint starts: it holds the left column unless the
// footprint starts left of it, and the upper row unless it starts above it.  So every (point, slot)
// has exactly one writer in the whole launch: the sums go there with plain stores, a bit marks the
// slot as written, and the per-point pass adds the slots in fixed order -- no floating-point
// atomics, the same gradient bits on every run.
__device__ __forceinline__ unsigned footprint_slot(float x, float y, int px0, int py0) {
    return (__float2int_rd(x - 0.5f) < px0 ? 1u : 0u) + (__float2int_rd(y - 0.5f) < py0 ? 2u : 0u);
}

// Lane j: the sums of instance j over its (up to) four pixels, in a fixed order.
__device__ __forceinline__ void add_fragments(const FragmentSlots& slots, const float4* pixel_grad, const unsigned (&pix)[4], const float4& wg, unsigned slot, uint32_t id, unsigned lane,
                                              float4* __restrict__ slot_grad, unsigned* __restrict__ slot_mask) {
    const float4 in01 = slots.in[lane][0], in23 = slots.in[lane][1], out01 = slots.out[lane][0], out23 = slots.out[lane][1];
    const float al[4] = {in01.x, in01.z, in23.x, in23.z}, G[4] = {in01.y, in01.w, in23.y, in23.w};
    const float met[4] = {out01.x, out01.z, out23.x, out23.z}, S[4] = {out01.y, out01.w, out23.y, out23.w};
    const float w[4] = {wg.x, wg.y, wg.z, wg.w};
    float4 sf = make_float4(0.f, 0.f, 0.f, 0.f);
    float so = 0.0f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        if (met[c] != 0.0f) {   // (a transmittance that is no number gives a gradient that is none, as in src/bilinear/kernels.cu:361-415)
            const float bw = met[c] * al[c];
            so += (met[c] * G[c] + S[c] * one_minus_alpha_reciprocal(1.0f - al[c])) * w[c];   // (two warps per item: 214 us with a division, 207 so)
            if (bw > 0.0f) {   // (zero times an upstream gradient that has overflowed would be no number)
                const float4 pg = pixel_grad[pix[c]];
                sf.x += bw * pg.x; sf.y += bw * pg.y; sf.z += bw * pg.z; sf.w += bw * pg.w;
            }
        }
    }
    if (sf.x != 0.0f || sf.y != 0.0f || sf.z != 0.0f || sf.w != 0.0f || so != 0.0f) {
        // one aligned 32-byte record per slot: a whole memory sector, written without reading it first
        float4* e = slot_grad + ((size_t)id * 4u + slot) * 2u;
        e[0] = sf;
        e[1] = make_float4(so, 0.0f, 0.0f, 0.0f);
        atomicOr(slot_mask + id, 1u << slot);
    }
}

// Shared memory of one warp of the backward pass.
struct __align__(16) WarpBackwardSmem {
    float4 ring_a[kGatherDepthBackward][32];   // records of the batches in flight (see the forward pass): position, alpha ...
    float4 ring_f[kGatherDepthBackward][32];   // ... and features
    float4 pixel_grad[32];                  // image gradient of the half's pixels
    FragmentSlots slots;
    uint32_t ring_id[kGatherDepthBackward][32];   // point ids of the batches in flight (0xFFFFFFFF: no instance)
};
constexpr size_t kWarpBackwardSmemBytes = kWarpBlendWarps * sizeof(WarpBackwardSmem);

__global__ void __launch_bounds__(kWarpBlendWarps * 32, kBackwardBlocks) blend_bilinear_warp_backward_kernel(
    const WarpItem* __restrict__ items0, const WarpItem* __restrict__ items1, const uint32_t* __restrict__ counts,
    unsigned* __restrict__ ticket, unsigned n_visits, const uint32_t* __restrict__ kept0,
    const uint32_t* __restrict__ kept1, const uint32_t* __restrict__ n_kept, const PointRec* __restrict__ rec,
    const float* __restrict__ seg_T, const float4* __restrict__ seg_C, const float* __restrict__ grad_image,
    const float* __restrict__ grad_alpha, const float* __restrict__ image, const float* __restrict__ alpha_image,
    float4* __restrict__ slot_grad, unsigned* __restrict__ slot_mask, int width, int height, int gw) {
    await_previous_kernel();
    constexpr unsigned kFull = 0xffffffffu;
    constexpr unsigned kNoInstance = 0xffffffffu;
    constexpr int kGatherDepth = kGatherDepthBackward;
    extern __shared__ __align__(16) unsigned char blend_smem[];
    const unsigned lane = lane_id();
    const unsigned parity = (lane & 1u) | ((lane >> 2) & 2u);   // of this lane's pixel: a footprint has each of the four once
    WarpBackwardSmem& sm = reinterpret_cast<WarpBackwardSmem*>(blend_smem)[threadIdx.x >> 5];
    const unsigned n_first = __ldg(counts) * 2u;
    const unsigned n_items = n_first + __ldg(counts + 1) * 2u;
    const unsigned n_rest = n_items - n_first;

    // the later segments first (they belong to the longest lists)
    ItemQueue queue(n_items, n_rest + __ldg(counts + kLongTiles + 1) * 2u, n_visits, kMostItemsBilinear);
    unsigned item;
    while (queue.take(ticket, lane, &item)) {
        const WarpItem it = load_item(item < n_rest ? items1 + (item >> 1) : items0 + ((item - n_rest) >> 1));
        const int half = (int)((item < n_rest ? item : item - n_rest) & 1u);
        const unsigned n_list = __ldg(n_kept + (size_t)(it.first + it.seg) * 2u + half);
        const unsigned tile = it.tile, seg = it.seg, n_seg = it.n_seg;
        const size_t sidx = (size_t)(it.first + seg) * 2u + half;
        if (n_list == 0u) continue;
        const uint32_t* list = (half ? kept1 : kept0) + it.begin;
        const int tx = (int)(tile % (unsigned)gw), ty = (int)(tile / (unsigned)gw);
        const int px0 = tx * 8, py0 = ty * 8 + 4 * half;
        const int px = px0 + (int)(lane & 7u), py = py0 + (int)(lane >> 3);

        float4 g = make_float4(0.f, 0.f, 0.f, 0.f), C_final = g, C_run = g;
        float K = 0.0f, Tr = 1.0f;
        bool done = !(px < width && py < height);
        if (!done) {
            const int64_t n_px = (int64_t)width * height;
            const int64_t pi = (int64_t)py * width + px;
            g = make_float4(__ldg(grad_image + pi), __ldg(grad_image + n_px + pi), __ldg(grad_image + 2 * n_px + pi),
                            __ldg(grad_image + 3 * n_px + pi));
            // what this segment and the ones behind it add to the pixel: the running colour starts at zero
            C_final = n_seg > 1u ? seg_C[sidx * 32 + lane]
                                 : make_float4(__ldg(image + pi), __ldg(image + n_px + pi), __ldg(image + 2 * n_px + pi), __ldg(image + 3 * n_px + pi));
            K = __ldg(grad_alpha + pi) * (1.0f - __ldg(alpha_image + pi));
            if (seg > 0u) Tr = seg_T[sidx * 32 + lane];
            done = Tr < kTransmittanceEps;
        }
        __syncwarp();   // the previous item's readers of pixel_grad are through
        sm.pixel_grad[lane] = g;
        __syncwarp();
        unsigned done_w = __ballot_sync(kFull, done);

        // ids kIdsAhead batches ahead of their gather, records kGatherDepth - 1 batches ahead of their use
        uint32_t idf[kIdsAhead];
#pragma unroll
        for (int k = 0; k < kIdsAhead; ++k) idf[k] = 32u * k + lane < n_list ? __ldg(list + 32u * k + lane) : 0u;
        unsigned issued = 0;   // instances whose gather has started
        auto gather = [&](unsigned stage) {
            const unsigned n = min(32u, n_list - issued);
            uint32_t id = kNoInstance;
            if (lane < n) {
                id = checked_point(idf[0]);
                const float4* p = reinterpret_cast<const float4*>(rec + id);
                async_copy_16(&sm.ring_a[stage][lane], p);
                async_copy_16(&sm.ring_f[stage][lane], p + 1);
            }
            sm.ring_id[stage][lane] = id;
            async_copy_commit();   // one group per batch, empty or not
#pragma unroll
            for (int k = 0; k + 1 < kIdsAhead; ++k) idf[k] = idf[k + 1];
            const unsigned nxt = issued + 32u * kIdsAhead + lane;
            idf[kIdsAhead - 1] = nxt < n_list ? __ldg(list + nxt) : 0u;
            issued += n;
        };
#pragma unroll
        for (int st = 0; st + 1 < kGatherDepth; ++st) gather((unsigned)st);
        for (unsigned batch = 0;; ++batch) {
            gather((batch + kGatherDepth - 1) & (kGatherDepth - 1));
            async_copy_wait<kGatherDepth - 1>();
            const unsigned stage = batch & (kGatherDepth - 1);
            const uint32_t id_cur = sm.ring_id[stage][lane];
            const bool staged = id_cur != kNoInstance;
            if (__ballot_sync(kFull, staged) == 0u) break;
            // ---- lane j: the fragments of staged instance j
            const float4 own = sm.ring_a[stage][lane], fo = sm.ring_f[stage][lane];
            float4 wg = make_float4(0.f, 0.f, 0.f, 0.f);
            unsigned pixels = 0u, pix[4];
            if (staged) pixels = footprint_weights(own.x, own.y, px0, py0, wg) & ~done_w;
            footprint_indices(own.x, own.y, px0, py0, pix);
            {
                float G[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float4 pg = sm.pixel_grad[pix[c]];
                    G[c] = fo.x * pg.x + fo.y * pg.y + fo.z * pg.z + fo.w * pg.w;
                }
                sm.slots.in[lane][0] = make_float4(rounded_alpha(own.z, wg.x), G[0], rounded_alpha(own.z, wg.y), G[1]);
                sm.slots.in[lane][1] = make_float4(rounded_alpha(own.z, wg.z), G[2], rounded_alpha(own.z, wg.w), G[3]);
                sm.slots.out[lane][0] = sm.slots.out[lane][1] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            const unsigned todo = warp_transpose_bits(pixels, lane);
            __syncwarp();   // (every lane sees the records the others have copied, too)
            // ---- every lane runs down the instances of its own pixel, front to back
            walk_backward(todo, sm.slots, sm.ring_f[stage], parity, g, C_final, K, Tr, C_run, done);
            __syncwarp();
            // ---- lane j: the sums of instance j
            if (pixels) add_fragments(sm.slots, sm.pixel_grad, pix, wg, footprint_slot(own.x, own.y, px0, py0), id_cur, lane, slot_grad, slot_mask);
            done_w = __ballot_sync(kFull, done);
            __syncwarp();
            if (done_w == kFull) break;
        }
        async_copy_wait<0>();   // whatever is still travelling lands before the next item reuses the ring
        __syncwarp();
    }
}

// The same by two warps per item (see blend_bilinear_pair_forward_kernel): one makes the fragments of a batch ready and, a batch later, adds up what the walk has left per instance,
// the other walks.  Slots and words of batch b lie in place b % 2: those of b - 1 are added up before those of b + 1 take their place.  2^23 samples at 1237x822 232 -> 207 us, 10^6 at
// 801x533 46 -> 42.  Where lists are short one warp per item is the faster form (see by_two_warps; 2^24 points crowding a corner of 3840x2160 382 against 456 us), and for feature rows and Gaussian
// splats at any number (2^23 samples of 16 channels 328 against 393, 2^22 splats 251 against 274, 288 with the sums where the ellipses are found), since their rings and sums
// leave room for too few items.  Three blocks per multiprocessor of 80 registers; four of 64 224 us.
struct __align__(16) PairBackwardSmem {
    float4 ring_a[3][32];     // records of the batches in flight: position, alpha ...
    float4 ring_f[3][32];     // ... and features
    float4 pixel_grad[32];    // image gradient of the half's pixels
    FragmentSlots slots[2];
    uint32_t ring_id[3][32];
    unsigned words[2][32];
    unsigned stopped[2], end[2], item;
};
constexpr size_t kPairBackwardSmemBytes = kPairs * sizeof(PairBackwardSmem);
constexpr int kPairBackwardBlocks = 3;

__global__ void __launch_bounds__(kWarpBlendWarps * 32, kPairBackwardBlocks) blend_bilinear_pair_backward_kernel(
    const WarpItem* __restrict__ items0, const WarpItem* __restrict__ items1, const uint32_t* __restrict__ counts,
    unsigned* __restrict__ ticket, unsigned n_visits, const uint32_t* __restrict__ kept0,
    const uint32_t* __restrict__ kept1, const uint32_t* __restrict__ n_kept, const PointRec* __restrict__ rec,
    const float* __restrict__ seg_T, const float4* __restrict__ seg_C, const float* __restrict__ grad_image,
    const float* __restrict__ grad_alpha, const float* __restrict__ image, const float* __restrict__ alpha_image,
    float4* __restrict__ slot_grad, unsigned* __restrict__ slot_mask, int width, int height, int gw) {
    await_previous_kernel();
    constexpr unsigned kFull = 0xffffffffu, kNoInstance = 0xffffffffu, kNoItem = 0xffffffffu;
    extern __shared__ __align__(16) unsigned char blend_smem[];
    const unsigned lane = lane_id(), pair = threadIdx.x >> 6;
    const bool prepares = ((threadIdx.x >> 5) & 1u) == 0u;
    const unsigned parity = (lane & 1u) | ((lane >> 2) & 2u);   // of this lane's pixel: a footprint has each of the four once
    PairBackwardSmem& sm = reinterpret_cast<PairBackwardSmem*>(blend_smem)[pair];
    const unsigned n_first = __ldg(counts) * 2u;
    const unsigned n_items = n_first + __ldg(counts + 1) * 2u;
    const unsigned n_rest = n_items - n_first;

    // the later segments first (they belong to the longest lists)
    ItemQueue queue(n_items, n_rest + __ldg(counts + kLongTiles + 1) * 2u, n_visits, kMostItemsBilinear);
    for (;;) {
        if (prepares) {
            unsigned taken;
            if (!queue.take(ticket, lane, &taken)) taken = kNoItem;
            if (lane == 0) sm.item = taken;
        }
        pair_barrier(pair);
        const unsigned item = sm.item;
        if (item == kNoItem) break;
        const WarpItem it = load_item(item < n_rest ? items1 + (item >> 1) : items0 + ((item - n_rest) >> 1));
        const int half = (int)((item < n_rest ? item : item - n_rest) & 1u);
        const size_t sidx = (size_t)(it.first + it.seg) * 2u + half;
        const unsigned n_list = __ldg(n_kept + sidx);
        const int tx = (int)(it.tile % (unsigned)gw), ty = (int)(it.tile / (unsigned)gw);
        const int px0 = tx * 8, py0 = ty * 8 + 4 * half;

        if (prepares) {
            const uint32_t* list = (half ? kept1 : kept0) + it.begin;
            // ids kIdsAhead batches ahead of their gather, records two batches ahead of their use
            uint32_t idf[kIdsAhead];
#pragma unroll
            for (int k = 0; k < kIdsAhead; ++k) idf[k] = 32u * k + lane < n_list ? __ldg(list + 32u * k + lane) : 0u;
            pair_barrier(pair);
            unsigned done_w = sm.stopped[0];
            if (n_list == 0u || done_w == kFull) continue;
            unsigned issued = 0;   // instances whose gather has started
            auto gather = [&](unsigned stage) {
                const unsigned n = min(32u, n_list - issued);
                uint32_t id = kNoInstance;
                if (lane < n) {
                    id = checked_point(idf[0]);
                    const float4* p = reinterpret_cast<const float4*>(rec + id);
                    async_copy_16(&sm.ring_a[stage][lane], p);
                    async_copy_16(&sm.ring_f[stage][lane], p + 1);
                }
                sm.ring_id[stage][lane] = id;
                async_copy_commit();   // one group per batch, empty or not
#pragma unroll
                for (int k = 0; k + 1 < kIdsAhead; ++k) idf[k] = idf[k + 1];
                const unsigned nxt = issued + 32u * kIdsAhead + lane;
                idf[kIdsAhead - 1] = nxt < n_list ? __ldg(list + nxt) : 0u;
                issued += n;
            };
            gather(0u);
            gather(1u);
            // lane j: instance j of the batch that is made ready, and of the one in front of it
            uint32_t id = kNoInstance, id_before = kNoInstance;
            unsigned pixels = 0u, pixels_before = 0u, pix[4], pix_before[4] = {0u, 0u, 0u, 0u};
            float4 wg = make_float4(0.f, 0.f, 0.f, 0.f), wg_before = wg;
            unsigned slot = 0u, slot_before = 0u;
            unsigned stage = 0u;   // of batch b
            for (unsigned b = 0;; ++b) {
                async_copy_wait<1>();   // all but the newest group: batch b has arrived
                id = sm.ring_id[stage][lane];
                const bool staged = id != kNoInstance, end = __ballot_sync(kFull, staged) == 0u;
                pixels = 0u;
                if (!end) {
                    // ---- lane j: the fragments of staged instance j
                    const float4 own = sm.ring_a[stage][lane], fo = sm.ring_f[stage][lane];
                    wg = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (staged) pixels = footprint_weights(own.x, own.y, px0, py0, wg) & ~done_w;
                    footprint_indices(own.x, own.y, px0, py0, pix);
                    slot = footprint_slot(own.x, own.y, px0, py0);
                    float G[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float4 pg = sm.pixel_grad[pix[c]];
                        G[c] = fo.x * pg.x + fo.y * pg.y + fo.z * pg.z + fo.w * pg.w;
                    }
                    FragmentSlots& slots = sm.slots[b & 1u];
                    slots.in[lane][0] = make_float4(rounded_alpha(own.z, wg.x), G[0], rounded_alpha(own.z, wg.y), G[1]);
                    slots.in[lane][1] = make_float4(rounded_alpha(own.z, wg.z), G[2], rounded_alpha(own.z, wg.w), G[3]);
                    slots.out[lane][0] = slots.out[lane][1] = make_float4(0.f, 0.f, 0.f, 0.f);
                    sm.words[b & 1u][lane] = warp_transpose_bits(pixels, lane);
                }
                if (lane == 0) sm.end[b & 1u] = end ? 1u : 0u;
                pair_barrier(pair);
                // batch b - 1: the walk is through with it
                if (pixels_before) add_fragments(sm.slots[(b + 1u) & 1u], sm.pixel_grad, pix_before, wg_before, slot_before, id_before, lane, slot_grad, slot_mask);
                if (end) break;
                done_w = sm.stopped[b & 1u];
                if (done_w == kFull) break;
                id_before = id; pixels_before = pixels; wg_before = wg; slot_before = slot;
#pragma unroll
                for (int c = 0; c < 4; ++c) pix_before[c] = pix[c];
                __syncwarp();   // batch b + 1 takes the place of b - 1
                stage = stage == 2u ? 0u : stage + 1u;
                gather(stage == 2u ? 0u : stage + 1u);   // batch b + 2
            }
            async_copy_wait<0>();   // whatever is still travelling lands before the next item reuses the ring
            __syncwarp();
            continue;
        }

        const int px = px0 + (int)(lane & 7u), py = py0 + (int)(lane >> 3);
        float4 g = make_float4(0.f, 0.f, 0.f, 0.f), C_final = g, C_run = g;
        float K = 0.0f, Tr = 1.0f;
        bool done = !(px < width && py < height);
        if (!done && n_list > 0u) {
            const int64_t n_px = (int64_t)width * height;
            const int64_t pi = (int64_t)py * width + px;
            g = make_float4(__ldg(grad_image + pi), __ldg(grad_image + n_px + pi), __ldg(grad_image + 2 * n_px + pi),
                            __ldg(grad_image + 3 * n_px + pi));
            // what this segment and the ones behind it add to the pixel: the running colour starts at zero
            C_final = it.n_seg > 1u ? seg_C[sidx * 32 + lane]
                                    : make_float4(__ldg(image + pi), __ldg(image + n_px + pi), __ldg(image + 2 * n_px + pi), __ldg(image + 3 * n_px + pi));
            K = __ldg(grad_alpha + pi) * (1.0f - __ldg(alpha_image + pi));
            if (it.seg > 0u) Tr = seg_T[sidx * 32 + lane];
            done = Tr < kTransmittanceEps;
        }
        sm.pixel_grad[lane] = g;
        unsigned done_w = __ballot_sync(kFull, done);
        if (lane == 0) sm.stopped[0] = done_w;
        pair_barrier(pair);
        if (n_list == 0u || done_w == kFull) continue;
        unsigned stage = 0u;
        for (unsigned b = 0;; ++b, stage = stage == 2u ? 0u : stage + 1u) {
            pair_barrier(pair);
            if (sm.end[b & 1u] || done_w == kFull) break;
            // ---- every lane runs down the instances of its own pixel, front to back
            walk_backward(done ? 0u : sm.words[b & 1u][lane], sm.slots[b & 1u], sm.ring_f[stage], parity, g, C_final, K, Tr, C_run, done);
            done_w = __ballot_sync(kFull, done);
            if (lane == 0) sm.stopped[(b + 1u) & 1u] = done_w;
        }
    }
}

// Backward pass over feature rows, the lists and the walk of the kernels above with a scalar in the place of the running colour: with
// G = <g, .> over the channels, dL/dalpha = T G(f) + (G(C_run) - G(C_final) + K) / (1 - alpha).  G(f) is formed per instance and pixel,
// and so is the gradient of a point's row, sum over its pixels of weight * g, with every staged lane busy.
// A splat whose 2x2 pixels all lie in this 8x4 half has no other writer in the launch and stores its row; the others
// (about a third) add theirs with one vector atomic per four channels.
// Records and rows are read once, where a batch is made ready: the next batch travels into their place while this one is walked and added up, which leaves the L1 cache more for the rows that
// neighbouring halves share (2^23 samples of 16 channels 330 -> 321 us against a ring of two batches, 4 channels 301 -> 296, 32 the same).
template <int C4>
struct __align__(16) RowsBackwardSmem {
    float4 ring_a[32];                            // records of the batch that is under way
    float4 ring_f[32 * feature_stride(C4)];       // ... and their rows
    float4 pixel_grad[32 * feature_stride(C4)];   // image gradient of the half's pixels
    FragmentSlots slots;
};
template <int C4>
constexpr size_t rows_warp_backward_smem_bytes() { return kWarpBlendWarps * sizeof(RowsBackwardSmem<C4>); }

template <int C4>
__global__ void __launch_bounds__(kWarpBlendWarps * 32, rows_backward_blocks(C4)) blend_rows_warp_backward_kernel(
    const WarpItem* __restrict__ items0, const WarpItem* __restrict__ items1, const uint32_t* __restrict__ counts,
    unsigned* __restrict__ ticket, unsigned n_visits, const uint32_t* __restrict__ kept0,
    const uint32_t* __restrict__ kept1, const uint32_t* __restrict__ n_kept, const PointRec* __restrict__ rec, const float4* __restrict__ rows,
    const float* __restrict__ seg_T, const float4* __restrict__ seg_C, const float* __restrict__ grad_image,
    const float* __restrict__ grad_alpha, const float* __restrict__ image, const float* __restrict__ alpha_image,
    float4* __restrict__ grad_rows, float* __restrict__ grad_opacity, int width, int height, int gw) {
    await_previous_kernel();
    constexpr unsigned kFull = 0xffffffffu;
    constexpr unsigned kNoInstance = 0xffffffffu;
    constexpr int kStride = feature_stride(C4);
    extern __shared__ __align__(16) unsigned char blend_smem[];
    const unsigned lane = lane_id();
    const unsigned parity = (lane & 1u) | ((lane >> 2) & 2u);   // of this lane's pixel: a footprint has each of the four once
    RowsBackwardSmem<C4>& sm = reinterpret_cast<RowsBackwardSmem<C4>*>(blend_smem)[threadIdx.x >> 5];
    const unsigned n_first = __ldg(counts) * 2u;
    const unsigned n_items = n_first + __ldg(counts + 1) * 2u;
    const unsigned n_rest = n_items - n_first;
    const int64_t n_px = (int64_t)width * height;

    ItemQueue queue(n_items, n_rest + __ldg(counts + kLongTiles + 1) * 2u, n_visits, kMostItems);
    unsigned item;
    while (queue.take(ticket, lane, &item)) {
        const WarpItem it = load_item(item < n_rest ? items1 + (item >> 1) : items0 + ((item - n_rest) >> 1));
        const int half = (int)((item < n_rest ? item : item - n_rest) & 1u);
        const unsigned n_list = __ldg(n_kept + (size_t)(it.first + it.seg) * 2u + half);
        const unsigned tile = it.tile, seg = it.seg, n_seg = it.n_seg;
        const size_t sidx = (size_t)(it.first + seg) * 2u + half;
        if (n_list == 0u) continue;
        const uint32_t* list = (half ? kept1 : kept0) + it.begin;
        const int tx = (int)(tile % (unsigned)gw), ty = (int)(tile / (unsigned)gw);
        const int px0 = tx * 8, py0 = ty * 8 + 4 * half;
        const int px = px0 + (int)(lane & 7u), py = py0 + (int)(lane >> 3);

        float4 g[C4];
        float G_final = 0.0f, G_run = 0.0f, K = 0.0f, Tr = 1.0f;
        bool done = !(px < width && py < height);
#pragma unroll
        for (int c = 0; c < C4; ++c) g[c] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!done) {
            const int64_t pi = (int64_t)py * width + px;
#pragma unroll
            for (int c = 0; c < C4; ++c) {
                const float* gp = grad_image + (int64_t)(4 * c) * n_px + pi;
                g[c] = make_float4(__ldg(gp), __ldg(gp + n_px), __ldg(gp + 2 * n_px), __ldg(gp + 3 * n_px));
                // what this segment and the ones behind it add to the pixel
                float4 v;
                if (n_seg > 1u) {
                    v = seg_C[(sidx * C4 + c) * 32 + lane];
                } else {
                    const float* ip = image + (int64_t)(4 * c) * n_px + pi;
                    v = make_float4(__ldg(ip), __ldg(ip + n_px), __ldg(ip + 2 * n_px), __ldg(ip + 3 * n_px));
                }
                G_final += v.x * g[c].x + v.y * g[c].y + v.z * g[c].z + v.w * g[c].w;
            }
            K = __ldg(grad_alpha + pi) * (1.0f - __ldg(alpha_image + pi));
            if (seg > 0u) Tr = seg_T[sidx * 32 + lane];
            done = Tr < kTransmittanceEps;
        }
        __syncwarp();   // the previous item's readers of pixel_grad are through
#pragma unroll
        for (int c = 0; c < C4; ++c) sm.pixel_grad[lane * kStride + c] = g[c];
        __syncwarp();
        unsigned done_w = __ballot_sync(kFull, done);

        uint32_t idf[kIdsAhead];
#pragma unroll
        for (int k = 0; k < kIdsAhead; ++k) idf[k] = 32u * k + lane < n_list ? __ldg(list + 32u * k + lane) : 0u;
        unsigned issued = 0;
        uint32_t id_next = kNoInstance;   // of the batch that is under way
        auto gather = [&]() {
            const unsigned n = min(32u, n_list - issued);
            uint32_t id = kNoInstance;
            if (lane < n) {
                id = checked_point(idf[0]);
                async_copy_16(&sm.ring_a[lane], reinterpret_cast<const float4*>(rec) + id);
            }
            gather_rows<C4>(sm.ring_f, rows, id, lane);
            id_next = id;
            async_copy_commit();
#pragma unroll
            for (int k = 0; k + 1 < kIdsAhead; ++k) idf[k] = idf[k + 1];
            const unsigned nxt = issued + 32u * kIdsAhead + lane;
            idf[kIdsAhead - 1] = nxt < n_list ? __ldg(list + nxt) : 0u;
            issued += n;
        };
        gather();
        for (;;) {
            async_copy_wait<0>();
            const uint32_t id_cur = id_next;
            const bool staged = id_cur != kNoInstance;
            if (__ballot_sync(kFull, staged) == 0u) break;
            __syncwarp();   // every lane sees what the others have copied
            // ---- lane j: the fragments of staged instance j in the pixels that have not stopped
            const float4 own = sm.ring_a[lane];
            float4 wg = make_float4(0.f, 0.f, 0.f, 0.f);
            unsigned pixels = 0u, pix[4];
            if (staged) pixels = footprint_weights(own.x, own.y, px0, py0, wg) & ~done_w;
            footprint_indices(own.x, own.y, px0, py0, pix);
            {
                float G[4] = {0.f, 0.f, 0.f, 0.f};
                const float4* row = sm.ring_f + lane * kStride;
#pragma unroll
                for (int c = 0; c < C4; ++c) {
                    const float4 f = row[c];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        // 32 channels: not for pixels outside the half or stopped (2^24 points at 3840x2160 1441 -> 1408 us; of 16 channels 824 -> 840)
                        if (C4 == 8 && !((pixels >> pix[q]) & 1u)) continue;
                        const float4 v = sm.pixel_grad[pix[q] * kStride + c];
                        G[q] += f.x * v.x + f.y * v.y + f.z * v.z + f.w * v.w;
                    }
                }
                sm.slots.in[lane][0] = make_float4(rounded_alpha(own.z, wg.x), G[0], rounded_alpha(own.z, wg.y), G[1]);
                sm.slots.in[lane][1] = make_float4(rounded_alpha(own.z, wg.z), G[2], rounded_alpha(own.z, wg.w), G[3]);
                sm.slots.out[lane][0] = sm.slots.out[lane][1] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            const unsigned todo = warp_transpose_bits(pixels, lane);
            __syncwarp();
            gather();   // the next batch, where this one lay: nobody reads its records and rows any more
            // ---- every lane runs down the instances of its own pixel, front to back
            walk_backward(todo, sm.slots, parity, G_final, K, Tr, G_run, done);
            __syncwarp();
            // ---- lane j: the sums of instance j over its (up to) four pixels, in a fixed order
            if (pixels) {
                const int qx = __float2int_rd(own.x - 0.5f) - px0, qy = __float2int_rd(own.y - 0.5f) - py0;
                const float4 in01 = sm.slots.in[lane][0], in23 = sm.slots.in[lane][1], out01 = sm.slots.out[lane][0], out23 = sm.slots.out[lane][1];
                const float al[4] = {in01.x, in01.z, in23.x, in23.z}, G[4] = {in01.y, in01.w, in23.y, in23.w};
                const float met[4] = {out01.x, out01.z, out23.x, out23.z}, S[4] = {out01.y, out01.w, out23.y, out23.w};
                const float w[4] = {wg.x, wg.y, wg.z, wg.w};
                float bw[4], so = 0.0f;
                bool any = false;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    // (no feature gradient from a weight that is not positive: a negative opacity, or not a number)
                    const float b = met[q] * al[q];
                    bw[q] = b > 0.0f ? b : 0.0f;
                    any = any || bw[q] != 0.0f;
                    if (met[q] != 0.0f) so += (met[q] * G[q] + S[q] * (1.0f / fmaxf(1.0f - al[q], kOneMinusAlphaEps))) * w[q];
                }
                const bool alone = qx >= 0 && qx < 7 && qy >= 0 && qy < 3;   // all four pixels in this half
                if (any) {
                    float4* dst = grad_rows + (size_t)id_cur * C4;
#pragma unroll
                    for (int c = 0; c < C4; ++c) {
                        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            if (bw[q] != 0.0f) {
                                const float4 v = sm.pixel_grad[pix[q] * kStride + c];
                                sum.x += bw[q] * v.x; sum.y += bw[q] * v.y; sum.z += bw[q] * v.z; sum.w += bw[q] * v.w;
                            }
                        }
                        if (alone) dst[c] = sum;
                        else if (sum.x != 0.0f || sum.y != 0.0f || sum.z != 0.0f || sum.w != 0.0f) atomicAdd(dst + c, sum);
                    }
                }
                if (so != 0.0f) {
                    if (alone) grad_opacity[id_cur] = so;
                    else atomicAdd(grad_opacity + id_cur, so);
                }
            }
            done_w = __ballot_sync(kFull, done);
            __syncwarp();
            if (done_w == kFull) break;
        }
        async_copy_wait<0>();   // whatever is still travelling lands before the next item reuses the ring
        __syncwarp();
    }
}

// ------------------------------------------------------------------------------------------------
// Bilinear blend over feature rows: every point carries C = 4 * C4 fp32 channels in the caller's
// (n, C) array and they are blended as they are, into a (C, H, W) image.  The walk, the stopping
// rule and the segment composition are those of the kernels above (src/bilinear/kernels.cu:241-420
// with the channel count as a parameter); the reference itself only has the 36-half -> 4-channel
// layout.  The transmittance pre-pass and the per-tile prefix do not look at features and are
// shared.  One instance per pixel thread and batch.
// ------------------------------------------------------------------------------------------------
template <int T, int C4>
constexpr size_t rows_forward_smem_bytes() {
    return (size_t)T * T * (16 + 16 * C4 + 4 * 4) + (size_t)(T * T / 32) * T * T * 4;
}

template <int T, int C4, int KIND>
__global__ void __launch_bounds__(T * T) blend_rows_forward_kernel(
    const Segment* __restrict__ segs, const uint32_t* __restrict__ n_segments, const uint32_t* __restrict__ inst_ids,
    const PointRec* __restrict__ rec, const float4* __restrict__ features, float* __restrict__ seg_T,
    float4* __restrict__ seg_C, float* __restrict__ seg_Z, float* __restrict__ image, float* __restrict__ depth_image,
    float* __restrict__ alpha_image, float* __restrict__ blending_weights, int width, int height, int gw) {
    await_previous_kernel();
    constexpr int P = T * T;
    constexpr int WORDS = P / 32;
    if (blockIdx.x >= *n_segments) return;
    const Segment sg = segs[blockIdx.x];
    const unsigned seg_idx = sg.info & 0xffffu, n_seg = sg.info >> 16;

    extern __shared__ __align__(16) unsigned char blend_smem[];
    float4* s_a = reinterpret_cast<float4*>(blend_smem);                        // [P]
    float4* s_f = s_a + P;                                                      // [C4][P]
    float* s_slot = reinterpret_cast<float*>(s_f + C4 * P);                     // [4][P] blending weight per footprint corner
    unsigned (*s_mask)[P] = reinterpret_cast<unsigned (*)[P]>(s_slot + 4 * P);  // [WORDS][P]

    const int t = threadIdx.x;
    const int tx = (int)(sg.tile % (unsigned)gw), ty = (int)(sg.tile / (unsigned)gw);
    const int px = tx * T + t % T, py = ty * T + t / T;
    const bool inside = px < width && py < height;
    const float pcx = (float)px + 0.5f, pcy = (float)py + 0.5f;
    const size_t state_idx = (size_t)blockIdx.x * P + t;

#pragma unroll
    for (int w = 0; w < WORDS; ++w) s_mask[w][t] = 0u;
#pragma unroll
    for (int q = 0; q < 4; ++q) s_slot[q * P + t] = 0.0f;
    float4 acc[C4];
#pragma unroll
    for (int c = 0; c < C4; ++c) acc[c] = make_float4(0.f, 0.f, 0.f, 0.f);
    float Z = 0.0f, Tr = 1.0f;
    if (seg_idx > 0u && inside) Tr = seg_T[state_idx];
    bool done = !inside || Tr < kTransmittanceEps;
    __syncthreads();

    uint32_t id = 0;
    int cnt = 0;
    auto flush_weights = [&]() {
        if (t < cnt) {
            const float sum = ((s_slot[t] + s_slot[P + t]) + s_slot[2 * P + t]) + s_slot[3 * P + t];
            if (sum > 0.0f) atomicAdd(blending_weights + id, sum);
            s_slot[t] = 0.0f; s_slot[P + t] = 0.0f; s_slot[2 * P + t] = 0.0f; s_slot[3 * P + t] = 0.0f;
        }
    };
    for (unsigned base = sg.begin; base < sg.end; base += P) {
        if (KIND == BLEND_TRAIN) flush_weights();
        cnt = (int)min((unsigned)P, sg.end - base);
        id = stage_instance<T, P, false>(t, cnt, base, inst_ids, rec, tx, ty, s_a, nullptr, s_mask);
        if (t < cnt) {
            const float4* row = features + (size_t)id * C4;
#pragma unroll
            for (int c = 0; c < C4; ++c) s_f[c * P + t] = __ldg(row + c);
        }
        __syncthreads();
#pragma unroll 1
        for (int w = 0; w < WORDS; ++w) {
            unsigned mbits = s_mask[w][t];
            if (mbits) s_mask[w][t] = 0u;
            while (mbits && !done) {
                const int j = w * 32 + __ffs(mbits) - 1;
                mbits &= mbits - 1u;
                const float4 a = s_a[j];
                const float dx = fabsf(a.x - pcx), dy = fabsf(a.y - pcy);
                if (dx >= 1.0f || dy >= 1.0f) continue;
                const float wgt = __saturatef(1.0f - dx) * __saturatef(1.0f - dy);
                const float al = rounded_alpha(a.z, wgt);
                const float bw = Tr * al;
                if (KIND == BLEND_TRAIN) {
                    if (bw > 0.0f) s_slot[((pcx > a.x ? 1 : 0) + (pcy > a.y ? 2 : 0)) * P + j] = bw * wgt;
                }
#pragma unroll
                for (int c = 0; c < C4; ++c) {
                    const float4 f = s_f[c * P + j];
                    acc[c].x += bw * f.x; acc[c].y += bw * f.y; acc[c].z += bw * f.z; acc[c].w += bw * f.w;
                }
                if (KIND == BLEND_INFER) Z += bw * a.w;
                Tr *= 1.0f - al;
                if (Tr < kTransmittanceEps) done = true;
            }
        }
        if (__syncthreads_count(done) == P) break;
    }
    if (KIND == BLEND_TRAIN) flush_weights();

    if (n_seg == 1u) {
        if (inside) {
            const int64_t n_px = (int64_t)width * height;
            const int64_t pi = (int64_t)py * width + px;
#pragma unroll
            for (int c = 0; c < C4; ++c) {
                image[(4 * c) * n_px + pi] = acc[c].x;
                image[(4 * c + 1) * n_px + pi] = acc[c].y;
                image[(4 * c + 2) * n_px + pi] = acc[c].z;
                image[(4 * c + 3) * n_px + pi] = acc[c].w;
            }
            if (KIND == BLEND_INFER) {
                const float A = 1.0f - Tr;
                depth_image[pi] = A > 0.0f ? Z / A : 0.0f;
                alpha_image[pi] = Tr < kTransmittanceEps ? 1.0f : A;
            } else {
                alpha_image[pi] = Tr < kTransmittanceEps ? 1.0f : 1.0f - Tr;
            }
        }
    } else {
#pragma unroll
        for (int c = 0; c < C4; ++c) seg_C[((size_t)blockIdx.x * C4 + c) * P + t] = acc[c];
        if (KIND == BLEND_INFER) {
            seg_Z[state_idx] = Z;
            seg_T[state_idx] = Tr;
        } else if (seg_idx == n_seg - 1u && inside) {
            alpha_image[(int64_t)py * width + px] = Tr < kTransmittanceEps ? 1.0f : 1.0f - Tr;
        }
    }
}

// Per tile with several segments, feature-row layout: image = sum of the segment colours in order;
// for training the running sum before each segment replaces the segment's own colour.
template <int T, int C4, int KIND>
__global__ void __launch_bounds__(T * T) blend_rows_combine_kernel(const Segment* __restrict__ segs, const uint32_t* __restrict__ tile_first,
                                                                   float4* __restrict__ seg_C, const float* __restrict__ seg_Z,
                                                                   const float* __restrict__ seg_T, float* __restrict__ image,
                                                                   float* __restrict__ depth_image, float* __restrict__ alpha_image,
                                                                   int width, int height, int gw) {
    await_previous_kernel();
    constexpr int P = T * T;
    const unsigned first = tile_first[blockIdx.x];
    const unsigned n_seg = segs[first].info >> 16;
    if (n_seg == 1u) return;
    const int t = threadIdx.x;
    const int tx = (int)(blockIdx.x % (unsigned)gw), ty = (int)(blockIdx.x / (unsigned)gw);
    const int px = tx * T + t % T, py = ty * T + t / T;
    const bool inside = px < width && py < height;
    const int64_t n_px = (int64_t)width * height;
    const int64_t pi = (int64_t)py * width + px;
#pragma unroll 1
    for (int c = 0; c < C4; ++c) {
        float4 run = make_float4(0.f, 0.f, 0.f, 0.f);
        for (unsigned s = 0; s < n_seg; ++s) {
            float4* slot = seg_C + ((size_t)(first + s) * C4 + c) * P + t;
            const float4 v = *slot;
            if (KIND == BLEND_TRAIN) *slot = run;
            run.x += v.x; run.y += v.y; run.z += v.z; run.w += v.w;
        }
        if (inside) {
            image[(4 * c) * n_px + pi] = run.x;
            image[(4 * c + 1) * n_px + pi] = run.y;
            image[(4 * c + 2) * n_px + pi] = run.z;
            image[(4 * c + 3) * n_px + pi] = run.w;
        }
    }
    if (KIND == BLEND_INFER) {
        float z = 0.0f, t_final = 1.0f;
        bool stopped = false;
        for (unsigned s = 0; s < n_seg; ++s) {
            z += seg_Z[(size_t)(first + s) * P + t];
            if (!stopped) {
                t_final = seg_T[(size_t)(first + s) * P + t];
                stopped = t_final < kTransmittanceEps;
            }
        }
        if (inside) {
            const float A = 1.0f - t_final;
            depth_image[pi] = A > 0.0f ? z / A : 0.0f;
            alpha_image[pi] = t_final < kTransmittanceEps ? 1.0f : A;
        }
    }
}

template <int T, int C4>
constexpr size_t rows_backward_smem_bytes() {
    return (size_t)T * T * (16 + 16 * C4 + 16 * C4 + 4 * 4 + 4 * 4) + (size_t)(T * T / 32) * T * T * 4;
}

// Backward over feature rows.  Per fragment only scalars are kept: with G = <g, .> over the channels,
// dL/dalpha = Tr * G(f) + (G(C_run) - G(C_final)) / (1 - alpha) + K / (1 - alpha), and G(C_run) is a
// running scalar.  The blending weight of each (instance, footprint corner) goes to a shared-memory
// slot; the thread that staged the instance then forms sum_corner bw * g(pixel of that corner) from
// the tile's pixel gradients in shared memory and issues one vector atomic per four channels.
template <int T, int C4>
__global__ void __launch_bounds__(T * T) blend_rows_backward_kernel(
    const Segment* __restrict__ segs, const uint32_t* __restrict__ n_segments, const uint32_t* __restrict__ inst_ids,
    const PointRec* __restrict__ rec, const float4* __restrict__ features, const float* __restrict__ seg_T,
    const float4* __restrict__ seg_C, const float* __restrict__ grad_image, const float* __restrict__ grad_alpha,
    const float* __restrict__ image, const float* __restrict__ alpha_image, float4* __restrict__ grad_features,
    float* __restrict__ grad_opacity, int width, int height, int gw) {
    await_previous_kernel();
    constexpr int P = T * T;
    constexpr int WORDS = P / 32;
    if (blockIdx.x >= *n_segments) return;
    const Segment sg = segs[blockIdx.x];
    const unsigned seg_idx = sg.info & 0xffffu;
    if (sg.begin == sg.end) return;

    extern __shared__ __align__(16) unsigned char blend_smem[];
    float4* s_a = reinterpret_cast<float4*>(blend_smem);                      // [P]
    float4* s_f = s_a + P;                                                    // [C4][P] staged feature rows
    float4* s_g = s_f + C4 * P;                                               // [C4][P] image gradient of the tile's pixels
    float* s_bw = reinterpret_cast<float*>(s_g + C4 * P);                     // [4][P]
    float* s_go = s_bw + 4 * P;                                               // [4][P]
    unsigned (*s_mask)[P] = reinterpret_cast<unsigned (*)[P]>(s_go + 4 * P);  // [WORDS][P]

    const int t = threadIdx.x;
    const int tx = (int)(sg.tile % (unsigned)gw), ty = (int)(sg.tile / (unsigned)gw);
    const int px = tx * T + t % T, py = ty * T + t / T;
    const bool inside = px < width && py < height;
    const float pcx = (float)px + 0.5f, pcy = (float)py + 0.5f;
    const size_t state_idx = (size_t)blockIdx.x * P + t;

#pragma unroll
    for (int w = 0; w < WORDS; ++w) s_mask[w][t] = 0u;
#pragma unroll
    for (int q = 0; q < 4; ++q) { s_bw[q * P + t] = 0.0f; s_go[q * P + t] = 0.0f; }

    float4 g[C4];
    float G_final = 0.0f, G_run = 0.0f, K = 0.0f, Tr = 1.0f;
#pragma unroll
    for (int c = 0; c < C4; ++c) g[c] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (inside) {
        const int64_t n_px = (int64_t)width * height;
        const int64_t pi = (int64_t)py * width + px;
#pragma unroll
        for (int c = 0; c < C4; ++c) {
            g[c] = make_float4(__ldg(grad_image + (4 * c) * n_px + pi), __ldg(grad_image + (4 * c + 1) * n_px + pi),
                               __ldg(grad_image + (4 * c + 2) * n_px + pi), __ldg(grad_image + (4 * c + 3) * n_px + pi));
            G_final += __ldg(image + (4 * c) * n_px + pi) * g[c].x + __ldg(image + (4 * c + 1) * n_px + pi) * g[c].y +
                       __ldg(image + (4 * c + 2) * n_px + pi) * g[c].z + __ldg(image + (4 * c + 3) * n_px + pi) * g[c].w;
        }
        K = __ldg(grad_alpha + pi) * (1.0f - __ldg(alpha_image + pi));
        if (seg_idx > 0u) {
            Tr = seg_T[state_idx];
#pragma unroll
            for (int c = 0; c < C4; ++c) {
                const float4 v = seg_C[((size_t)blockIdx.x * C4 + c) * P + t];
                G_run += v.x * g[c].x + v.y * g[c].y + v.z * g[c].z + v.w * g[c].w;
            }
        }
    }
#pragma unroll
    for (int c = 0; c < C4; ++c) s_g[c * P + t] = g[c];
    bool done = !inside || Tr < kTransmittanceEps;
    __syncthreads();

    uint32_t id = 0;
    int cnt = 0;
    auto flush_gradients = [&]() {
        if (t < cnt) {
            const float4 a = s_a[t];
            const int qx = __float2int_rd(a.x - 0.5f) - tx * T;
            const int qy = __float2int_rd(a.y - 0.5f) - ty * T;
            float bw[4];
            float so = 0.0f;
            bool any = false;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                bw[q] = s_bw[q * P + t];
                so += s_go[q * P + t];
                any = any || bw[q] != 0.0f;
                s_bw[q * P + t] = 0.0f;
                s_go[q * P + t] = 0.0f;
            }
            if (any) {
                // a corner slot is only ever written by the pixel thread of that corner, so a filled
                // slot names a pixel of this tile
                float4* dst = grad_features + (size_t)id * C4;
#pragma unroll
                for (int c = 0; c < C4; ++c) {
                    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        if (bw[q] != 0.0f) {
                            const float4 v = s_g[c * P + (qy + (q >> 1)) * T + qx + (q & 1)];
                            sum.x += bw[q] * v.x; sum.y += bw[q] * v.y; sum.z += bw[q] * v.z; sum.w += bw[q] * v.w;
                        }
                    }
                    if (sum.x != 0.0f || sum.y != 0.0f || sum.z != 0.0f || sum.w != 0.0f) atomicAdd(dst + c, sum);
                }
            }
            if (so != 0.0f) atomicAdd(grad_opacity + id, so);
        }
    };
    for (unsigned base = sg.begin; base < sg.end; base += P) {
        flush_gradients();
        cnt = (int)min((unsigned)P, sg.end - base);
        id = stage_instance<T, P, false>(t, cnt, base, inst_ids, rec, tx, ty, s_a, nullptr, s_mask);
        if (t < cnt) {
            const float4* row = features + (size_t)id * C4;
#pragma unroll
            for (int c = 0; c < C4; ++c) s_f[c * P + t] = __ldg(row + c);
        }
        __syncthreads();
#pragma unroll 1
        for (int w = 0; w < WORDS; ++w) {
            unsigned mbits = s_mask[w][t];
            if (mbits) s_mask[w][t] = 0u;
            while (mbits && !done) {
                const int j = w * 32 + __ffs(mbits) - 1;
                mbits &= mbits - 1u;
                const float4 a = s_a[j];
                const float dx = fabsf(a.x - pcx), dy = fabsf(a.y - pcy);
                if (dx >= 1.0f || dy >= 1.0f) continue;
                const float wgt = __saturatef(1.0f - dx) * __saturatef(1.0f - dy);
                const float al = rounded_alpha(a.z, wgt);
                const float bw = Tr * al;
                const int q = (pcx > a.x ? 1 : 0) + (pcy > a.y ? 2 : 0);
                if (bw > 0.0f) s_bw[q * P + j] = bw;
                float fg = 0.0f;
#pragma unroll
                for (int c = 0; c < C4; ++c) {
                    const float4 f = s_f[c * P + j];
                    fg += f.x * g[c].x + f.y * g[c].y + f.z * g[c].z + f.w * g[c].w;
                }
                G_run += bw * fg;
                const float oma = 1.0f - al;
                const float rcp = 1.0f / fmaxf(oma, kOneMinusAlphaEps);
                const float dalpha = Tr * fg + (G_run - G_final) * rcp + K * rcp;
                const float dop = dalpha * wgt;
                if (dop != 0.0f) s_go[q * P + j] = dop;
                Tr *= oma;
                if (Tr < kTransmittanceEps) done = true;
            }
        }
        if (__syncthreads_count(done) == P) break;
    }
    flush_gradients();
}

// ------------------------------------------------------------------------------------------------
// Gaussian blend on 16x16 tiles (src/gaussian/kernels.cu:401-474 forward, :476-579 backward, :581-660 inference).
// A footprint is an ellipse of a few pixels, not a fixed 2x2: the staging thread sets its instance's bit
// for the pixels of the ellipse's bounding box inside the tile (slightly widened, so a superset of the
// pixels that pass the reference's tests), and every pixel thread walks only its set bits and applies
// the reference's tests and arithmetic unchanged.  Per-point sums (blending weight, gradients) are
// accumulated with shared-memory atomics per staged instance and leave with one global atomic per
// instance (the reference issues global atomics per fragment).
// ------------------------------------------------------------------------------------------------
template <int T>
__device__ __forceinline__ void gaussian_mask_bits(int j, const float4& a, const float4& c, float neg_log_threshold, int tile_x, int tile_y,
                                                   unsigned (*s_mask)[T * T]) {
    // points with  -0.5 d^T Conic d >= -L  lie within |dx| <= sqrt(2 L cov_xx), |dy| <= sqrt(2 L cov_yy),
    // cov = Conic^-1
    const float det = c.x * c.z - c.y * c.y;
    int x0 = 0, x1 = T - 1, y0 = 0, y1 = T - 1;
    if (det > 0.0f) {
        const float s = 2.0f * neg_log_threshold / det;
        const float rx = sqrtf(fmaxf(s * c.z, 0.0f)) * 1.001f + 0.01f;
        const float ry = sqrtf(fmaxf(s * c.x, 0.0f)) * 1.001f + 0.01f;
        // (an ellipse that reaches beyond the integers, as with a cut-off whose threshold underflows to zero, must not wrap round)
        constexpr float kFar = 1e9f;
        x0 = max(0, __float2int_ru(fmaxf(a.x - rx - 0.5f, -kFar)) - tile_x * T);
        x1 = min(T - 1, __float2int_rd(fminf(a.x + rx - 0.5f, kFar)) - tile_x * T);
        y0 = max(0, __float2int_ru(fmaxf(a.y - ry - 0.5f, -kFar)) - tile_y * T);
        y1 = min(T - 1, __float2int_rd(fminf(a.y + ry - 0.5f, kFar)) - tile_y * T);
    }
    const unsigned bit = 1u << (j & 31);
    unsigned* mrow = s_mask[j >> 5];
    for (int y = y0; y <= y1; ++y)
        for (int x = x0; x <= x1; ++x) atomicOr(mrow + y * T + x, bit);
}

// Pass 1 of the segmented gaussian blend (tiles with several segments only): per-pixel product of
// (1 - alpha) over one segment; FAST selects the exponential of the inference kernels.
template <int T, bool FAST>
__global__ void __launch_bounds__(T * T) blend_gaussian_transmittance_kernel(
    const Segment* __restrict__ segs, const uint32_t* __restrict__ n_segments, const uint32_t* __restrict__ inst_ids,
    const PointRec* __restrict__ rec, const float4* __restrict__ conic, float* __restrict__ seg_T, int width, int height, int gw,
    float threshold, float neg_log_threshold) {
    await_previous_kernel();
    constexpr int B = T * T;
    constexpr int WORDS = B / 32;
    if (blockIdx.x >= *n_segments) return;
    const Segment sg = segs[blockIdx.x];
    const unsigned seg_idx = sg.info & 0xffffu, n_seg = sg.info >> 16;
    if (n_seg == 1u || seg_idx == n_seg - 1u) return;
    __shared__ float4 s_a[B];
    __shared__ float4 s_c[B];
    __shared__ unsigned s_mask[WORDS][B];
    const int t = threadIdx.x;
    const int tx = (int)(sg.tile % (unsigned)gw), ty = (int)(sg.tile / (unsigned)gw);
    const int px = tx * T + t % T, py = ty * T + t / T;
    const float pcx = (float)px + 0.5f, pcy = (float)py + 0.5f;
#pragma unroll
    for (int w = 0; w < WORDS; ++w) s_mask[w][t] = 0u;
    float Tr = 1.0f;
    bool done = !(px < width && py < height);
    for (unsigned base = sg.begin; base < sg.end; base += B) {
        if (__syncthreads_count(done) == B) break;
        const int cnt = (int)min((unsigned)B, sg.end - base);
        if (t < cnt) {
            const uint32_t id = checked_point(__ldg(inst_ids + base + t));
            const float4 a = __ldg(reinterpret_cast<const float4*>(rec + id));
            const float4 c = __ldg(conic + id);
            s_a[t] = a;
            s_c[t] = c;
            gaussian_mask_bits<T>(t, a, c, neg_log_threshold, tx, ty, s_mask);
        }
        __syncthreads();
#pragma unroll 1
        for (int w = 0; w < WORDS; ++w) {
            unsigned mbits = s_mask[w][t];
            if (mbits) s_mask[w][t] = 0u;
            while (mbits && !done) {
                const int j = w * 32 + __ffs(mbits) - 1;
                mbits &= mbits - 1u;
                const float4 a = s_a[j];
                const float4 c = s_c[j];
                const float dx = a.x - pcx, dy = a.y - pcy;
                const float e = -0.5f * (c.x * dx * dx + c.z * dy * dy) - c.y * dx * dy;
                if (e > 0.0f) continue;
                const float G = FAST ? __expf(e) : expf(e);
                if (G < threshold) continue;
                Tr *= 1.0f - rounded_alpha(a.z, G);
                if (Tr < kTransmittanceEps) done = true;
            }
        }
    }
    seg_T[(size_t)blockIdx.x * B + t] = Tr;
}

// Main pass: one block per (tile, segment), starting from the segment's incoming transmittance.
template <int T, int KIND>
__global__ void __launch_bounds__(T * T) blend_gaussian_forward_kernel(
    const Segment* __restrict__ segs, const uint32_t* __restrict__ n_segments, const uint32_t* __restrict__ inst_ids,
    const PointRec* __restrict__ rec, const float4* __restrict__ conic, float* __restrict__ seg_T, float4* __restrict__ seg_C,
    float* __restrict__ seg_Z, float* __restrict__ image, float* __restrict__ depth_image,
    float* __restrict__ alpha_image, float* __restrict__ blending_weights, int width, int height, int gw,
    float threshold, float neg_log_threshold) {
    await_previous_kernel();
    constexpr int B = T * T;
    constexpr int WORDS = B / 32;
    if (blockIdx.x >= *n_segments) return;
    const Segment sg = segs[blockIdx.x];
    const unsigned seg_idx = sg.info & 0xffffu, n_seg = sg.info >> 16;
    __shared__ float4 s_a[B];
    __shared__ float4 s_f[B];
    __shared__ float4 s_c[B];
    __shared__ uint32_t s_id[B];
    __shared__ unsigned s_mask[WORDS][B];
    __shared__ float s_bw[KIND == BLEND_TRAIN ? B : 1];
    const int t = threadIdx.x;
    const int tx = (int)(sg.tile % (unsigned)gw), ty = (int)(sg.tile / (unsigned)gw);
    const int px = tx * T + t % T, py = ty * T + t / T;
    const bool inside = px < width && py < height;
    const float pcx = (float)px + 0.5f, pcy = (float)py + 0.5f;
    const size_t state_idx = (size_t)blockIdx.x * B + t;
#pragma unroll
    for (int w = 0; w < WORDS; ++w) s_mask[w][t] = 0u;
    if (KIND == BLEND_TRAIN) s_bw[t] = 0.0f;
    float C0 = 0.f, C1 = 0.f, C2 = 0.f, C3 = 0.f, Z = 0.f, Tr = 1.0f;
    if (seg_idx > 0u && inside) Tr = seg_T[state_idx];
    bool done = !inside || Tr < kTransmittanceEps;
    int cnt = 0;
    auto flush_weights = [&]() {
        if (t < cnt) {
            const float sum = s_bw[t];
            if (sum > 0.0f) atomicAdd(blending_weights + s_id[t], sum);
            s_bw[t] = 0.0f;
        }
    };
    for (unsigned base = sg.begin; base < sg.end; base += B) {
        if (__syncthreads_count(done) == B) break;     // also: every thread has finished the batch before
        if (KIND == BLEND_TRAIN) flush_weights();
        cnt = (int)min((unsigned)B, sg.end - base);
        if (t < cnt) {
            const uint32_t id = checked_point(__ldg(inst_ids + base + t));
            const float4* r = reinterpret_cast<const float4*>(rec + id);
            const float4 a = __ldg(r);
            const float4 c = __ldg(conic + id);
            s_a[t] = a;
            s_f[t] = __ldg(r + 1);
            s_c[t] = c;
            s_id[t] = id;
            gaussian_mask_bits<T>(t, a, c, neg_log_threshold, tx, ty, s_mask);
        }
        __syncthreads();
#pragma unroll 1
        for (int w = 0; w < WORDS; ++w) {
            unsigned mbits = s_mask[w][t];
            if (mbits) s_mask[w][t] = 0u;
            while (mbits && !done) {
                const int j = w * 32 + __ffs(mbits) - 1;
                mbits &= mbits - 1u;
                const float4 a = s_a[j];
                const float4 c = s_c[j];
                const float dx = a.x - pcx, dy = a.y - pcy;
                const float e = -0.5f * (c.x * dx * dx + c.z * dy * dy) - c.y * dx * dy;
                if (e > 0.0f) continue;
                const float G = KIND == BLEND_INFER ? __expf(e) : expf(e);
                if (G < threshold) continue;
                const float al = rounded_alpha(a.z, G);
                const float bw = Tr * al;
                if (KIND == BLEND_TRAIN) {
                    if (bw > 0.0f) atomicAdd(&s_bw[j], G * bw);
                }
                const float4 f = s_f[j];
                C0 += bw * f.x; C1 += bw * f.y; C2 += bw * f.z; C3 += bw * f.w;
                if (KIND == BLEND_INFER) Z += bw * a.w;
                Tr *= 1.0f - al;
                if (Tr < kTransmittanceEps) done = true;
            }
        }
    }
    if (KIND == BLEND_TRAIN) {
        __syncthreads();
        flush_weights();
    }
    if (n_seg == 1u) {
        if (inside) {
            const int64_t n_px = (int64_t)width * height;
            const int64_t pi = (int64_t)py * width + px;
            image[pi] = C0;
            image[n_px + pi] = C1;
            image[2 * n_px + pi] = C2;
            image[3 * n_px + pi] = C3;
            if (KIND == BLEND_INFER) {
                const float A = 1.0f - Tr;
                depth_image[pi] = A > 0.0f ? Z / A : 0.0f;
                alpha_image[pi] = Tr < kTransmittanceEps ? 1.0f : A;
            } else {
                alpha_image[pi] = Tr < kTransmittanceEps ? 1.0f : 1.0f - Tr;
            }
        }
    } else {
        seg_C[state_idx] = make_float4(C0, C1, C2, C3);
        if (KIND == BLEND_INFER) {
            seg_Z[state_idx] = Z;
            seg_T[state_idx] = Tr;
        } else if (seg_idx == n_seg - 1u && inside) {
            alpha_image[(int64_t)py * width + px] = Tr < kTransmittanceEps ? 1.0f : 1.0f - Tr;
        }
    }
}

template <int T>
__global__ void __launch_bounds__(T * T) blend_gaussian_backward_kernel(
    const Segment* __restrict__ segs, const uint32_t* __restrict__ n_segments, const uint32_t* __restrict__ inst_ids,
    const PointRec* __restrict__ rec, const float4* __restrict__ conic, const float* __restrict__ seg_T,
    const float4* __restrict__ seg_C, const float* __restrict__ grad_image, const float* __restrict__ grad_alpha,
    const float* __restrict__ image, const float* __restrict__ alpha_image, float4* __restrict__ grad_feat_view,
    float* __restrict__ grad_opacity, int width, int height, int gw) {
    await_previous_kernel();
    constexpr int B = T * T;
    constexpr int WORDS = B / 32;
    if (blockIdx.x >= *n_segments) return;
    const Segment sg = segs[blockIdx.x];
    const unsigned seg_idx = sg.info & 0xffffu;
    if (sg.begin == sg.end) return;
    __shared__ float4 s_a[B];
    __shared__ float4 s_f[B];
    __shared__ float4 s_c[B];
    __shared__ uint32_t s_id[B];
    __shared__ unsigned s_mask[WORDS][B];
    __shared__ float s_gf[4][B];   // per staged instance: view-space feature gradient ...
    __shared__ float s_go[B];      // ... and opacity gradient, summed with shared-memory atomics
    const int t = threadIdx.x;
    const int tx = (int)(sg.tile % (unsigned)gw), ty = (int)(sg.tile / (unsigned)gw);
    const size_t state_idx = (size_t)blockIdx.x * B + t;
    const int px = tx * T + t % T, py = ty * T + t / T;
    const bool inside = px < width && py < height;
    const float pcx = (float)px + 0.5f, pcy = (float)py + 0.5f;
#pragma unroll
    for (int w = 0; w < WORDS; ++w) s_mask[w][t] = 0u;
#pragma unroll
    for (int q = 0; q < 4; ++q) s_gf[q][t] = 0.0f;
    s_go[t] = 0.0f;
    float4 g = make_float4(0.f, 0.f, 0.f, 0.f), Cfin = make_float4(0.f, 0.f, 0.f, 0.f);
    float K = 0.0f;
    if (inside) {
        const int64_t n_px = (int64_t)width * height;
        const int64_t pi = (int64_t)py * width + px;
        g = make_float4(__ldg(grad_image + pi), __ldg(grad_image + n_px + pi), __ldg(grad_image + 2 * n_px + pi),
                        __ldg(grad_image + 3 * n_px + pi));
        Cfin = make_float4(__ldg(image + pi), __ldg(image + n_px + pi), __ldg(image + 2 * n_px + pi),
                           __ldg(image + 3 * n_px + pi));
        K = __ldg(grad_alpha + pi) * (1.0f - __ldg(alpha_image + pi));
    }
    float4 Crun = make_float4(0.f, 0.f, 0.f, 0.f);
    float Tr = 1.0f;
    if (inside && seg_idx > 0u) { Tr = seg_T[state_idx]; Crun = seg_C[state_idx]; }
    bool done = !inside || Tr < kTransmittanceEps;
    int cnt = 0;
    auto flush_gradients = [&]() {
        if (t < cnt) {
            const float4 sf = make_float4(s_gf[0][t], s_gf[1][t], s_gf[2][t], s_gf[3][t]);
            const float so = s_go[t];
            const uint32_t id = s_id[t];
            if (sf.x != 0.0f || sf.y != 0.0f || sf.z != 0.0f || sf.w != 0.0f) atomicAdd(grad_feat_view + id, sf);
            if (so != 0.0f) atomicAdd(grad_opacity + id, so);
            s_gf[0][t] = 0.0f; s_gf[1][t] = 0.0f; s_gf[2][t] = 0.0f; s_gf[3][t] = 0.0f;
            s_go[t] = 0.0f;
        }
    };
    constexpr float kNegLogThreshold = 4.5f;   // -ln(kTrainGaussThreshold)
    for (unsigned base = sg.begin; base < sg.end; base += B) {
        if (__syncthreads_count(done) == B) break;
        flush_gradients();
        cnt = (int)min((unsigned)B, sg.end - base);
        if (t < cnt) {
            const uint32_t id = checked_point(__ldg(inst_ids + base + t));
            const float4* r = reinterpret_cast<const float4*>(rec + id);
            const float4 a = __ldg(r);
            const float4 c = __ldg(conic + id);
            s_a[t] = a;
            s_f[t] = __ldg(r + 1);
            s_c[t] = c;
            s_id[t] = id;
            gaussian_mask_bits<T>(t, a, c, kNegLogThreshold, tx, ty, s_mask);
        }
        __syncthreads();
#pragma unroll 1
        for (int w = 0; w < WORDS; ++w) {
            unsigned mbits = s_mask[w][t];
            if (mbits) s_mask[w][t] = 0u;
            while (mbits && !done) {
                const int j = w * 32 + __ffs(mbits) - 1;
                mbits &= mbits - 1u;
                const float4 a = s_a[j];
                const float4 c = s_c[j];
                const float dx = a.x - pcx, dy = a.y - pcy;
                const float e = -0.5f * (c.x * dx * dx + c.z * dy * dy) - c.y * dx * dy;
                if (e > 0.0f) continue;
                const float G = expf(e);
                if (G < kTrainGaussThreshold) continue;
                const float al = rounded_alpha(a.z, G);
                const float bw = Tr * al;
                if (bw > 0.0f) {
                    atomicAdd(&s_gf[0][j], bw * g.x); atomicAdd(&s_gf[1][j], bw * g.y);
                    atomicAdd(&s_gf[2][j], bw * g.z); atomicAdd(&s_gf[3][j], bw * g.w);
                }
                const float4 f = s_f[j];
                Crun.x += bw * f.x; Crun.y += bw * f.y; Crun.z += bw * f.z; Crun.w += bw * f.w;
                const float oma = 1.0f - al;
                const float rcp = 1.0f / fmaxf(oma, kOneMinusAlphaEps);
                const float from_features = (Tr * f.x + (Crun.x - Cfin.x) * rcp) * g.x +
                                            (Tr * f.y + (Crun.y - Cfin.y) * rcp) * g.y +
                                            (Tr * f.z + (Crun.z - Cfin.z) * rcp) * g.z +
                                            (Tr * f.w + (Crun.w - Cfin.w) * rcp) * g.w;
                const float dalpha = from_features + K * rcp;
                const float dop = dalpha * G;
                if (dop != 0.0f) atomicAdd(&s_go[j], dop);
                Tr *= oma;
                if (Tr < kTransmittanceEps) done = true;
            }
        }
    }
    __syncthreads();
    flush_gradients();
}

// ------------------------------------------------------------------------------------------------
// Gaussian blend on 8x8 tiles, one warp per work item: the passes, lists and segments of the bilinear warp blend above.
// (Arithmetic per fragment: src/gaussian/kernels.cu:401-474 forward, :476-579 backward, :581-660 inference.)
//
// A footprint is an ellipse instead of 2x2 pixels.  The key says which 2x2-pixel cells of the tile it can reach (a column range
// and a row range, see cell_code), so that dead instances are dropped unread like bilinear ones.  Of a batch of 32 staged
// instances, lane j first finds the pixels of the half inside the ellipse of instance j, row by row and slightly widened (a
// superset of what passes the reference's tests); a 32x32 bit transposition over the warp turns these masks into one word per
// pixel with the instances that reach it, and every lane walks down the set bits of its own pixel.  What a fragment adds to its
// point is left in shared memory, the words of accepted fragments are transposed back, and lane j adds up the sums of
// instance j: no shared-memory floating-point atomics (compare-and-swap loops, five per fragment of the backward pass), one
// global atomic per instance and half.
//
// Bound by the chain of instructions of a batch (masks, transposition, the pixels' lists, the sums) and by the passes draining while
// their longest items finish (6 to 10 of 64 warps of a multiprocessor active on average).  Against one block of 64 threads per
// (tile, segment) that staged every instance: 2^22 samples at 1237x822, forward and backward 1680 -> 990 us; 2 * 10^6 splats
// with sizes at 1297x840, inference 511 -> 200 us.
// ------------------------------------------------------------------------------------------------
// Pixels of the tile (bit = row * 8 + column) in the cells of a code.
__device__ __forceinline__ unsigned long long cell_pixels(unsigned code) {
    if (code >= 100u) return 0ull;
    unsigned c0, c1, r0, r1;
    cell_range(code % 10u, &c0, &c1);
    cell_range(code / 10u, &r0, &r1);
    const unsigned row = ((1u << (2u * c1 + 2u)) - 1u) & ~((1u << (2u * c0)) - 1u);
    unsigned long long m = 0ull;
    for (unsigned y = 2u * r0; y < 2u * r1 + 2u; ++y) m |= (unsigned long long)row << (8u * y);
    return m;
}

// Pixels of the 8x4 half at (px0, py0) (bit = row * 8 + column) that a splat at `a` with conic `c` can reach: a superset of
// those with  c.x dx^2 + 2 c.y dx dy + c.z dy^2 <= reach  (reach = -2 log threshold).  The widening by a thousandth covers what the approximate roots and quotients are off by
// (a few parts in 10^7).
__device__ __forceinline__ float approximate_root(float x) {
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ unsigned ellipse_pixels(const float4& a, const float4& c, float reach, int px0, int py0) {
    const float det = c.x * c.z - c.y * c.y;
    if (!(det > 0.0f)) return 0xffffffffu;   // degenerate (or not a number): the per-pixel tests decide
    const float inv = __fdividef(1.0f, c.x), peak = reach * c.x;
    const float ry = approximate_root(__fdividef(peak, det)) * 1.001f + 0.01f;
    const float x0 = a.x - 0.5f - (float)px0, y0 = a.y - 0.5f - (float)py0;
    unsigned m = 0u;
#pragma unroll
    for (int y = 0; y < 4; ++y) {
        const float dy = y0 - (float)y;
        // the rounding of det of a long ellipse (a thousandth at most) is covered by the widening, as is that of the root
        const float r = approximate_root(fmaxf(peak * 1.002f - det * dy * dy, 0.0f)) * inv * 1.001f + 0.01f;
        const float mid = x0 + c.y * dy * inv;
        const int lo = __float2int_ru(fminf(fmaxf(mid - r, 0.0f), 8.0f)), hi = __float2int_rd(fminf(fmaxf(mid + r, -1.0f), 7.0f));
        if (fabsf(dy) <= ry && lo <= hi) m |= ((2u << hi) - (1u << lo)) << (8 * y);
    }
    return m;
}

// One warp per item: training passes over short lists (see by_two_warps), the products, and all passes of inference, which have less to do per fragment (2^22 splats: products 184 us, 199 with two
// warps; 2 * 10^6 splats of a frame, first segments 151 and 194).
template <bool BLEND, bool WEIGHTS>
struct __align__(16) GaussForwardSmem {
    float4 ring_a[2][32], ring_c[2][32];              // records and conics of the batches in flight
    float4 ring_f[BLEND ? 2 : 1][BLEND ? 32 : 1];     // ... and features
    float out[WEIGHTS ? 32 : 1][33];                  // [staged instance][pixel]: what the fragment adds to the blending weight
    uint32_t ring_id[2][32];
    uint32_t queue[kQueueCap];
};
template <int PASS, int KIND>
constexpr size_t gauss_forward_smem_bytes() {
    return 2 * 256 * sizeof(unsigned) + kWarpBlendWarps * sizeof(GaussForwardSmem<PASS != PASS_PRODUCT, PASS != PASS_PRODUCT && KIND == BLEND_TRAIN>);
}

template <int PASS, int KIND>
__global__ void __launch_bounds__(kWarpBlendWarps * 32, kGaussForwardBlocks) blend_gaussian_warp_forward_kernel(
    const WarpItem* __restrict__ items, const uint32_t* __restrict__ counts, unsigned* __restrict__ ticket, unsigned n_visits, const uint32_t* __restrict__ inst_keys,
    const uint32_t* __restrict__ inst_ids, const PointRec* __restrict__ rec, const float4* __restrict__ conic, float* __restrict__ seg_T,
    float4* __restrict__ seg_C, float* __restrict__ seg_Z, float* __restrict__ seg_E, float* __restrict__ image, float* __restrict__ depth_image,
    float* __restrict__ alpha_image, float* __restrict__ blending_weights, uint32_t* kept0, uint32_t* kept1, uint32_t* __restrict__ n_kept,
    int width, int height, int gw, float threshold, float reach) {
    await_previous_kernel();
    constexpr unsigned kFull = 0xffffffffu;
    constexpr unsigned kNoInstance = 0xffffffffu;
    constexpr bool kBlend = PASS != PASS_PRODUCT;
    constexpr bool kWeights = kBlend && KIND == BLEND_TRAIN;
    constexpr bool kDepth = kBlend && KIND == BLEND_INFER;
    using Smem = GaussForwardSmem<kBlend, kWeights>;
    extern __shared__ __align__(16) unsigned char blend_smem[];
    unsigned* s_reach = reinterpret_cast<unsigned*>(blend_smem);     // [half][key code] -> pixels of the half reached
    Smem& sm = reinterpret_cast<Smem*>(blend_smem + 2 * 256 * sizeof(unsigned))[threadIdx.x >> 5];
    const unsigned lane = lane_id();
    const unsigned lt_mask = (1u << lane) - 1u;
    {
        const unsigned long long m = cell_pixels(threadIdx.x);
        s_reach[threadIdx.x] = (unsigned)m;
        s_reach[256 + threadIdx.x] = (unsigned)(m >> 32);
    }
    __syncthreads();
    const unsigned n_items = __ldg(counts + (PASS == PASS_FIRST ? 0 : 1)) * 2u;
    ItemQueue queue(n_items, PASS == PASS_FIRST ? __ldg(counts + kLongTiles + 1) * 2u : 0u, n_visits, kMostItems);
    unsigned item;
    while (queue.take(ticket, lane, &item)) {
        const WarpItem it = load_item(items + (item >> 1));
        const unsigned tile = it.tile, seg = it.seg, n_seg = it.n_seg, first = it.first;
        const int half = (int)(item & 1u);
        const size_t sidx = (size_t)(first + seg) * 2u + half;      // this item's slot in the per-segment arrays
        const size_t sidx0 = (size_t)first * 2u + half;             // segment 0 of the same tile half
        const uint2 rg = make_uint2(it.begin, it.end);
        const int tx = (int)(tile % (unsigned)gw), ty = (int)(tile / (unsigned)gw);
        const int px0 = tx * 8, py0 = ty * 8 + 4 * half;            // first pixel of this half
        const int px = px0 + (int)(lane & 7u), py = py0 + (int)(lane >> 3);
        const bool inside = px < width && py < height;
        const float pcx = (float)px + 0.5f, pcy = (float)py + 0.5f;

        float Tr = 1.0f, Z = 0.0f, stop = kTransmittanceEps;
        float4 C = make_float4(0.f, 0.f, 0.f, 0.f);
        bool done = !inside;
        if (PASS == PASS_PRODUCT) {
            // product of (1 - alpha) over the segment, until it would carry the state segment 0 left below the threshold; the
            // margin keeps a pixel open when rounding, of this product or of REST's, could be what carries it over the line
            const float T0 = seg_T[sidx0 * 32 + lane];
            done = done || T0 < kTransmittanceEps;
            if (!done) stop = kTransmittanceEps / T0 * (1.0f - stop_margin(rg.y - rg.x));
        } else if (PASS == PASS_REST) {
            Tr = seg_T[sidx * 32 + lane];
            done = done || Tr < kTransmittanceEps;
        }
        unsigned done_w = __ballot_sync(kFull, done);   // bit l = pixel of lane l has stopped (warp-uniform)

        uint32_t* kept = half ? kept1 : kept0;
        unsigned n_out = 0;
        if (done_w != kFull) {
            CandidateStream in;
            const unsigned* reach_of_key = s_reach + 256 * half;
            auto fill = [&]() {
                if (PASS != PASS_REST) in.fill(reach_of_key, done_w, sm.queue, lane, lt_mask);
                __syncwarp();
            };
            uint32_t idf[kIdsAhead];
            if (PASS == PASS_REST) {
                in.head = 0u;
                in.tail = n_kept[sidx];     // length of PRODUCT's list; the list itself starts at kept[rg.x]
#pragma unroll
                for (int k = 0; k < kIdsAhead; ++k) idf[k] = 32u * k + lane < in.tail ? kept[rg.x + 32u * k + lane] : 0u;
            } else {
                in.start(inst_keys, inst_ids, rg.x, rg.y, lane);
            }
            auto gather = [&](unsigned stage) {
                const unsigned n = min(32u, in.tail - in.head);
                uint32_t id = kNoInstance;
                if (lane < n) {
                    id = checked_point(PASS == PASS_REST ? idf[0] : sm.queue[(in.head + lane) & (kQueueCap - 1)]);
                    const float4* p = reinterpret_cast<const float4*>(rec + id);
                    async_copy_16(&sm.ring_a[stage][lane], p);
                    async_copy_16(&sm.ring_c[stage][lane], conic + id);
                    if (kBlend) async_copy_16(&sm.ring_f[stage][lane], p + 1);
                }
                sm.ring_id[stage][lane] = id;
                async_copy_commit();   // one group per batch, empty or not: the waits below count groups
                if (PASS == PASS_REST) {
#pragma unroll
                    for (int k = 0; k + 1 < kIdsAhead; ++k) idf[k] = idf[k + 1];
                    const unsigned nxt = in.head + 32u * kIdsAhead + lane;
                    idf[kIdsAhead - 1] = nxt < in.tail ? kept[rg.x + nxt] : 0u;
                }
                in.head += n;
            };
            fill();
            gather(0u);
            fill();
            for (unsigned batch = 0;; ++batch) {
                gather((batch + 1u) & 1u);
                async_copy_wait<1>();   // all but the newest group: this batch has arrived
                const unsigned stage = batch & 1u;
                const uint32_t id_cur = sm.ring_id[stage][lane];
                const bool staged = id_cur != kNoInstance;
                if (__ballot_sync(kFull, staged) == 0u) break;   // batches are filled in order: nothing is left
                // ---- lane j: the pixels instance j can reach that have not stopped
                unsigned pixels = 0u;
                if (staged) pixels = ellipse_pixels(sm.ring_a[stage][lane], sm.ring_c[stage][lane], reach, px0, py0) & ~done_w;
                fill();   // (its __syncwarp also shows every lane the records the others have copied)
                if (PASS == PASS_PRODUCT || kWeights) {
                    // the list of this item: see the bilinear kernel
                    const unsigned b = __ballot_sync(kFull, pixels != 0u);
                    if (pixels) kept[rg.x + n_out + __popc(b & lt_mask)] = id_cur;
                    n_out += __popc(b);
                }
                // ---- every lane runs down the instances of its own pixel, front to back
                unsigned todo = warp_transpose_bits(pixels, lane);
                unsigned taken = 0u;   // instances whose blending weight this pixel adds to
                while (todo) {
                    // a few at a time: their exponentials do not wait for one another (products, three for two: 188 -> 183 us; the other passes the same or slower)
                    constexpr int kPair = PASS == PASS_PRODUCT ? 3 : 2;
                    int j[kPair];
                    float al[kPair], G[kPair];
                    bool ok[kPair];
#pragma unroll
                    for (int u = 0; u < kPair; ++u) {
                        ok[u] = todo != 0u;
                        j[u] = ok[u] ? __ffs(todo) - 1 : j[0];
                        todo &= todo - 1u;
                        const float4 a = sm.ring_a[stage][j[u]], c = sm.ring_c[stage][j[u]];
                        const float dx = a.x - pcx, dy = a.y - pcy;
                        const float e = -0.5f * (c.x * dx * dx + c.z * dy * dy) - c.y * dx * dy;
                        G[u] = KIND == BLEND_INFER ? __expf(e) : expf(e);
                        ok[u] = ok[u] && !(e > 0.0f) && !(G[u] < threshold);
                        al[u] = rounded_alpha(a.z, G[u]);
                    }
#pragma unroll
                    for (int u = 0; u < kPair; ++u) {
                        if (!ok[u] || done) continue;
                        if (kBlend) {
                            const float bw = Tr * al[u];
                            if (kWeights && bw > 0.0f) {
                                sm.out[j[u]][lane] = G[u] * bw;
                                taken |= 1u << j[u];
                            }
                            const float4 f = sm.ring_f[stage][j[u]];
                            C.x += bw * f.x; C.y += bw * f.y; C.z += bw * f.z; C.w += bw * f.w;
                            if (kDepth) Z += bw * sm.ring_a[stage][j[u]].w;
                        }
                        Tr *= 1.0f - al[u];
                        if (Tr < stop) done = true;
                    }
                    if (done) todo = 0u;
                }
                __syncwarp();
                if (kWeights) {
                    unsigned from = warp_transpose_bits(taken, lane);
                    float sum = 0.0f;
                    while (from) {
                        sum += sm.out[lane][__ffs(from) - 1];
                        from &= from - 1u;
                    }
                    if (sum > 0.0f) atomicAdd(blending_weights + id_cur, sum);
                }
                done_w = __ballot_sync(kFull, done);
                __syncwarp();
                if (done_w == kFull) break;   // every pixel has stopped: the rest of the list has no effect
            }
            async_copy_wait<0>();   // whatever is still travelling lands before the next item reuses the ring
            __syncwarp();
        }
        if ((PASS == PASS_PRODUCT || kWeights) && lane == 0) n_kept[sidx] = n_out;

        if (PASS == PASS_PRODUCT) {
            seg_T[sidx * 32 + lane] = Tr;   // this segment's product
            finish_products(items, item >> 1, (unsigned)half, seg, n_seg, seg_T, first, inside, lane);
            continue;
        }
        const int64_t n_px = (int64_t)width * height;
        const int64_t pi = (int64_t)py * width + px;
        if (n_seg == 1u) {
            if (inside) {
                image[pi] = C.x;
                image[n_px + pi] = C.y;
                image[2 * n_px + pi] = C.z;
                image[3 * n_px + pi] = C.w;
                const float A = 1.0f - Tr;
                if (kDepth) depth_image[pi] = A > 0.0f ? Z / A : 0.0f;
                alpha_image[pi] = Tr < kTransmittanceEps ? 1.0f : A;
            }
        } else {
            // partial colour of this segment; the per-tile combine adds the segments up in order
            const size_t si = sidx * 32 + lane;
            seg_C[si] = C;
            if (PASS == PASS_FIRST) seg_T[si] = Tr;   // the exact state behind segment 0
            if (kDepth) {
                seg_Z[si] = Z;
                seg_E[si] = Tr;
            } else if (seg + 1u == n_seg && inside) {
                alpha_image[pi] = Tr < kTransmittanceEps ? 1.0f : 1.0f - Tr;
            }
        }
    }
}

// First and later segments of a training pass by two warps per item, as in blend_bilinear_pair_forward_kernel: 2^22 splats at 1237x822 129 / 274 -> 98 / 200 us, the step at 3840x2160
// (129,600 tiles) 1880 -> 1800.
struct __align__(16) GaussPairSmem {
    float4 ring_a[3][32], ring_c[3][32], ring_f[3][32];   // records and conics of the batches in flight
    float out[32][33];                                    // [staged instance][pixel]: what the fragment adds to the blending weight
    uint32_t ring_id[3][32];
    unsigned words[2][32];
    unsigned stopped[2], end[2], item;
    uint32_t queue[kQueueCap];
};
constexpr size_t kGaussPairSmemBytes = 2 * 256 * sizeof(unsigned) + kPairs * sizeof(GaussPairSmem);
constexpr int kGaussPairBlocks = 3;
template <int PASS>
__global__ void __launch_bounds__(kWarpBlendWarps * 32, kGaussPairBlocks) blend_gaussian_pair_forward_kernel(
    const WarpItem* __restrict__ items, const uint32_t* __restrict__ counts, unsigned* __restrict__ ticket, unsigned n_visits, const uint32_t* __restrict__ inst_keys,
    const uint32_t* __restrict__ inst_ids, const PointRec* __restrict__ rec, const float4* __restrict__ conic, float* __restrict__ seg_T, float4* __restrict__ seg_C,
    float* __restrict__ image, float* __restrict__ alpha_image, float* __restrict__ blending_weights, uint32_t* kept0, uint32_t* kept1,
    uint32_t* __restrict__ n_kept, int width, int height, int gw, float reach) {
    await_previous_kernel();
    static_assert(PASS != PASS_PRODUCT, "blends");
    constexpr unsigned kFull = 0xffffffffu, kNoInstance = 0xffffffffu, kNoItem = 0xffffffffu;
    using Smem = GaussPairSmem;
    extern __shared__ __align__(16) unsigned char blend_smem[];
    unsigned* s_reach = reinterpret_cast<unsigned*>(blend_smem);     // [half][key code] -> pixels of the half reached
    const unsigned lane = lane_id(), pair = threadIdx.x >> 6;
    const bool prepares = ((threadIdx.x >> 5) & 1u) == 0u;
    Smem& sm = reinterpret_cast<Smem*>(blend_smem + 2 * 256 * sizeof(unsigned))[pair];
    const unsigned lt_mask = (1u << lane) - 1u;
    {
        const unsigned long long m = cell_pixels(threadIdx.x);
        s_reach[threadIdx.x] = (unsigned)m;
        s_reach[256 + threadIdx.x] = (unsigned)(m >> 32);
    }
    __syncthreads();
    const unsigned n_items = __ldg(counts + (PASS == PASS_FIRST ? 0 : 1)) * 2u;
    ItemQueue queue(n_items, PASS == PASS_FIRST ? __ldg(counts + kLongTiles + 1) * 2u : 0u, n_visits, kMostItems);
    for (;;) {
        if (prepares) {
            unsigned taken;
            if (!queue.take(ticket, lane, &taken)) taken = kNoItem;
            if (lane == 0) sm.item = taken;
        }
        pair_barrier(pair);
        const unsigned item = sm.item;
        if (item == kNoItem) break;
        const WarpItem it = load_item(items + (item >> 1));
        const unsigned tile = it.tile, seg = it.seg, n_seg = it.n_seg, first = it.first;
        const int half = (int)(item & 1u);
        const size_t sidx = (size_t)(first + seg) * 2u + half;      // this item's slot in the per-segment arrays
        const uint2 rg = make_uint2(it.begin, it.end);
        const int tx = (int)(tile % (unsigned)gw), ty = (int)(tile / (unsigned)gw);
        const int px0 = tx * 8, py0 = ty * 8 + 4 * half;            // first pixel of this half
        const int px = px0 + (int)(lane & 7u), py = py0 + (int)(lane >> 3);
        const bool inside = px < width && py < height;

        if (prepares) {
            // ---- where the instances come from.  FIRST filters the item's keys; REST blends the list PRODUCT
            // compacted for this item (a superset of what is still alive at the true transmittance, see above), its ids
            // loaded kIdsAhead batches ahead of their gather.
            uint32_t* kept = half ? kept1 : kept0;
            const unsigned* reach_of_key = s_reach + 256 * half;
            CandidateStream in;
            uint32_t idf[kIdsAhead];
            if (PASS == PASS_REST) {
                in.head = 0u;
                in.tail = n_kept[sidx];     // length of PRODUCT's list; the list itself starts at kept[rg.x]
#pragma unroll
                for (int k = 0; k < kIdsAhead; ++k) idf[k] = 32u * k + lane < in.tail ? kept[rg.x + 32u * k + lane] : 0u;
            } else {
                in.start(inst_keys, inst_ids, rg.x, rg.y, lane);
            }
            pair_barrier(pair);
            unsigned done_w = sm.stopped[0], n_out = 0;
            if (done_w != kFull) {   // else: nothing in this list can have an effect
                auto fill = [&]() {
                    if (PASS != PASS_REST) in.fill(reach_of_key, done_w, sm.queue, lane, lt_mask);
                    __syncwarp();
                };
                // the next (up to) 32 candidates become a batch: their records start to travel into `stage` of the ring
                auto gather = [&](unsigned stage) {
                    const unsigned n = min(32u, in.tail - in.head);
                    uint32_t id = kNoInstance;
                    if (lane < n) {
                        id = checked_point(PASS == PASS_REST ? idf[0] : sm.queue[(in.head + lane) & (kQueueCap - 1)]);
                        const float4* p = reinterpret_cast<const float4*>(rec + id);
                        async_copy_16(&sm.ring_a[stage][lane], p);
                        async_copy_16(&sm.ring_c[stage][lane], conic + id);
                        async_copy_16(&sm.ring_f[stage][lane], p + 1);
                    }
                    sm.ring_id[stage][lane] = id;
                    async_copy_commit();   // one group per batch, empty or not: the waits below count groups
                    if (PASS == PASS_REST) {
#pragma unroll
                        for (int k = 0; k + 1 < kIdsAhead; ++k) idf[k] = idf[k + 1];
                        const unsigned nxt = in.head + 32u * kIdsAhead + lane;
                        idf[kIdsAhead - 1] = nxt < in.tail ? kept[rg.x + nxt] : 0u;
                    }
                    in.head += n;
                };
                fill();
                gather(0u);
                fill();
                gather(1u);
                unsigned stage = 0u;   // of batch b
                for (unsigned b = 0;; ++b) {
                    fill();
                    async_copy_wait<1>();   // all but the newest group: batch b has arrived
                    const uint32_t id_cur = sm.ring_id[stage][lane];
                    const bool staged = id_cur != kNoInstance;
                    const bool end = __ballot_sync(kFull, staged) == 0u;   // batches are filled in order: nothing is left
                    if (!end) {
                        // ---- lane j: the pixels of staged instance j that have not stopped
                        const unsigned pixels = staged ? ellipse_pixels(sm.ring_a[stage][lane], sm.ring_c[stage][lane], reach, px0, py0) & ~done_w : 0u;
                        // what reaches a pixel that has not stopped goes into the list of this item, as in blend_bilinear_warp_forward_kernel
                        const unsigned alive = __ballot_sync(kFull, pixels != 0u);
                        if (pixels) kept[rg.x + n_out + __popc(alive & lt_mask)] = id_cur;
                        n_out += __popc(alive);
                        sm.words[b & 1u][lane] = warp_transpose_bits(pixels, lane);
                    }
                    if (lane == 0) sm.end[b & 1u] = end ? 1u : 0u;
                    pair_barrier(pair);
                    if (end) break;
                    done_w = sm.stopped[b & 1u];
                    if (done_w == kFull) break;   // every pixel has stopped: the rest of the list has no effect
                    stage = stage == 2u ? 0u : stage + 1u;
                    gather(stage == 2u ? 0u : stage + 1u);   // batch b + 2, where batch b - 1 lay
                }
                async_copy_wait<0>();   // whatever is still travelling lands before the next item reuses the ring
                __syncwarp();
            }
            if (lane == 0) n_kept[sidx] = n_out;
            continue;
        }

        const float pcx = (float)px + 0.5f, pcy = (float)py + 0.5f;
        float Tr = 1.0f;
        float4 C = make_float4(0.f, 0.f, 0.f, 0.f);
        bool done = !inside;
        if (PASS == PASS_REST) {
            Tr = seg_T[sidx * 32 + lane];
            done = done || Tr < kTransmittanceEps;
        }
        unsigned done_w = __ballot_sync(kFull, done);   // bit l = pixel of lane l has stopped (warp-uniform)
        if (lane == 0) sm.stopped[0] = done_w;
        pair_barrier(pair);
        if (done_w != kFull) {
            unsigned stage = 0u;
            for (unsigned b = 0;; ++b, stage = stage == 2u ? 0u : stage + 1u) {
                pair_barrier(pair);
                if (sm.end[b & 1u] || done_w == kFull) break;
                // ---- every lane runs down the instances of its own pixel, front to back
                unsigned todo = done ? 0u : sm.words[b & 1u][lane];   // (made before the pixels that stopped in the batch in front of it were known)
                unsigned taken = 0u;   // instances whose blending weight this pixel adds to
                while (todo) {
                    constexpr int kPair = 2;
                    int j[kPair];
                    float al[kPair], G[kPair];
                    bool ok[kPair];
#pragma unroll
                    for (int u = 0; u < kPair; ++u) {
                        ok[u] = todo != 0u;
                        j[u] = ok[u] ? __ffs(todo) - 1 : j[0];
                        todo &= todo - 1u;
                        const float4 a = sm.ring_a[stage][j[u]], c = sm.ring_c[stage][j[u]];
                        const float dx = a.x - pcx, dy = a.y - pcy;
                        const float e = -0.5f * (c.x * dx * dx + c.z * dy * dy) - c.y * dx * dy;
                        G[u] = expf(e);
                        ok[u] = ok[u] && !(e > 0.0f) && !(G[u] < kTrainGaussThreshold);
                        al[u] = rounded_alpha(a.z, G[u]);
                    }
#pragma unroll
                    for (int u = 0; u < kPair; ++u) {
                        if (!ok[u] || done) continue;
                        const float bw = Tr * al[u];
                        if (bw > 0.0f) {
                            sm.out[j[u]][lane] = G[u] * bw;
                            taken |= 1u << j[u];
                        }
                        const float4 f = sm.ring_f[stage][j[u]];
                        C.x += bw * f.x; C.y += bw * f.y; C.z += bw * f.z; C.w += bw * f.w;
                        Tr *= 1.0f - al[u];
                        if (Tr < kTransmittanceEps) done = true;
                    }
                    if (done) todo = 0u;
                }
                __syncwarp();
                unsigned from = warp_transpose_bits(taken, lane);
                float sum = 0.0f;
                while (from) {
                    sum += sm.out[lane][__ffs(from) - 1];
                    from &= from - 1u;
                }
                if (sum > 0.0f) atomicAdd(blending_weights + sm.ring_id[stage][lane], sum);
                done_w = __ballot_sync(kFull, done);
                if (lane == 0) sm.stopped[(b + 1u) & 1u] = done_w;
            }
        }
        const int64_t n_px = (int64_t)width * height, pi = (int64_t)py * width + px;
        const float alpha = Tr < kTransmittanceEps ? 1.0f : 1.0f - Tr;
        if (n_seg == 1u) {
            if (inside) {
                image[pi] = C.x;
                image[n_px + pi] = C.y;
                image[2 * n_px + pi] = C.z;
                image[3 * n_px + pi] = C.w;
                alpha_image[pi] = alpha;
            }
        } else {
            // partial colour of this segment; the per-tile combine adds the segments up in order
            seg_C[sidx * 32 + lane] = C;
            if (PASS == PASS_FIRST) seg_T[sidx * 32 + lane] = Tr;   // the exact state behind segment 0
            if (seg + 1u == n_seg && inside) alpha_image[pi] = alpha;
        }
    }
}

struct __align__(16) GaussBackwardSmem {
    float4 ring_a[2][32], ring_c[2][32], ring_f[2][32];
    float4 pixel_grad[32];      // image gradient of the half's pixels
    float out_bw[32][33];       // [staged instance][pixel]: blending weight of the fragment ...
    float out_go[32][33];       // ... and what it adds to the opacity gradient
    uint32_t ring_id[2][32];
};
constexpr size_t kGaussBackwardSmemBytes = kWarpBlendWarps * sizeof(GaussBackwardSmem);

__global__ void __launch_bounds__(kWarpBlendWarps * 32, kGaussBackwardBlocks) blend_gaussian_warp_backward_kernel(
    const WarpItem* __restrict__ items0, const WarpItem* __restrict__ items1, const uint32_t* __restrict__ counts,
    unsigned* __restrict__ ticket, unsigned n_visits, const uint32_t* __restrict__ kept0, const uint32_t* __restrict__ kept1, const uint32_t* __restrict__ n_kept,
    const PointRec* __restrict__ rec, const float4* __restrict__ conic, const float* __restrict__ seg_T, const float4* __restrict__ seg_C,
    const float* __restrict__ grad_image, const float* __restrict__ grad_alpha, const float* __restrict__ image,
    const float* __restrict__ alpha_image, float4* __restrict__ grad_feat_view, float* __restrict__ grad_opacity, int width, int height, int gw,
    float reach) {
    await_previous_kernel();
    constexpr unsigned kFull = 0xffffffffu;
    constexpr unsigned kNoInstance = 0xffffffffu;
    extern __shared__ __align__(16) unsigned char blend_smem[];
    const unsigned lane = lane_id();
    GaussBackwardSmem& sm = reinterpret_cast<GaussBackwardSmem*>(blend_smem)[threadIdx.x >> 5];
    const unsigned n_first = __ldg(counts) * 2u;
    const unsigned n_items = n_first + __ldg(counts + 1) * 2u;
    const unsigned n_rest = n_items - n_first;
    ItemQueue queue(n_items, n_rest + __ldg(counts + kLongTiles + 1) * 2u, n_visits, kMostItems);
    unsigned item;
    while (queue.take(ticket, lane, &item)) {
        const WarpItem it = load_item(item < n_rest ? items1 + (item >> 1) : items0 + ((item - n_rest) >> 1));
        const int half = (int)((item < n_rest ? item : item - n_rest) & 1u);
        const unsigned n_list = __ldg(n_kept + (size_t)(it.first + it.seg) * 2u + half);
        const unsigned tile = it.tile, seg = it.seg, n_seg = it.n_seg;
        const size_t sidx = (size_t)(it.first + seg) * 2u + half;
        if (n_list == 0u) continue;
        const uint32_t* list = (half ? kept1 : kept0) + it.begin;
        const int tx = (int)(tile % (unsigned)gw), ty = (int)(tile / (unsigned)gw);
        const int px0 = tx * 8, py0 = ty * 8 + 4 * half;
        const int px = px0 + (int)(lane & 7u), py = py0 + (int)(lane >> 3);
        const float pcx = (float)px + 0.5f, pcy = (float)py + 0.5f;

        float4 g = make_float4(0.f, 0.f, 0.f, 0.f), Cfin = g, Crun = g;
        float K = 0.0f, Tr = 1.0f;
        bool done = !(px < width && py < height);
        if (!done) {
            const int64_t n_px = (int64_t)width * height;
            const int64_t pi = (int64_t)py * width + px;
            g = make_float4(__ldg(grad_image + pi), __ldg(grad_image + n_px + pi), __ldg(grad_image + 2 * n_px + pi),
                            __ldg(grad_image + 3 * n_px + pi));
            // what this segment and the ones behind it add to the pixel: the running colour starts at zero
            Cfin = n_seg > 1u ? seg_C[sidx * 32 + lane]
                              : make_float4(__ldg(image + pi), __ldg(image + n_px + pi), __ldg(image + 2 * n_px + pi), __ldg(image + 3 * n_px + pi));
            K = __ldg(grad_alpha + pi) * (1.0f - __ldg(alpha_image + pi));
            if (seg > 0u) Tr = seg_T[sidx * 32 + lane];
            done = Tr < kTransmittanceEps;
        }
        __syncwarp();   // the previous item's readers of pixel_grad are through
        sm.pixel_grad[lane] = g;
        unsigned done_w = __ballot_sync(kFull, done);

        uint32_t idf[kIdsAhead];
#pragma unroll
        for (int k = 0; k < kIdsAhead; ++k) idf[k] = 32u * k + lane < n_list ? __ldg(list + 32u * k + lane) : 0u;
        unsigned issued = 0;   // instances whose gather has started
        auto gather = [&](unsigned stage) {
            const unsigned n = min(32u, n_list - issued);
            uint32_t id = kNoInstance;
            if (lane < n) {
                id = checked_point(idf[0]);
                const float4* p = reinterpret_cast<const float4*>(rec + id);
                async_copy_16(&sm.ring_a[stage][lane], p);
                async_copy_16(&sm.ring_c[stage][lane], conic + id);
                async_copy_16(&sm.ring_f[stage][lane], p + 1);
            }
            sm.ring_id[stage][lane] = id;
            async_copy_commit();   // one group per batch, empty or not
#pragma unroll
            for (int k = 0; k + 1 < kIdsAhead; ++k) idf[k] = idf[k + 1];
            const unsigned nxt = issued + 32u * kIdsAhead + lane;
            idf[kIdsAhead - 1] = nxt < n_list ? __ldg(list + nxt) : 0u;
            issued += n;
        };
        gather(0u);
        for (unsigned batch = 0;; ++batch) {
            gather((batch + 1u) & 1u);
            async_copy_wait<1>();
            const unsigned stage = batch & 1u;
            const uint32_t id_cur = sm.ring_id[stage][lane];
            const bool staged = id_cur != kNoInstance;
            if (__ballot_sync(kFull, staged) == 0u) break;
            unsigned pixels = 0u;
            if (staged) pixels = ellipse_pixels(sm.ring_a[stage][lane], sm.ring_c[stage][lane], reach, px0, py0) & ~done_w;
            __syncwarp();   // every lane sees the records the others have copied
            unsigned todo = warp_transpose_bits(pixels, lane);
            unsigned taken = 0u;   // instances this pixel hands a gradient to
            while (todo) {
                // three at a time: their exponentials and reciprocals do not wait for one another (one at a time 260 us, two 239, three 234)
                constexpr int kPair = 3;
                int j[kPair];
                float al[kPair], G[kPair], rcp[kPair];
                bool ok[kPair];
#pragma unroll
                for (int u = 0; u < kPair; ++u) {
                    ok[u] = todo != 0u;
                    j[u] = ok[u] ? __ffs(todo) - 1 : j[0];
                    todo &= todo - 1u;
                    const float4 a = sm.ring_a[stage][j[u]], c = sm.ring_c[stage][j[u]];
                    const float dx = a.x - pcx, dy = a.y - pcy;
                    const float e = -0.5f * (c.x * dx * dx + c.z * dy * dy) - c.y * dx * dy;
                    G[u] = expf(e);
                    ok[u] = ok[u] && !(e > 0.0f || G[u] < kTrainGaussThreshold);
                    al[u] = rounded_alpha(a.z, G[u]);
                    rcp[u] = one_minus_alpha_reciprocal(1.0f - al[u]);
                }
#pragma unroll
                for (int u = 0; u < kPair; ++u) {
                    if (!ok[u] || done) continue;
                    const float bw = Tr * al[u];
                    const float4 f = sm.ring_f[stage][j[u]];
                    Crun.x += bw * f.x; Crun.y += bw * f.y; Crun.z += bw * f.z; Crun.w += bw * f.w;
                    const float from_features = (Tr * f.x + (Crun.x - Cfin.x) * rcp[u]) * g.x +
                                                (Tr * f.y + (Crun.y - Cfin.y) * rcp[u]) * g.y +
                                                (Tr * f.z + (Crun.z - Cfin.z) * rcp[u]) * g.z +
                                                (Tr * f.w + (Crun.w - Cfin.w) * rcp[u]) * g.w;
                    sm.out_bw[j[u]][lane] = bw;
                    sm.out_go[j[u]][lane] = (from_features + K * rcp[u]) * G[u];
                    taken |= 1u << j[u];
                    Tr *= 1.0f - al[u];
                    if (Tr < kTransmittanceEps) done = true;
                }
                if (done) todo = 0u;
            }
            __syncwarp();
            // ---- lane j: the sums of instance j over its pixels
            unsigned from = warp_transpose_bits(taken, lane);
            if (from) {
                float4 sf = make_float4(0.f, 0.f, 0.f, 0.f);
                float so = 0.0f;
                do {
                    const int p = __ffs(from) - 1;
                    from &= from - 1u;
                    const float bw = sm.out_bw[lane][p];
                    if (bw > 0.0f) {   // (zero times an upstream gradient that has overflowed would be no number)
                        const float4 pg = sm.pixel_grad[p];
                        sf.x += bw * pg.x; sf.y += bw * pg.y; sf.z += bw * pg.z; sf.w += bw * pg.w;
                    }
                    so += sm.out_go[lane][p];
                } while (from);
                if (sf.x != 0.0f || sf.y != 0.0f || sf.z != 0.0f || sf.w != 0.0f) atomicAdd(grad_feat_view + id_cur, sf);
                if (so != 0.0f) atomicAdd(grad_opacity + id_cur, so);
            }
            done_w = __ballot_sync(kFull, done);
            __syncwarp();
            if (done_w == kFull) break;
        }
        async_copy_wait<0>();   // whatever is still travelling lands before the next item reuses the ring
        __syncwarp();
    }
}

// SH chain rule for every point, zero rows for culled ones, written as 72 contiguous bytes per point
// through a shared-memory slab so the stores are coalesced 16-byte vectors.
// src/bilinear/kernels.cu:86-104 + include/sh_utils.cuh:44-62; the zero rows replace the
// torch::zeros of src/rasterization_api.cu:139.
// SLOTS (warp blend): the view-space gradient of a point is the sum of its (up to four) written slots in slot order,
// see blend_bilinear_warp_backward_kernel; the opacity gradient is formed here too and written for every point.
struct GradientSlots {
    const float4* grad;      // [4 n][2]: {feature gradient}, {opacity gradient, -, -, -}
    const unsigned* mask;    // [n] bit s: slot s was written
};
// Bound by the 76 bytes a point's gradients take (97 us of 162 for 2^23 samples) and by waiting for the slots of the touched
// ones: eight blocks per multiprocessor (32 registers) keep more of them in flight (without the bound 180 us; 2^24
// points 318 -> 285).
template <bool SLOTS>
__global__ void __launch_bounds__(kPreThreads, 8) preprocess_backward_kernel(
    const float* __restrict__ positions, const float* __restrict__ cam, const uint2* __restrict__ bounds,
    const float4* __restrict__ grad_feat_view, GradientSlots slots, float* __restrict__ grad_opacities,
    __half* __restrict__ grad_features, int64_t n, bool bulk_ok) {
    await_previous_kernel();
    __shared__ __align__(16) __half s_out[kPreThreads * 36];
    const int64_t block_first = (int64_t)blockIdx.x * kPreThreads;
    const int in_block = (int)min((int64_t)kPreThreads, n - block_first);
    const int64_t i = block_first + threadIdx.x;
    __half* o = s_out + threadIdx.x * 36;
    // With slots the mask alone says whether a point received anything: most points of a dense scene lie behind stopped pixels,
    // and neither their bounds nor their positions are read (2^23 samples: 184 -> 165 us).
    bool touched = false;
    unsigned m = 0;
    if (i < n) {
        if (SLOTS) touched = (m = __ldg(slots.mask + i)) != 0u;
        else touched = tiles_of(__ldg(bounds + i)) != 0u;
    }
    if (touched) {
        float b[9];
        sh_basis(__ldg(positions + 3 * i), __ldg(positions + 3 * i + 1), __ldg(positions + 3 * i + 2), cam, b);
        b[1] = -b[1]; b[3] = -b[3]; b[5] = -b[5]; b[7] = -b[7];
        float4 gv = make_float4(0.f, 0.f, 0.f, 0.f);
        if (SLOTS) {
            float go = 0.0f;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if ((m >> q) & 1u) {
                    const float4 v = __ldg(slots.grad + (i * 4 + q) * 2);
                    gv.x += v.x; gv.y += v.y; gv.z += v.z; gv.w += v.w;
                    go += __ldg(slots.grad + (i * 4 + q) * 2 + 1).x;
                }
            }
            grad_opacities[i] = go;
        } else {
            gv = __ldg(grad_feat_view + i);
        }
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const __half2 xy = __float22half2_rn(make_float2(b[k] * gv.x, b[k] * gv.y));
            const __half2 zw = __float22half2_rn(make_float2(b[k] * gv.z, b[k] * gv.w));
            *reinterpret_cast<__half2*>(o + 4 * k) = xy;
            *reinterpret_cast<__half2*>(o + 4 * k + 2) = zw;
        }
    } else {
#pragma unroll
        for (int k = 0; k < 18; ++k) *reinterpret_cast<unsigned*>(o + 2 * k) = 0u;
        if (SLOTS && i < n) grad_opacities[i] = 0.0f;
    }
    unsigned char* dst = reinterpret_cast<unsigned char*>(grad_features) + block_first * 72;
    const int bytes = in_block * 72;
    // one bulk asynchronous store of the block's contiguous 72-byte rows when base and size are multiples
    // of 16 bytes; 16-byte stores through registers otherwise
    const bool bulk = bulk_ok && (bytes & 15) == 0;
    if (bulk) fence_shared_for_bulk();
    __syncthreads();
    if (bulk) {
        if (threadIdx.x == 0) bulk_store_from_shared(dst, s_out, (unsigned)bytes);
        return;
    }
    const int n16 = bytes / 16;
    uint4* dst16 = reinterpret_cast<uint4*>(dst);
    const uint4* src16 = reinterpret_cast<const uint4*>(s_out);
    for (int k = threadIdx.x; k < n16; k += kPreThreads) dst16[k] = src16[k];
    for (int k = n16 * 16 + 2 * threadIdx.x; k < bytes; k += 2 * kPreThreads)
        *reinterpret_cast<unsigned short*>(dst + k) = *reinterpret_cast<const unsigned short*>(reinterpret_cast<const unsigned char*>(s_out) + k);
}

// ------------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------------
struct PointBlob {
    PointRec* rec;
    uint2* bounds;                        // tile bounds per point; none where they follow from `quad`
    uint32_t* quad;                       // bilinear, warp blend: packed footprint origin per point (see pack_quad), else none
    float4* conic;
    uint4* foot;                          // gaussian, warp blend: tile bounds and ellipse per point (see pack_footprint)
    uint32_t* keys[2];
    uint32_t* ids[2];
    unsigned* inst_block_sums;
    unsigned* state;                      // words that start at zero: [0] finished blocks of the instance count, then
    unsigned long long* counters;         // visible, instances; deferred: instances emitted
    void* sort_ws;                        // directly behind `state`: cleared together
    size_t total;
};

// Which of the two blend organisations a call uses: one warp per tile part with the dead-instance filter
// (8x8 tiles) or one block per (tile, segment).
bool uses_warp_blend(int tile) { return tile == 8; }

// Sized by the number of input points (every per-visible array gets room for all of them), so
// that the layout is known before the visible count has been read back.
PointBlob carve_point_blob(void* p, int64_t n, int mode, int tile) {
    PointBlob b;
    Carver c(p);
    b.rec = c.take<PointRec>(n);
    const bool quads = mode == INPC_MODE_BILINEAR && uses_warp_blend(tile);
    b.bounds = quads ? nullptr : c.take<uint2>(n);
    b.quad = quads ? c.take<uint32_t>(n) : nullptr;
    b.conic = mode == INPC_MODE_GAUSSIAN ? c.take<float4>(n) : nullptr;
    b.foot = mode == INPC_MODE_GAUSSIAN && uses_warp_blend(tile) ? c.take<uint4>(n) : nullptr;
    for (int k = 0; k < 2; ++k) b.keys[k] = c.take<uint32_t>(n);
    for (int k = 0; k < 2; ++k) b.ids[k] = c.take<uint32_t>(n);
    b.inst_block_sums = c.take<unsigned>(ceil_div<int64_t>(n > 0 ? n : 1, kInstThreads));
    b.state = c.take<unsigned>(64);
    b.counters = reinterpret_cast<unsigned long long*>(b.state + 16);
    c.off = align_up(c.off);
    b.sort_ws = c.base + c.off;
    c.off += sort_workspace_bytes(n, n);
    b.total = c.used();
    return b;
}

struct InstanceBlob {
    uint32_t* keys[2];
    uint32_t* ids[2];
    uint2* ranges;
    Segment* segs;
    uint32_t* tile_first;
    uint32_t* n_segments;
    float* seg_T;
    float4* seg_C;
    float* seg_Z;
    float* seg_E;         // warp blend, inference: transmittance at the end of every segment
    int64_t max_segments;
    uint32_t* tile_rank;  // warp blend: per block of 1024 tiles, the segments and the non-empty tiles of each class before it
    WarpItem* items0;     // warp blend: segment 0 of the non-empty tiles
    WarpItem* items1;     // warp blend: every segment behind a tile's first
    uint32_t* n_kept;     // warp blend: per item, length of the compacted list the forward pass blended
    void* sort_ws;
    size_t total;
};

// Upper bound on the segments of the warp blend for up to n_instances instances (see segment_lengths): one per tile, one more
// for every tile that is longer than a first segment, and the later segments that are full.
int64_t max_warp_segments(int64_t n_instances, int n_tiles, const SegmentLimits limits) {
    const int64_t target = limits.target;
    const int64_t by_first = ceil_div<int64_t>(n_instances, limits.first_max), by_later = ceil_div<int64_t>(n_instances, limits.later_max);
    const int64_t longer = by_first > 2 * target ? by_first : 2 * target;
    return n_tiles + (longer < n_tiles ? longer : n_tiles) + (by_later > target ? by_later : target) + 1;
}

// Upper bound on the number of (tile, segment) work items, known from the instance count alone.
int blend_batch(int tile);
int64_t max_segments(int64_t n_instances, int n_tiles, int tile) {
    return (int64_t)n_tiles + ceil_div<int64_t>(n_instances, (int64_t)blend_batch(tile) * kMinBatchesPerSegment);
}

constexpr int kWarpBlendParts = 2;   // work items of the warp blend per (tile, segment): the two 8x4 halves
// Bilinear splats touch at most 2x2 tiles.
bool has_instance_bound(int mode, int tile) { return mode == INPC_MODE_BILINEAR && uses_warp_blend(tile); }

// Whether a call sizes everything for that bound and leaves its counts on the device.  Feature rows do so only where nothing can be read
// back, while their stream is being captured: the bound takes three times the instance scratch the counts ask for (64 bytes per
// point against about 20), and with C / 4 times the segment colours that is memory a scene of wide rows has better use for; the
// counts are also part of what their forward returns.
bool defers_counts(int mode, int tile, bool rows, int64_t n, cudaStream_t stream) {
    if (!has_instance_bound(mode, tile) || n <= 0 || n >= ((int64_t)1 << 28)) return false;
    if (!rows) return true;
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    return status == cudaStreamCaptureStatusActive;
}

// The bounded path sizes its arrays for 4 instances per point; most splats touch one tile of four or none twice, about 1.3
// on average (2^23 samples at 1237x822: 1.26; at 3840x2160 less).  Only picks tile sizes.
int64_t likely_instances(int64_t capacity, bool deferred) { return deferred ? capacity / 3 : capacity; }

// `deferred`: n_instances is the bound, not a count.
InstanceBlob carve_instance_blob(void* p, int64_t n_instances, bool deferred, int n_tiles, int tile, int mode, bool with_depth, int c4 = 1) {
    InstanceBlob b;
    Carver c(p);
    const bool warp_blend = uses_warp_blend(tile);
    // [0] segments (block blend) or non-empty tiles (warp blend), [1] later segments (warp blend), [2..5] work tickets of
    // the warp blend passes FIRST, PRODUCT, REST and of its backward pass, [6] blocks of warp_items_count_kernel that are done, [8..9] tiles of
    // the longest class and of the two longer ones (kLongTiles).  Counters, tile ranges and the sort's state lie side
    // by side: they are cleared together.
    b.n_segments = c.take<uint32_t>(64);
    b.ranges = c.take<uint2>(n_tiles);
    c.off = align_up(c.off);
    b.sort_ws = c.base + c.off;
    c.off += sort_workspace_bytes(n_instances, likely_instances(n_instances, deferred));
    for (int k = 0; k < 2; ++k) b.keys[k] = c.take<uint32_t>(n_instances);
    for (int k = 0; k < 2; ++k) b.ids[k] = c.take<uint32_t>(n_instances);
    // upper bound on the number of (tile, segment) pairs, known from the instance count alone
    b.max_segments = warp_blend ? max_warp_segments(n_instances, n_tiles, segment_limits(mode, !with_depth)) : max_segments(n_instances, n_tiles, tile);
    const size_t px = (size_t)b.max_segments * tile * tile;
    b.segs = c.take<Segment>(warp_blend ? 0 : b.max_segments);
    b.tile_first = c.take<uint32_t>(n_tiles);
    b.seg_T = c.take<float>(px);
    b.seg_C = c.take<float4>(px * (size_t)c4);
    b.seg_Z = c.take<float>(with_depth ? px : 0);
    b.seg_E = c.take<float>(with_depth && warp_blend ? px : 0);
    b.tile_rank = c.take<uint32_t>(warp_blend ? (size_t)n_tiles + 8 : 0);   // four words per block of 1024 tiles
    b.items0 = c.take<WarpItem>(warp_blend ? (size_t)n_tiles : 0);
    b.items1 = c.take<WarpItem>(warp_blend ? (size_t)b.max_segments : 0);
    b.n_kept = c.take<uint32_t>(warp_blend ? (size_t)b.max_segments * kWarpBlendParts : 0);
    b.total = c.used();
    return b;
}

// The state handed back to the caller only stores blob bases and counts; which ping-pong buffer holds
// a sorted result follows from the number of radix passes, which follows from the bits of the keys.
int tile_buffer_of(int n_tiles) { return sort_pass_count(bit_length((uint32_t)(n_tiles - 1))) & 1; }
int depth_buffer_of(const inpc_raster_state* st) { return sort_pass_count(st->depth_key_bits) & 1; }
// Instance capacity the blobs of `st` were carved for.
int64_t instance_capacity(const inpc_raster_state* st) { return (st->deferred_counts & 1) ? 4 * st->n_points : st->n_instances; }

// One event per host thread and device: an event belongs to the device that was current when it was made.
cudaEvent_t counters_event() {
    static thread_local cudaEvent_t events[kMaxDevices] = {nullptr};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    if (!events[dev] && cudaEventCreateWithFlags(&events[dev], cudaEventDisableTiming) != cudaSuccess) events[dev] = nullptr;
    return events[dev];
}

unsigned long long* pinned_counters() {
    static thread_local unsigned long long* p = nullptr;
    if (!p && cudaHostAlloc(reinterpret_cast<void**>(&p), 4 * sizeof(unsigned long long), cudaHostAllocDefault) != cudaSuccess) p = nullptr;
    return p;
}

int check_view(const inpc_view* v, int tile_size, int mode, int64_t n) {
    if (!v || !v->w2c || !v->cam_position) { set_error("view, view.w2c and view.cam_position must be non-null"); return INPC_E_INVALID; }
    if (mode != INPC_MODE_BILINEAR && mode != INPC_MODE_GAUSSIAN) { set_error("unsupported rasterizer mode %d", mode); return INPC_E_INVALID; }
    if (tile_size != 8 && tile_size != 16) { set_error("tile_size must be 8 or 16, got %d", tile_size); return INPC_E_INVALID; }
    if (v->width <= 0 || v->height <= 0 || v->width > 65535 * tile_size || v->height > 65535 * tile_size) {
        set_error("image size %dx%d out of range", v->width, v->height);
        return INPC_E_INVALID;
    }
    if (mode == INPC_MODE_BILINEAR && tile_size == 8 && (v->width > kMaxCodedSide || ceil_div(v->height, 8) > kMaxCodedTileRows)) {
        set_error("image size %dx%d exceeds the %d x %d pixels of the 8x8-tile bilinear path (use tile_size 16)", v->width, v->height, kMaxCodedSide,
                  kMaxCodedTileRows * 8);
        return INPC_E_INVALID;
    }
    // tile indices live in the low kTileKeyBits bits of the instance keys
    const int64_t tiles = (int64_t)ceil_div(v->width, tile_size) * ceil_div(v->height, tile_size);
    if (tiles > ((int64_t)1 << kTileKeyBits)) {
        set_error("image size %dx%d gives %lld tiles of %d pixels, more than the supported 2^%u", v->width, v->height, (long long)tiles, tile_size, kTileKeyBits);
        return INPC_E_INVALID;
    }
    if (n < 0 || n >= ((int64_t)1 << 30)) { set_error("n=%lld out of range [0, 2^30)", (long long)n); return INPC_E_INVALID; }
    return INPC_OK;
}

// Checked build: publish the index limit before a call's kernels / collect the failure count after them.
int begin_index_checks(int64_t n_points, cudaStream_t stream) {
#ifdef INPC_CHECK_INDICES
    const unsigned long long limit = (unsigned long long)n_points;
    const unsigned zero = 0;
    INPC_CUDA_TRY(cudaMemcpyToSymbolAsync(g_check_n_points, &limit, sizeof(limit), 0, cudaMemcpyHostToDevice, stream));
    INPC_CUDA_TRY(cudaMemcpyToSymbolAsync(g_check_failures, &zero, sizeof(zero), 0, cudaMemcpyHostToDevice, stream));
#else
    (void)n_points; (void)stream;
#endif
    return INPC_OK;
}

int end_index_checks(cudaStream_t stream) {
#ifdef INPC_CHECK_INDICES
    unsigned failures = 0;
    INPC_CUDA_TRY(cudaMemcpyFromSymbolAsync(&failures, g_check_failures, sizeof(failures), 0, cudaMemcpyDeviceToHost, stream));
    INPC_CUDA_TRY(cudaStreamSynchronize(stream));
    if (failures) {
        set_error("checked build: %u point indices read from the sorted lists were out of range (accesses skipped)", failures);
        return INPC_E_DEVICE;
    }
#else
    (void)stream;
#endif
    return INPC_OK;
}

int launch_clear(const ClearList& list, cudaStream_t stream) {
    if (list.count == 0) return INPC_OK;
    size_t total = 0;
    for (int k = 0; k < list.count; ++k) total += list.bytes[k];
    const size_t blocks = ceil_div<size_t>(total, 256 * 16 * 4), cap = (size_t)sm_count() * 8;
    launch_chained(clear_kernel, (unsigned)(blocks < 1 ? 1 : blocks < cap ? blocks : cap), 256, 0, stream, list);
    INPC_LAUNCH_CHECK("clear_kernel");
    return INPC_OK;
}

template <int MODE, int VARIANT>
int run_front(const RasterParams& rp, int64_t n, const float* positions, const void* features, const float* opacities,
              inpc_alloc_fn alloc_point, inpc_alloc_fn alloc_instance, void* user, inpc_raster_state* st,
              bool with_depth, PointBlob* pb_out, InstanceBlob* ib_out, cudaStream_t stream, const char* entry, ClearList clear, int c4 = 1,
              const PointSets* sets = nullptr) {
    // `clear`: outputs of the call that have to start at zero
    // `sets`: the input of a batched multi-set call (then n is the virtual total and the three pointers are unused)
    const int n_tiles = rp.gw * rp.gh * rp.n_sets;
    PointSets ps;
    if (sets) {
        ps = *sets;
    } else {
        ps.count = 1;
        ps.start[0] = 0; ps.start[1] = n;
        ps.size[0] = n;
        ps.positions[0] = positions; ps.features[0] = features; ps.opacities[0] = opacities;
    }
    {
        // a failure an earlier call of this thread reported from the device surfaces here at the latest
        const int rc_prev = check_previous_calls();
        if (rc_prev != INPC_OK) return rc_prev;
    }
    unsigned* status = acquire_status(entry);
    if (!status) return INPC_E_CUDA;
    const bool warp_blend = uses_warp_blend(rp.tile);
    const PointBlob sizing = carve_point_blob(nullptr, n, MODE, rp.tile);
    void* pblob = alloc_point(user, sizing.total);
    if (!pblob) { set_error("point allocator returned NULL for %zu bytes", sizing.total); return INPC_E_ALLOC; }
    const PointBlob pb = carve_point_blob(pblob, n, MODE, rp.tile);
    {
        const int rc_check = begin_index_checks(n, stream);
        if (rc_check != INPC_OK) return rc_check;
    }

    // Bilinear splats touch at most 2x2 tiles, so the warp-blend path sizes everything behind the projection
    // for 4 n instances and lets the kernels read the two counts from device memory: no host synchronisation at
    // all (the reference reads both counts back with blocking copies, src/bilinear/forward.cu:86-89).  The other
    // paths (gaussian splats have no such bound, feature rows keep their scratch small) read the counts back once.
    const bool deferred = defers_counts(MODE, rp.tile, VARIANT == VAR_ROWS, n, stream);
    int64_t n_visible = 0, n_instances = 0;
    // depth keys are offsets from the near plane's bit pattern, bounded by the far plane's: nothing is measured.  (Where the range of the depths was measured first, in a pass that also counted and
    // compacted, planes 0.01 and 100 / 0.01 and 1000 / 0 and 100: step of 2^22 gaussian splats 1482 / 1479 / 1479 us, 1235 / 1272 / 1272 so; of 2^23 rows of 16 channels 1553 / 1556 / 1557,
    // 1399 / 1430 / 1522; of 2^22 bilinear splats on 16x16 tiles 1475 / 1480 / 1476, 1457 / 1472 / 1486.)
    const float near_depth = rp.v.near_plane > 0.0f ? rp.v.near_plane : 0.0f;
    const float far_depth = rp.v.far_plane != rp.v.far_plane ? INFINITY   // a far plane that is no number culls nothing
                                                             : rp.v.far_plane > near_depth ? rp.v.far_plane : near_depth;
    uint32_t key_base, last_key;
    memcpy(&key_base, &near_depth, 4);
    memcpy(&last_key, &far_depth, 4);
    if (!(rp.v.near_plane > 0.0f)) { key_base = 0u; last_key = 0xFFFFFFFFu; }
    int key_bits = bit_length(last_key - key_base);
    if (key_bits == 0) key_bits = 1;
    // with offsets of up to 2^30 - 1, a splat of four tiles at the far plane would have the key of a culled point
    if (key_bits == (int)kCountShift && last_key - key_base == (1u << kCountShift) - 1u) ++key_bits;
    const bool counts_in_keys = key_bits <= (int)(MODE == INPC_MODE_BILINEAR ? kCountShift : kGaussCountShift);
    const int tile_bits = bit_length((uint32_t)(n_tiles - 1));
    CarriedCodes codes;   // the depth sort carries the footprints along where they fit
    if (MODE == INPC_MODE_BILINEAR && warp_blend) codes = carried_codes(pb.quad, n, key_bits, (int64_t)n_tiles * 64);
    const bool carried = codes.bits > 0;
    void* iblob = nullptr;
    InstanceBlob ib;
    auto make_instance_blob = [&]() -> int {
        const InstanceBlob isz = carve_instance_blob(nullptr, n_instances, deferred, n_tiles, rp.tile, MODE, with_depth, c4);
        iblob = alloc_instance(user, isz.total);
        if (!iblob) { set_error("instance allocator returned NULL for %zu bytes", isz.total); return INPC_E_ALLOC; }
        ib = carve_instance_blob(iblob, n_instances, deferred, n_tiles, rp.tile, MODE, with_depth, c4);
        return INPC_OK;
    };
    auto clear_instance_blob = [&](ClearList& list) {
        list.add(ib.n_segments, (size_t)(static_cast<char*>(ib.sort_ws) - reinterpret_cast<char*>(ib.n_segments)) +
                                    sort_zero_bytes(n_instances, likely_instances(n_instances, deferred), tile_bits));
    };
    int rc, in_alt = 0;
    // read from here by everything behind the sorts, also where the host knows the counts: zero if a sort has failed
    unsigned long long* n_visible_dev = n > 0 ? pb.counters : nullptr;
    unsigned long long* n_instances_dev = n > 0 ? pb.counters + 1 : nullptr;
    if (n > 0) {
        unsigned long long* host = nullptr;
        cudaEvent_t ready = nullptr;
        if (deferred) {
            n_visible = n;                // capacities from here on
            n_instances = 4 * n;
            rc = make_instance_blob();
            if (rc != INPC_OK) return rc;
            clear_instance_blob(clear);
        } else {
            host = pinned_counters();
            ready = counters_event();
            if (!host || !ready) return cuda_fail(cudaGetLastError(), "cudaHostAlloc / cudaEventCreate (counters)");
        }
        {
            StageScope scope(STAGE_PREPROCESS, stream);
            clear.add(pb.state, (size_t)(static_cast<char*>(pb.sort_ws) - reinterpret_cast<char*>(pb.state)) + sort_zero_bytes(n, n, key_bits));
            rc = launch_clear(clear, stream);
            if (rc != INPC_OK) return rc;
            const int64_t chunks = ceil_div<int64_t>(n, kPreThreads), resident = (int64_t)sm_count() * projection_blocks(MODE);
            auto* project = preprocess_kernel<MODE, VARIANT>;
            launch_chained(project, (unsigned)(chunks < resident ? chunks : resident), kPreThreads, 0, stream,
                ps, rp, (unsigned)chunks, key_base, pb.rec, pb.bounds, pb.quad, pb.conic, pb.foot, pb.keys[0], counts_in_keys ? 1 : 0, VARIANT == VAR_ROWS && warp_blend ? 1 : 2,
                key_histogram(pb.sort_ws, n, n, key_bits), pb.counters, deferred ? nullptr : pb.counters + 1, status);
            INPC_LAUNCH_CHECK("preprocess_kernel");
            if (!deferred) {
                INPC_CUDA_TRY(cudaMemcpyAsync(host, pb.counters, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, stream));
                INPC_CUDA_TRY(cudaEventRecord(ready, stream));
            }
        }
        {
            // needs nothing from the host: it runs while the host waits for the counters
            StageScope scope(STAGE_SORT_DEPTH, stream);
            rc = carried ? sort_marked_keys_with_codes(pb.keys[0], pb.keys[1], pb.ids[0], pb.ids[1], n, pb.counters, key_bits, codes, pb.sort_ws, status, &in_alt, stream)
                         : sort_marked_keys(pb.keys[0], pb.keys[1], pb.ids[0], pb.ids[1], n, pb.counters, key_bits, pb.sort_ws, status, &in_alt, stream);
            if (rc != INPC_OK) return rc;
        }
        if (!deferred) {
            INPC_CUDA_TRY(cudaEventSynchronize(ready));
            n_visible = (int64_t)host[0];
            n_instances = (int64_t)host[1];
            // counts that cannot be: more survivors than points, or (bilinear: at most 2x2 tiles per splat)
            // more instances than four per survivor, or instances without survivors
            if (n_visible > n || (n_visible == 0 && n_instances != 0) || (MODE == INPC_MODE_BILINEAR && n_instances > 4 * n_visible)) {
                set_error("inconsistent counts from the projection pass: %lld visible of %lld points, %lld instances", (long long)n_visible,
                          (long long)n, (long long)n_instances);
                return INPC_E_DEVICE;
            }
        }
    }
    if (n_instances >= ((int64_t)1 << 30)) {
        set_error("%lld (point, tile) instances exceed the 2^30 capacity", (long long)n_instances);
        return INPC_E_CAPACITY;
    }

    if (!deferred) {
        // (n == 0: the outputs are cleared here, nothing has launched yet)
        rc = make_instance_blob();
        if (rc != INPC_OK) return rc;
        ClearList rest;
        if (n == 0) rest = clear;
        clear_instance_blob(rest);
        rc = launch_clear(rest, stream);
        if (rc != INPC_OK) return rc;
    }

    const bool counted = MODE == INPC_MODE_BILINEAR && warp_blend;   // the emission counts the digits of its keys
    const uint32_t* sorted_ids = pb.ids[in_alt];
    if (n_visible > 0 && n_instances > 0) {
        const int64_t ibk = ceil_div<int64_t>(n_visible, kInstThreads), count_need = carried || counts_in_keys ? ceil_div<int64_t>(ibk, kInstThreads / 4 / 32) : ibk, count_cap = (int64_t)sm_count() * 8;
        const unsigned count_blocks = (unsigned)(count_need < count_cap ? count_need : count_cap);
        {
            StageScope scope(STAGE_INSTANCES, stream);
            // the count of touched tiles follows from the codes, or rides in the top key bits where the depth offsets leave them free
            auto* count = carried ? instance_count_kernel<COUNTS_IN_CODES> : !counts_in_keys ? instance_count_kernel<COUNTS_GATHERED>
                          : MODE == INPC_MODE_BILINEAR ? instance_count_kernel<COUNTS_IN_KEYS> : instance_count_kernel<COUNTS_IN_GAUSS_KEYS>;
            launch_chained(count, count_blocks, kInstThreads / 4, 0, stream, pb.keys[in_alt], sorted_ids, pb.bounds, pb.quad, n_visible_dev, pb.inst_block_sums, (unsigned)ibk, pb.state, n_instances_dev, codes.escape);
            INPC_LAUNCH_CHECK("instance_count_kernel");
            if (counted) {
                const KeyHistogram digits = key_histogram(ib.sort_ws, n_instances, likely_instances(n_instances, deferred), tile_bits);
                unsigned long long* n_emitted = deferred && tile_bits > 0 ? pb.counters + 2 : nullptr;
                if (carried) {
                    static bool attr_set[kMaxDevices] = {false};
                    rc = opt_in_dynamic_smem(emit_coded_kernel, sizeof(EmitCodedSmem), attr_set);
                    if (rc != INPC_OK) return rc;
                    const int64_t need = ceil_div<int64_t>(n_visible, kCodedThreads * kCodedPoints), cap = (int64_t)sm_count() * kCodedBlocks;
                    launch_chained(emit_coded_kernel, (unsigned)(need < cap ? need : cap), kCodedThreads, sizeof(EmitCodedSmem), stream, sorted_ids, pb.keys[in_alt], codes, n_visible_dev,
                        pb.inst_block_sums, rp.gw, digits, n_emitted, ib.keys[0], ib.ids[0]);
                } else {
                    const int64_t cap = (int64_t)sm_count() * 2;   // two blocks of 1024 threads fill a multiprocessor
                    launch_chained(emit_quads_kernel, (unsigned)(ibk < cap ? ibk : cap), kInstThreads, 0, stream, sorted_ids, pb.quad, n_visible_dev, pb.inst_block_sums,
                        rp.gw, digits, n_emitted, ib.keys[0], ib.ids[0]);
                }
            } else {
                launch_chained(warp_blend ? emit_instances_kernel<true> : emit_instances_kernel<false>, (unsigned)ibk, kInstThreads, 0, stream, sorted_ids, pb.bounds, pb.foot,
                    n_visible_dev, pb.inst_block_sums, rp.gw, ib.keys[0], ib.ids[0]);
            }
            INPC_LAUNCH_CHECK(carried ? "emit_coded_kernel" : counted ? "emit_quads_kernel" : "emit_instances_kernel");
        }
        StageScope scope(STAGE_SORT_TILE, stream);
        int t_alt = 0;
        rc = sort_pairs_device_count(ib.keys[0], ib.keys[1], ib.ids[0], ib.ids[1], n_instances, likely_instances(n_instances, deferred), n_instances_dev, tile_bits, ib.sort_ws, true, status, &t_alt, stream, counted);
        if (rc != INPC_OK) return rc;
        const int64_t range_blocks = ceil_div<int64_t>(n_instances, 256 * (int64_t)kRangeKeysFew), range_cap = (int64_t)sm_count() * 8;
        launch_chained(tile_ranges_kernel, (unsigned)(range_blocks < range_cap ? range_blocks : range_cap), 256, 0, stream, ib.keys[t_alt], n_instances_dev, ib.ranges);
        INPC_LAUNCH_CHECK("tile_ranges_kernel");
    }
    if (warp_blend) {
        StageScope scope(STAGE_SORT_TILE, stream);
        const int item_blocks = ceil_div(n_tiles, kItemTilesPerBlock);
        uint4* item_sums = reinterpret_cast<uint4*>(ib.tile_rank);
        launch_chained(warp_items_count_kernel, item_blocks, kItemThreads, 0, stream, ib.ranges, n_tiles, segment_limits(MODE, !with_depth), VARIANT != VAR_ROWS, (unsigned long long)n_instances, n_instances_dev, item_sums, ib.n_segments + 6, ib.n_segments);
        INPC_LAUNCH_CHECK("warp_items_count_kernel");
        launch_chained(warp_items_fill_kernel, item_blocks, kItemThreads, 0, stream, ib.ranges, n_tiles, segment_limits(MODE, !with_depth), VARIANT != VAR_ROWS, (unsigned long long)n_instances, n_instances_dev, item_sums, ib.n_segments, ib.items0, ib.items1);
        INPC_LAUNCH_CHECK("warp_items_fill_kernel");
    } else {
        StageScope scope(STAGE_SORT_TILE, stream);
        launch_chained(count_segments_kernel, 1, kScanThreads, 0, stream, ib.ranges, n_tiles, blend_batch(rp.tile), ib.tile_first, ib.n_segments);
        INPC_LAUNCH_CHECK("count_segments_kernel");
        launch_chained(emit_segments_kernel, ceil_div(n_tiles, 256), 256, 0, stream, ib.ranges, n_tiles, blend_batch(rp.tile), ib.tile_first, ib.segs);
        INPC_LAUNCH_CHECK("emit_segments_kernel");
    }
    st->point_blob = pblob;
    st->instance_blob = iblob;
    st->n_points = n;
    st->n_visible = deferred ? -1 : n_visible;       // -1: still on the device, see inpc_raster_resolve
    st->n_instances = deferred ? -1 : n_instances;
    st->tile_size = rp.tile;
    st->mode = MODE;
    st->depth_key_base = key_base;
    st->depth_key_bits = key_bits;
    st->channels = VARIANT == VAR_ROWS ? 4 * c4 : 4;
    st->deferred_counts = (deferred ? 1 : 0) | (VARIANT == VAR_ROWS && warp_blend ? 2 : 0);   // bit 1: records 16 bytes apart, without features
    *pb_out = pb;
    *ib_out = ib;
    return INPC_OK;
}

RasterParams make_params(const inpc_view* view, int tile_size, float sigma_world, float sigma_cutoff, const float* scales) {
    RasterParams rp;
    rp.v = to_params(view);
    rp.tile = tile_size;
    rp.inv_tile = 1.0f / (float)tile_size;
    rp.gw = ceil_div(view->width, tile_size);
    rp.gh = ceil_div(view->height, tile_size);
    rp.n_sets = 1;
    rp.sigma_world = sigma_world;
    rp.sigma_cutoff = sigma_cutoff;
    rp.scales = scales;
    rp.reach = -2.0f * logf(expf(-0.5f * sigma_cutoff * sigma_cutoff));
    return rp;
}

// Instances staged per pixel thread and batch.  Measured on B200 (2^23 points, clustered and uniform
// scenes): one per thread is fastest for both tile sizes; deeper batches lose more to mask traffic
// and same-word atomicOr contention than they gain from fewer barriers.
template <int T> struct BlendConfig;
template <> struct BlendConfig<16> { static constexpr int kIpt = 1; };

int blend_batch(int tile) { return tile * tile * BlendConfig<16>::kIpt; }

// Grid of a persistent pass (the item counts live on the device): the blocks that are resident, which registers limit for some kernels and shared memory for
// others, and not more than the launch bounds ask for (in passes of gaussian splats over later segments, of 63 registers, four would fit: the products of a training
// step of 2^22 samples take 206 to 217 us with three and 204 to 213 with four, but a frame of 2 * 10^6 splats, where they are short, 581 and 585).  With four per multiprocessor for all passes, blocks that found nothing left came last, and a warp's share of the items (see ItemQueue) was
// counted too small: step of 2^24 points crowding a corner of 3840x2160 2633 -> 2540 us (first pass 347 -> 297, backward 441 -> 392), of 2^23 samples
// at 1237x822 1623 -> 1608.
// `takers`: warps of a block that take items, or pairs of warps; `visits_each`: of a resident one, 0 for the rule of gaussian splats and rows (see ItemQueue); `pass`: of the forward
// passes (PASS_FIRST also for a backward pass).
constexpr unsigned kVisits = 4, kVisitsPairBackward = 6;   // bilinear splats of four channels
struct BlendGrid {
    unsigned blocks = 1, visits = 1;
};
template <typename Kernel>
int warp_blend_grid(Kernel kernel, size_t smem, int most, unsigned takers, unsigned visits_each, int pass, int (&known)[kMaxDevices], BlendGrid* grid) {
    int blocks = 1;
    const int rc = resident_blocks(kernel, kWarpBlendWarps * 32, smem, known, &blocks);
    grid->blocks = (unsigned)(sm_count() * min(blocks, most));
    grid->visits = visits_each ? grid->blocks * takers * visits_each : (unsigned)sm_count() * (pass == PASS_FIRST ? 4u : 3u) * takers * 8u;
    return rc;
}
// Where in the counts the number of tiles is among which those of several segments lie: they are longer than a first segment, i.e. in the first class where the tiles lie by
// length, and the combine kernel looks at no others then (129,600 tiles, few of which have more than one segment: 12 -> 5 us, before it blanked empty tiles).
constexpr int tiles_with_segments(bool by_length) { return by_length ? kLongTiles : 0; }
unsigned small_grid() { return (unsigned)(sm_count() * 4); }   // of the combine kernel

struct ForwardPassArgs {
    const uint32_t *keys, *ids;
    const PointRec* rec;
    const float4* rows;   // feature rows, or nullptr
    float* seg_T;
    float4* seg_C;
    float *seg_Z, *seg_E, *image, *depth, *alpha, *blending_weights;
    uint32_t *kept0, *kept1, *n_kept;
    int W, H, gw, gh;
};

// One pass of the warp blend's forward: its shared memory (the per-warp rings) is above the 48 KB a kernel gets unasked.
template <int PASS, int KIND, int C4, bool ROWS>
int launch_warp_forward_pass(const WarpItem* items, const uint32_t* counts, unsigned* ticket, const ForwardPassArgs& a,
                             cudaStream_t stream) {
    static int known[kMaxDevices] = {0};
    constexpr size_t smem = warp_forward_smem_bytes<PASS, KIND, C4>();
    BlendGrid grid;
    const int rc = warp_blend_grid(blend_bilinear_warp_forward_kernel<PASS, KIND, C4, ROWS>, smem, forward_blocks(PASS, C4), kWarpBlendWarps, ROWS ? 0u : kVisits, PASS, known, &grid);
    if (rc != INPC_OK) return rc;
    launch_chained(blend_bilinear_warp_forward_kernel<PASS, KIND, C4, ROWS>, grid.blocks, kWarpBlendWarps * 32, smem, stream,
        items, counts, ticket, grid.visits, a.keys, a.ids, a.rec, a.rows, a.seg_T, a.seg_C, a.seg_Z, a.seg_E, a.image, a.depth, a.alpha, a.blending_weights,
        a.kept0, a.kept1, a.n_kept, a.W, a.H, a.gw, a.gh);
    INPC_LAUNCH_CHECK("blend_bilinear_warp_forward_kernel");
    return INPC_OK;
}

// The same with two warps per item.
template <int PASS, int C4, bool ROWS>
int launch_pair_forward_pass(const WarpItem* items, const uint32_t* counts, unsigned* ticket, const ForwardPassArgs& a, cudaStream_t stream) {
    static int known[kMaxDevices] = {0};
    constexpr size_t smem = pair_forward_smem_bytes<C4>();
    BlendGrid grid;
    const int rc = warp_blend_grid(blend_bilinear_pair_forward_kernel<PASS, C4, ROWS>, smem, pair_forward_blocks(C4), kPairs, ROWS ? 0u : kVisits, PASS, known, &grid);
    if (rc != INPC_OK) return rc;
    launch_chained(blend_bilinear_pair_forward_kernel<PASS, C4, ROWS>, grid.blocks, kWarpBlendWarps * 32, smem, stream,
        items, counts, ticket, grid.visits, a.keys, a.ids, a.rec, a.rows, a.seg_T, a.seg_C, a.image, a.alpha, a.blending_weights, a.kept0, a.kept1, a.n_kept, a.W, a.H, a.gw);
    INPC_LAUNCH_CHECK("blend_bilinear_pair_forward_kernel");
    return INPC_OK;
}
template <int PASS, int KIND, int C4, bool ROWS>
int launch_forward_pass(const WarpItem* items, const uint32_t* counts, unsigned* ticket, const ForwardPassArgs& a, bool pairs, cudaStream_t stream) {
    if constexpr (KIND == BLEND_TRAIN) {
        if (pairs) return launch_pair_forward_pass<PASS, C4, ROWS>(items, counts, ticket, a, stream);
    }
    return launch_warp_forward_pass<PASS, KIND, C4, ROWS>(items, counts, ticket, a, stream);
}

// C4, `rows`: feature rows of 4 C4 channels (ROWS), or one group of four channels in the records.
template <int KIND, int C4 = 1, bool ROWS = false>
int launch_bilinear_warp_forward(const RasterParams& rp, int64_t n_points, const PointBlob& pb, const InstanceBlob& ib, int t_alt, const float4* rows, float* image,
                                 float* depth, float* alpha, float* blending_weights, cudaStream_t stream) {
    const unsigned grid = small_grid();
    const int W = rp.v.width, H = rp.v.height;
    // the ping-pong buffers the tile sort left unused receive the compacted lists (part 0: ids, part 1: keys)
    const uint32_t* keys = ib.keys[t_alt];
    const uint32_t* ids = ib.ids[t_alt];
    uint32_t* kept0 = ib.ids[1 - t_alt];
    uint32_t* kept1 = ib.keys[1 - t_alt];
    const unsigned threads = kWarpBlendWarps * 32;
    const ForwardPassArgs a{keys, ids, pb.rec, rows, ib.seg_T, ib.seg_C, ib.seg_Z, ib.seg_E, image, depth, alpha, blending_weights,
                            kept0, kept1, ib.n_kept, W, H, rp.gw, rp.gh};
    const bool pairs = by_two_warps(INPC_MODE_BILINEAR, ROWS, (int64_t)rp.gw * rp.gh, n_points);
    int rc_pass = launch_forward_pass<PASS_FIRST, KIND, C4, ROWS>(ib.items0, ib.n_segments, ib.n_segments + 2, a, pairs, stream);
    if (rc_pass != INPC_OK) return rc_pass;
    rc_pass = launch_warp_forward_pass<PASS_PRODUCT, KIND, 1, ROWS>(ib.items1, ib.n_segments, ib.n_segments + 3, a, stream);
    if (rc_pass != INPC_OK) return rc_pass;
    rc_pass = launch_forward_pass<PASS_REST, KIND, C4, ROWS>(ib.items1, ib.n_segments, ib.n_segments + 4, a, pairs, stream);
    if (rc_pass != INPC_OK) return rc_pass;
    launch_chained(warp_blend_combine_kernel<KIND, C4>, grid, threads, 0, stream, ib.items0, ib.n_segments, tiles_with_segments(!ROWS), ib.seg_C, ib.seg_Z, ib.seg_E,
                                                                      image, depth, alpha, W, H, rp.gw, rp.gh, ROWS ? 0 : rp.gw * rp.gh * rp.n_sets);
    INPC_LAUNCH_CHECK("warp_blend_combine_kernel");
    return INPC_OK;
}

int launch_bilinear_warp_backward(const RasterParams& rp, int64_t n_points, const PointBlob& pb, const InstanceBlob& ib, int t_alt, const float* grad_image,
                                  const float* grad_alpha, const float* image, const float* alpha, float4* slot_grad,
                                  unsigned* slot_mask, cudaStream_t stream) {
    auto launch = [&](auto kernel, const char* name, size_t smem, int most, unsigned takers, unsigned visits_each, int (&known)[kMaxDevices]) -> int {
        BlendGrid grid;
        const int rc = warp_blend_grid(kernel, smem, most, takers, visits_each, PASS_FIRST, known, &grid);
        if (rc != INPC_OK) return rc;
        launch_chained(kernel, grid.blocks, kWarpBlendWarps * 32, smem, stream,
            ib.items0, ib.items1, ib.n_segments, ib.n_segments + 5, grid.visits, ib.ids[1 - t_alt], ib.keys[1 - t_alt], ib.n_kept, pb.rec,
            ib.seg_T, ib.seg_C, grad_image, grad_alpha, image, alpha, slot_grad, slot_mask, rp.v.width, rp.v.height, rp.gw);
        INPC_LAUNCH_CHECK(name);
        return INPC_OK;
    };
    static int known[kMaxDevices] = {0}, known_pairs[kMaxDevices] = {0};
    return by_two_warps(INPC_MODE_BILINEAR, false, (int64_t)rp.gw * rp.gh, n_points)
               ? launch(blend_bilinear_pair_backward_kernel, "blend_bilinear_pair_backward_kernel", kPairBackwardSmemBytes, kPairBackwardBlocks, kPairs, kVisitsPairBackward, known_pairs)
               : launch(blend_bilinear_warp_backward_kernel, "blend_bilinear_warp_backward_kernel", kWarpBackwardSmemBytes, kBackwardBlocks, kWarpBlendWarps, kVisits, known);
}

template <int T, int KIND>
int launch_bilinear_forward(const RasterParams& rp, const PointBlob& pb, const InstanceBlob& ib, const uint32_t* ids, float* image,
                            float* depth, float* alpha, float* blending_weights, cudaStream_t stream) {
    constexpr int IPT = BlendConfig<T>::kIpt;
    const int n_tiles = rp.gw * rp.gh * rp.n_sets;
    const int W = rp.v.width, H = rp.v.height;
    const unsigned grid = (unsigned)ib.max_segments;
    launch_chained(blend_bilinear_transmittance_kernel<T, IPT>, grid, T * T, 0, stream, ib.segs, ib.n_segments, ids, pb.rec, ib.seg_T, W, H, rp.gw);
    INPC_LAUNCH_CHECK("blend_bilinear_transmittance_kernel");
    launch_chained(blend_prefix_kernel<T>, n_tiles, T * T, 0, stream, ib.segs, ib.tile_first, ib.seg_T);
    INPC_LAUNCH_CHECK("blend_prefix_kernel");
    launch_chained(blend_bilinear_forward_kernel<T, IPT, KIND>, grid, T * T, 0, stream, ib.segs, ib.n_segments, ids, pb.rec, ib.seg_T, ib.seg_C, ib.seg_Z,
                                                                           image, depth, alpha, blending_weights, W, H, rp.gw);
    INPC_LAUNCH_CHECK("blend_bilinear_forward_kernel");
    launch_chained(blend_combine_kernel<T, KIND>, n_tiles, T * T, 0, stream, ib.segs, ib.tile_first, ib.seg_C, ib.seg_Z, ib.seg_T, image, depth, alpha,
                                                                W, H, rp.gw);
    INPC_LAUNCH_CHECK("blend_combine_kernel");
    return INPC_OK;
}

template <int T>
int launch_bilinear_backward(const RasterParams& rp, const PointBlob& pb, const InstanceBlob& ib, const uint32_t* ids,
                             const float* grad_image, const float* grad_alpha, const float* image, const float* alpha, float4* gfv,
                             float* grad_opacities, cudaStream_t stream) {
    constexpr int IPT = BlendConfig<T>::kIpt;
    constexpr size_t smem = backward_smem_bytes<T, IPT>();
    static bool attr_set[kMaxDevices] = {false};
    {
        const int rc_attr = opt_in_dynamic_smem(blend_bilinear_backward_kernel<T, IPT>, smem, attr_set);
        if (rc_attr != INPC_OK) return rc_attr;
    }
    launch_chained(blend_bilinear_backward_kernel<T, IPT>, (unsigned)ib.max_segments, T * T, smem, stream,
        ib.segs, ib.n_segments, ids, pb.rec, ib.seg_T, ib.seg_C, grad_image, grad_alpha, image, alpha, gfv, grad_opacities,
        rp.v.width, rp.v.height, rp.gw);
    INPC_LAUNCH_CHECK("blend_bilinear_backward_kernel");
    return INPC_OK;
}

template <int PASS, int KIND>
int launch_gaussian_warp_forward_pass(const WarpItem* items, const uint32_t* counts, unsigned* ticket, const float4* conic,
                                      const ForwardPassArgs& a, float threshold, float reach, cudaStream_t stream) {
    static int known[kMaxDevices] = {0};
    constexpr size_t smem = gauss_forward_smem_bytes<PASS, KIND>();
    BlendGrid grid;
    const int rc = warp_blend_grid(blend_gaussian_warp_forward_kernel<PASS, KIND>, smem, kGaussForwardBlocks, kWarpBlendWarps, 0u, PASS, known, &grid);
    if (rc != INPC_OK) return rc;
    launch_chained(blend_gaussian_warp_forward_kernel<PASS, KIND>, grid.blocks, kWarpBlendWarps * 32, smem, stream,
        items, counts, ticket, grid.visits, a.keys, a.ids, a.rec, conic, a.seg_T, a.seg_C, a.seg_Z, a.seg_E, a.image, a.depth, a.alpha, a.blending_weights,
        a.kept0, a.kept1, a.n_kept, a.W, a.H, a.gw, threshold, reach);
    INPC_LAUNCH_CHECK("blend_gaussian_warp_forward_kernel");
    return INPC_OK;
}

template <int PASS>
int launch_gaussian_pair_forward_pass(const WarpItem* items, const uint32_t* counts, unsigned* ticket, const float4* conic, const ForwardPassArgs& a, float reach, cudaStream_t stream) {
    static int known[kMaxDevices] = {0};
    BlendGrid grid;
    const int rc = warp_blend_grid(blend_gaussian_pair_forward_kernel<PASS>, kGaussPairSmemBytes, kGaussPairBlocks, kPairs, 0u, PASS, known, &grid);
    if (rc != INPC_OK) return rc;
    launch_chained(blend_gaussian_pair_forward_kernel<PASS>, grid.blocks, kWarpBlendWarps * 32, kGaussPairSmemBytes, stream,
        items, counts, ticket, grid.visits, a.keys, a.ids, a.rec, conic, a.seg_T, a.seg_C, a.image, a.alpha, a.blending_weights, a.kept0, a.kept1, a.n_kept, a.W, a.H, a.gw, reach);
    INPC_LAUNCH_CHECK("blend_gaussian_pair_forward_kernel");
    return INPC_OK;
}

template <int KIND>
int launch_gaussian_warp_forward(const RasterParams& rp, int64_t n_points, const PointBlob& pb, const InstanceBlob& ib, int t_alt, float* image, float* depth,
                                 float* alpha, float* blending_weights, float threshold, cudaStream_t stream) {
    const unsigned grid = small_grid();
    int rc;
    const int W = rp.v.width, H = rp.v.height;
    const unsigned threads = kWarpBlendWarps * 32;
    const ForwardPassArgs a{ib.keys[t_alt], ib.ids[t_alt], pb.rec, nullptr, ib.seg_T, ib.seg_C, ib.seg_Z, ib.seg_E, image, depth, alpha, blending_weights,
                            ib.ids[1 - t_alt], ib.keys[1 - t_alt], ib.n_kept, W, H, rp.gw, rp.gh};
    const bool pairs = by_two_warps(INPC_MODE_GAUSSIAN, false, (int64_t)rp.gw * rp.gh, n_points);
    auto blend = [&](auto which, const WarpItem* items, int at) -> int {
        constexpr int kPass = decltype(which)::value;
        if constexpr (KIND == BLEND_TRAIN) {
            if (pairs) return launch_gaussian_pair_forward_pass<kPass>(items, ib.n_segments, ib.n_segments + at, pb.conic, a, rp.reach, stream);
        }
        return launch_gaussian_warp_forward_pass<kPass, KIND>(items, ib.n_segments, ib.n_segments + at, pb.conic, a, threshold, rp.reach, stream);
    };
    rc = blend(std::integral_constant<int, PASS_FIRST>{}, ib.items0, 2);
    if (rc != INPC_OK) return rc;
    rc = launch_gaussian_warp_forward_pass<PASS_PRODUCT, KIND>(ib.items1, ib.n_segments, ib.n_segments + 3, pb.conic, a, threshold, rp.reach, stream);
    if (rc != INPC_OK) return rc;
    rc = blend(std::integral_constant<int, PASS_REST>{}, ib.items1, 4);
    if (rc != INPC_OK) return rc;
    launch_chained(warp_blend_combine_kernel<KIND, 1>, grid, threads, 0, stream, ib.items0, ib.n_segments, tiles_with_segments(true), ib.seg_C, ib.seg_Z, ib.seg_E, image, depth, alpha, W, H,
                                                                     rp.gw, rp.gh, rp.gw * rp.gh * rp.n_sets);
    INPC_LAUNCH_CHECK("warp_blend_combine_kernel");
    return INPC_OK;
}

int launch_gaussian_warp_backward(const RasterParams& rp, const PointBlob& pb, const InstanceBlob& ib, int t_alt, const float* grad_image,
                                  const float* grad_alpha, const float* image, const float* alpha, float4* gfv, float* grad_opacities,
                                  cudaStream_t stream) {
    static int known[kMaxDevices] = {0};
    BlendGrid grid;
    const int rc = warp_blend_grid(blend_gaussian_warp_backward_kernel, kGaussBackwardSmemBytes, kGaussBackwardBlocks, kWarpBlendWarps, 0u, PASS_FIRST, known, &grid);
    if (rc != INPC_OK) return rc;
    launch_chained(blend_gaussian_warp_backward_kernel, grid.blocks, kWarpBlendWarps * 32, kGaussBackwardSmemBytes, stream,
        ib.items0, ib.items1, ib.n_segments, ib.n_segments + 5, grid.visits, ib.ids[1 - t_alt], ib.keys[1 - t_alt], ib.n_kept, pb.rec, pb.conic, ib.seg_T, ib.seg_C,
        grad_image, grad_alpha, image, alpha, gfv, grad_opacities, rp.v.width, rp.v.height, rp.gw, rp.reach);
    INPC_LAUNCH_CHECK("blend_gaussian_warp_backward_kernel");
    return INPC_OK;
}

template <int T, int KIND>
int launch_gaussian_forward(const RasterParams& rp, const PointBlob& pb, const InstanceBlob& ib, const uint32_t* ids, float* image,
                            float* depth, float* alpha, float* blending_weights, float threshold, cudaStream_t stream) {
    const int n_tiles = rp.gw * rp.gh * rp.n_sets;
    const int W = rp.v.width, H = rp.v.height;
    const unsigned grid = (unsigned)ib.max_segments;
    const float neg_log_threshold = -logf(threshold);
    launch_chained(blend_gaussian_transmittance_kernel<T, KIND == BLEND_INFER>, grid, T * T, 0, stream, ib.segs, ib.n_segments, ids, pb.rec, pb.conic, ib.seg_T, W, H,
                                                                                          rp.gw, threshold, neg_log_threshold);
    INPC_LAUNCH_CHECK("blend_gaussian_transmittance_kernel");
    launch_chained(blend_prefix_kernel<T>, n_tiles, T * T, 0, stream, ib.segs, ib.tile_first, ib.seg_T);
    INPC_LAUNCH_CHECK("blend_prefix_kernel");
    launch_chained(blend_gaussian_forward_kernel<T, KIND>, grid, T * T, 0, stream, ib.segs, ib.n_segments, ids, pb.rec, pb.conic, ib.seg_T, ib.seg_C, ib.seg_Z, image,
                                                                      depth, alpha, blending_weights, W, H, rp.gw, threshold, neg_log_threshold);
    INPC_LAUNCH_CHECK("blend_gaussian_forward_kernel");
    launch_chained(blend_combine_kernel<T, KIND>, n_tiles, T * T, 0, stream, ib.segs, ib.tile_first, ib.seg_C, ib.seg_Z, ib.seg_T, image, depth, alpha, W, H, rp.gw);
    INPC_LAUNCH_CHECK("blend_combine_kernel");
    return INPC_OK;
}

template <int KIND>
int launch_blend_forward(int mode, const RasterParams& rp, const PointBlob& pb, const InstanceBlob& ib, const inpc_raster_state* st,
                         float* image, float* depth, float* alpha, float* blending_weights, float threshold,
                         cudaStream_t stream) {
    const int n_tiles = rp.gw * rp.gh * rp.n_sets;
    const int t_alt = tile_buffer_of(n_tiles);
    const uint32_t* ids = ib.ids[t_alt];
    StageScope scope(STAGE_BLEND_FWD, stream);
    if (mode == INPC_MODE_BILINEAR) {
        if (rp.tile == 8) return launch_bilinear_warp_forward<KIND>(rp, st->n_points, pb, ib, t_alt, nullptr, image, depth, alpha, blending_weights, stream);
        return launch_bilinear_forward<16, KIND>(rp, pb, ib, ids, image, depth, alpha, blending_weights, stream);
    }
    if (rp.tile == 8) return launch_gaussian_warp_forward<KIND>(rp, st->n_points, pb, ib, t_alt, image, depth, alpha, blending_weights, threshold, stream);
    return launch_gaussian_forward<16, KIND>(rp, pb, ib, ids, image, depth, alpha, blending_weights, threshold, stream);
}

template <int T, int C4, int KIND>
int launch_rows_forward(const RasterParams& rp, const PointBlob& pb, const InstanceBlob& ib, const uint32_t* ids, const float* features,
                        float* image, float* depth, float* alpha, float* blending_weights, cudaStream_t stream) {
    static_assert(T == 16, "8x8 tiles take the warp blend");
    constexpr size_t smem = rows_forward_smem_bytes<T, C4>();
    static bool attr_set[kMaxDevices] = {false};
    {
        const int rc_attr = opt_in_dynamic_smem(blend_rows_forward_kernel<T, C4, KIND>, smem, attr_set);
        if (rc_attr != INPC_OK) return rc_attr;
    }
    const int n_tiles = rp.gw * rp.gh * rp.n_sets;
    const int W = rp.v.width, H = rp.v.height;
    const unsigned grid = (unsigned)ib.max_segments;
    launch_chained(blend_bilinear_transmittance_kernel<T, 1>, grid, T * T, 0, stream, ib.segs, ib.n_segments, ids, pb.rec, ib.seg_T, W, H, rp.gw);
    INPC_LAUNCH_CHECK("blend_bilinear_transmittance_kernel");
    launch_chained(blend_prefix_kernel<T>, n_tiles, T * T, 0, stream, ib.segs, ib.tile_first, ib.seg_T);
    INPC_LAUNCH_CHECK("blend_prefix_kernel");
    launch_chained(blend_rows_forward_kernel<T, C4, KIND>, grid, T * T, smem, stream, ib.segs, ib.n_segments, ids, pb.rec, reinterpret_cast<const float4*>(features),
                                                                         ib.seg_T, ib.seg_C, ib.seg_Z, image, depth, alpha, blending_weights, W, H, rp.gw);
    INPC_LAUNCH_CHECK("blend_rows_forward_kernel");
    launch_chained(blend_rows_combine_kernel<T, C4, KIND>, n_tiles, T * T, 0, stream, ib.segs, ib.tile_first, ib.seg_C, ib.seg_Z, ib.seg_T, image, depth, alpha,
                                                                         W, H, rp.gw);
    INPC_LAUNCH_CHECK("blend_rows_combine_kernel");
    return INPC_OK;
}

template <int C4>
int launch_rows_warp_backward(const RasterParams& rp, const PointBlob& pb, const InstanceBlob& ib, int t_alt, const float* features,
                              const float* grad_image, const float* grad_alpha, const float* image, const float* alpha,
                              float* grad_features, float* grad_opacities, cudaStream_t stream) {
    static int known[kMaxDevices] = {0};
    constexpr size_t smem = rows_warp_backward_smem_bytes<C4>();
    BlendGrid grid;
    const int rc = warp_blend_grid(blend_rows_warp_backward_kernel<C4>, smem, rows_backward_blocks(C4), kWarpBlendWarps, 0u, PASS_FIRST, known, &grid);
    if (rc != INPC_OK) return rc;
    launch_chained(blend_rows_warp_backward_kernel<C4>, grid.blocks, kWarpBlendWarps * 32, smem, stream,
        ib.items0, ib.items1, ib.n_segments, ib.n_segments + 5, grid.visits, ib.ids[1 - t_alt], ib.keys[1 - t_alt], ib.n_kept, pb.rec,
        reinterpret_cast<const float4*>(features), ib.seg_T, ib.seg_C, grad_image, grad_alpha, image, alpha,
        reinterpret_cast<float4*>(grad_features), grad_opacities, rp.v.width, rp.v.height, rp.gw);
    INPC_LAUNCH_CHECK("blend_rows_warp_backward_kernel");
    return INPC_OK;
}

template <int T, int C4>
int launch_rows_backward(const RasterParams& rp, const PointBlob& pb, const InstanceBlob& ib, const uint32_t* ids, const float* features,
                         const float* grad_image, const float* grad_alpha, const float* image, const float* alpha,
                         float* grad_features, float* grad_opacities, cudaStream_t stream) {
    constexpr size_t smem = rows_backward_smem_bytes<T, C4>();
    static bool attr_set[kMaxDevices] = {false};
    {
        const int rc_attr = opt_in_dynamic_smem(blend_rows_backward_kernel<T, C4>, smem, attr_set);
        if (rc_attr != INPC_OK) return rc_attr;
    }
    launch_chained(blend_rows_backward_kernel<T, C4>, (unsigned)ib.max_segments, T * T, smem, stream,
        ib.segs, ib.n_segments, ids, pb.rec, reinterpret_cast<const float4*>(features), ib.seg_T, ib.seg_C, grad_image, grad_alpha, image, alpha,
        reinterpret_cast<float4*>(grad_features), grad_opacities, rp.v.width, rp.v.height, rp.gw);
    INPC_LAUNCH_CHECK("blend_rows_backward_kernel");
    return INPC_OK;
}

// The channel count is a template parameter of the kernels: one switch for all of them.
template <typename F>
int dispatch_rows(int channels, F&& f) {
    if (channels == 4) return f(std::integral_constant<int, 1>());
    if (channels == 8) return f(std::integral_constant<int, 2>());
    if (channels == 16) return f(std::integral_constant<int, 4>());
    if (channels == 32) return f(std::integral_constant<int, 8>());
    set_error("feature rows: channels must be 4, 8, 16 or 32 (got %d)", channels);
    return INPC_E_INVALID;
}

// The outputs of a call that start at zero.  Images do so for feature rows on 8x8 tiles alone: of 16 planes the empty tiles take longer to blank (28 us of a
// 1237x822 image, warp_blend_combine_kernel) than everything to clear (10); with four channels and the alpha 3840x2160 pixels take 25 us to clear, the empty tiles 8.
ClearList weights_to_clear(float* weights, int64_t n) {
    ClearList list;
    list.add(weights, sizeof(float) * (size_t)n);
    return list;
}
ClearList rows_to_clear(const RasterParams& rp, int channels, float* image, float* depth, float* alpha, float* weights, int64_t n) {
    ClearList list = weights_to_clear(weights, n);
    if (uses_warp_blend(rp.tile)) {
        const size_t n_px = (size_t)rp.v.width * rp.v.height;
        list.add(image, sizeof(float) * channels * n_px);
        list.add(depth, sizeof(float) * n_px);
        list.add(alpha, sizeof(float) * n_px);
    }
    return list;
}

template <int KIND>
int rows_forward(int tile_size, const inpc_view* view, int64_t n, const float* positions, const float* features, int channels,
                 const float* opacities, float* image, float* depth, float* alpha, float* blending_weights,
                 inpc_alloc_fn alloc_point, inpc_alloc_fn alloc_instance, void* alloc_user, inpc_raster_state* state, cudaStream_t stream) {
    const RasterParams rp = make_params(view, tile_size, 0.0f, 3.0f, nullptr);
    PointBlob pb;
    InstanceBlob ib;
    int rc = run_front<INPC_MODE_BILINEAR, VAR_ROWS>(rp, n, positions, nullptr, opacities, alloc_point, alloc_instance, alloc_user, state,
                                                     KIND == BLEND_INFER, &pb, &ib, stream, KIND == BLEND_INFER ? "inpc_render_rows" : "inpc_rasterize_rows_forward",
                                                     rows_to_clear(rp, channels, image, depth, alpha, blending_weights, n), channels / 4);
    if (rc != INPC_OK) return rc;
    const int t_alt = tile_buffer_of(rp.gw * rp.gh);
    {
        StageScope scope(STAGE_BLEND_FWD, stream);
        rc = dispatch_rows(channels, [&](auto c4) {
            constexpr int kC4 = decltype(c4)::value;
            if (tile_size == 8)
                return launch_bilinear_warp_forward<KIND, kC4, true>(rp, n, pb, ib, t_alt, reinterpret_cast<const float4*>(features), image, depth, alpha, blending_weights, stream);
            return launch_rows_forward<16, kC4, KIND>(rp, pb, ib, ib.ids[t_alt], features, image, depth, alpha, blending_weights, stream);
        });
    }
    return rc != INPC_OK ? rc : end_index_checks(stream);
}

}  // namespace

}  // namespace inpc

using namespace inpc;

extern "C" int inpc_rasterize_forward(int mode, int tile_size, const inpc_view* view, int64_t n, const float* positions,
                                      const void* features, const float* opacities, float* image, float* alpha,
                                      float* blending_weights, inpc_alloc_fn alloc_point, inpc_alloc_fn alloc_instance,
                                      void* alloc_user, inpc_raster_state* state, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    int rc = check_view(view, tile_size, mode, n);
    if (rc != INPC_OK) return rc;
    if (!state || !alloc_point || !alloc_instance || !image || !alpha || (n > 0 && (!positions || !features || !opacities || !blending_weights))) {
        set_error("inpc_rasterize_forward: null argument");
        return INPC_E_INVALID;
    }
    const RasterParams rp = make_params(view, tile_size, 0.0f, 3.0f, nullptr);
    PointBlob pb;
    InstanceBlob ib;
    if (mode == INPC_MODE_BILINEAR)
        rc = run_front<INPC_MODE_BILINEAR, VAR_TRAIN>(rp, n, positions, features, opacities, alloc_point, alloc_instance, alloc_user, state, false, &pb, &ib, stream, "inpc_rasterize_forward", weights_to_clear(blending_weights, n));
    else
        rc = run_front<INPC_MODE_GAUSSIAN, VAR_TRAIN>(rp, n, positions, features, opacities, alloc_point, alloc_instance, alloc_user, state, false, &pb, &ib, stream, "inpc_rasterize_forward", weights_to_clear(blending_weights, n));
    if (rc != INPC_OK) return rc;
    rc = launch_blend_forward<BLEND_TRAIN>(mode, rp, pb, ib, state, image, nullptr, alpha, blending_weights, kTrainGaussThreshold, stream);
    return rc != INPC_OK ? rc : end_index_checks(stream);
}

extern "C" int inpc_rasterize_backward(const inpc_raster_state* state, const inpc_view* view, const float* grad_image,
                                       const float* grad_alpha, const float* image, const float* alpha,
                                       const float* positions, const float* opacities, float* grad_features_view,
                                       void* grad_features, float* grad_opacities, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (!state) { set_error("inpc_rasterize_backward: null state"); return INPC_E_INVALID; }
    int rc = check_view(view, state->tile_size, state->mode, state->n_points);
    if (rc != INPC_OK) return rc;
    const int64_t n = state->n_points;
    if (!grad_image || !grad_alpha || !image || !alpha || (n > 0 && (!positions || !grad_features_view || !grad_features || !grad_opacities || !state->point_blob || !state->instance_blob))) {
        set_error("inpc_rasterize_backward: null argument");
        return INPC_E_INVALID;
    }
    (void)opacities;   // the opacity travels in the point record
    if (n == 0) return INPC_OK;
    rc = begin_index_checks(n, stream);
    if (rc != INPC_OK) return rc;
    const RasterParams rp = make_params(view, state->tile_size, 0.0f, 3.0f, nullptr);
    const int n_tiles = rp.gw * rp.gh * rp.n_sets;
    const PointBlob pb = carve_point_blob(state->point_blob, n, state->mode, state->tile_size);
    const InstanceBlob ib = carve_instance_blob(state->instance_blob, instance_capacity(state), state->deferred_counts & 1, n_tiles, state->tile_size, state->mode, false);
    const uint32_t* ids = ib.ids[tile_buffer_of(n_tiles)];
    float4* gfv = reinterpret_cast<float4*>(grad_features_view);
    const int W = rp.v.width, H = rp.v.height;
    // the caller's scratch holds 33 floats per point: four 32-byte slot records and one mask word for the warp blend
    // or, for the other paths, the (n,4) accumulation buffer of their atomics
    const bool slots = has_instance_bound(state->mode, state->tile_size);
    if (slots && (reinterpret_cast<uintptr_t>(grad_features_view) & 31u)) {
        set_error("inpc_rasterize_backward: grad_features_view must be 32-byte aligned");
        return INPC_E_INVALID;
    }
    float4* slot_grad = gfv;
    unsigned* slot_mask = reinterpret_cast<unsigned*>(grad_features_view + 32 * (size_t)n);
    ClearList clear;
    if (slots) {
        clear.add(slot_mask, sizeof(unsigned) * (size_t)n);
    } else {
        clear.add(grad_features_view, sizeof(float4) * (size_t)n);
        clear.add(grad_opacities, sizeof(float) * (size_t)n);
    }
    if (uses_warp_blend(state->tile_size)) clear.add(ib.n_segments + 5, sizeof(uint32_t));   // the work ticket
    rc = launch_clear(clear, stream);
    if (rc != INPC_OK) return rc;
    {
        StageScope scope(STAGE_BLEND_BWD, stream);
        if (state->mode == INPC_MODE_BILINEAR) {
            rc = rp.tile == 8 ? launch_bilinear_warp_backward(rp, n, pb, ib, tile_buffer_of(n_tiles), grad_image, grad_alpha, image, alpha, slot_grad, slot_mask, stream)
                              : launch_bilinear_backward<16>(rp, pb, ib, ids, grad_image, grad_alpha, image, alpha, gfv, grad_opacities, stream);
            if (rc != INPC_OK) return rc;
        } else {
            if (rp.tile == 8) {
                rc = launch_gaussian_warp_backward(rp, pb, ib, tile_buffer_of(n_tiles), grad_image, grad_alpha, image, alpha, gfv, grad_opacities, stream);
                if (rc != INPC_OK) return rc;
            } else {
                launch_chained(blend_gaussian_backward_kernel<16>, (unsigned)ib.max_segments, 256, 0, stream, ib.segs, ib.n_segments, ids, pb.rec, pb.conic, ib.seg_T, ib.seg_C, grad_image, grad_alpha, image, alpha, gfv, grad_opacities, W, H, rp.gw);
                INPC_LAUNCH_CHECK("blend_gaussian_backward_kernel");
            }
        }
    }
    StageScope scope(STAGE_PREPROCESS_BWD, stream);
    const GradientSlots gs{slot_grad, slot_mask};
    const bool bulk_ok = (reinterpret_cast<uintptr_t>(grad_features) & 15u) == 0;
    if (slots)
        launch_chained(preprocess_backward_kernel<true>, (unsigned)ceil_div<int64_t>(n, kPreThreads), kPreThreads, 0, stream,
            positions, view->cam_position, pb.bounds, gfv, gs, grad_opacities, static_cast<__half*>(grad_features), n, bulk_ok);
    else
        launch_chained(preprocess_backward_kernel<false>, (unsigned)ceil_div<int64_t>(n, kPreThreads), kPreThreads, 0, stream,
            positions, view->cam_position, pb.bounds, gfv, gs, grad_opacities, static_cast<__half*>(grad_features), n, bulk_ok);
    INPC_LAUNCH_CHECK("preprocess_backward_kernel");
    return end_index_checks(stream);
}

extern "C" int inpc_render(int mode, int tile_size, const inpc_view* view, int64_t n, const float* positions,
                           const void* features_raw, float sigma_world, float sigma_cutoff, float* image, float* depth,
                           float* alpha, inpc_alloc_fn alloc_point, inpc_alloc_fn alloc_instance, void* alloc_user,
                           void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    int rc = check_view(view, tile_size, mode, n);
    if (rc != INPC_OK) return rc;
    if (!alloc_point || !alloc_instance || !image || !depth || !alpha || (n > 0 && (!positions || !features_raw))) {
        set_error("inpc_render: null argument");
        return INPC_E_INVALID;
    }
    const RasterParams rp = make_params(view, tile_size, sigma_world, sigma_cutoff, nullptr);
    inpc_raster_state st;
    PointBlob pb;
    InstanceBlob ib;
    if (mode == INPC_MODE_BILINEAR)
        rc = run_front<INPC_MODE_BILINEAR, VAR_RAW37>(rp, n, positions, features_raw, nullptr, alloc_point, alloc_instance, alloc_user, &st, true, &pb, &ib, stream, "inpc_render", ClearList());
    else
        rc = run_front<INPC_MODE_GAUSSIAN, VAR_RAW37>(rp, n, positions, features_raw, nullptr, alloc_point, alloc_instance, alloc_user, &st, true, &pb, &ib, stream, "inpc_render", ClearList());
    if (rc != INPC_OK) return rc;
    // runtime cut-off exp(-cutoff^2/2): src/gaussian/inference.cu:171
    const float threshold = expf(-0.5f * sigma_cutoff * sigma_cutoff);
    rc = launch_blend_forward<BLEND_INFER>(mode, rp, pb, ib, &st, image, depth, alpha, nullptr, threshold, stream);
    return rc != INPC_OK ? rc : end_index_checks(stream);
}

extern "C" int inpc_render_preextracted(int mode, int tile_size, const inpc_view* view, int64_t n, const float* positions,
                                        const void* features, const float* opacities, const float* scales,
                                        float sigma_world, float sigma_cutoff, float* image, float* depth, float* alpha,
                                        inpc_alloc_fn alloc_point, inpc_alloc_fn alloc_instance, void* alloc_user,
                                        void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    int rc = check_view(view, tile_size, mode, n);
    if (rc != INPC_OK) return rc;
    if (!alloc_point || !alloc_instance || !image || !depth || !alpha || (n > 0 && (!positions || !features || !opacities))) {
        set_error("inpc_render_preextracted: null argument");
        return INPC_E_INVALID;
    }
    const RasterParams rp = make_params(view, tile_size, sigma_world, sigma_cutoff, scales);
    inpc_raster_state st;
    PointBlob pb;
    InstanceBlob ib;
    if (mode == INPC_MODE_BILINEAR)
        rc = run_front<INPC_MODE_BILINEAR, VAR_PREEXTRACTED>(rp, n, positions, features, opacities, alloc_point, alloc_instance, alloc_user, &st, true, &pb, &ib, stream, "inpc_render_preextracted", ClearList());
    else
        rc = run_front<INPC_MODE_GAUSSIAN, VAR_PREEXTRACTED>(rp, n, positions, features, opacities, alloc_point, alloc_instance, alloc_user, &st, true, &pb, &ib, stream, "inpc_render_preextracted", ClearList());
    if (rc != INPC_OK) return rc;
    const float threshold = expf(-0.5f * sigma_cutoff * sigma_cutoff);
    rc = launch_blend_forward<BLEND_INFER>(mode, rp, pb, ib, &st, image, depth, alpha, nullptr, threshold, stream);
    return rc != INPC_OK ? rc : end_index_checks(stream);
}

extern "C" int inpc_render_multi(int tile_size, const inpc_view* view, int n_sets, const int64_t* n_points, const float* const* positions,
                                 const void* const* features_raw, float* images, float* depths, float* alphas,
                                 inpc_alloc_fn alloc_point, inpc_alloc_fn alloc_instance, void* alloc_user, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (n_sets < 1 || n_sets > kMaxSets) { set_error("inpc_render_multi: n_sets=%d outside [1, %d]", n_sets, kMaxSets); return INPC_E_INVALID; }
    if (!n_points || !positions || !features_raw || !alloc_point || !alloc_instance || !images || !depths || !alphas) {
        set_error("inpc_render_multi: null argument");
        return INPC_E_INVALID;
    }
    if (tile_size != 8) { set_error("inpc_render_multi: bilinear splats on 8x8 tiles only (tile_size %d)", tile_size); return INPC_E_INVALID; }
    PointSets ps;
    ps.count = n_sets;
    int64_t cursor = 0;
    for (int j = 0; j < n_sets; ++j) {
        if (n_points[j] < 0 || (n_points[j] > 0 && (!positions[j] || !features_raw[j]))) { set_error("inpc_render_multi: bad set %d", j); return INPC_E_INVALID; }
        ps.start[j] = cursor;
        ps.size[j] = n_points[j];
        ps.positions[j] = positions[j];
        ps.features[j] = features_raw[j];
        ps.opacities[j] = nullptr;
        cursor = (cursor + n_points[j] + kSetAlign - 1) / kSetAlign * kSetAlign;   // every set starts a block of the input passes
    }
    ps.start[n_sets] = cursor;
    const int64_t n_virtual = cursor;
    int rc = check_view(view, tile_size, INPC_MODE_BILINEAR, n_virtual);
    if (rc != INPC_OK) return rc;
    RasterParams rp = make_params(view, tile_size, 0.0f, 3.0f, nullptr);
    rp.n_sets = n_sets;
    // the stacked grid has to fit what a single image may use: tile indices in 24 bits, tile rows in 11
    if ((int64_t)rp.gw * rp.gh * n_sets > ((int64_t)1 << kTileKeyBits) || (int64_t)rp.gh * n_sets > kMaxCodedTileRows) {
        set_error("inpc_render_multi: %d images of %dx%d exceed the stacked tile grid", n_sets, view->width, view->height);
        return INPC_E_INVALID;
    }
    inpc_raster_state st;
    PointBlob pb;
    InstanceBlob ib;
    rc = run_front<INPC_MODE_BILINEAR, VAR_RAW37>(rp, n_virtual, nullptr, nullptr, nullptr, alloc_point, alloc_instance, alloc_user, &st, true, &pb, &ib,
                                                  stream, "inpc_render_multi", ClearList(), 1, &ps);
    if (rc != INPC_OK) return rc;
    rc = launch_blend_forward<BLEND_INFER>(INPC_MODE_BILINEAR, rp, pb, ib, &st, images, depths, alphas, nullptr, 0.0f, stream);
    return rc != INPC_OK ? rc : end_index_checks(stream);
}

namespace {
int check_rows(const inpc_view* view, int tile_size, int64_t n, int channels) {
    const int rc = check_view(view, tile_size, INPC_MODE_BILINEAR, n);
    if (rc != INPC_OK) return rc;
    if (channels != 4 && channels != 8 && channels != 16 && channels != 32) { set_error("feature rows: channels must be 4, 8, 16 or 32, got %d", channels); return INPC_E_INVALID; }
    return INPC_OK;
}
}  // namespace

extern "C" int inpc_rasterize_rows_forward(int tile_size, const inpc_view* view, int64_t n, const float* positions,
                                           const float* features, int channels, const float* opacities, float* image,
                                           float* alpha, float* blending_weights, inpc_alloc_fn alloc_point,
                                           inpc_alloc_fn alloc_instance, void* alloc_user, inpc_raster_state* state, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    int rc = check_rows(view, tile_size, n, channels);
    if (rc != INPC_OK) return rc;
    if (!state || !alloc_point || !alloc_instance || !image || !alpha || (n > 0 && (!positions || !features || !opacities || !blending_weights))) {
        set_error("inpc_rasterize_rows_forward: null argument");
        return INPC_E_INVALID;
    }
    if (reinterpret_cast<uintptr_t>(features) & 15u) { set_error("inpc_rasterize_rows_forward: features must be 16-byte aligned"); return INPC_E_INVALID; }
    return rows_forward<BLEND_TRAIN>(tile_size, view, n, positions, features, channels, opacities, image, nullptr, alpha, blending_weights,
                                     alloc_point, alloc_instance, alloc_user, state, stream);
}

extern "C" int inpc_render_rows(int tile_size, const inpc_view* view, int64_t n, const float* positions, const float* features,
                                int channels, const float* opacities, float* image, float* depth, float* alpha,
                                inpc_alloc_fn alloc_point, inpc_alloc_fn alloc_instance, void* alloc_user, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    int rc = check_rows(view, tile_size, n, channels);
    if (rc != INPC_OK) return rc;
    if (!alloc_point || !alloc_instance || !image || !depth || !alpha || (n > 0 && (!positions || !features || !opacities))) {
        set_error("inpc_render_rows: null argument");
        return INPC_E_INVALID;
    }
    if (reinterpret_cast<uintptr_t>(features) & 15u) { set_error("inpc_render_rows: features must be 16-byte aligned"); return INPC_E_INVALID; }
    inpc_raster_state st;
    return rows_forward<BLEND_INFER>(tile_size, view, n, positions, features, channels, opacities, image, depth, alpha, nullptr,
                                     alloc_point, alloc_instance, alloc_user, &st, stream);
}

extern "C" int inpc_rasterize_rows_backward(const inpc_raster_state* state, const inpc_view* view, const float* grad_image,
                                            const float* grad_alpha, const float* image, const float* alpha, const float* features,
                                            float* grad_features, float* grad_opacities, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (!state) { set_error("inpc_rasterize_rows_backward: null state"); return INPC_E_INVALID; }
    int rc = check_rows(view, state->tile_size, state->n_points, state->channels);
    if (rc != INPC_OK) return rc;
    if (state->mode != INPC_MODE_BILINEAR) { set_error("inpc_rasterize_rows_backward: state is not from inpc_rasterize_rows_forward"); return INPC_E_INVALID; }
    const int64_t n = state->n_points;
    const int channels = state->channels;
    if (!grad_image || !grad_alpha || !image || !alpha || (n > 0 && (!features || !grad_features || !grad_opacities || !state->point_blob || !state->instance_blob))) {
        set_error("inpc_rasterize_rows_backward: null argument");
        return INPC_E_INVALID;
    }
    if ((reinterpret_cast<uintptr_t>(features) | reinterpret_cast<uintptr_t>(grad_features)) & 15u) {
        set_error("inpc_rasterize_rows_backward: features and grad_features must be 16-byte aligned");
        return INPC_E_INVALID;
    }
    if (n == 0) return INPC_OK;
    const RasterParams rp = make_params(view, state->tile_size, 0.0f, 3.0f, nullptr);
    const int n_tiles = rp.gw * rp.gh * rp.n_sets;
    const PointBlob pb = carve_point_blob(state->point_blob, n, state->mode, state->tile_size);
    const InstanceBlob ib = carve_instance_blob(state->instance_blob, instance_capacity(state), state->deferred_counts & 1, n_tiles, state->tile_size, state->mode, false, channels / 4);
    const int t_alt = tile_buffer_of(n_tiles);
    ClearList clear;
    clear.add(grad_features, sizeof(float) * (size_t)n * channels);
    clear.add(grad_opacities, sizeof(float) * (size_t)n);
    if (state->tile_size == 8) clear.add(ib.n_segments + 5, sizeof(uint32_t));   // the work ticket
    rc = launch_clear(clear, stream);
    if (rc != INPC_OK) return rc;
    rc = begin_index_checks(n, stream);
    if (rc != INPC_OK) return rc;
    {
        StageScope scope(STAGE_BLEND_BWD, stream);
        rc = dispatch_rows(channels, [&](auto c4) {
            constexpr int kC4 = decltype(c4)::value;
            if (state->tile_size == 8)
                return launch_rows_warp_backward<kC4>(rp, pb, ib, t_alt, features, grad_image, grad_alpha, image, alpha, grad_features, grad_opacities, stream);
            return launch_rows_backward<16, kC4>(rp, pb, ib, ib.ids[t_alt], features, grad_image, grad_alpha, image, alpha, grad_features, grad_opacities, stream);
        });
    }
    return rc != INPC_OK ? rc : end_index_checks(stream);
}

extern "C" int inpc_raster_resolve(inpc_raster_state* state, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (!state) { set_error("inpc_raster_resolve: null state"); return INPC_E_INVALID; }
    if (!(state->deferred_counts & 1) || state->n_points == 0) return INPC_OK;
    if (!state->point_blob) { set_error("inpc_raster_resolve: state without a point blob"); return INPC_E_INVALID; }
    const PointBlob pb = carve_point_blob(state->point_blob, state->n_points, state->mode, state->tile_size);
    unsigned long long host[3];
    INPC_CUDA_TRY(cudaMemcpyAsync(host, pb.counters, sizeof(host), cudaMemcpyDeviceToHost, stream));
    INPC_CUDA_TRY(cudaStreamSynchronize(stream));
    // a call whose sort has failed has counted nothing, and says so here
    const int rc_prev = check_previous_calls();
    if (rc_prev != INPC_OK) return rc_prev;
    state->n_visible = (int64_t)host[0];
    state->n_instances = (int64_t)host[1];
    if (state->n_visible == 0) state->depth_key_base = 0u;
    // three counts made independently: by the depth sort's histogram, from the sorted keys, and of the instances written
    if (state->n_visible < 0 || state->n_visible > state->n_points || state->n_instances < state->n_visible || state->n_instances > 4 * state->n_visible || host[2] != host[1]) {
        set_error("inconsistent counts: %lld of %lld points in the depth sort, %lld instances by its keys, %lld emitted", (long long)state->n_visible,
                  (long long)state->n_points, (long long)state->n_instances, (long long)host[2]);
        return INPC_E_DEVICE;
    }
    return INPC_OK;
}

namespace inpc_debug {
__global__ void sorted_depths_kernel(const uint32_t* __restrict__ ids, const PointRec* __restrict__ rec, int rec_stride, int64_t n, uint32_t* __restrict__ dst) {
    await_previous_kernel();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = __float_as_uint(reinterpret_cast<const float4*>(rec)[(int64_t)ids[i] * rec_stride].w);
}

__global__ void unpack_points_kernel(const PointRec* __restrict__ rec, int rec_stride, const uint2* __restrict__ bounds, const uint32_t* __restrict__ quad, int64_t n, int which,
                                     int gw, void* __restrict__ dst) {
    await_previous_kernel();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint2 b = quad ? quad_bounds(quad[i], gw) : bounds[i];
    const bool vis = tiles_of(b) != 0u;
    const float4* r = reinterpret_cast<const float4*>(rec) + i * rec_stride;
    if (which == 4) static_cast<unsigned*>(dst)[i] = tiles_of(b);
    else if (which == 5) { const float4 a = vis ? r[0] : make_float4(0, 0, 0, 0); static_cast<float2*>(dst)[i] = make_float2(a.x, a.y); }
    else if (which == 6) static_cast<float*>(dst)[i] = vis ? r[0].w : 0.0f;
    else if (which == 7) static_cast<float4*>(dst)[i] = vis && rec_stride == 2 ? r[1] : make_float4(0, 0, 0, 0);
    else if (which == 8) {
        unsigned short* o = static_cast<unsigned short*>(dst) + 4 * i;
        o[0] = (unsigned short)(b.x & 0xffffu); o[1] = (unsigned short)(b.x >> 16);
        o[2] = (unsigned short)(b.y & 0xffffu); o[3] = (unsigned short)(b.y >> 16);
    }
}

__global__ void arithmetic_kernel(int which, int64_t n, const float* __restrict__ in, void* __restrict__ out) {
    await_previous_kernel();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (which == 0) {
        static_cast<float*>(out)[i] = one_minus_alpha_reciprocal(in[i]);
    } else {
        const float* v = in + 8 * i;
        static_cast<unsigned*>(out)[i] = ellipse_pixels(make_float4(v[0], v[1], 0.0f, 0.0f), make_float4(v[2], v[3], v[4], 0.0f), v[5], (int)v[6], (int)v[7]);
    }
}
}  // namespace inpc_debug

extern "C" int inpc_debug_arithmetic(int which, int64_t n, const float* in, void* out, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (which < 0 || which > 1 || n < 0 || n >= ((int64_t)1 << 30) || (n > 0 && (!in || !out))) { set_error("inpc_debug_arithmetic: bad argument"); return INPC_E_INVALID; }
    if (n == 0) return INPC_OK;
    launch_chained(inpc_debug::arithmetic_kernel, (unsigned)ceil_div<int64_t>(n, 256), 256, 0, stream, which, n, in, out);
    INPC_LAUNCH_CHECK("arithmetic_kernel");
    return INPC_OK;
}

extern "C" int inpc_raster_debug_copy(const inpc_raster_state* state, const inpc_view* view, int which, void* dst,
                                      void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (!state || !view || !dst) { set_error("inpc_raster_debug_copy: null argument"); return INPC_E_INVALID; }
    const int gw = ceil_div(view->width, state->tile_size), gh = ceil_div(view->height, state->tile_size);
    const int n_tiles = gw * gh;
    const PointBlob pb = carve_point_blob(state->point_blob, state->n_points, state->mode, state->tile_size);
    if (state->n_visible < 0 || state->n_instances < 0) { set_error("inpc_raster_debug_copy: the counts of this state are still on the device; call inpc_raster_resolve first"); return INPC_E_INVALID; }
    const InstanceBlob ib = carve_instance_blob(state->instance_blob, instance_capacity(state), state->deferred_counts & 1, n_tiles, state->tile_size, state->mode, false);
    const int d = depth_buffer_of(state);
    const int ti = tile_buffer_of(n_tiles);
    switch (which) {
        case 0: INPC_CUDA_TRY(cudaMemcpyAsync(dst, pb.ids[d], 4 * (size_t)state->n_visible, cudaMemcpyDeviceToDevice, stream)); break;
        case 1:   // not every sort keeps its keys: the depths of the points in their order
            if (state->n_visible > 0) {
                launch_chained(inpc_debug::sorted_depths_kernel, (unsigned)ceil_div<int64_t>(state->n_visible, 256), 256, 0, stream,
                    pb.ids[d], pb.rec, (state->deferred_counts & 2) ? 1 : 2, state->n_visible, static_cast<uint32_t*>(dst));
                INPC_LAUNCH_CHECK("sorted_depths_kernel");
            }
            break;
        case 2: INPC_CUDA_TRY(cudaMemcpyAsync(dst, ib.ids[ti], 4 * (size_t)state->n_instances, cudaMemcpyDeviceToDevice, stream)); break;
        case 3: INPC_CUDA_TRY(cudaMemcpyAsync(dst, ib.ranges, 8 * (size_t)n_tiles, cudaMemcpyDeviceToDevice, stream)); break;
        case 4: case 5: case 6: case 7: case 8:
            if (state->n_points > 0) {
                launch_chained(inpc_debug::unpack_points_kernel, (unsigned)ceil_div<int64_t>(state->n_points, 256), 256, 0, stream, pb.rec, (state->deferred_counts & 2) ? 1 : 2, pb.bounds, pb.quad, state->n_points, which, gw, dst);
                INPC_LAUNCH_CHECK("unpack_points_kernel");
            }
            break;
        default: set_error("inpc_raster_debug_copy: unknown array %d", which); return INPC_E_INVALID;
    }
    return INPC_OK;
}

