// Onesweep least-significant-digit radix sort of (u32 key, u32 value) pairs for sm_100a.
//
// One up-front kernel builds the digit histograms of every pass in a single read of the keys; each
// pass is then ONE kernel that reads the pairs once and writes them once.  Inside a pass every tile
// ranks its keys stably (per-warp match-any ranking), publishes its per-digit counts and resolves
// its global offsets with a decoupled look-back over the tiles before it.  Tiles take their index
// from a ticket counter, so a tile a later one waits for is always already running; every wait is
// nevertheless bounded and reports through the status word instead of spinning for ever.
//
// Replaces cub::DeviceRadixSort::SortPairs as used in rasterization/src/bilinear/forward.cu:91-98
// (32-bit depth keys) and :132-139 (tile keys) of the reference.
#include "common.cuh"
#include <mutex>

namespace inpc {

namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kLargeItems = 16;          // pairs per thread and tile, see tile_items
constexpr int kLargeTile = kThreads * kLargeItems;
static_assert(kRadix <= kThreads, "a thread owns at most one digit");
static_assert(kLargeTile < 65536, "tile-local positions fit 16 bits");

constexpr unsigned kFlagAggregate = 1u << 30;
constexpr unsigned kFlagPrefix = 2u << 30;
constexpr unsigned kFlagMask = 3u << 30;
constexpr unsigned kValueMask = ~kFlagMask;
constexpr int kSpinLimit = 1 << 22;

// ---- histogram of every pass in one read ---------------------------------------------------
constexpr int kHistThreads = 512;
constexpr int kHistItemsPerBlock = kHistThreads * 4 * 8;   // 8 uint4 loads per thread

// `n_dev` (optional): the number of pairs lives on the device (the grid is then sized for an upper bound).
// The kernel is bound by its shared-memory atomics (up to four per key), not by how the keys arrive: a variant that
// brought them in with bulk asynchronous copies (cp.async.bulk into two 16 KB slabs per block, an mbarrier per slab)
// measured the same on B200 -- whole sort of 2^23 pairs, 32 / 27 / 24 key bits: 316 / 271 / 241 us against
// 314 / 267 / 239 us with the plain 16-byte loads below; 2^25 pairs, 25 bits: 794 against 799 us.
// The block that finishes last turns the counts of every pass into digit bases (exclusive scans): no launch of its own.
__global__ void __launch_bounds__(kHistThreads) radix_histogram_kernel(
    const uint32_t* __restrict__ keys, int64_t n_arg, const unsigned long long* __restrict__ n_dev, KeyHistogram out) {
    await_previous_kernel();
    const int64_t n = n_dev ? (int64_t)*n_dev : n_arg;
    if ((int64_t)blockIdx.x * kHistItemsPerBlock >= n) return;
    __shared__ BlockHistogram s_hist;
    clear_histogram(s_hist);
    __syncthreads();

    auto count = [&](uint32_t k) { count_key(s_hist, out.pt, k); };
    for (int64_t block_base = (int64_t)blockIdx.x * kHistItemsPerBlock; block_base < n; block_base += (int64_t)gridDim.x * kHistItemsPerBlock) {
        const int64_t block_end = min(n, block_base + (int64_t)kHistItemsPerBlock);
        // keys is 16-byte aligned (carved at 256 bytes) and block_base is a multiple of 4
        const uint4* keys4 = reinterpret_cast<const uint4*>(keys + block_base);
        const int n_vec = (int)((block_end - block_base) / 4);
        for (int v = threadIdx.x; v < n_vec; v += kHistThreads) {
            const uint4 k = __ldg(keys4 + v);
            count(k.x); count(k.y); count(k.z); count(k.w);
        }
        for (int64_t i = block_base + (int64_t)n_vec * 4 + threadIdx.x; i < block_end; i += kHistThreads) count(keys[i]);
    }
    const int64_t all = ceil_div<int64_t>(n, kHistItemsPerBlock);
    finish_histogram(s_hist, out, (unsigned)min(all, (int64_t)gridDim.x), nullptr);
}

// ---- one pass ---------------------------------------------------------------------------------
// Bound by shared-memory wavefronts (63 % of the LSU data pipe over the whole pass, 39 wavefronts per 32 pairs) and by
// the phases of a tile waiting on one another, not by DRAM (16 bytes per pair, 15 % of its peak).  Persistent blocks take
// tiles from a ticket counter: the grid fits the chip whatever the bound on n is (a grid sized for an upper bound of a
// device-side count was mostly empty blocks).  Per tile:
//   1. rank: every lane ORs its bit into its warp's match word of its digit; the word then names the lanes that hold the
//      digit, and the last of them advances the warp's counter and clears the word.  (One ballot per digit bit instead
//      keeps the integer pipe busy for 9.5 thousand cycles per tile of 9-bit digits, this takes 8.)
//   2. thread d adds up digit d over the warps and publishes the tile's count; directly behind it -- so that few tiles are
//      ever between their count and their prefix -- the decoupled look-back;
//   3. the pairs go to their tile-local slots in shared memory as 8-byte words;
//   4. coalesced write-out: consecutive slots of one digit go to consecutive addresses.
// Measured against the pass before it (ballots, one block per possible tile): 2^23 pairs of 27 bits 265 -> 228 us, 10.6 M of 14
// bits 190 -> 167, 2^25 of 30 bits 976 -> 860.  Without any look-back the same passes take 214, 167 and 860: the waiting is
// hidden.  Tried and not kept: the next tile's ticket and keys asked for before the write-out (tiles then publish later
// and less evenly: 2^25 pairs 978 us), look-back windows of 16 and 32 (234 and 269), 256 x 24 / 256 x 32 / 384 x 20 threads x
// items (243, 230, 243).
template <int BITS, int ITEMS>
struct PassSmem {
    static constexpr int kBins = BITS > 0 ? 1 << BITS : kRadix;
    union {
        struct {                        // steps 1 and 2
            unsigned count[kWarps][kBins];
            unsigned match[kWarps][kBins];
        };
        uint2 pairs[kThreads * ITEMS];  // steps 3 and 4; the two never live at the same time
    };
    unsigned global_off[kBins];         // global position of a digit's first pair minus its tile-local one
    unsigned scan[kWarps + 1];
    unsigned tile_id;
};

// What a pass reads and writes.
//   PASS_PAIRS    keys and values, as they are.
//   PASS_MARKED   (a first pass) keys of kNoKey take no part, and the values are the positions.
//   PASS_PACK     (a first pass) the same, and the position is written as a 64-bit word with the key bits above this pass's digit on top, then the code
//                 of the point's footprint word: its upper half goes where the keys go and its lower half where the values go, so
//                 that the passes behind it sort by bits of the upper half and need not know.
//   PASS_UNPACK   (the last pass behind it) the values written are the positions, the keys the codes.
enum { PASS_PAIRS = 0, PASS_MARKED = 1, PASS_PACK = 2, PASS_UNPACK = 3 };

// Widths of the fields of such a word; `codes` for PASS_PACK only.
struct PackedFields {
    int key_bits, position_bits;
    CarriedCodes codes;
};

// log2 of the tiles a splat touches, of a footprint word with bit 31 set.
__device__ __forceinline__ unsigned tiles_log2_of_escaped(uint32_t q) { return ((q & 0xFu) == 9u ? 1u : 0u) + ((q >> 16 & 0xFu) == 9u ? 1u : 0u); }

// A look-back that has given up: reported, and the count withdrawn.  What is sorted now has holes that hold whatever lay there: whoever reads the count finds nothing to read.
// (Not inlined: the passes over large tiles, which use all the registers there are, then spill nothing; inlined up to 8 bytes.  2^25 pairs of 30 bits 570 -> 566 us, the depth and tile
// sorts of 2^24 points at 3840x2160 672 -> 662.)
__device__ __noinline__ void give_up(volatile unsigned* status, unsigned long long* withdraw) {
    status[STATUS_LOOKBACK_TIMEOUT] = 1u;
    if (withdraw) *withdraw = 0ull;
}

// BITS > 0 fixes the digit width at compile time; BITS == 0 takes it from `bits_arg`.
// PASS_MARKED: keys of kNoKey take no part, and the values are the positions.  Points that are culled get such a key where they lie, which
// spares the projection a pass that counts the visible ones beforehand, a scan and the point ids: training step of 2^23 samples at 1237x822
// 1684 -> 1639 us, of 2^24 points at 3840x2160 2795 -> 2703, 2^25 points of a cloud at 1920x1080 3158 -> 3008.
template <int BITS, int ITEMS, int FORM>
__global__ void __launch_bounds__(kThreads, 2) radix_onesweep_pass_kernel(
    const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
    uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, int64_t n_arg, const unsigned long long* n_dev,
    int shift, int bits_arg, const unsigned* __restrict__ digit_base, volatile unsigned* tile_state, unsigned* ticket, unsigned long long* withdraw,
    volatile unsigned* status, int spin_limit, unsigned mute_tile, const PackedFields fields) {
    await_previous_kernel();
    constexpr bool MARKED = FORM == PASS_MARKED || FORM == PASS_PACK;
    constexpr int kLocalBits = ITEMS == kLargeItems ? 13 : 11;   // of a position in the tile
    static_assert(kThreads * ITEMS == 1 << kLocalBits, "positions of a tile");
    using Smem = PassSmem<BITS, ITEMS>;
    constexpr int kBins = Smem::kBins;
    constexpr unsigned kTile = kThreads * ITEMS;
    constexpr unsigned kFull = 0xffffffffu;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem& s = *reinterpret_cast<Smem*>(smem_raw);

    const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const unsigned digit_mask = (1u << (BITS > 0 ? BITS : bits_arg)) - 1u;
    const unsigned lt_mask = (1u << lane) - 1u;
    const unsigned n = n_dev ? (unsigned)*n_dev : (unsigned)n_arg;   // < 2^30
    const unsigned n_tiles = (n + kTile - 1u) / kTile;
    unsigned *const my_count = s.count[warp], *const my_match = s.match[warp];
    // warp-striped layout: warp w owns [w*32*ITEMS, (w+1)*32*ITEMS) of the tile, item i of lane l
    // is element i*32+l of that segment, so (warp, item, lane) order is the input order.
    const unsigned local = warp * (32u * ITEMS) + lane;

    uint32_t key[ITEMS];
    auto load_keys = [&](unsigned tile) {
        if (tile >= n_tiles) return;
        const unsigned first = tile * kTile + local;
        const uint32_t* kp = keys_in + first;
        if (tile * kTile + kTile <= n) {
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) key[i] = __ldg(kp + i * 32);
        } else {
            // padding ranks behind every real key of its digit: it is last in the tile, and its digit is the largest
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) key[i] = first + i * 32u < n ? __ldg(kp + i * 32) : 0xFFFFFFFFu;
        }
    };

    if (tid == 0) s.tile_id = atomicAdd(ticket, 1u);
    __syncthreads();
    unsigned tile = s.tile_id;
    // `mute_tile` (no tile in normal operation) is dropped without publishing anything: the tiles behind it then
    // run into the limit of their look-back wait, which is how the tests exercise that path
    if (tile == mute_tile) return;
    load_keys(tile);
    while (tile < n_tiles) {
        const unsigned valid = min(kTile, n - tile * kTile);
        const bool full = valid == kTile;
#pragma unroll
        for (int i = 0; i < kBins / 32; ++i) my_count[i * 32 + lane] = my_match[i * 32 + lane] = 0u;
        __syncwarp();

        // 1. stable rank within the warp's segment, per digit
        // Two 16-bit positions in a word: 64 registers do not hold keys, values and positions otherwise, and what they spilled
        // (13 of them) went through the unit the pass is bound by.  10.6 M pairs of 14 bits 130.5 -> 126.5 us, 2^25 of 30 bits 594 -> 573.
        unsigned pos2[ITEMS / 2];
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const unsigned d = (key[i] >> shift) & digit_mask;
            const unsigned before = my_count[d];
            unsigned pos;
            const bool in = !MARKED || key[i] != kNoKey;
            const unsigned first_digit = __shfl_sync(kFull, d, 0);   // (by every lane: not behind an &&)
            if (__all_sync(kFull, in && d == first_digit)) {
                // one digit in the whole row, as in keys that are nearly in order: 32 atomics on one word would go one by one
                pos = before + lane;
                __syncwarp();
                if (lane == 31u) my_count[d] = before + 32u;
            } else {
                if (in) atomicOr(my_match + d, 1u << lane);
                __syncwarp();
                const unsigned peers = my_match[d];
                pos = before + __popc(peers & lt_mask);
                __syncwarp();
                if (in && (peers >> lane) == 1u) { my_count[d] = pos + 1u; my_match[d] = 0u; }   // the last lane with this digit
            }
            pos2[i / 2] = i & 1 ? pos2[i / 2] | (pos << 16) : pos;
            __syncwarp();
        }
        uint32_t val[ITEMS];
        {
            const unsigned first = tile * kTile + local;
            const uint32_t* vp = vals_in + first;
            if (FORM == PASS_PACK) {
                // the words of marked points are not used
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) val[i] = full || first + i * 32u < n ? __ldg(fields.codes.quad + first + i * 32u) : 0u;
#pragma unroll
                for (int i = 0; i < ITEMS; ++i)
                    if (val[i] >> 31) val[i] = fields.codes.escape + tiles_log2_of_escaped(val[i]);
            } else if (MARKED || !vals_in) {   // the values are the positions
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) val[i] = first + i * 32u;
            } else if (full) {
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) val[i] = __ldg(vp + i * 32);
            } else {
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) val[i] = first + i * 32u < n ? __ldg(vp + i * 32) : 0u;
            }
        }
        __syncthreads();

        // 2. digit `tid` over the warps
        unsigned total = 0;
        if (tid < (unsigned)kBins) {
#pragma unroll
            for (int w = 0; w < kWarps; ++w) total += s.count[w][tid];
            // publish this tile's digit count before any waiting
            tile_state[tile * kBins + tid] = total | (tile == 0 ? kFlagPrefix : kFlagAggregate);
        }
        unsigned block_total;
        const unsigned start = block_exclusive_scan(total, s.scan, &block_total);
        if (tid < (unsigned)kBins) {
            unsigned run = start;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
                const unsigned c = s.count[w][tid];
                s.count[w][tid] = run;
                run += c;
            }
            // decoupled look-back, a window of predecessors per round trip: the loads of a window are
            // independent, so their latencies overlap; entries are then consumed nearest-first
            unsigned exclusive = 0;
            if (tile > 0) {
                constexpr int kWindow = 8;
                int j = (int)tile - 1;
                bool gave_up = false, finished = false;
                while (j >= 0 && !finished && !gave_up) {
                    unsigned v[kWindow];
                    volatile unsigned* sp = tile_state + j * kBins + tid;
#pragma unroll
                    for (int k = 0; k < kWindow; ++k) {
                        v[k] = kFlagPrefix;   // beyond tile 0: an empty inclusive prefix
                        if (j - k >= 0) v[k] = sp[-k * kBins];
                    }
#pragma unroll
                    for (int k = 0; k < kWindow; ++k) {
                        if (finished || gave_up) break;
                        unsigned x = v[k];
                        int spins = 0;
                        while ((x & kFlagMask) == 0u && spins < spin_limit) {   // not published yet: poll this one
                            __nanosleep(20);
                            x = sp[-k * kBins];
                            ++spins;
                        }
                        if ((x & kFlagMask) == 0u) { gave_up = true; break; }
                        exclusive += x & kValueMask;
                        if (x & kFlagPrefix) finished = true;
                    }
                    j -= kWindow;
                }
                if (gave_up) give_up(status, withdraw);
                tile_state[tile * kBins + tid] = ((exclusive + total) & kValueMask) | kFlagPrefix;
            }
            s.global_off[tid] = __ldg(digit_base + tid) + exclusive - start;
        }
        __syncthreads();

        // 3. tile-local slots
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) pos2[i / 2] += (unsigned)my_count[(key[i] >> shift) & digit_mask] << (16 * (i & 1));
        __syncthreads();   // the counters are dead from here on: their storage holds the staged pairs
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
            if (!MARKED || key[i] != kNoKey) {
                uint2 staged = make_uint2(key[i], val[i]);
                if (FORM == PASS_PACK) {   // key, code and position in the tile: with the pass's digit the word has no room for the whole position
                    const unsigned long long word = ((unsigned long long)(key[i] & (0xFFFFFFFFu >> (32 - fields.key_bits))) << (fields.codes.bits + kLocalBits)) |
                                                    ((unsigned long long)val[i] << kLocalBits) | (local + i * 32u);
                    staged = make_uint2((unsigned)(word >> 32), (unsigned)word);
                }
                s.pairs[i & 1 ? pos2[i / 2] >> 16 : pos2[i / 2] & 0xFFFFu] = staged;
            }
        __syncthreads();

        // 4. write-out.  Padding ranks behind every real pair of the last tile, i.e. at slots >= valid.  dst < n always holds
        // in a healthy sort; after a look-back that gave up, a later pass meets keys whose digits no longer match the
        // histogram taken up front, and its positions can then run past the end: those are dropped.
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const unsigned q = tid + i * kThreads;
            if (MARKED ? q < block_total : full || q < valid) {
                uint2 kv = s.pairs[q];
                unsigned digit = (kv.x >> shift) & digit_mask;
                if (FORM == PASS_PACK) {   // shift is 0: the digit lies at the lower end of the key
                    const unsigned long long word = ((unsigned long long)kv.x << 32) | kv.y;
                    digit = (unsigned)(word >> (fields.codes.bits + kLocalBits)) & digit_mask;
                    const int rest = fields.key_bits - (BITS > 0 ? BITS : bits_arg);
                    const unsigned long long out = ((word >> (fields.codes.bits + kLocalBits + (BITS > 0 ? BITS : bits_arg))) << (64 - rest)) |
                                                   (((word >> kLocalBits) & ((1ull << fields.codes.bits) - 1ull)) << fields.position_bits) |
                                                   (tile * kTile + (kv.y & (kTile - 1u)));
                    kv = make_uint2((unsigned)(out >> 32), (unsigned)out);
                }
                if (FORM == PASS_UNPACK) {
                    const unsigned long long word = ((unsigned long long)kv.x << 32) | kv.y;
                    kv = make_uint2((unsigned)(word >> fields.position_bits) & ((1u << fields.codes.bits) - 1u), kv.y & ((1u << fields.position_bits) - 1u));
                }
                const unsigned dst = s.global_off[digit] + q;
                if (dst < n) {
                    keys_out[dst] = kv.x;
                    vals_out[dst] = kv.y;
                }
            }
        }
        __syncthreads();   // everybody has read the staged pairs
        if (tid == 0) s.tile_id = atomicAdd(ticket, 1u);
        __syncthreads();
        tile = s.tile_id;
        load_keys(tile);
    }
}

// Pairs per thread of a tile, from the number of pairs a call most likely sorts.  Large tiles have longer output runs, less
// bookkeeping per pair and a shorter chain of look-backs; small ones have less to do one after the other.  Measured, tiles of
// 8192 / 2048 pairs, 27 key bits: 2^14 pairs 50 / 40 us, 2^17 56 / 48, 2^18 58 / 50, 2^19 62 / 64, 2^20 62 / 87.
constexpr int kSmallItems = 4;
constexpr int64_t kSmallMax = 1 << 18;
int tile_items(int64_t n_likely) { return n_likely > kSmallMax ? kLargeItems : kSmallItems; }

// Digit bins a pass keeps per tile: digits of 7, 8 and 9 bits (depth keys 9 or 8, tile keys 7 to 9) have unrolled kernels.
int pass_bins(int bits) { return bits >= 7 && bits <= 9 ? 1 << bits : kRadix; }

struct SortWorkspace {
    unsigned* hist;     // [kMaxPasses][kRadix]
    unsigned* ticket;   // [kMaxPasses] tickets, then the histogram's count of finished blocks
    unsigned* base;     // [kMaxPasses][kRadix]
    unsigned* state;    // [passes][tiles][bins]
    size_t zero_bytes;  // leading bytes that must be cleared per sort (hist + ticket), the state follows them
    size_t total;
};

SortWorkspace carve_sort_workspace(void* ws, int64_t n, int items) {
    SortWorkspace w;
    const int64_t tiles = n > 0 ? ceil_div<int64_t>(n, (int64_t)kThreads * items) : 1;
    Carver c(ws);
    w.hist = c.take<unsigned>(kMaxPasses * kRadix);
    w.ticket = c.take<unsigned>(64);
    w.zero_bytes = c.used();
    w.state = c.take<unsigned>((size_t)kMaxPasses * tiles * kRadix);
    w.base = c.take<unsigned>(kMaxPasses * kRadix);
    w.total = c.used();
    return w;
}

struct PassArgs {
    int64_t tiles;         // upper bound
    const uint32_t *kin, *vin;   // vin may be null: the values are the positions 0, 1, ...
    uint32_t *kout, *vout;
    int64_t n;
    const unsigned long long* n_dev;
    int shift, bits;
    const unsigned* base;
    unsigned *state, *ticket, *status;
    unsigned long long* withdraw;   // the count in device memory, or null: zero once a tile has given up
    int form;              // PASS_...
    PackedFields fields;   // of PASS_PACK and PASS_UNPACK
    int spin_limit;        // polls a tile spends on one unpublished predecessor before it gives up
    unsigned mute_tile;    // tile that never publishes (tests only); 0xFFFFFFFF = none
};

template <int BITS, int ITEMS, int FORM>
int launch_onesweep_instance(const PassArgs& a, cudaStream_t stream) {
    static bool attr_set[kMaxDevices] = {false};
    constexpr size_t kSmemBytes = sizeof(PassSmem<BITS, ITEMS>);
    const int rc = opt_in_dynamic_smem(radix_onesweep_pass_kernel<BITS, ITEMS, FORM>, kSmemBytes, attr_set);
    if (rc != INPC_OK) return rc;
    const int64_t resident = (int64_t)sm_count() * 2;
    launch_chained(radix_onesweep_pass_kernel<BITS, ITEMS, FORM>, (unsigned)(a.tiles < resident ? a.tiles : resident), kThreads, kSmemBytes, stream,
        a.kin, a.vin, a.kout, a.vout, a.n, a.n_dev, a.shift, a.bits, a.base, a.state, a.ticket, a.withdraw, a.status, a.spin_limit, a.mute_tile, a.fields);
    INPC_LAUNCH_CHECK("radix_onesweep_pass_kernel");
    return INPC_OK;
}

template <int ITEMS, int FORM>
int launch_onesweep_form(const PassArgs& a, cudaStream_t stream) {
    switch (a.bits) {
        case 7: return launch_onesweep_instance<7, ITEMS, FORM>(a, stream);
        case 8: return launch_onesweep_instance<8, ITEMS, FORM>(a, stream);
        case 9: return launch_onesweep_instance<9, ITEMS, FORM>(a, stream);
        default: return launch_onesweep_instance<0, ITEMS, FORM>(a, stream);
    }
}

template <int ITEMS>
int launch_onesweep_pass(const PassArgs& a, cudaStream_t stream) {
    switch (a.form) {
        case PASS_MARKED: return launch_onesweep_form<ITEMS, PASS_MARKED>(a, stream);
        case PASS_PACK: return launch_onesweep_form<ITEMS, PASS_PACK>(a, stream);
        case PASS_UNPACK: return launch_onesweep_form<ITEMS, PASS_UNPACK>(a, stream);
        default: return launch_onesweep_form<ITEMS, PASS_PAIRS>(a, stream);
    }
}

}  // namespace

static size_t state_words(int64_t tiles, int end_bit) {
    const int n_passes = ceil_div(end_bit, kRadixBits);
    size_t words = 0;
    for (int p = 0, bit = 0; p < n_passes; ++p) {
        const int b = (end_bit - bit + (n_passes - p) - 1) / (n_passes - p);
        words += (size_t)tiles * pass_bins(b);
        bit += b;
    }
    return words;
}

static PassTable pass_table(int end_bit) {
    PassTable pt;
    pt.n_passes = ceil_div(end_bit, kRadixBits);
    int bit = 0;
    for (int p = 0; p < kMaxPasses; ++p) { pt.shift[p] = 0; pt.bits[p] = 0; }
    for (int p = 0; p < pt.n_passes; ++p) {
        // spread the bits evenly over the passes (e.g. 12 bits -> 6 + 6): fewer digits per pass
        // means longer, better-coalesced output runs
        const int b = (end_bit - bit + (pt.n_passes - p) - 1) / (pt.n_passes - p);
        pt.shift[p] = bit;
        pt.bits[p] = b;
        bit += b;
    }
    return pt;
}

static KeyHistogram histogram_of(const SortWorkspace& w, int end_bit) { return {pass_table(end_bit), w.hist, w.base, w.ticket + kMaxPasses}; }

KeyHistogram key_histogram(void* workspace, int64_t n, int64_t n_likely, int end_bit) {
    return histogram_of(carve_sort_workspace(workspace, n, tile_items(n_likely)), end_bit);
}

// Histograms, tickets and the look-back state lie at the front of the workspace.
size_t sort_zero_bytes(int64_t n, int64_t n_likely, int end_bit) {
    if (n <= 0 || end_bit <= 0) return 0;
    const int items = tile_items(n_likely);
    return carve_sort_workspace(nullptr, n, items).zero_bytes + state_words(ceil_div<int64_t>(n, (int64_t)kThreads * items), end_bit) * sizeof(unsigned);
}

// A workspace serves every smaller sort as well.  The look-back state of kSmallMax pairs in small tiles is larger than that of
// up to four times as many in large ones (1.07 MB against 0.29 MB just above), so from there on the size does not fall below it.
size_t sort_workspace_bytes(int64_t n, int64_t n_likely) {
    const size_t own = carve_sort_workspace(nullptr, n, tile_items(n_likely)).total;
    if (tile_items(n_likely) == kSmallItems) return own;
    const size_t small = carve_sort_workspace(nullptr, kSmallMax, kSmallItems).total;
    return own > small ? own : small;
}

int sort_pass_count(int end_bit) { return end_bit > 0 ? ceil_div(end_bit, kRadixBits) : 0; }

// Argument checks shared by the entry points; *nothing_to_do is set when the call is valid but makes no pass.
static int check_sort_args(const char* who, const uint32_t* keys, const uint32_t* keys_alt, const uint32_t* values, const uint32_t* values_alt,
                           int64_t n, int end_bit, bool* nothing_to_do) {
    *nothing_to_do = false;
    if (n < 0 || n >= (int64_t)1 << 30) { set_error("%s: n=%lld out of range [0, 2^30)", who, (long long)n); return INPC_E_INVALID; }
    if (end_bit < 0 || end_bit > 32) { set_error("%s: end_bit=%d out of range", who, end_bit); return INPC_E_INVALID; }
    if (n <= 1 || end_bit == 0) { *nothing_to_do = true; return INPC_OK; }
    if (!keys || !keys_alt || !values || !values_alt) { set_error("%s: null pointer", who); return INPC_E_INVALID; }
    if ((reinterpret_cast<uintptr_t>(keys) | reinterpret_cast<uintptr_t>(keys_alt)) & 15u) {
        set_error("%s: key buffers must be 16-byte aligned", who);
        return INPC_E_INVALID;
    }
    return INPC_OK;
}

// The sort proper: `workspace` holds sort_workspace_bytes(n) bytes, `status` is the device address of the
// status words a tile that gives up its look-back writes to.  Every entry point ends up here.
// `items`: pairs per thread of a tile, the value the workspace was sized with.
static int sort_pairs_with(const char* who, uint32_t* keys, uint32_t* keys_alt, uint32_t* values, uint32_t* values_alt, int64_t n, int end_bit,
                           int items, void* workspace, bool zeroed, unsigned* status, int* result_in_alt, cudaStream_t stream, int spin_limit = kSpinLimit,
                           unsigned mute_tile = 0xFFFFFFFFu, unsigned long long* n_dev = nullptr, bool position_values = false, unsigned long long* marked_count = nullptr, bool counted = false, const CarriedCodes* codes = nullptr) {
    if (result_in_alt) *result_in_alt = 0;
    if (!workspace || !status) { set_error("%s: null workspace", who); return INPC_E_INVALID; }

    const PassTable pt = pass_table(end_bit);
    SortWorkspace w = carve_sort_workspace(workspace, n, items);
    const int64_t tiles = ceil_div<int64_t>(n, (int64_t)kThreads * items);
    // a workspace that is reused keeps the previous call's contents, so everything this call reads is cleared first
    if (!zeroed) INPC_CUDA_TRY(cudaMemsetAsync(workspace, 0, w.zero_bytes + state_words(tiles, end_bit) * sizeof(unsigned), stream));

    if (!counted) {
        const int64_t hist_blocks = ceil_div<int64_t>(n, kHistItemsPerBlock), hist_cap = (int64_t)sm_count() * 4;
        const unsigned hist_grid = (unsigned)(hist_blocks < hist_cap ? hist_blocks : hist_cap);
        launch_chained(radix_histogram_kernel, hist_grid, kHistThreads, 0, stream, keys, n, n_dev, histogram_of(w, end_bit));
        INPC_LAUNCH_CHECK("radix_histogram_kernel");
    }

    PassArgs a;
    a.tiles = tiles; a.n = n; a.n_dev = n_dev; a.status = status;
    a.spin_limit = spin_limit; a.mute_tile = mute_tile;
    a.withdraw = marked_count ? marked_count : n_dev;
    a.kin = keys; a.kout = keys_alt; a.vin = position_values || marked_count ? nullptr : values; a.vout = values_alt;
    a.state = w.state;
    a.fields = {end_bit, bit_length((uint32_t)(n - 1)), codes ? *codes : CarriedCodes{}};
    for (int p = 0; p < pt.n_passes; ++p) {
        a.shift = pt.shift[p]; a.bits = pt.bits[p];
        a.form = p == 0 && marked_count ? (codes ? PASS_PACK : PASS_MARKED) : codes && p == pt.n_passes - 1 ? PASS_UNPACK : PASS_PAIRS;
        if (codes && p > 0) a.shift += 32 - end_bit;   // the key's upper bits lie at the upper end of the first word
        a.base = w.base + p * kRadix;
        a.ticket = w.ticket + p;
        const int rc = items == kLargeItems ? launch_onesweep_pass<kLargeItems>(a, stream) : launch_onesweep_pass<kSmallItems>(a, stream);
        if (rc != INPC_OK) return rc;
        if (p == 0 && marked_count) a.n_dev = marked_count;   // the passes behind the first find only the keys that take part
        a.state += (size_t)tiles * pass_bins(a.bits);
        const uint32_t* t = a.kin; a.kin = a.kout; a.kout = const_cast<uint32_t*>(t);
        a.vin = a.vout; a.vout = a.vout == values ? values_alt : values;
    }
    if (result_in_alt) *result_in_alt = pt.n_passes & 1;
    return INPC_OK;
}

// `position_values`: the values to be sorted are 0 .. n - 1 and need not lie in `values` (with fewer than two pairs, where nothing
// is done, they do).
int sort_pairs(uint32_t* keys, uint32_t* keys_alt, uint32_t* values, uint32_t* values_alt, int64_t n, int64_t n_likely,
               int end_bit, void* workspace, bool zeroed, unsigned* status, int* result_in_alt, cudaStream_t stream, bool position_values, bool counted) {
    if (result_in_alt) *result_in_alt = 0;
    bool nothing = false;
    const int rc = check_sort_args("sort_pairs", keys, keys_alt, values, values_alt, n, end_bit, &nothing);
    if (rc != INPC_OK || nothing) return rc;
    if (!workspace) { set_error("sort_pairs: null workspace"); return INPC_E_INVALID; }
    return sort_pairs_with("sort_pairs", keys, keys_alt, values, values_alt, n, end_bit, tile_items(n_likely), workspace, zeroed, status, result_in_alt, stream, kSpinLimit,
                           0xFFFFFFFFu, nullptr, position_values, nullptr, counted);
}

CarriedCodes carried_codes(const uint32_t* quad, int64_t n, int end_bit, int64_t words) {
    CarriedCodes c;
    if (n < 1 || end_bit < 1 || end_bit > 32 || words < 1 || words > (int64_t)1 << 30) return c;
    const PassTable pt = pass_table(end_bit);
    const int bits = bit_length((uint32_t)(words + 2));
    // behind the first pass: the key bits that are left, code, position; staged in the first one: key, code, position in the tile
    if (pt.n_passes < 2 || end_bit - pt.bits[0] + bits + bit_length((uint32_t)(n - 1)) > 64 || end_bit + bits + bit_length(kLargeTile - 1) > 64) return c;
    c.quad = quad;
    c.bits = bits;
    c.escape = (uint32_t)words;
    return c;
}

// (one pair is sorted like more: how many take part is not known here)
static int sort_marked(uint32_t* keys, uint32_t* keys_alt, uint32_t* values, uint32_t* values_alt, int64_t n, unsigned long long* count, int end_bit, const CarriedCodes* codes,
                       void* workspace, unsigned* status, int* result_in_alt, cudaStream_t stream) {
    if (result_in_alt) *result_in_alt = 0;
    bool nothing = false;
    const int rc = check_sort_args("sort_marked_keys", keys, keys_alt, values, values_alt, n < 2 ? 2 : n, end_bit, &nothing);
    if (rc != INPC_OK) return rc;
    if (n < 1 || nothing || !workspace || !count || (codes && (!codes->quad || codes->bits < 1 || sort_pass_count(end_bit) < 2))) {
        set_error("sort_marked_keys: needs keys, key bits, a workspace, the count and codes that fit");
        return INPC_E_INVALID;
    }
    return sort_pairs_with("sort_marked_keys", keys, keys_alt, values, values_alt, n, end_bit, tile_items(n), workspace, true, status, result_in_alt, stream, kSpinLimit,
                           0xFFFFFFFFu, nullptr, true, count, true, codes);
}

int sort_marked_keys(uint32_t* keys, uint32_t* keys_alt, uint32_t* values, uint32_t* values_alt, int64_t n, unsigned long long* count, int end_bit, void* workspace,
                     unsigned* status, int* result_in_alt, cudaStream_t stream) {
    return sort_marked(keys, keys_alt, values, values_alt, n, count, end_bit, nullptr, workspace, status, result_in_alt, stream);
}

int sort_marked_keys_with_codes(uint32_t* keys, uint32_t* keys_alt, uint32_t* values, uint32_t* values_alt, int64_t n, unsigned long long* count, int end_bit, const CarriedCodes& codes,
                                void* workspace, unsigned* status, int* result_in_alt, cudaStream_t stream) {
    return sort_marked(keys, keys_alt, values, values_alt, n, count, end_bit, &codes, workspace, status, result_in_alt, stream);
}

// The same sort with the number of pairs in device memory (*n_dev <= n_max): grids and the look-back state are
// sized for n_max, the kernels read the count themselves, and the result is always in the alternate buffers iff
// the number of passes is odd.  No host synchronisation anywhere.
int sort_pairs_device_count(uint32_t* keys, uint32_t* keys_alt, uint32_t* values, uint32_t* values_alt, int64_t n_max, int64_t n_likely,
                            unsigned long long* n_dev, int end_bit, void* workspace, bool zeroed, unsigned* status, int* result_in_alt,
                            cudaStream_t stream, bool counted) {
    if (result_in_alt) *result_in_alt = 0;
    if (n_max <= 0 || end_bit == 0) return INPC_OK;
    bool nothing = false;
    const int rc = check_sort_args("sort_pairs", keys, keys_alt, values, values_alt, n_max < 2 ? 2 : n_max, end_bit, &nothing);
    if (rc != INPC_OK) return rc;
    if (!workspace || !n_dev) { set_error("sort_pairs: null workspace or count"); return INPC_E_INVALID; }
    return sort_pairs_with("sort_pairs", keys, keys_alt, values, values_alt, n_max, end_bit, tile_items(n_likely), workspace, zeroed, status, result_in_alt, stream, kSpinLimit,
                           0xFFFFFFFFu, n_dev, false, nullptr, counted);
}

}  // namespace inpc

// ---- sorting without any allocation -------------------------------------------------------------
// Scratch for inpc_sort_pairs_static lives in this fixed device array: every GPU that loads the library
// holds it (about 1 MB) until the process exits.  Layout = the ordinary sort workspace for
// kStaticMaxPairs pairs, followed by one 256-byte status area.
namespace inpc {
namespace {
constexpr int64_t kStaticMaxPairs = 1 << 20;
constexpr size_t kStaticTiles = (kStaticMaxPairs + kLargeTile - 1) / kLargeTile;   // the static sort always takes large tiles: its scratch stays small
constexpr size_t kStaticWorkspaceBytes = (kMaxPasses * kRadix * 4 + 256)            // histograms + tickets
                                         + kMaxPasses * kStaticTiles * kRadix * 4   // look-back state
                                         + kMaxPasses * kRadix * 4;                 // digit bases
constexpr size_t kStaticScratchBytes = kStaticWorkspaceBytes + 256;
static_assert(kStaticWorkspaceBytes % 256 == 0, "status area must stay 256-byte aligned");

static __device__ __align__(256) unsigned char g_static_sort_scratch[kStaticScratchBytes];

std::mutex g_static_mutex;
void* g_static_scratch_ptr[kMaxDevices] = {nullptr};   // device address of the array, per device

// Once per device, with that device current: resolve the array's device address.  In host code the
// array's name is only a handle for the runtime, not an address a kernel could use.
int static_scratch_for_current_device(void** out) {
    int dev = -1;
    INPC_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) { set_error("device index %d outside the supported range", dev); return INPC_E_INVALID; }
    std::lock_guard<std::mutex> lock(g_static_mutex);
    if (!g_static_scratch_ptr[dev]) {
        void* p = nullptr;
        INPC_CUDA_TRY(cudaGetSymbolAddress(&p, g_static_sort_scratch));
        g_static_scratch_ptr[dev] = p;
    }
    *out = g_static_scratch_ptr[dev];
    return INPC_OK;
}
}  // namespace
}  // namespace inpc

extern "C" int inpc_sort_pairs_static(uint32_t* keys, uint32_t* keys_alt, uint32_t* values, uint32_t* values_alt,
                                      int64_t n, int end_bit, int* result_in_alt, void* stream_) {
    using namespace inpc;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (result_in_alt) *result_in_alt = 0;
    if (n > kStaticMaxPairs) {
        set_error("inpc_sort_pairs_static: n=%lld exceeds the fixed capacity of %lld pairs; use inpc_sort_pairs with a caller workspace",
                  (long long)n, (long long)kStaticMaxPairs);
        return INPC_E_CAPACITY;
    }
    // the hand-written size of the fixed array must be what the ordinary workspace layout needs at capacity
    const size_t needed = carve_sort_workspace(nullptr, kStaticMaxPairs, kLargeItems).total;
    if (needed != kStaticWorkspaceBytes) {
        set_error("inpc_sort_pairs_static: fixed scratch of %zu bytes does not match the workspace layout (%zu bytes)",
                  kStaticWorkspaceBytes, needed);
        return INPC_E_INVALID;
    }
    bool nothing = false;
    int rc = check_sort_args("inpc_sort_pairs_static", keys, keys_alt, values, values_alt, n, end_bit, &nothing);
    if (rc != INPC_OK || nothing) return rc;
    void* scratch = nullptr;
    rc = static_scratch_for_current_device(&scratch);
    if (rc != INPC_OK) return rc;
    // the status words of this entry point live behind the workspace, inside the same fixed array
    unsigned* status = reinterpret_cast<unsigned*>(static_cast<unsigned char*>(scratch) + kStaticWorkspaceBytes);
    INPC_CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(unsigned) * STATUS_WORDS, stream));
    return sort_pairs_with("inpc_sort_pairs_static", keys, keys_alt, values, values_alt, n, end_bit, kLargeItems, scratch, false, status, result_in_alt, stream);
}

extern "C" size_t inpc_sort_workspace_bytes(int64_t n) { return inpc::sort_workspace_bytes(n < 0 ? 0 : n, n); }

extern "C" int inpc_sort_pairs(uint32_t* keys, uint32_t* keys_alt, uint32_t* values, uint32_t* values_alt,
                               int64_t n, int end_bit, void* workspace, int* result_in_alt, void* stream) {
    using namespace inpc;
    if (result_in_alt) *result_in_alt = 0;
    bool nothing = false;
    int rc = check_sort_args("inpc_sort_pairs", keys, keys_alt, values, values_alt, n, end_bit, &nothing);
    if (rc != INPC_OK || nothing) return rc;
    if (!workspace) { set_error("inpc_sort_pairs: null workspace"); return INPC_E_INVALID; }
    rc = check_previous_calls();
    if (rc != INPC_OK) return rc;
    unsigned* status = acquire_status("inpc_sort_pairs");
    if (!status) return INPC_E_CUDA;
    return sort_pairs(keys, keys_alt, values, values_alt, n, n, end_bit, workspace, false, status, result_in_alt, static_cast<cudaStream_t>(stream));
}

// Test hook: inpc_sort_pairs with tile 0 of every pass leaving before it publishes its digit counts and a
// look-back limit of 2^10 polls.  The tiles behind it give up within microseconds, report through the call's
// status words, publish what they have and finish: every access stays inside the buffers (the write-out
// checks its destination against n), the output is simply not sorted.  Returns the call's status ticket in *ticket.
extern "C" int inpc_debug_sort_lookback_timeout(uint32_t* keys, uint32_t* keys_alt, uint32_t* values, uint32_t* values_alt,
                                                int64_t n, int end_bit, void* workspace, long long* ticket, void* stream) {
    using namespace inpc;
    bool nothing = false;
    int rc = check_sort_args("inpc_debug_sort_lookback_timeout", keys, keys_alt, values, values_alt, n, end_bit, &nothing);
    if (rc != INPC_OK) return rc;
    if (nothing || !workspace || !ticket) { set_error("inpc_debug_sort_lookback_timeout: needs n > 1, end_bit > 0, a workspace and a ticket pointer"); return INPC_E_INVALID; }
    unsigned* status = acquire_status("inpc_debug_sort_lookback_timeout", ticket);
    if (!status) return INPC_E_CUDA;
    return sort_pairs_with("inpc_debug_sort_lookback_timeout", keys, keys_alt, values, values_alt, n, end_bit, tile_items(n), workspace, false, status, nullptr,
                           static_cast<cudaStream_t>(stream), 1 << 10, 0u);
}

// The same for the sorts whose count is in device memory: all n keys, of which *count say there are n; `marked` as in a depth sort (no key equals kNoKey, the values are the
// positions).  The tiles that give up leave *count at zero, and the passes behind them, and whoever else reads the count, find nothing to do.
extern "C" int inpc_debug_counted_sort_lookback_timeout(uint32_t* keys, uint32_t* keys_alt, uint32_t* values, uint32_t* values_alt, int64_t n, unsigned long long* count,
                                                        int marked, int end_bit, void* workspace, long long* ticket, void* stream) {
    using namespace inpc;
    bool nothing = false;
    int rc = check_sort_args("inpc_debug_counted_sort_lookback_timeout", keys, keys_alt, values, values_alt, n, end_bit, &nothing);
    if (rc != INPC_OK) return rc;
    if (nothing || !workspace || !count || !ticket) { set_error("inpc_debug_counted_sort_lookback_timeout: needs n > 1, end_bit > 0, a workspace, a count and a ticket pointer"); return INPC_E_INVALID; }
    unsigned* status = acquire_status("inpc_debug_counted_sort_lookback_timeout", ticket);
    if (!status) return INPC_E_CUDA;
    return sort_pairs_with("inpc_debug_counted_sort_lookback_timeout", keys, keys_alt, values, values_alt, n, end_bit, tile_items(n), workspace, false, status, nullptr,
                           static_cast<cudaStream_t>(stream), 1 << 10, 0u, marked ? nullptr : count, false, marked ? count : nullptr);
}

// Status words of the last inpc_sort_pairs_static call on the current device, copied out of the fixed array
// after `stream` has been synchronised (no allocation here either).
extern "C" int inpc_sort_pairs_static_status(void* stream_, unsigned* words) {
    using namespace inpc;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (!words) { set_error("inpc_sort_pairs_static_status: null argument"); return INPC_E_INVALID; }
    void* scratch = nullptr;
    const int rc = static_scratch_for_current_device(&scratch);
    if (rc != INPC_OK) return rc;
    unsigned host[STATUS_WORDS];
    INPC_CUDA_TRY(cudaMemcpyAsync(host, static_cast<unsigned char*>(scratch) + kStaticWorkspaceBytes, sizeof(host), cudaMemcpyDeviceToHost, stream));
    INPC_CUDA_TRY(cudaStreamSynchronize(stream));
    for (int k = 0; k < (int)STATUS_WORDS; ++k) words[k] = host[k];
    if (host[STATUS_LOOKBACK_TIMEOUT]) {
        set_error("inpc_sort_pairs_static: a radix-sort tile gave up waiting for a predecessor tile; the results of that call are invalid");
        return INPC_E_DEVICE;
    }
    return INPC_OK;
}
