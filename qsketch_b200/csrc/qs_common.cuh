// qs_common.cuh — constants, device layout and helpers shared by the sm_100a kernels.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace qsb {

// Reference constants (lib/default.cu:39-54, device_sketch_v3.h:160).
constexpr uint32_t START = 1024;       // NEXT_LEVEL_ID_START: ids <= START are reserved
constexpr uint32_t FIRST_ID = START + 1;  // Device_Hash_Table::resize sets 1025 (device_sketch.h:109)
constexpr uint32_t LIMIT = 128;        // a selected 8-bit counter > LIMIT triggers the high level
constexpr uint32_t CROSS = LIMIT + 2;  // a byte reaching 130 under all-adds means order matters
constexpr uint32_t SATURATED = 2;      // word-7 value of a bucket whose link failed (pool full)
constexpr uint32_t FLAG = 0x80000000u; // word-7 bit: bucket crossed during the current chunk
constexpr int LOW_WORDS = 8;           // 32 B low bucket: 7 words of packed counters + index
constexpr int LOW_COUNTERS = 28;       // generate_hashmask(..., 32, 3, 4): bits 0..27
constexpr int HIGH_WORDS = 32;         // 128 B high bucket of u32 counters

// Status bits latched in Ctl::status.
constexpr uint32_t ST_POOL_FULL = 1u;
constexpr uint32_t ST_TIMEOUT = 2u;
constexpr uint32_t ST_CAPACITY = 4u;
constexpr uint32_t ST_BAD_OFFSETS = 8u;  // batched streams: offsets not non-decreasing from 0

// a % d by a 32-bit reciprocal (in place of the two run-time `%` of device_sketch_v3.h:42-44 per
// key).  With M = floor(2^32 / d), q = (a * M) >> 32 is floor(a / d) or one less for every 32-bit
// a: a / d - a * M / 2^32 = a * (2^32 / d - M) / 2^32 < 1.  So r = a - q * d lies in [0, 2d) and
// one conditional subtraction (min(r, r - d) in unsigned arithmetic: r - d wraps when r < d)
// finishes: a high multiply, a multiply-add, an add and a min, where the 64-bit direct
// remainder (Lemire, Kaser, Kurz 2019) takes two 32-bit wide and two high multiplies.
struct FastMod {
    uint32_t M, d;
};

inline FastMod make_fastmod(uint32_t d) {
    FastMod f;
    f.M = d < 2 ? 0xffffffffu : (uint32_t)((1ull << 32) / d);  // d = 1: q = a - 1 (a > 0), r = 1 -> 0
    f.d = d;
    return f;
}

__host__ __device__ __forceinline__ uint64_t umin64(uint64_t a, uint64_t b) { return a < b ? a : b; }

__device__ __forceinline__ uint32_t fast_mod(const FastMod& f, uint32_t a) {
    const uint32_t r = a - __umulhi(a, f.M) * f.d;
    return min(r, r - f.d);
}

// Per-sketch device control block.
struct Ctl {
    uint32_t next_id;      // bump allocator (atomic_malloc, device_sketch_v3.h:69-85)
    uint32_t status;       // latched ST_* bits
    uint32_t n_flagged;    // buckets flagged in the current chunk
    uint32_t n_records;    // records gathered for the ordered replay
    uint32_t n_long;       // slots whose segment needed a grid-wide count
    uint32_t bar_count;    // blocks that finished the current repair (its last block resets)
    uint32_t link_gen;     // repairs that linked buckets since the create/clear (never reset
                           // otherwise): tags the per-stream link ranks of batched streams
    uint32_t n_switch;     // partitioned insert: buckets that switched in the current chunk
    uint32_t link_base;    // and the allocator when the chunk began
    unsigned long long bar_arrive;  // grid barrier arrivals (a barrier ends at the next multiple
                                    // of the grid size)
    unsigned long long dropped;
    unsigned long long repaired_buckets;
    unsigned long long repaired_keys;
    unsigned long long inserted;
    unsigned long long repairs;        // repair invocations that had flagged buckets
    unsigned long long phase_t;        // globaltimer at the last phase mark
    unsigned long long phase_ns[12];   // accumulated time per repair phase
};

// Everything a MSWS kernel needs, passed by value.
struct MswsDev {
    uint32_t* low;           // n_low * 8 words
    uint32_t* high;          // n_high * 32 words
    const uint32_t* masks;   // n_masks mask words (bit i selects counter i)
    const uint32_t* codes;   // masks of three counters: the counters' numbers, 5 bits each (!wide)
    Ctl* ctl;
    uint64_t n_low;
    uint64_t n_high;
    FastMod fm_low;
    FastMod fm_mask;
    uint32_t seed;
    uint32_t n_masks;
    uint32_t compat_v3;
    uint32_t wide;           // some mask does not select exactly three counters
    uint32_t flag_cap;       // capacity of flag_list / per-slot arrays
    // ordered-replay scratch
    uint32_t* flag_list;     // slot -> bucket
    uint32_t* tile_counts;   // per key tile of the chunk
    uint2* rec[2];           // (slot, mask) records, ping-pong for the radix passes
    uint32_t* hist;          // 256 * max record tiles
    uint32_t* seg_beg;       // per slot: first record of its segment
    uint32_t* totals;        // long_cap slots * 28 counts
    uint32_t long_cap;       // slots whose per-counter totals are computed grid-wide
    uint32_t route;          // 0 adaptive, 1 preload, 2 fused (pass-1 routing)
    const uint32_t* skip;    // optional: bit i set = key i of the chunk is not for this sketch
    uint32_t max_tiles;      // tiles of REPAIR_TILE elements in a chunk
    // learned split, pass 1 only: keys found in this exact table count there instead of in
    // the sketch, and pass 1 sets their bits in skip_out (null tbl_keys: no table)
    const uint32_t* tbl_keys;
    uint32_t* tbl_counts;
    uint32_t* skip_out;
    uint32_t tbl_slots;
    uint32_t ins_tile;       // pass-1 keys per tile (0: the stage size)
    uint32_t prof;           // repair phase timers on (qs_set_profiling); off they cost nothing
    // Link order.  One-key-at-a-time insertion hands out high ids in the array order of the
    // keys that switch buckets to the high level; the ordered replay does the same:
    uint32_t* rpos[2];       // per record: its position in array order, carried through the
                             // radix passes beside rec[]
    uint2* sw;               // per slot: the switch key's position (then its rank) or NONE, and
                             // the bucket's keys at or after the switch
    uint32_t* sw_base;       // per slot, batched streams: the stream's allocator before the repair
                             // (partitioned insert: per row, its stream)
    uint32_t* sw_bits;       // one bit per record position: a bucket switches there
    uint32_t* sw_cnt;        // switches per SW_BLOCK positions
};
constexpr uint32_t SW_BLOCK = 4096;  // positions per switch count (128 bit words)

// Scratch of the partitioned insert (qs_part.cu); its tiles share the memory of the ordered
// replay's records.
struct PartDev {
    uint32_t* ent;    // entries, each tile's at its own place, ordered by partition
    uint16_t* idx;    // each entry's key: its index in the tile
    uint16_t* off;    // [parts + 1][stride] first entry of each partition's run in each tile
    uint32_t* hot;    // [PART_HOT] the current call's heavy keys, two per set
    uint32_t stride;  // tiles a chunk can have
    uint32_t shift;   // a partition is 2^shift consecutive buckets
    uint32_t parts;
    uint32_t tiles;   // this chunk's tiles, of `tile` keys
    uint32_t tile;
};
constexpr uint32_t PART_TILE = 16384, PART_TILE_SMALL = 2048;
// Chunks below this many keys (half a large tile per SM) take small tiles.  Uniform calls of 2^20 keys
// 34 us with small tiles, 36 with large ones; 1.3M 42 / 36; 2.4M 83 / 65.
constexpr uint64_t PART_SMALL_MAX = 74ull * PART_TILE;
constexpr uint32_t PART_MAX_PARTS = 2048, PART_MAX_SHIFT = 11;
// Buckets of a partition, as a shift: 64, more while that makes 640 partitions, and down to 16 for small
// tables while that makes fewer than 256, because a partition is one block's (2^24 uniform keys, warm:
// 1,021 buckets in 16 partitions 1049 us, in 64 306; 2,039 527 -> 216; 4,093 332 -> 204; 8,191 306 -> 268;
// but 16,381 in 512 instead of 256 314 -> 348).
__host__ __device__ constexpr uint32_t part_shift(uint64_t n_low) {
    uint32_t s = 4;
    while (s < 6 && (n_low >> s) >= 256) ++s;
    while (s < PART_MAX_SHIFT && (n_low >> s) >= 640) ++s;
    return s;
}
// Tables of fewer partitions stay with pass 1: at 509 buckets 2^24 uniform keys 407 us through pass 1, 525
// in 32 partitions (cleared 655 / 579; Zipf 1.4 417 / 155, cleared 854 / 297), 1980 in eight of 64 buckets.
constexpr uint64_t PART_MIN_PARTS = 32;
constexpr uint32_t PART_MAX_MASKS = 2048;         // mask tables the apply step keeps in shared memory
constexpr uint64_t PART_MAX_CHUNK = 1ull << 26;
constexpr uint32_t PART_HOT = 2048;               // heavy keys of a call
// Calls of at least this many keys into a warm sketch are sampled for them by a kernel of its own
// (9-12 us a call with the lookups): 1.6M Zipf 1.1 keys 140 -> 59 us, Zipf 0.8 67 -> 65, uniform 36 -> 47.
// Shorter ones by each block of the split for itself: at 2^20 Zipf 1.1 the call's sample gave 95 -> 61
// us and uniform 34 -> 43, the blocks' 107 -> 44 and 30 -> 32.
constexpr uint64_t PART_HOT_MIN = 3ull << 19;

// Batched streams: many per-stream MSWS sketches share one low-table arena and one high
// pool arena.  A stream's sketch is the bucket range [low_base, low_base + fm_low.d) of the
// low arena and the id range (high_base + START, high_base + START + n_high) of the pool, so
// a bucket or a high id is one global number and pass 1, the flag machinery and the
// ordered replay work unchanged; only hashing and allocation read the stream's descriptor.
struct StreamDesc {
    FastMod fm_low;      // d = the stream's low bucket count
    uint32_t seed;       // the stream's hash multiplier
    uint32_t low_base;   // first bucket of the stream's sketch in the low arena
    uint32_t high_base;  // global high id = high_base + the stream's own id (from FIRST_ID)
    uint32_t n_high;     // the stream's pool size in buckets (own ids < START + n_high)
    uint32_t shift;      // partitioned insert: 2^shift buckets to the smallest partition
    uint32_t parts;      // and the partitions then (0: not for this stream)
};

struct BatchDev {
    const StreamDesc* desc;   // [n_streams]
    const uint64_t* key_off;  // [n_streams + 1] caller's offsets: stream s = keys[off[s], off[s+1])
    uint64_t* lo;             // [n_streams] first flat key of each stream's slice in the window
    uint64_t* hi;             // [n_streams] end of that slice
    uint32_t* item_off;       // [n_streams + 1] prefix of work items (key tiles) per stream
    uint32_t* wpre;           // [n_streams + 1] prefix of the slices' key counts: window key i of
                              // stream s is flat key lo[s] + i - wpre[s]
    uint64_t* win;            // [2] 0 and the window's key count
    uint32_t* work;           // work-queue heads, one per size-class launch of pass 1
    const uint32_t* cls_streams; // [n_streams] the streams grouped by size class (pass-1 launches)
    uint32_t* cls_item_off;   // [n_streams + 1] prefix of work items in the grouped order
    uint32_t* next_id;        // [n_streams] per-stream bump allocators (from FIRST_ID)
    uint32_t* status;         // [n_streams] latched ST_* bits per stream
    unsigned long long* first;// [n_streams] (repair generation << 32) | ~(lowest rank of the
                              // stream's links in that repair): ranks within each stream
    // partitioned insert (its plan fills item_off with its own tiles)
    uint32_t* part_shift;     // [n_streams] buckets of a partition in this window (batch_shift)
    uint32_t* part_off;       // [n_streams + 1] prefix of the streams' partitions in this window
    uint32_t* run_off;        // [n_streams + 1] prefix of the streams' run bounds in PartDev::off
    uint32_t* base_id;        // [n_streams] next_id when the window began
    uint32_t* hot;            // [n_streams][BATCH_HOT] heavy keys of each stream in this call
    uint32_t* hot_mul;        // [n_streams] the multiplier of each stream's sets in `hot`
    uint32_t n_streams;       // 0: not a batch
    uint32_t pad;
};
constexpr uint32_t BATCH_HOT = 128;

// Which keys one batched launch sequence covers: flat mode, the keys [c0, c1) of the caller's
// flat array; else, for the streams [s_lo, s_hi), each stream's keys [rel_lo, rel_hi) counted
// from the stream's start (the per-stream chunk ramp).
struct BatchWindow {
    uint64_t c0, c1;
    uint64_t rel_lo, rel_hi;
    uint32_t s_lo, s_hi;
    uint32_t flat;
    uint64_t fold;   // dense streams: one with at most this many keys from rel_hi on has them in the window
                     // that ends at rel_hi, and none in the one that begins there
    uint32_t coarse; // dense streams: partitions of at least about 2,048 keys (batch_shift)
    uint32_t which;  // all streams, or only the dense or the sparse ones (batch_dense), or (flat)
                     // work items only for the slices of more than SMALL_STREAM keys
};
enum { STREAMS_ALL = 0, STREAMS_DENSE = 1, STREAMS_SPARSE = 2, STREAMS_LONG = 3 };
// Keys of a stream in one call that one block takes by itself (k_msws_small).
constexpr uint64_t SMALL_STREAM = 4096;
// Buckets of a partition of such a stream, of `keys` keys in the window, as a shift: as many as it takes
// for 2,048 keys to a partition, down to eight of them, in windows of more than BATCH_PARTS partitions (few
// would leave the chip idle: 44 streams of up to 84,000 keys 409 -> 423 us).  A block per partition is 20 to 30 ns of the
// chip, whatever its keys: 512 streams of 33,000 keys, 1,024 to 8,192 buckets, cleared / warm, in 32 to 64
// partitions each 0.89 / 0.96 ms uniform and 1.60 / 1.13 Zipf 1.2; so 0.54 / 0.58 and 1.51 / 0.71 (pass 1
// 0.64 / 0.94 and 1.23 / 0.88).
constexpr uint64_t BATCH_PARTS = 2560;  // eight or nine waves of blocks
__host__ __device__ __forceinline__ uint32_t batch_shift(uint32_t shift, uint32_t n_low, uint64_t keys, bool coarse) {
    while (coarse && shift < PART_MAX_SHIFT && (n_low >> shift) > 8 && (n_low >> shift) > (keys >> 11)) ++shift;
    return shift;
}
__host__ __device__ __forceinline__ uint32_t batch_parts(uint32_t shift, uint32_t n_low) {
    return (uint32_t)(((uint64_t)n_low + (1ull << shift) - 1) >> shift);
}
// Streams whose keys go through the partitioned insert: at least a key to a bucket and 2^15 keys in
// the call.  The partitioned insert streams a sketch's table twice (about 46 ps a bucket) and takes
// 20-30 ps a key; pass 1 and the replay take 66 ps a key.  (From 1.5 keys a bucket on only: 64 streams of
// 135,000 keys, up to 262,144 buckets, warm, 503 -> 489 us uniform, but 667 -> 682 at exponent 0.6.)
__host__ __device__ __forceinline__ bool batch_dense(uint64_t keys, uint32_t n_low, uint32_t parts) {
    return parts && keys >= (1ull << 15) && keys >= n_low;
}

// Plain count-min (rows x n counters, one seed per row) or, when `masks` is set, a one-level
// bucket sketch: n buckets of `rows` u32 counters, a key's mask (of rows bits) selecting its
// counters in its bucket hv % n (the reference's warp and sub-warp sketches, v1/v2).
struct CmDev {
    uint32_t* table;  // rows * n
    uint64_t n;
    FastMod fm;
    uint32_t rows;
    uint32_t n_masks;       // bucket sketch: mask count H
    uint32_t seeds[16];
    const uint32_t* masks;  // bucket sketch: H mask words (bit i selects counter i), else null
    FastMod fm_mask;
};

constexpr int REPAIR_TILE = 4096;   // elements per tile in the ordered-replay passes
constexpr int REPAIR_THREADS = 512; // 16 warps x 256 elements
constexpr int MAX_CM_ROWS = 16;
constexpr uint32_t MAX_SIZE_CLASSES = 64;  // floor(log2 n_low) of a batched stream's sketch

// Spread a 4-bit nibble to the low bit of each byte: b0->bit0, b1->bit8, b2->bit16, b3->bit24.
__device__ __forceinline__ uint32_t expand_nibble(uint32_t nib) {
    return (nib * 0x00204081u) & 0x01010101u;
}

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(r));
    return r;
}

}  // namespace qsb
