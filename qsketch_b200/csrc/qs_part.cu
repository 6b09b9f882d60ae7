// qs_part.cu — the partitioned MSWS insert: large chunks, bucket by bucket in shared memory.
//
// Pass 1 of qs_msws.cu sends every key to its bucket in L2 with returning atomics and merges
// equal keys of a warp first (__match_any_sync: 64 SM cycles for 32 distinct values); the
// ordered replay then reads the whole chunk again to find the keys of the buckets that
// crossed.  A chunk with enough keys per bucket is instead split by bucket range:
//   1. k_part_split: tiles of the chunk are ordered by partition (2^shift consecutive buckets)
//      in shared memory and written out with each key's index in its tile.  An entry is the
//      bucket within the partition and the number of the key's mask; nothing is hashed again.
//   2. k_part_apply: one block per partition holds the partition's 32-byte buckets in shared
//      memory and applies the entries tile by tile with shared-memory atomics.  A bucket whose
//      selected counter would pass the threshold is replayed on the spot: the entries of the
//      flagged buckets in the current run of tiles are sorted by array position and the exact
//      sequential rule of qs_replay.cuh finds the switching key.  The new high bucket is a
//      temporary row; the index word names it until the link order is known.
//   3. k_part_link: high ids in the array order of the switching keys, as one-key-at-a-time
//      insertion hands them out; rows move to their high buckets.
// Nothing waits across blocks: the order between the steps is the order of the launches.
//
// What bounds it (2^24-key chunks): the split, instruction issue and the shared-memory pipe, each
// half busy between its barriers (88-96 warp instructions per 32 keys; 86-93 us); the apply step, the latency of a unit's dependent
// shared-memory steps with 32 warps an SM (95 us for uniform keys, 155 us for Zipf 1.1 with the
// heavy keys counted in the split).  Against pass 1 and the replay: 2^24 uniform keys into 8 MB
// 0.55 -> 0.21 ms, 2^27 Zipf 1.1 keys into 64 MB 6.4 -> 2.2 ms (both with default knobs).
#include "qs_kernels.h"
#include "qs_replay.cuh"

namespace qsb {

constexpr int AP_THREADS = 512;
constexpr int AP_WARPS = AP_THREADS / 32;
constexpr uint32_t AP_TILES = AP_THREADS;   // tiles whose run bounds are staged at a time
// A unit: the entries applied between two looks at the flagged buckets (whole runs; a longer run is
// a unit of its own).  A thread holds its share of the unit in registers, so the records of the
// flagged buckets are gathered without reading the entries again, and always fit the
// shared memory they are sorted in.  Half the size beside the 2048-bucket partitions of the
// largest tables, so that two blocks fit an SM.
__host__ __device__ constexpr uint32_t ap_unit(uint32_t shift) { return shift > 10 ? 2048u : 4096u; }
// A partition that gets far more than its share starts with short units, doubling: the buckets of
// its heavy keys link in them, with few records each.
constexpr uint32_t AP_FIRST = 256;
constexpr uint32_t ENT_MASK_BITS = 14;      // entry = bucket in partition << 14 | mask number
constexpr uint32_t ENT_MASK = (1u << ENT_MASK_BITS) - 1u;
// Index words while a partition is in shared memory, beside 0, FLAG | slot and real ids (below
// ACC: the path takes pools of less than 2^28 buckets):
//   ACC | a        linked; its high increments collect in row a of the block's accumulators
//   ACC | NEW | a  the same for a bucket linked in this chunk, whose id is not known yet
//   TEMP | row     linked in this chunk with no accumulator left: a row in global memory (from
//                  long_cap on there is none: counted again when the id is known)
constexpr uint32_t ACC = 0x20000000u, NEW = 0x10000000u, TEMP = 0x40000000u;
constexpr uint32_t ACC_WORDS = LOW_COUNTERS + 1;  // 28 counters and the keys of a NEW bucket
// Accumulator rows of a block: the linked buckets of a partition, a few per cent of its buckets.
__host__ __device__ constexpr uint32_t ap_accs(uint32_t shift) { return shift > 10 ? 80u : 192u; }
// ---- 0: the heavy keys of a call ---------------------------------------------------------

constexpr uint32_t HOT_SETS = PART_HOT / 2;  // two keys per set
constexpr uint32_t HOT_BLOCKS = 64, HOT_THREADS = 1024;
constexpr uint32_t HOT_SAMPLES = 16384, HOT_SLOTS = 1024, HOT_MIN = 3;
constexpr uint32_t HOT_EMPTY = 0xffffffffu, IN_TABLE = 0x80000000u;

__device__ __forceinline__ uint32_t hot_set(uint32_t key) { return (key * 0x9E3779B1u) >> 22; }
static_assert(HOT_SETS == 1024, "hot_set yields 10 bits");

// Keys seen at least HOT_MIN times among HOT_SAMPLES evenly spaced ones (a share of about 2e-4).
// Every block reads the whole sample and counts the keys of its own sets.  What bounds it is the
// latency of one block's steps: 16 blocks of 512 threads with a sector per key 19 us, with a sector
// per four keys 13 us, 64 blocks of 1024 threads 7 us.  Which keys the table keeps when a set
// overflows (the heaviest go first) does not change any result.
__global__ void __launch_bounds__(HOT_THREADS) k_part_hot(const uint32_t* __restrict__ keys, uint64_t n, uint32_t* hot) {
    __shared__ uint32_t s_key[HOT_SLOTS], s_cnt[HOT_SLOTS];
    constexpr uint32_t SETS = HOT_SETS / HOT_BLOCKS;  // this block's sets
    __shared__ uint32_t s_hot[2 * SETS];
    const uint32_t tid = threadIdx.x, set0 = blockIdx.x * SETS;
    for (uint32_t i = tid; i < HOT_SLOTS; i += HOT_THREADS) s_key[i] = HOT_EMPTY, s_cnt[i] = 0u;
    for (uint32_t i = tid; i < 2 * SETS; i += HOT_THREADS) s_hot[i] = HOT_EMPTY;
    // four neighbouring keys per place: the scattered sectors bound the reads (an SM takes one in
    // about two cycles), not the keys
    const uint32_t* base = reinterpret_cast<const uint32_t*>((reinterpret_cast<uintptr_t>(keys) + 15) & ~(uintptr_t)15);
    const uint64_t step = (n - 3) / HOT_SAMPLES;  // in units of four keys, times four places
    uint32_t k[HOT_SAMPLES / HOT_THREADS];
#pragma unroll
    for (uint32_t j = 0; j < HOT_SAMPLES / HOT_THREADS / 4; ++j) {
        const uint4 q = __ldg(reinterpret_cast<const uint4*>(base) + step * (uint64_t)(j * HOT_THREADS + tid));
        k[4 * j] = q.x, k[4 * j + 1] = q.y, k[4 * j + 2] = q.z, k[4 * j + 3] = q.w;
    }
    __syncthreads();
#pragma unroll
    for (uint32_t j = 0; j < HOT_SAMPLES / HOT_THREADS; ++j) {
        if (k[j] == HOT_EMPTY || hot_set(k[j]) - set0 >= SETS) continue;
        const uint32_t h = mix32(k[j]);
        for (uint32_t q = 0; q < 8; ++q) {  // a heavy key finds a slot early; a lone one may be left out
            const uint32_t s = (h + q) & (HOT_SLOTS - 1);
            uint32_t seen = reinterpret_cast<volatile uint32_t*>(s_key)[s];
            if (seen == HOT_EMPTY) seen = atomicCAS(s_key + s, HOT_EMPTY, k[j]);
            if (seen == HOT_EMPTY || seen == k[j]) {
                atomicAdd(s_cnt + s, 1u);
                break;
            }
        }
    }
    __syncthreads();
    uint32_t hi = 0xffffffffu;
    for (uint32_t lo : {64u, 8u, HOT_MIN}) {  // the heaviest first
        for (uint32_t i = tid; i < HOT_SLOTS; i += HOT_THREADS) {
            if (s_cnt[i] < lo || s_cnt[i] >= hi) continue;
            const uint32_t s = 2 * (hot_set(s_key[i]) - set0);
            if (atomicCAS(s_hot + s, HOT_EMPTY, s_key[i]) != HOT_EMPTY) atomicCAS(s_hot + s + 1, HOT_EMPTY, s_key[i]);
        }
        hi = lo;
        __syncthreads();
    }
    for (uint32_t i = tid; i < 2 * SETS; i += HOT_THREADS) hot[2 * set0 + i] = s_hot[i];
}

// ---- the sketch a tile or a partition belongs to ----------------------------------------------

// One sketch, or stream s of a batch: the window's slices are cut into tiles stream after stream,
// each stream with its own partitions and run bounds; everything else is the single-sketch path.
struct PartView {
    FastMod fm;
    uint32_t seed, low_base, shift, parts;
    uint32_t tile0, tiles;  // its tiles in the chunk
    uint16_t* off;          // [parts + 1][tiles of `stride`]
    uint32_t stride;
};
template <bool BATCH>
__device__ __forceinline__ PartView part_view(const MswsDev& D, const PartDev& Q, const BatchDev& B, uint32_t s) {
    PartView V;
    if (!BATCH) {
        V.fm = D.fm_low, V.seed = D.seed, V.low_base = 0, V.shift = Q.shift, V.parts = Q.parts;
        V.tile0 = 0, V.tiles = Q.tiles, V.off = Q.off, V.stride = Q.stride;
        return V;
    }
    const StreamDesc* sd = B.desc + s;
    V.fm = FastMod{__ldg(&sd->fm_low.M), __ldg(&sd->fm_low.d)};
    V.seed = __ldg(&sd->seed), V.low_base = __ldg(&sd->low_base);
    V.shift = __ldg(B.part_shift + s), V.parts = batch_parts(V.shift, V.fm.d);
    V.tile0 = __ldcg(B.item_off + s), V.tiles = __ldcg(B.item_off + s + 1) - V.tile0;
    V.off = Q.off + __ldcg(B.run_off + s), V.stride = V.tiles;
    return V;
}

// One block: the slices of the window's streams (offsets checked by the host), their tiles of
// `tile` keys and run bounds, and the allocators as the window begins.
__global__ void __launch_bounds__(1024) k_part_plan(BatchDev B, BatchWindow W, uint32_t tile, Ctl* ctl) {
    const uint32_t S = B.n_streams;
    for (uint32_t s = threadIdx.x; s < S; s += blockDim.x) {
        const uint64_t o0 = __ldcg(B.key_off + s), len = __ldcg(B.key_off + s + 1) - o0;
        const bool in = s >= W.s_lo && s < W.s_hi && in_window(B, W, s, len);
        auto cut = [&](uint64_t rel) { return rel && len - umin64(rel, len) <= W.fold ? len : umin64(rel, len); };
        const uint64_t lo = in ? o0 + cut(W.rel_lo) : o0, hi = in ? o0 + cut(W.rel_hi) : o0;
        const uint32_t t = (uint32_t)((hi - lo + tile - 1) / tile);
        B.lo[s] = lo;
        B.hi[s] = hi;
        B.item_off[s] = t;
        const uint32_t n_low = B.desc[s].fm_low.d, shift = batch_shift(B.desc[s].shift, n_low, hi - lo, W.coarse);
        const uint32_t parts = t ? batch_parts(shift, n_low) : 0u;
        B.part_shift[s] = shift;
        B.part_off[s] = parts;
        B.run_off[s] = t * (parts + 1u);
        B.base_id[s] = __ldcg(B.next_id + s);
    }
    __syncthreads();
    const uint32_t tiles = block_scan_array(B.item_off, S), runs = block_scan_array(B.run_off, S);
    const uint32_t parts = block_scan_array(B.part_off, S);
    if (threadIdx.x == 0) {
        B.part_off[S] = parts;
        B.item_off[S] = tiles;
        B.run_off[S] = runs;
        ctl->n_switch = 0;
    }
}

// The set of a key in a stream's table, under the multiplier its stream was given.
__device__ __forceinline__ uint32_t batch_hot_set(uint32_t key, uint32_t mul) { return (key * mul) >> 26; }
static_assert(BATCH_HOT == 2 * 64, "batch_hot_set yields 6 bits, two keys per set");

// A block per dense stream: keys seen at least four times in 4096 samples of its keys from `first` on
// (short streams: none).  Sets are few, and a heavy key that finds its set full would go through
// one block entry by entry (0.5 M of them, 0.9 ms), so each of the eight warps tries a multiplier
// and the one that leaves the least weight out is kept with the stream.
__global__ void __launch_bounds__(256) k_part_hot_batch(const uint32_t* __restrict__ keys, BatchDev B, uint64_t first,
                                                        uint64_t fold) {
    constexpr uint32_t N = 4096, SLOTS = 4096, LIST = 512;
    __shared__ uint32_t s_key[SLOTS], s_cnt[SLOTS], s_hot[BATCH_HOT];
    const uint32_t tid = threadIdx.x, s = blockIdx.x;
    const uint64_t o0 = __ldcg(B.key_off + s), all = __ldcg(B.key_off + s + 1) - o0;
    if (!batch_dense(all, B.desc[s].fm_low.d, B.desc[s].parts) || all <= first + fold) return;
    const uint64_t lo = o0 + first, len = all - first;
    for (uint32_t i = tid; i < BATCH_HOT; i += 256) s_hot[i] = HOT_EMPTY;
    if (len >= 8 * N) {
        for (uint32_t i = tid; i < SLOTS; i += 256) s_key[i] = HOT_EMPTY, s_cnt[i] = 0u;
        const uint64_t step = len / N;
        uint32_t k[N / 256];
#pragma unroll
        for (uint32_t j = 0; j < N / 256; ++j) k[j] = __ldg(keys + lo + step * (uint64_t)(j * 256 + tid));
        __syncthreads();
#pragma unroll
        for (uint32_t j = 0; j < N / 256; ++j) {
            if (k[j] == HOT_EMPTY) continue;
            const uint32_t h = mix32(k[j]);
            for (uint32_t q = 0; q < 4; ++q) {
                const uint32_t i = (h + q) & (SLOTS - 1);
                uint32_t seen = reinterpret_cast<volatile uint32_t*>(s_key)[i];
                if (seen == HOT_EMPTY) seen = atomicCAS(s_key + i, HOT_EMPTY, k[j]);
                if (seen == HOT_EMPTY || seen == k[j]) {
                    atomicAdd(s_cnt + i, 1u);
                    break;
                }
            }
        }
        __syncthreads();
        // the candidates, the heaviest tier first
        __shared__ uint32_t s_list[LIST], s_n, s_occ[8][BATCH_HOT / 2], s_lost[8];
        if (tid == 0) s_n = 0;
        for (uint32_t i = tid; i < 8 * BATCH_HOT / 2; i += 256) (&s_occ[0][0])[i] = 0u;
        __syncthreads();
        uint32_t hi = 0xffffffffu;
        for (uint32_t least : {64u, 16u, 4u}) {
            for (uint32_t i = tid; i < SLOTS; i += 256)
                if (s_cnt[i] >= least && s_cnt[i] < hi) {
                    const uint32_t at = atomicAdd(&s_n, 1u);
                    if (at < LIST) s_list[at] = i;
                }
            hi = least;
            __syncthreads();
        }
        const uint32_t n = min(s_n, LIST), wid = tid >> 5, lane = tid & 31;
        auto mul = [](uint32_t w) { return 0x9E3779B1u + w * 0x3C6EF372u; };  // odd
        uint32_t lost = 0;
        for (uint32_t i0 = 0; i0 < n; i0 += 32) {
            const uint32_t i = i0 + lane;
            if (i < n && atomicAdd(&s_occ[wid][batch_hot_set(s_key[s_list[i]], mul(wid))], 1u) >= 2u) lost += s_cnt[s_list[i]];
            __syncwarp();
        }
        lost = __reduce_add_sync(0xffffffffu, lost);
        if (lane == 0) s_lost[wid] = lost;
        __syncthreads();
        uint32_t best = 0;
        for (uint32_t w = 1; w < 8; ++w) best = s_lost[w] < s_lost[best] ? w : best;
        if (wid == 0) {
            for (uint32_t i0 = 0; i0 < n; i0 += 32) {
                if (i0 + lane < n) {
                    const uint32_t key = s_key[s_list[i0 + lane]], h = 2 * batch_hot_set(key, mul(best));
                    if (atomicCAS(s_hot + h, HOT_EMPTY, key) != HOT_EMPTY) atomicCAS(s_hot + h + 1, HOT_EMPTY, key);
                }
                __syncwarp();
            }
            if (lane == 0) B.hot_mul[s] = mul(best);
        }
    } else if (tid == 0) {
        B.hot_mul[s] = 1u;
    }
    __syncthreads();
    for (uint32_t i = tid; i < BATCH_HOT; i += 256) B.hot[(uint64_t)s * BATCH_HOT + i] = s_hot[i];
}

// ---- 1: tiles ordered by partition ---------------------------------------------------------

enum { HOT_NONE = 0, HOT_CALL = 1, HOT_OWN = 2 };

// The whole block: the keys seen at least `least` times among 1,024 of the tile's, PER of each thread
// (the first `cnt` of the tile are there), into their sets of hkey[PART_HOT]; tmp: 2,048 words.
template <int THREADS, int PER, int KPT>
__device__ __forceinline__ void sample_hot(const uint32_t (&e)[KPT], uint32_t cnt, uint32_t least, uint32_t* tmp,
                                           uint32_t* hkey) {
    constexpr uint32_t SLOTS = 1024;
    static_assert(THREADS * PER == SLOTS, "a slot per sample");
    const uint32_t tid = threadIdx.x;
    uint32_t *key = tmp, *num = tmp + SLOTS;
    for (uint32_t i = tid; i < SLOTS; i += THREADS) key[i] = HOT_EMPTY, num[i] = 0u;
    for (uint32_t i = tid; i < PART_HOT; i += THREADS) hkey[i] = HOT_EMPTY;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const uint32_t k = e[j];
        if (4 * tid + j >= cnt || k == HOT_EMPTY) continue;
        const uint32_t h = mix32(k);
        for (uint32_t p = 0; p < 8; ++p) {
            const uint32_t i = (h + p) & (SLOTS - 1);
            uint32_t seen = reinterpret_cast<volatile uint32_t*>(key)[i];
            if (seen == HOT_EMPTY) seen = atomicCAS(key + i, HOT_EMPTY, k);
            if (seen == HOT_EMPTY || seen == k) {
                atomicAdd(num + i, 1u);
                break;
            }
        }
    }
    __syncthreads();
    for (uint32_t i = tid; i < SLOTS; i += THREADS) {
        if (num[i] < least) continue;
        const uint32_t s = 2 * hot_set(key[i]);
        if (atomicCAS(hkey + s, HOT_EMPTY, key[i]) != HOT_EMPTY) atomicCAS(hkey + s + 1, HOT_EMPTY, key[i]);
    }
    __syncthreads();
}

// HOT: keys of a hot table whose bucket is linked when the chunk begins are counted in shared memory
// (high-level additions commute) and never become entries.  HOT_CALL: the table that k_part_hot (or
// k_part_hot_batch) left for the call.  HOT_OWN, for calls too short for a launch of its own: each
// block samples its first tile and finds the keys of about 4,096 entries and more, which would
// otherwise pass through one block of the apply step, unit after unit: warm sketches, 10^6 equal
// keys 476 -> 26 us, Zipf 1.1 107 -> 44 (0.5 MB) and 127 -> 52 (8 MB), exponent 0.9 75 -> 50, uniform
// 30 -> 32 (sampling 1,024 keys of the whole chunk in every block 34: its sectors are the same for all).
// TABLE (learned split): keys of the exact table count there (D.tbl_keys, D.tbl_counts) and never
// become entries; four lookups of a thread are in flight at a time, and the table's heavy keys are
// counted in shared memory with the others.
// Bound by the random 32-byte sectors of the table in L2 (1 MB table, 2^24 keys: 263 us against 92
// without); 8,192-key tiles and whole-warp probing of every key took 302 us.
template <int PT_THREADS, int KPT, int HOT, bool BATCH, bool TABLE>
__global__ void __launch_bounds__(PT_THREADS, 1024 / PT_THREADS) k_part_split(const uint32_t* __restrict__ keys, uint64_t n, MswsDev D,
                                                              PartDev Q, BatchDev B) {
    constexpr uint32_t R = PT_THREADS * KPT, HOTS = BATCH ? BATCH_HOT : PART_HOT;
    extern __shared__ __align__(16) uint32_t sm[];
    uint32_t* s_ent = sm;                                          // [R]
    uint16_t* s_idx = reinterpret_cast<uint16_t*>(sm + R);         // [R]
    uint32_t* s_hkey = sm + R + R / 2;                             // HOT: [HOTS] keys, counts, high ids
    uint32_t* s_hcnt = s_hkey + HOTS;
    uint32_t* s_hid = s_hcnt + HOTS;
    uint32_t* s_hist = HOT ? s_hid + HOTS : s_hkey;                // [parts] counts, then first positions
    __shared__ uint32_t s_dead[TABLE ? R / 32 : 1], s_more;  // TABLE: keys found after their first sector
    const int tid = threadIdx.x;
    if (!BATCH && blockIdx.x == 0 && tid == 0) {
        D.ctl->n_switch = 0;
        D.ctl->link_base = D.ctl->next_id;
    }
    uint32_t stream = 0, hot_mul = 0;
    PartView V = part_view<false>(D, Q, B, 0);
    // Learned chunks skip the lookups while no hot key is linked or in the table (0.45 -> 0.44 ms a pass);
    // for plain ones the branch costs Zipf streams more (1 %) than it gives uniform ones.
    bool any_hot = !TABLE && HOT != HOT_OWN;
    auto load_hot = [&] {  // the hot keys whose buckets are linked
        bool mine = false;
        const uint32_t* hot = BATCH ? B.hot + (uint64_t)stream * BATCH_HOT : Q.hot;
        if (BATCH) hot_mul = __ldcg(B.hot_mul + stream);
        for (uint32_t i = tid; i < HOTS; i += PT_THREADS) {
            uint32_t key = HOT == HOT_OWN ? s_hkey[i] : __ldcg(hot + i), id = 0;
            if (HOT == HOT_OWN && key == HOT_EMPTY) continue;
            const int ts = TABLE && key != HOT_EMPTY ? table_find(D.tbl_keys, D.tbl_slots, key) : -1;
            if (ts >= 0) {
                id = IN_TABLE | (uint32_t)ts;
            } else if (key != HOT_EMPTY) {
                id = __ldcg(D.low + (uint64_t)(V.low_base + fast_mod(V.fm, key * V.seed)) * LOW_WORDS + 7);
                if (!is_linked(D, id)) key = HOT_EMPTY;
            }
            s_hkey[i] = key;
            s_hcnt[i] = 0u;
            s_hid[i] = id;
            mine |= key != HOT_EMPTY;
        }
        if (TABLE || HOT == HOT_OWN) any_hot = __syncthreads_or(mine);
    };
    auto flush_hot = [&] {  // their counts: one add per counter
        for (uint32_t i = tid; i < HOTS; i += PT_THREADS) {
            if (HOT == HOT_OWN && s_hkey[i] == HOT_EMPTY) continue;
            const uint32_t c = s_hcnt[i];
            if (!c) continue;
            if (TABLE && (s_hid[i] & IN_TABLE)) {
                atomicAdd(D.tbl_counts + (s_hid[i] & ~IN_TABLE), c);
                continue;
            }
            uint32_t* hb = D.high + (uint64_t)(s_hid[i] - START) * HIGH_WORDS;
            for (uint32_t m = __ldg(D.masks + fast_mod(D.fm_mask, s_hkey[i] * V.seed)); m; m &= m - 1)
                atomicAdd(hb + (__ffs(m) - 1), c);
        }
    };
    if (HOT == HOT_CALL && !BATCH) load_hot();
    if (BATCH) stream = NONE;
    for (uint32_t t = blockIdx.x; t < Q.tiles; t += gridDim.x) {
        if (BATCH) {
            const uint32_t s = stream_of_item_warp(B, t);
            if (s != stream) {  // uniform over the block
                if (HOT && stream != NONE) {
                    flush_hot();
                    __syncthreads();
                }
                stream = s;
                V = part_view<true>(D, Q, B, s);
                if (HOT) load_hot();
            }
        }
        const uint32_t parts = V.parts, per = (parts + PT_THREADS - 1) / PT_THREADS, lt = t - V.tile0;
        const uint64_t p0 = (uint64_t)t * R;                                             // its place and positions
        const uint64_t k0 = BATCH ? __ldcg(B.lo + stream) + (uint64_t)lt * R : p0;       // its first key
        const uint32_t cnt = (uint32_t)umin64(R, (BATCH ? __ldcg(B.hi + stream) : n) - k0);
        const bool vec = (reinterpret_cast<uintptr_t>(keys + k0) & 15u) == 0;
        for (uint32_t i = tid; i < parts; i += PT_THREADS) s_hist[i] = 0u;
        // the link order's switch bits and counts of this tile's positions
        for (uint32_t i = tid; i < R / 32; i += PT_THREADS) __stcg(D.sw_bits + (p0 >> 5) + i, 0u);
        if (R >= SW_BLOCK) {
            if (tid < (int)(R / SW_BLOCK)) __stcg(D.sw_cnt + p0 / SW_BLOCK + tid, 0u);
        } else if (tid == 0 && (p0 % SW_BLOCK) == 0) {
            __stcg(D.sw_cnt + p0 / SW_BLOCK, 0u);
        }
        uint32_t e[KPT], pr[KPT];  // the key, then its entry; partition << 16 | rank
        // thread's keys: vector v of 4 at tile index v * 4 * PT_THREADS + 4 * tid
        if (vec && cnt == R) {
#pragma unroll
            for (int v = 0; v < KPT / 4; ++v) {
                const uint4 q = __ldcs(reinterpret_cast<const uint4*>(keys + k0) + v * PT_THREADS + tid);
                e[4 * v] = q.x, e[4 * v + 1] = q.y, e[4 * v + 2] = q.z, e[4 * v + 3] = q.w;
            }
        } else {
#pragma unroll
            for (int j = 0; j < KPT; ++j) {
                const uint32_t i = (j / 4) * 4 * PT_THREADS + 4 * tid + (j & 3);
                e[j] = i < cnt ? __ldg(keys + k0 + i) : 0u;
            }
        }
        __syncthreads();
        if (HOT == HOT_OWN && t == blockIdx.x) {
            // about a unit's worth of entries in the chunk, and no chance repetition
            const uint32_t least = max(4u, (uint32_t)((4096ull << 10) / n));
            sample_hot<PT_THREADS, 1024 / PT_THREADS>(e, cnt, least, s_ent, s_hkey);
            load_hot();
        }
        uint32_t live = 0;  // bit j: key j goes to the sketch
#pragma unroll
        for (int j = 0; j < KPT; ++j) {
            const uint32_t i = (j / 4) * 4 * PT_THREADS + 4 * tid + (j & 3);
            bool on = i < cnt;
            if (!BATCH && !TABLE && D.skip && on) on = !((__ldg(D.skip + ((k0 + i) >> 5)) >> ((k0 + i) & 31)) & 1u);
            live |= on ? 1u << j : 0u;
        }
        if (HOT && any_hot) {  // four sets' loads in flight: a thread otherwise waits one shared-memory round per key
#pragma unroll
            for (int j0 = 0; j0 < KPT; j0 += 4) {
                uint32_t set[4];
                uint2 hk[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    set[j] = 2 * (BATCH ? batch_hot_set(e[j0 + j], hot_mul) : hot_set(e[j0 + j]));
                    hk[j] = *reinterpret_cast<const uint2*>(s_hkey + set[j]);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t key = e[j0 + j], bit = 1u << (j0 + j);
                    const bool x = hk[j].x == key, y = hk[j].y == key;
                    if ((x || y) && key != HOT_EMPTY && (live & bit)) {
                        atomicAdd(s_hcnt + set[j] + (x ? 0u : 1u), 1u);
                        live &= ~bit;
                    }
                }
            }
        }
        if (TABLE) {
            // Each key's first sector; the few whose sector is full without the key (one in
            // five at the table's highest fill) are listed and probed on by whole warps.
            uint32_t* l_key = s_ent;   // free until the scatter
            uint16_t* l_idx = s_idx;
            if (tid == 0) s_more = 0;
            for (uint32_t i = tid; i < R / 32; i += PT_THREADS) s_dead[i] = 0u;
            __syncthreads();
#pragma unroll
            for (int j0 = 0; j0 < KPT; j0 += 4) {
                uint4 a[4], c[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t sec = mix32(e[j0 + j]) & (D.tbl_slots / TBL_SECTOR - 1u);
                    const uint4* q = reinterpret_cast<const uint4*>(D.tbl_keys + (uint64_t)sec * TBL_SECTOR);
                    const bool on = (live >> (j0 + j)) & 1u;
                    a[j] = on ? __ldg(q) : make_uint4(HOT_EMPTY, 0, 0, 0);
                    c[j] = on ? __ldg(q + 1) : make_uint4(0, 0, 0, 0);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t key = e[j0 + j], bit = 1u << (j0 + j);
                    const uint32_t k8[8] = {a[j].x, a[j].y, a[j].z, a[j].w, c[j].x, c[j].y, c[j].z, c[j].w};
                    uint32_t at = 8;
                    bool room = false;
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        at = k8[q] == key ? (uint32_t)q : at;
                        room |= k8[q] == HOT_EMPTY;
                    }
                    const bool on = (live & bit) && key != HOT_EMPTY;
                    if (on && at < 8u) {
                        atomicAdd(D.tbl_counts + (mix32(key) & (D.tbl_slots / TBL_SECTOR - 1u)) * TBL_SECTOR + at, 1u);
                        live &= ~bit;
                    } else if (on && !room) {
                        const uint32_t l = atomicAdd(&s_more, 1u);
                        l_key[l] = key;
                        l_idx[l] = (uint16_t)((j0 / 4) * 4 * PT_THREADS + 4 * tid + j);
                    }
                }
            }
            __syncthreads();
            for (uint32_t l = tid; l < s_more; l += PT_THREADS) {
                const int ts = table_find(D.tbl_keys, D.tbl_slots, l_key[l]);
                if (ts >= 0) {
                    atomicAdd(D.tbl_counts + ts, 1u);
                    atomicOr(s_dead + (l_idx[l] >> 5), 1u << (l_idx[l] & 31));
                }
            }
            __syncthreads();
#pragma unroll
            for (int v = 0; v < KPT / 4; ++v) {
                const uint32_t i = v * 4 * PT_THREADS + 4 * tid;
                live &= ~(((s_dead[i >> 5] >> (i & 31)) & 0xfu) << (4 * v));
            }
        }
#pragma unroll
        for (int j = 0; j < KPT; ++j) {
            const uint32_t hv = e[j] * V.seed;
            const uint32_t b = fast_mod(V.fm, hv), p = b >> V.shift;
            e[j] = ((b & ((1u << V.shift) - 1u)) << ENT_MASK_BITS) | fast_mod(D.fm_mask, hv);
            pr[j] = (live >> j) & 1u ? (p << 16) | atomicAdd(s_hist + p, 1u) : NONE;
        }
        __syncthreads();
        {  // first position of each partition; its row of the run bounds
            constexpr uint32_t PER = PART_MAX_PARTS / PT_THREADS;
            uint32_t c[PER], sum = 0, total;
#pragma unroll
            for (uint32_t j = 0; j < PER; ++j) {
                const uint32_t p = tid * per + j;
                c[j] = j < per && p < parts ? s_hist[p] : 0u;
                sum += c[j];
            }
            uint32_t run = block_exclusive_scan(sum, &total);
#pragma unroll
            for (uint32_t j = 0; j < PER; ++j) {
                const uint32_t p = tid * per + j;
                if (j < per && p < parts) {
                    s_hist[p] = run;
                    V.off[(uint64_t)p * V.stride + lt] = (uint16_t)run;
                    run += c[j];
                }
            }
            if (tid == 0) V.off[(uint64_t)parts * V.stride + lt] = (uint16_t)total;
            __syncthreads();
#pragma unroll
            for (int j0 = 0; j0 < KPT; j0 += 4) {
                uint32_t pos[4];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    pos[j] = pr[j0 + j] == NONE ? NONE : s_hist[pr[j0 + j] >> 16] + (pr[j0 + j] & 0xffffu);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (pos[j] == NONE) continue;
                    s_ent[pos[j]] = e[j0 + j];
                    s_idx[pos[j]] = (uint16_t)((j0 / 4) * 4 * PT_THREADS + 4 * tid + j);
                }
            }
            __syncthreads();
            uint4* ge = reinterpret_cast<uint4*>(Q.ent + p0);
            uint4* gi = reinterpret_cast<uint4*>(Q.idx + p0);
            for (uint32_t i = tid; i * 4 < total; i += PT_THREADS) __stcg(ge + i, reinterpret_cast<const uint4*>(s_ent)[i]);
            for (uint32_t i = tid; i * 8 < total; i += PT_THREADS) __stcg(gi + i, reinterpret_cast<const uint4*>(s_idx)[i]);
        }
        __syncthreads();
    }
    if (HOT && (HOT == HOT_OWN ? any_hot : !BATCH || stream != NONE)) flush_hot();
}

// ---- 2: one partition per block ------------------------------------------------------------

struct ApShared {
    uint32_t* tab;             // [2^shift][8] the partition's buckets (word 7: flagged buckets by slot)
    uint32_t* w7;              // [2^shift] their index words
    uint32_t* mk;              // [n_masks] mask_codes
    uint32_t* acc;             // [ap_accs][ACC_WORDS]
    uint32_t* accid;           // [ap_accs] a row's high id, or (NEW) its switch position
    uint16_t* accb;            // [ap_accs] and its bucket
    unsigned long long* recs;  // [ap_unit]
    uint32_t* before;          // [AP_TILES + 1] entries of the staged runs before run r
    uint32_t* dlt;             // [AP_TILES] run r: its first entry minus before[r]
    uint16_t* map;             // [ap_unit] the run of each entry of the unit
    uint32_t stream;           // batch: whose partition this is
};

__host__ __device__ inline size_t apply_smem(uint32_t shift, uint32_t n_masks) {
    const size_t pb = (size_t)1 << shift;
    return (size_t)ap_unit(shift) * 10 + pb * 36 + (size_t)((n_masks + 1) & ~1u) * 4 + AP_TILES * 8 + 8 +
           ap_accs(shift) * (ACC_WORDS * 4 + 6);
}

__device__ __forceinline__ ApShared ap_carve(uint8_t* p, uint32_t shift, uint32_t n_masks) {
    const size_t pb = (size_t)1 << shift;
    ApShared S;
    S.recs = reinterpret_cast<unsigned long long*>(p);
    p += ap_unit(shift) * 8;
    S.tab = reinterpret_cast<uint32_t*>(p);
    p += pb * 32;
    S.mk = reinterpret_cast<uint32_t*>(p);
    p += (size_t)((n_masks + 1) & ~1u) * 4;  // what follows stays 8-byte aligned (replay_warp uses the run map's memory)
    S.acc = reinterpret_cast<uint32_t*>(p);
    p += ap_accs(shift) * ACC_WORDS * 4;
    S.accid = reinterpret_cast<uint32_t*>(p);
    p += ap_accs(shift) * 4;
    S.w7 = reinterpret_cast<uint32_t*>(p);
    p += pb * 4;
    S.dlt = reinterpret_cast<uint32_t*>(p);
    p += AP_TILES * 4;
    S.before = reinterpret_cast<uint32_t*>(p);
    p += AP_TILES * 4 + 8;
    S.map = reinterpret_cast<uint16_t*>(p);
    p += ap_unit(shift) * 2;
    S.accb = reinterpret_cast<uint16_t*>(p);
    return S;
}

// c occurrences to the selected low counters of a bucket, any mask; whether one crosses.
__device__ __forceinline__ bool part_low_add(uint32_t* bw, uint32_t mm, uint32_t c) {
    bool cross = false;
    while (mm) {
        const uint32_t w = (uint32_t)(__ffs(mm) - 1) >> 2, nib = (mm >> (4u * w)) & 0xfu;
        mm &= ~(nib << (4u * w));
        cross |= crosses(atomicAdd(bw + w, expand_nibble(nib) * c), nib, c);
    }
    return cross;
}

// One entry (MANY: c merged occurrences; else c = 1) of the chunk.
template <bool MANY, bool WIDE>
__device__ __forceinline__ void part_apply_entry(const MswsDev& D, const ApShared& S, uint32_t e, uint32_t c,
                                                 uint32_t* s_nflag, uint32_t* s_drop) {
    const uint32_t lb = e >> ENT_MASK_BITS;
    const uint32_t q = S.mk[e & ENT_MASK];
    const uint32_t w7 = S.w7[lb];
    if ((int32_t)w7 <= 0) {  // not linked, or flagged in this run of tiles
        bool cross;
        uint32_t* bw = S.tab + lb * LOW_WORDS;
        if (MANY || WIDE) {
            cross = part_low_add(bw, code_mask<WIDE>(q), c);
        } else {
            // counter i: byte i & 3 of word i >> 2.  One more makes 130 of 129, so no byte below
            // 128 can cross; counters that share a word see each other's additions only in the
            // other's byte.
            const uint32_t sx = (q & 3u) * 8u, sy = ((q >> 5) & 3u) * 8u, sz = ((q >> 10) & 3u) * 8u;
            const uint32_t ox = atomicAdd(bw + ((q >> 2) & 7u), 1u << sx);
            const uint32_t oy = atomicAdd(bw + ((q >> 7) & 7u), 1u << sy);
            const uint32_t oz = atomicAdd(bw + (q >> 12), 1u << sz);
            cross = ((ox & (0x80u << sx)) | (oy & (0x80u << sy)) | (oz & (0x80u << sz))) != 0u;
            if (cross)
                cross = ((ox >> sx) & 0xffu) >= CROSS - 1u || ((oy >> sy) & 0xffu) >= CROSS - 1u ||
                        ((oz >> sz) & 0xffu) >= CROSS - 1u;
        }
        if (cross && !(atomicOr(S.w7 + lb, FLAG) & FLAG)) {
            const uint32_t slot = atomicAdd(s_nflag, 1u);
            S.tab[slot * LOW_WORDS + 7] = lb;
            atomicExch(S.w7 + lb, FLAG | slot);
        }
        return;
    }
    if ((w7 & (ACC | TEMP)) == ACC) {
        uint32_t* row = S.acc + (w7 & 0xffffu) * ACC_WORDS;
        if (WIDE) {
            for (uint32_t mm = q; mm; mm &= mm - 1) atomicAdd(row + (__ffs(mm) - 1), c);
        } else {
            atomicAdd(row + (q & 31u), c);
            atomicAdd(row + ((q >> 5) & 31u), c);
            atomicAdd(row + (q >> 10), c);
        }
        if (w7 & NEW) atomicAdd(row + LOW_COUNTERS, c);
        return;
    }
    uint32_t* hb;
    if (w7 & TEMP) {
        const uint32_t r = w7 & ~TEMP;
        if (r >= D.long_cap) return;
        hb = D.totals + (uint64_t)r * LOW_COUNTERS;
        atomicAdd(&D.sw[r].y, c);
    } else if (is_linked(D, w7)) {
        hb = D.high + (uint64_t)(w7 - START) * HIGH_WORDS;
    } else {  // saturated: the pool ran out
        atomicAdd(s_drop, c);
        return;
    }
    for (uint32_t mm = code_mask<WIDE>(q); mm; mm &= mm - 1) atomicAdd(hb + (__ffs(mm) - 1), c);
}

// A thread's share of up to U * AP_THREADS entries: entry u * AP_THREADS + tid for u < U, `sub` in
// all.  Heavy: one key fills most of the partition, so a warp counts the entries equal to one of
// its first ones and adds them at once.
template <bool WIDE, int U>
__device__ __forceinline__ void part_apply_batch(const MswsDev& D, const ApShared& S, const uint32_t (&e)[U], uint32_t sub,
                                                 bool heavy, uint32_t* s_nflag, uint32_t* s_drop) {
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    uint32_t skip = HOT_EMPTY;  // no entry
    if (heavy && tid - lane < sub) {  // warp-uniform
        const uint32_t have = __ballot_sync(0xffffffffu, tid < sub);
        uint32_t x = __shfl_sync(0xffffffffu, e[0], 0);
        const uint32_t other = __ballot_sync(0xffffffffu, tid < sub && e[0] != x);
        if (__popc(other) > 16) x = __shfl_sync(0xffffffffu, e[0], __ffs(other) - 1);
        uint32_t c = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) c += e[u] == x && u * AP_THREADS + tid < sub;
        c = __reduce_add_sync(0xffffffffu, c);
        if (c >= 2) {
            skip = x;
            if (lane == (uint32_t)__ffs(have) - 1) part_apply_entry<true, WIDE>(D, S, x, c, s_nflag, s_drop);
        }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const uint32_t k = u * AP_THREADS + tid;
        if (k - lane >= sub) break;  // warp-uniform
        if (k < sub && e[u] != skip) part_apply_entry<false, WIDE>(D, S, e[u], 1u, s_nflag, s_drop);
    }
}

// A bucket that switched at array position pos, with n_after keys from there on: its increments
// collect in an accumulator (or a row) until the link order is known.  Called by a whole warp,
// lane c with counter c's high increment H.
__device__ __forceinline__ void put_row(const MswsDev& D, uint32_t r, uint32_t stream, uint32_t bucket, uint32_t pos,
                                        uint32_t n_after, uint32_t H) {
    const int lane = threadIdx.x & 31;
    if (r < D.long_cap && lane < LOW_COUNTERS) __stcg(D.totals + (uint64_t)r * LOW_COUNTERS + lane, H);
    if (lane == 0) {
        __stcg(D.flag_list + r, bucket);  // sized, as sw and sw_base, for every bucket a chunk can link
        __stcg(D.sw_base + r, stream);    // (batch)
        __stcg(D.sw + r, make_uint2(pos, n_after));
        atomicOr(D.sw_bits + (pos >> 5), 1u << (pos & 31));
        atomicAdd(D.sw_cnt + pos / SW_BLOCK, 1u);
    }
}
__device__ __forceinline__ void open_row(const MswsDev& D, const ApShared& S, uint32_t accs, uint32_t* s_nacc, uint32_t lb,
                                         uint32_t b0, uint32_t pos, uint32_t n_after, uint32_t H) {
    const int lane = threadIdx.x & 31;
    uint32_t a = 0;
    if (lane == 0) a = atomicAdd(s_nacc, 1u);
    a = __shfl_sync(0xffffffffu, a, 0);
    if (a < accs) {
        if (lane < LOW_COUNTERS) S.acc[a * ACC_WORDS + lane] = H;
        if (lane == 0) {
            S.acc[a * ACC_WORDS + LOW_COUNTERS] = n_after;
            S.accid[a] = pos;
            S.accb[a] = (uint16_t)lb;
            S.w7[lb] = ACC | NEW | a;
        }
        return;
    }
    uint32_t r = 0;
    if (lane == 0) r = atomicAdd(&D.ctl->n_switch, 1u);
    r = __shfl_sync(0xffffffffu, r, 0);
    put_row(D, r, S.stream, b0 + lb, pos, n_after, H);
    if (lane == 0) S.w7[lb] = TEMP | r;
}

// Pre-chunk counter of lane i: the bucket's words minus the packed increments T (counter c in
// lane c), as pre_counters of the grid-wide replay.
__device__ __forceinline__ uint32_t part_pre(const uint32_t* bw, uint32_t T) {
    const int lane = threadIdx.x & 31;
    const uint32_t fw = lane < 7 ? bw[lane] : 0u;
    uint32_t sw = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) sw += __shfl_sync(0xffffffffu, T, (4 * (lane & 7) + k) & 31) << (8 * k);
    const uint32_t pwi = __shfl_sync(0xffffffffu, fw - sw, (lane >> 2) & 7);
    return lane < LOW_COUNTERS ? (pwi >> (8 * (lane & 3))) & 0xffu : 0u;
}

__device__ __forceinline__ void part_write_low(uint32_t* bw, uint32_t cur) {
    const int lane = threadIdx.x & 31;
    uint32_t word = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) word |= __shfl_sync(0xffffffffu, cur, (4 * (lane & 7) + k) & 31) << (8 * k);
    if (lane < 7) bw[lane] = word;
}

// Ascending sort of recs[0, K) (at most ap_unit) by the whole block: bitonic over the next power
// of two, padded with all ones.
__device__ __forceinline__ void block_sort(unsigned long long* recs, uint32_t K) {
    uint32_t N = 32;
    while (N < K) N <<= 1;
    for (uint32_t i = K + threadIdx.x; i < N; i += AP_THREADS) recs[i] = ~0ull;
    __syncthreads();
    for (uint32_t k = 2; k <= N; k <<= 1)
        for (uint32_t j = k >> 1; j; j >>= 1) {
            for (uint32_t i = threadIdx.x; i < N / 2; i += AP_THREADS) {
                const uint32_t a = ((i & ~(j - 1)) << 1) | (i & (j - 1)), b = a | j;
                const unsigned long long x = recs[a], y = recs[b];
                if ((x > y) == ((a & k) == 0)) {
                    recs[a] = y;
                    recs[b] = x;
                }
            }
            __syncthreads();
        }
}

// Flagged bucket `s` replayed by one warp from recs[0, K), which hold the unit's records in the order
// of their entries: tile after tile, but in any order within a tile.  Counts over whole tiles do not
// need the order, so the warp adds the bucket's records up, 32 at a time, to the record with which
// some counter passes the threshold; the switching key is in that record's tile, and only that
// tile's records (all of them, if there are at most 32) are put in order.  False, with nothing
// changed, if there are more than 32.  buf: 32 words of the warp (the run map's memory, which is
// done with by then); cnt: 32 counts of the warp.
static_assert(ap_unit(11) * 2 >= AP_WARPS * 32 * 8, "the run map holds every warp's 32 records");
template <bool WIDE>
__device__ __forceinline__ void count_record(const ApShared& S, uint32_t* cnt, uint32_t x) {
    const uint32_t q = S.mk[x & ENT_MASK];
    if (WIDE) {
        for (uint32_t mm = q; mm; mm &= mm - 1) atomicAdd(cnt + (__ffs(mm) - 1), 1u);
    } else {
        atomicAdd(cnt + (q & 31u), 1u);
        atomicAdd(cnt + ((q >> 5) & 31u), 1u);
        atomicAdd(cnt + (q >> 10), 1u);
    }
}
template <bool WIDE>
__device__ __forceinline__ bool replay_warp(const MswsDev& D, const PartDev& Q, const ApShared& S,
                                            unsigned long long* buf, uint32_t* cnt, uint32_t accs, uint32_t* s_nacc,
                                            uint32_t s, uint32_t K, uint32_t b0, uint32_t* s_rb, uint32_t* s_rk) {
    const uint32_t lane = threadIdx.x & 31, in_tile = Q.tile - 1u;
    auto record = [&](uint32_t k, bool& mine) {
        const unsigned long long r = k < K ? S.recs[k] : ~0ull;
        mine = (uint32_t)(r >> 46) == s;
        return r;
    };
    auto tile_of = [&](unsigned long long r) { return (uint32_t)(r >> ENT_MASK_BITS) & ~in_tile; };
    // adds a record's counters to cnt; lane c then reads counter c
    auto add = [&](unsigned long long r) { count_record<WIDE>(S, cnt, (uint32_t)r); };
    auto start = [&](uint32_t v) {
        __syncwarp();
        cnt[lane] = v;
        __syncwarp();
    };
    auto counted = [&] {
        __syncwarp();
        return reinterpret_cast<volatile uint32_t*>(cnt)[lane];
    };
    // lane c: the records of a group (bit i: lane i's, mask mm) that select counter c
    auto selecting = [&](uint32_t mm) {
        uint32_t occ = 0;
#pragma unroll
        for (uint32_t c = 0; c < LOW_COUNTERS; ++c) {
            const uint32_t bal = __ballot_sync(0xffffffffu, (mm >> c) & 1u);
            if (lane == c) occ = bal;
        }
        return occ;
    };
    bool mine;
    uint32_t n = 0;
    ReplayOut o;
    if (s < AP_WARPS) {  // counted as the records were gathered (cnt is this slot's row)
        n = __shfl_sync(0xffffffffu, cnt[lane], LOW_COUNTERS);
    } else {
        start(0u);
        for (uint32_t k0 = 0; k0 < K; k0 += 32) {
            const unsigned long long r = record(k0 + lane, mine);
            n += __popc(__ballot_sync(0xffffffffu, mine));
            if (mine) add(r);
        }
        __syncwarp();
    }
    o.T = lane < LOW_COUNTERS ? cnt[lane] : 0u;
    const uint32_t lb = S.tab[s * LOW_WORDS + 7];
    uint32_t* bw = S.tab + lb * LOW_WORDS;
    o.P = part_pre(bw, o.T);
    // the tile that crosses (n > 32), the counters and records before it
    uint32_t cur = o.P, before = 0, x = NONE, from = 0;  // from: the first group with records of tile x
    if (n > 32) {
        start(o.P);
        for (uint32_t k0 = 0; k0 < K; k0 += 32) {
            const unsigned long long r = record(k0 + lane, mine);
            const uint32_t bal = __ballot_sync(0xffffffffu, mine);
            if (!bal) continue;
            if (mine) add(r);
            const uint32_t now = counted();
            if (!__any_sync(0xffffffffu, now != cur && now > LIMIT + 1)) {
                cur = now;
                before += __popc(bal);
                continue;
            }
            // the record that takes a counter to LIMIT + 2, the first of all counters'
            const uint32_t occ = selecting(mine ? code_mask<WIDE>(S.mk[(uint32_t)r & ENT_MASK]) : 0u);
            const uint32_t need = LIMIT + 2 - cur;  // (cur <= LIMIT + 1 so far)
            const uint32_t j = __reduce_min_sync(0xffffffffu, now > LIMIT + 1 && now != cur ? __fns(occ, 0, need) : 32u);
            x = __shfl_sync(0xffffffffu, tile_of(r), j);
            const uint32_t first = __shfl_sync(0xffffffffu, tile_of(r), __ffs(bal) - 1);
            const uint32_t lt = __ballot_sync(0xffffffffu, mine && tile_of(r) < x);
            cur += __popc(occ & lt);
            before += __popc(lt);
            from = k0;
            if (x == first && k0) {  // it may have begun in earlier groups
                start(0u);
                for (uint32_t q = k0; q > 0;) {
                    from = q -= 32;
                    const unsigned long long e = record(q + lane, mine);
                    const bool in = mine && tile_of(e) == x;
                    if (in) add(e);
                    before -= __popc(__ballot_sync(0xffffffffu, in));
                    if (__any_sync(0xffffffffu, mine && !in)) break;  // records of an earlier tile
                }
                cur -= counted();
            }
            break;
        }
    }
    uint32_t m = 0;
    if (n <= 32 || x != NONE) {
        uint32_t c = 0;
        for (uint32_t k0 = from; k0 < K; k0 += 32) {
            const unsigned long long r = record(k0 + lane, mine);
            const bool in = mine && (x == NONE || tile_of(r) == x);
            const uint32_t bal = __ballot_sync(0xffffffffu, in);
            if (x != NONE && __any_sync(0xffffffffu, mine && tile_of(r) > x) && !bal) break;
            if (c + __popc(bal) > 32) return false;
            if (in) buf[c + __popc(bal & lanemask_lt())] = r;
            c += __popc(bal);
        }
        __syncwarp();
        // in array order: by tile and index in it
        unsigned long long r = ~0ull;
        if (lane < c) {
            r = buf[lane];
            const uint32_t at = (uint32_t)(r >> ENT_MASK_BITS);
            r = (unsigned long long)((at & ~in_tile) + __ldcg(Q.idx + at)) << ENT_MASK_BITS | (r & ENT_MASK);
        }
        __syncwarp();
        buf[lane] = r;
        __syncwarp();
        uint32_t rank = 0;
        for (uint32_t k = 0; k < c; ++k) rank += buf[k] < r;
        __syncwarp();
        if (lane < c) buf[rank] = r;  // positions are distinct
        __syncwarp();
        r = buf[lane];
        m = lane < c ? code_mask<WIDE>(S.mk[(uint32_t)r & ENT_MASK]) : 0u;
        o.L = (uint32_t)(r >> ENT_MASK_BITS);  // lane i: the i-th record's position
    }
    const uint32_t occ = selecting(m);
    bool trig = false;
    for (uint32_t mm = m; __any_sync(0xffffffffu, mm != 0); mm &= mm - 1) {
        const int c = mm ? __ffs(mm) - 1 : 0;
        const uint32_t bal = __shfl_sync(0xffffffffu, occ, c), P = __shfl_sync(0xffffffffu, cur, c);
        trig |= mm && P + __popc(bal & lanemask_lt()) > LIMIT;
    }
    const uint32_t tb = __ballot_sync(0xffffffffu, trig);
    if (tb) {
        const int j = __ffs(tb) - 1;
        o.cur = cur + __popc(occ & ((1u << j) - 1u));
        o.mL = __shfl_sync(0xffffffffu, m, j);
        const uint32_t pos = __shfl_sync(0xffffffffu, o.L, j);
        const uint32_t H = high_increments(D, o);
        __syncwarp();
        part_write_low(bw, o.cur);
        open_row(D, S, accs, s_nacc, lb, b0, pos, n - before - j, H);
    } else if (lane == 0) {
        S.w7[lb] = 0u;  // every key added low
    }
    if (lane == 0) {
        atomicAdd(s_rb, 1u);
        atomicAdd(s_rk, n);
    }
    __syncwarp();
    return true;
}

// The partition `p` (batch: of the window's) that a block works on.  (The plan wrote the offsets in an
// earlier kernel: the search goes through the L1.)
template <bool BATCH>
__device__ __forceinline__ PartView part_of_block(const MswsDev& D, const PartDev& Q, const BatchDev& B, uint32_t& p,
                                                  uint32_t& stream) {
    stream = 0;
    if (BATCH) {
        uint32_t lo = 0, hi = B.n_streams;  // part_off[lo] <= p < part_off[hi]: the last such lo has partitions
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (__ldg(B.part_off + mid) <= p) lo = mid;
            else hi = mid;
        }
        stream = lo;
        p -= __ldg(B.part_off + lo);
    }
    return part_view<BATCH>(D, Q, B, stream);
}

template <bool WIDE, bool BATCH>
__global__ void __launch_bounds__(AP_THREADS, 2) k_part_apply(MswsDev D, PartDev Q, BatchDev B) {
    extern __shared__ __align__(128) uint8_t smem[];
    uint32_t p = blockIdx.x, stream;
    const PartView V = part_of_block<BATCH>(D, Q, B, p, stream);
    if (V.tiles == 0) return;
    ApShared S = ap_carve(smem, V.shift, D.n_masks);
    S.stream = stream;
    __shared__ uint32_t s_nflag, s_nrec, s_many, s_drop, s_rb, s_rk, s_nacc, s_new, s_row;
    __shared__ uint32_t s_cnt[LOW_COUNTERS + 2];  // bisection: counts per counter, keys, mask
    __shared__ uint32_t s_pre[LOW_COUNTERS];
    __shared__ uint32_t s_wcnt[4096 / 32];  // records of each warp's 32 entries, then those before them
    __shared__ uint32_t s_rcnt[AP_WARPS][32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (uint32_t i = tid; i < D.n_masks; i += AP_THREADS) S.mk[i] = __ldg(mask_codes<WIDE>(D) + i);
    const uint32_t accs = ap_accs(V.shift);
    for (uint32_t i = tid; i < accs * ACC_WORDS; i += AP_THREADS) S.acc[i] = 0u;
    if (tid == 0) s_nflag = s_nrec = s_many = s_drop = s_rb = s_rk = s_nacc = s_new = 0;
    __syncthreads();
    const uint64_t b0 = V.low_base + ((uint64_t)p << V.shift);
    const uint32_t nb = (uint32_t)umin64((uint64_t)1 << V.shift, V.fm.d - ((uint64_t)p << V.shift));
    uint4* gt = reinterpret_cast<uint4*>(D.low + b0 * LOW_WORDS);
    {
        uint4* st = reinterpret_cast<uint4*>(S.tab);
        for (uint32_t i0 = tid; i0 < nb * 2; i0 += 4 * AP_THREADS) {
            uint4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (i0 + u * AP_THREADS < nb * 2) v[u] = __ldcg(gt + i0 + u * AP_THREADS);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t i = i0 + u * AP_THREADS;
                if (i < nb * 2) {
                    st[i] = v[u];
                    if (i & 1u) {
                        uint32_t w7 = v[u].w;
                        if (is_linked(D, w7)) {
                            const uint32_t a = atomicAdd(&s_nacc, 1u);
                            if (a < accs) {
                                S.accid[a] = w7;
                                S.accb[a] = (uint16_t)(i >> 1);
                                w7 = ACC | a;
                            }
                        }
                        S.w7[i >> 1] = w7;
                    }
                }
            }
        }
    }
    const uint16_t* o0 = V.off + (uint64_t)p * V.stride;
    const uint16_t* o1 = o0 + V.stride;
    const uint32_t tile = Q.tile, cap = ap_unit(V.shift), mean = max(1u, tile / V.parts);
    constexpr int U = 4096 / AP_THREADS;  // a thread's entries of a unit, at most
    uint32_t units = 0;
    for (uint32_t ts = 0; ts < V.tiles; ts += AP_TILES) {
        // the run bounds of the next AP_TILES tiles
        __syncthreads();
        const uint32_t nr = min(AP_TILES, V.tiles - ts), tile_s = V.tile0 + ts;
        uint32_t a = 0, len = 0, total;
        if (tid < nr) {
            a = __ldcg(o0 + ts + tid);
            len = __ldcg(o1 + ts + tid) - a;
        }
        const uint32_t before = block_exclusive_scan(len, &total);
        S.dlt[tid] = (tile_s + tid) * tile + a - before;
        S.before[tid] = before;
        if (tid == 0) S.before[nr] = total;  // (entry nr < AP_TILES already holds it)
        // far above an even share, a heavy key is likely, maybe of a bucket that is not linked yet
        const bool heavy = total > 4u * mean * nr;
        for (uint32_t r0 = 0; r0 < nr;) {
            __syncthreads();
            const uint32_t base = S.before[r0];
            const uint32_t most = heavy ? min(cap, AP_FIRST << min(units++, 4u)) : cap;
            const uint32_t r1 =
                r0 + __syncthreads_count(tid >= r0 && tid < nr && (tid == r0 || before + len - base <= most));
            const uint32_t sub = S.before[r1] - base;
            const uint32_t rb = r0;
            r0 = r1;
            if (sub == 0) continue;
            const bool one_run = sub > cap;  // then r1 == rb + 1: no map needed
            uint32_t e[U];
            if (!one_run) {
                // the run of each entry: eight lanes per run, a warp or the whole block where a unit
                // has few long ones (eight lanes alone take 10 k cycles for 3,000 entries)
                const uint32_t nruns = r1 - rb, G = nruns > 4 * AP_WARPS ? 8u : nruns > 2 ? 32u : (uint32_t)AP_THREADS;
                for (uint32_t r = rb + tid / G; r < r1; r += AP_THREADS / G) {
                    const uint32_t k1 = S.before[r + 1] - base;
                    for (uint32_t k = S.before[r] - base + (tid & (G - 1u)); k < k1; k += G) S.map[k] = (uint16_t)r;
                }
                __syncthreads();
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t k = u * AP_THREADS + tid;
                    e[u] = k < sub ? __ldcg(Q.ent + S.dlt[S.map[k]] + base + k) : 0u;
                }
                part_apply_batch<WIDE, U>(D, S, e, sub, heavy, &s_nflag, &s_drop);
            } else {
                const uint32_t* run = Q.ent + S.dlt[rb] + base;
                for (uint32_t k0 = 0; k0 < sub; k0 += U * AP_THREADS) {
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const uint32_t k = k0 + u * AP_THREADS + tid;
                        e[u] = k < sub ? __ldcg(run + k) : 0u;
                    }
                    part_apply_batch<WIDE, U>(D, S, e, sub - k0, true, &s_nflag, &s_drop);
                }
            }
            __syncthreads();
            const uint32_t F = s_nflag;
            if (F == 0) continue;
            // the records of the flagged buckets (slot, entry, mask number), in the entries' order
            auto put = [&](uint32_t k, uint32_t x, uint32_t at) {
                const uint32_t slot = S.w7[x >> ENT_MASK_BITS] & ~FLAG;
                S.recs[k] = (unsigned long long)slot << 46 | (unsigned long long)at << ENT_MASK_BITS | (x & ENT_MASK);
                if (slot < AP_WARPS) {  // the totals of the first slots, one per warp
                    count_record<WIDE>(S, s_rcnt[slot], x);
                    atomicAdd(&s_rcnt[slot][LOW_COUNTERS], 1u);
                }
            };
            s_rcnt[wid][lane] = 0u;
            if (!one_run) {
                uint32_t hits = 0;  // bit u: entry u
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const bool hit = u * AP_THREADS + tid < sub && (S.w7[e[u] >> ENT_MASK_BITS] & FLAG);
                    const uint32_t bal = __ballot_sync(0xffffffffu, hit);
                    hits |= hit ? 1u << u : 0u;
                    if (lane == 0) s_wcnt[u * AP_WARPS + wid] = __popc(bal);
                }
                __syncthreads();
                if (wid == 0) {
                    uint32_t c[4], sum = 0;
#pragma unroll
                    for (int i = 0; i < 4; ++i) sum += c[i] = s_wcnt[4 * lane + i];
                    uint32_t v = sum;
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) {
                        const uint32_t y = __shfl_up_sync(0xffffffffu, v, d);
                        if (lane >= d) v += y;
                    }
                    if (lane == 31) s_nrec = v;
                    v -= sum;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        s_wcnt[4 * lane + i] = v;
                        v += c[i];
                    }
                }
                __syncthreads();
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t bal = __ballot_sync(0xffffffffu, (hits >> u) & 1u), k = u * AP_THREADS + tid;
                    if ((hits >> u) & 1u)
                        put(s_wcnt[u * AP_WARPS + wid] + __popc(bal & lanemask_lt()), e[u], S.dlt[S.map[k]] + base + k);
                }
            } else {
                __syncthreads();
                for (uint32_t k = tid; k < sub; k += AP_THREADS) {
                    const uint32_t at = S.dlt[rb] + base + k, x = __ldcg(Q.ent + at);
                    if (!(S.w7[x >> ENT_MASK_BITS] & FLAG)) continue;
                    const uint32_t i = atomicAdd(&s_nrec, 1u);
                    if (i < cap) put(i, x, at);
                }
            }
            __syncthreads();
            const uint32_t K = s_nrec;
            if (K <= cap) {
                for (uint32_t s = wid; s < F; s += AP_WARPS)
                    if (!replay_warp<WIDE>(D, Q, S, reinterpret_cast<unsigned long long*>(S.map) + wid * 32, s_rcnt[wid], accs,
                                           &s_nacc, s, K, (uint32_t)b0, &s_rb, &s_rk) && lane == 0)
                        s_many = 1;
                __syncthreads();
            }
            // a bucket with more than 32 records of the tile that crosses: all records sorted by
            // position (12 k cycles for 300 of them), then a warp each
            if (K <= cap && s_many) {
                for (uint32_t k = tid; k < K; k += AP_THREADS) {
                    const unsigned long long r = S.recs[k];
                    const uint32_t at = (uint32_t)(r >> ENT_MASK_BITS);
                    S.recs[k] = (r >> 46) << 46 |
                                (unsigned long long)((at & ~(tile - 1u)) + __ldcg(Q.idx + at)) << ENT_MASK_BITS |
                                (r & ENT_MASK);
                }
                block_sort(S.recs, K);
                for (uint32_t s = wid; s < F; s += AP_WARPS) {
                    const uint32_t lb = S.tab[s * LOW_WORDS + 7];
                    if (S.w7[lb] != (FLAG | s)) continue;  // replayed above
                    uint32_t beg = 0, end = 0;  // the slot's records
                    {
                        uint32_t lo = 0, hi = K;
                        while (lo < hi) {
                            const uint32_t mid = (lo + hi) >> 1;
                            if ((uint32_t)(S.recs[mid] >> 46) < s) lo = mid + 1;
                            else hi = mid;
                        }
                        beg = lo, hi = K;
                        while (lo < hi) {
                            const uint32_t mid = (lo + hi) >> 1;
                            if ((uint32_t)(S.recs[mid] >> 46) <= s) lo = mid + 1;
                            else hi = mid;
                        }
                        end = lo;
                    }
                    uint32_t* bw = S.tab + lb * LOW_WORDS;
                    ReplayOut o;
                    o.T = 0;
                    for (uint32_t q = beg; q < end; q += 32)
                        o.T += group_counts(q + lane < end ? code_mask<WIDE>(S.mk[(uint32_t)S.recs[q + lane] & ENT_MASK]) : 0u);
                    o.P = part_pre(bw, o.T);
                    o.cur = o.P;
                    o.mL = 0;
                    o.found = false;
                    o.L = 0;
                    for (uint32_t q = beg; q < end; q += 32) {
                        const uint32_t m = q + lane < end ? code_mask<WIDE>(S.mk[(uint32_t)S.recs[q + lane] & ENT_MASK]) : 0u;
                        const int j = link_step(m, o.cur);
                        if (j >= 0) {
                            o.found = true;
                            o.L = q + j;
                            o.mL = __shfl_sync(0xffffffffu, m, j);
                            break;
                        }
                    }
                    if (o.found) {
                        const uint32_t pos = (uint32_t)(S.recs[o.L] >> ENT_MASK_BITS);
                        const uint32_t H = high_increments(D, o);
                        __syncwarp();
                        part_write_low(bw, o.cur);
                        open_row(D, S, accs, &s_nacc, lb, (uint32_t)b0, pos, end - o.L, H);
                    } else if (lane == 0) {
                        S.w7[lb] = 0u;  // every key added low
                    }
                    if (lane == 0) {
                        atomicAdd(&s_rb, 1u);
                        atomicAdd(&s_rk, end - beg);
                    }
                }
            } else if (K > cap) {
                // More records than fit, all of one tile (a very heavy key that is not linked
                // yet): per flagged bucket, bisect the array position of the switching key, the
                // first position x such that some counter has 130 - P occurrences up to x (the key
                // that sees 129 = P + its earlier occurrences).
                const uint32_t plo = (tile_s + rb) * tile, phi = plo + tile - 1;
                for (uint32_t s = 0; s < F; ++s) {
                    const uint32_t lb = S.tab[s * LOW_WORDS + 7];
                    uint32_t* bw = S.tab + lb * LOW_WORDS;
                    auto count = [&](uint32_t upto) {  // occurrences per counter (and keys) at positions <= upto
                        __syncthreads();
                        if (tid < LOW_COUNTERS + 2) s_cnt[tid] = 0u;
                        __syncthreads();
                        for (uint32_t k = tid; k < sub; k += AP_THREADS) {
                            const uint32_t at = S.dlt[rb] + base + k, x = __ldcg(Q.ent + at);
                            if ((x >> ENT_MASK_BITS) != lb) continue;
                            const uint32_t pos = plo + __ldcg(Q.idx + at);
                            if (pos > upto) continue;
                            const uint32_t m = code_mask<WIDE>(S.mk[x & ENT_MASK]);
                            for (uint32_t mm = m; mm; mm &= mm - 1) atomicAdd(s_cnt + (__ffs(mm) - 1), 1u);
                            atomicAdd(s_cnt + LOW_COUNTERS, 1u);
                            if (pos == upto) s_cnt[LOW_COUNTERS + 1] = m;
                        }
                        __syncthreads();
                    };
                    count(phi);
                    const uint32_t n_total = s_cnt[LOW_COUNTERS];
                    uint32_t T = lane < LOW_COUNTERS ? s_cnt[lane] : 0u;
                    if (wid == 0) {
                        const uint32_t P = part_pre(bw, T);
                        if (lane < LOW_COUNTERS) s_pre[lane] = P;
                    }
                    __syncthreads();
                    const uint32_t P = lane < LOW_COUNTERS ? s_pre[lane] : 0u;
                    auto reached = [&](uint32_t c) { return __any_sync(0xffffffffu, c && P + c > LIMIT + 1); };
                    const bool found = reached(T);
                    uint32_t lo = plo, hi = phi;  // uniform over the block
                    while (found && lo < hi) {
                        const uint32_t mid = lo + (hi - lo) / 2;
                        count(mid);
                        if (reached(lane < LOW_COUNTERS ? s_cnt[lane] : 0u)) hi = mid;
                        else lo = mid + 1;
                    }
                    if (found) count(lo);
                    if (wid == 0) {
                        if (found) {
                            ReplayOut o;
                            o.T = T;
                            o.P = P;
                            o.mL = s_cnt[LOW_COUNTERS + 1];
                            const uint32_t upto = lane < LOW_COUNTERS ? s_cnt[lane] : 0u;
                            o.cur = P + upto - (lane < LOW_COUNTERS ? (o.mL >> lane) & 1u : 0u);
                            const uint32_t n_after = n_total - s_cnt[LOW_COUNTERS] + 1u;
                            const uint32_t H = high_increments(D, o);
                            part_write_low(bw, o.cur);
                            open_row(D, S, accs, &s_nacc, lb, (uint32_t)b0, lo, n_after, H);
                        } else if (lane == 0) {
                            S.w7[lb] = 0u;
                        }
                        if (lane == 0) {
                            s_rb += 1u;
                            s_rk += n_total;
                        }
                    }
                    __syncthreads();
                }
            }
            __syncthreads();
            if (tid == 0) s_nflag = s_nrec = s_many = 0;
        }
    }
    __syncthreads();
    // the accumulators: linked buckets' counts to their high buckets, new ones to rows
    const uint32_t na = min(s_nacc, accs);
    for (uint32_t a = tid; a < na; a += AP_THREADS)
        if (S.w7[S.accb[a]] & NEW) atomicAdd(&s_new, 1u);
    __syncthreads();
    if (tid == 0 && s_new) s_row = atomicAdd(&D.ctl->n_switch, s_new);
    __syncthreads();
    for (uint32_t a = wid; a < na; a += AP_WARPS) {
        const uint32_t lb = S.accb[a], id = S.accid[a];
        const uint32_t v = lane < LOW_COUNTERS ? S.acc[a * ACC_WORDS + lane] : 0u;
        if (S.w7[lb] & NEW) {
            uint32_t r = 0;
            if (lane == 0) r = atomicAdd(&s_row, 1u);
            r = __shfl_sync(0xffffffffu, r, 0);
            put_row(D, r, S.stream, (uint32_t)b0 + lb, id, S.acc[a * ACC_WORDS + LOW_COUNTERS], v);
            if (lane == 0 && r >= D.long_cap) S.w7[lb] = TEMP | r;
        } else {
            if (v) atomicAdd(D.high + (uint64_t)(id - START) * HIGH_WORDS + lane, v);
            if (lane == 0) S.w7[lb] = id;
        }
    }
    __syncthreads();
    {
        const uint4* st = reinterpret_cast<const uint4*>(S.tab);
        for (uint32_t i = tid; i < nb * 2; i += AP_THREADS) {
            uint4 v = st[i];
            if (i & 1u) v.w = S.w7[i >> 1];  // a new bucket's is set with its id
            __stcg(gt + i, v);
        }
    }
    if (tid == 0) {
        if (s_drop) atomicAdd(&D.ctl->dropped, (unsigned long long)s_drop);
        if (s_rb) {
            atomicAdd(&D.ctl->repaired_buckets, (unsigned long long)s_rb);
            atomicAdd(&D.ctl->repaired_keys, (unsigned long long)s_rk);
        }
    }
}

// ---- 3: high ids in the array order of the switching keys -----------------------------------

// The id of a bucket that switched at position pos, ranked by spre and the switch bits (a batch:
// within the stream, whose positions are contiguous, on its own allocator); ok: inside the pool.
// Called by a whole warp.
template <bool BATCH>
__device__ __forceinline__ uint32_t part_link_id(const MswsDev& D, const PartDev& Q, const BatchDev& B, const uint32_t* spre,
                                                 uint32_t base, uint32_t stream, uint32_t pos, bool& ok) {
    const uint32_t id = base + switch_rank(D, spre, pos);
    if (!BATCH) {
        ok = (uint64_t)(id - START) < D.n_high;
        return id;
    }
    const uint32_t own = __ldcg(B.base_id + stream) + (id - base) - switch_rank(D, spre, __ldcg(B.item_off + stream) * Q.tile);
    const uint32_t nh = __ldg(&B.desc[stream].n_high);
    ok = (uint64_t)(own - START) < nh;
    if ((threadIdx.x & 31) == 0) {
        atomicMax(B.next_id + stream, (uint32_t)min((unsigned long long)own + 1ull, (unsigned long long)START + nh));
        if (!ok) atomicOr(B.status + stream, ST_POOL_FULL);
    }
    return own + __ldg(&B.desc[stream].high_base);
}

// More buckets linked in the chunk than there are rows of counts: the others' index words still hold
// their rows' numbers.  A block takes a partition, links its buckets of that kind and counts their
// entries from the switches on again, all in one pass over the partition's entries.  (Bucket by
// bucket, each by a warp over the partition's entries, 2^24 keys that link most of 2^19 uniform
// buckets took 9.4 ms and 0.6 M buckets of equal keys 184 ms; so 0.93 and 5.1, the ranks of the ids.)
template <bool BATCH>
__device__ __forceinline__ void part_link_rest(const MswsDev& D, const PartDev& Q, const BatchDev& B, const uint32_t* spre,
                                               uint32_t base, uint32_t parts) {
    __shared__ uint32_t s_pos[1u << PART_MAX_SHIFT], s_id[1u << PART_MAX_SHIFT];  // by bucket; id 0: dropped
    __shared__ uint16_t s_list[1u << PART_MAX_SHIFT];
    __shared__ uint32_t s_n, s_first;
    const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    bool full = false;  // a bucket found the pool exhausted
    for (uint32_t q = blockIdx.x; q < parts; q += gridDim.x) {
        uint32_t p = q, stream;
        const PartView V = part_of_block<BATCH>(D, Q, B, p, stream);
        if (V.tiles == 0) continue;
        const uint64_t b0 = V.low_base + ((uint64_t)p << V.shift);
        const uint32_t nb = (uint32_t)umin64((uint64_t)1 << V.shift, V.fm.d - ((uint64_t)p << V.shift));
        __syncthreads();
        if (tid == 0) s_n = 0, s_first = NONE;
        __syncthreads();
        for (uint32_t i = tid; i < nb; i += AP_THREADS) {
            const uint32_t w7 = __ldcg(D.low + (b0 + i) * LOW_WORDS + 7), r = w7 & ~TEMP;
            uint32_t pos = NONE;
            if (w7 < FLAG && (w7 & TEMP) && r >= D.long_cap) {
                pos = __ldcg(&D.sw[r].x);
                atomicMin(&s_first, pos);
                s_list[atomicAdd(&s_n, 1u)] = (uint16_t)i;
            }
            s_pos[i] = pos;
        }
        __syncthreads();
        const uint32_t n = s_n;
        if (n == 0) continue;
        for (uint32_t l = wid; l < n; l += AP_WARPS) {
            const uint32_t i = s_list[l];
            bool ok;
            const uint32_t id = part_link_id<BATCH>(D, Q, B, spre, base, stream, s_pos[i], ok);
            if (ok) {
                link_bucket(D, (uint32_t)(b0 + i), id, true, 0u, 0u);
            } else if (lane == 0) {
                __stcg(D.low + (b0 + i) * LOW_WORDS + 7, SATURATED);
                full = true;
            }
            if (lane == 0) s_id[i] = ok ? id : 0u;
        }
        __syncthreads();
        const uint16_t* o0 = V.off + (uint64_t)p * V.stride - V.tile0;
        constexpr uint32_t G = 8;  // lanes per run
        uint32_t dropped = 0;
        for (uint32_t t = s_first / Q.tile + tid / G; t < V.tile0 + V.tiles; t += AP_THREADS / G) {
            const uint32_t e1 = t * Q.tile + __ldcg(o0 + V.stride + t);
            for (uint32_t i = t * Q.tile + __ldcg(o0 + t) + (tid & (G - 1u)); i < e1; i += G) {
                const uint32_t e = __ldcg(Q.ent + i), first = s_pos[e >> ENT_MASK_BITS];
                if (first == NONE) continue;
                const uint32_t pos = t * Q.tile + __ldcg(Q.idx + i), id = s_id[e >> ENT_MASK_BITS];
                if (pos < first) continue;
                if (id == 0u) {
                    ++dropped;
                    continue;
                }
                uint32_t* hb = D.high + (uint64_t)(id - START) * HIGH_WORDS;
                const uint32_t wrap = D.compat_v3 && pos == first ? 7u : 31u;  // the switching key lands on bit % 8
                for (uint32_t m = __ldg(D.masks + (e & ENT_MASK)); m; m &= m - 1) atomicAdd(hb + ((__ffs(m) - 1) & wrap), 1u);
            }
        }
        if (dropped) atomicAdd(&D.ctl->dropped, (unsigned long long)dropped);
    }
    if (full) atomicOr(&D.ctl->status, ST_POOL_FULL);
}

template <bool BATCH>
__global__ void __launch_bounds__(AP_THREADS, 2) k_part_link(MswsDev D, PartDev Q, BatchDev B, uint32_t parts) {
    extern __shared__ __align__(16) uint32_t spre[];  // switches per SW_BLOCK positions, then their prefix
    Ctl* ctl = D.ctl;
    const uint32_t ns = __ldcg(&ctl->n_switch);
    if (ns == 0) return;
    const uint32_t base = __ldcg(&ctl->link_base);
    const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (!BATCH && blockIdx.x == 0 && tid == 0)  // the allocator stops at the pool's end, as the oracle's
        ctl->next_id = (uint32_t)min((unsigned long long)base + ns, (unsigned long long)START + D.n_high);
    if (blockIdx.x * AP_WARPS >= ns) return;
    const uint32_t nq = (uint32_t)(((uint64_t)Q.tiles * Q.tile + SW_BLOCK - 1) / SW_BLOCK);
    for (uint32_t i = tid; i < nq; i += AP_THREADS) spre[i] = __ldcg(D.sw_cnt + i);
    __syncthreads();
    block_scan_smem(spre, nq);
    const uint32_t rows = min(ns, D.long_cap);
    for (uint32_t r = blockIdx.x * AP_WARPS + wid; r < rows; r += gridDim.x * AP_WARPS) {
        const uint2 w = __ldcg(D.sw + r);
        const uint32_t stream = BATCH ? __ldcg(D.sw_base + r) : 0u, b = __ldcg(D.flag_list + r);
        bool ok;
        const uint32_t id = part_link_id<BATCH>(D, Q, B, spre, base, stream, w.x, ok);
        const uint32_t H = lane < LOW_COUNTERS ? __ldcg(D.totals + (uint64_t)r * LOW_COUNTERS + lane) : 0u;
        link_bucket(D, b, id, ok, H, w.y);
    }
    if (ns > rows) part_link_rest<BATCH>(D, Q, B, spre, base, parts);
}

// ---- launchers ------------------------------------------------------------------------------

static size_t split_smem(uint32_t tile, uint32_t parts, uint32_t hot) {
    return (size_t)tile * 6 + parts * 4 + hot * 12;
}

// Kernel and threads of a split by tile size.
template <int HOT, bool BATCH, bool TABLE>
static const void* split_of(bool small) {
    return small ? (const void*)k_part_split<512, 4, HOT, BATCH, TABLE> : (const void*)k_part_split<1024, 16, HOT, BATCH, TABLE>;
}
static const void* split_fn(uint32_t tile, int hot, bool batch, bool table) {
    const bool small = tile == PART_TILE_SMALL;
    if (batch)  // small tiles without, large ones with heavy keys
        return small ? (const void*)k_part_split<512, 4, HOT_NONE, true, false> : (const void*)k_part_split<1024, 16, HOT_CALL, true, false>;
    if (table)
        return hot == HOT_OWN    ? split_of<HOT_OWN, false, true>(small)
               : hot == HOT_CALL ? split_of<HOT_CALL, false, true>(small)
                                 : split_of<HOT_NONE, false, true>(small);
    return hot == HOT_OWN    ? split_of<HOT_OWN, false, false>(small)
           : hot == HOT_CALL ? split_of<HOT_CALL, false, false>(small)
                             : split_of<HOT_NONE, false, false>(small);
}

static const void* apply_fn(bool wide, bool batch) {
    return batch ? (wide ? (const void*)k_part_apply<true, true> : (const void*)k_part_apply<false, true>)
                 : (wide ? (const void*)k_part_apply<true, false> : (const void*)k_part_apply<false, false>);
}

size_t part_apply_smem(uint32_t shift, uint32_t n_masks) { return apply_smem(shift, n_masks); }

cudaError_t part_configure(int num_sms, PartLaunch* L) {
    // the dynamic shared-memory cap is a per-kernel attribute shared by every sketch of the
    // process: the largest any of them may ask for; a launch passes its own size
    const size_t split_max = split_smem(PART_TILE, PART_MAX_PARTS, PART_HOT);
    const size_t apply_max = std::max(apply_smem(PART_MAX_SHIFT, PART_MAX_MASKS), apply_smem(PART_MAX_SHIFT - 1, PART_MAX_MASKS));
    const size_t link_max = PART_MAX_CHUNK / SW_BLOCK * 4;
    cudaError_t e = cudaSuccess;
    auto cap = [&](const void* fn, size_t bytes) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    };
    for (int batch = 0; batch < 2; ++batch) {
        for (int hot = 0; hot < 3; ++hot)
            for (int i = 0; i < 4; ++i) cap(split_fn(i & 1 ? PART_TILE : PART_TILE_SMALL, hot, batch != 0, i & 2), split_max);
        for (int wide = 0; wide < 2; ++wide) cap(apply_fn(wide != 0, batch != 0), apply_max);
    }
    cap((const void*)k_part_link<false>, link_max);
    cap((const void*)k_part_link<true>, link_max);
    L->num_sms = num_sms;
    return e;
}

cudaError_t part_hot(const uint32_t* d_keys, uint64_t n, const PartDev& part, cudaStream_t st) {
    uint32_t* hot = part.hot;
    void* args[] = {(void*)&d_keys, (void*)&n, (void*)&hot};
    return cudaLaunchKernel((const void*)k_part_hot, dim3(HOT_BLOCKS), dim3(HOT_THREADS), args, 0, st);
}

// Split, apply and link of a chunk (or a batch's window) whose tiles Q names.
static cudaError_t part_steps(const uint32_t* d_keys, uint64_t n, const MswsDev& D, const PartDev& Q, const BatchDev& B,
                              const PartLaunch& L, int hot, uint32_t blocks, cudaStream_t st) {
    MswsDev Dc = D;
    PartDev Qc = Q;
    BatchDev Bc = B;
    const bool batch = B.n_streams != 0;
    {
        void* args[] = {(void*)&d_keys, (void*)&n, (void*)&Dc, (void*)&Qc, (void*)&Bc};
        const bool small = Q.tile == PART_TILE_SMALL;
        const int grid = (int)std::min<uint64_t>(Q.tiles, (uint64_t)(small ? 2 * L.num_sms : L.num_sms));
        const cudaError_t e = cudaLaunchKernel(split_fn(Q.tile, hot, batch, D.tbl_keys != nullptr), dim3(grid), dim3(small ? 512 : 1024), args,
                                               split_smem(Q.tile, Q.parts, hot ? (batch ? BATCH_HOT : PART_HOT) : 0), st);
        if (e != cudaSuccess) return e;
    }
    void* args[] = {(void*)&Dc, (void*)&Qc, (void*)&Bc};
    const cudaError_t e = cudaLaunchKernel(apply_fn(D.wide != 0, batch), dim3(blocks), dim3(AP_THREADS), args, L.apply_smem, st);
    if (e != cudaSuccess) return e;
    const uint64_t nq = ((uint64_t)Q.tiles * Q.tile + SW_BLOCK - 1) / SW_BLOCK;
    void* largs[] = {(void*)&Dc, (void*)&Qc, (void*)&Bc, (void*)&blocks};
    return cudaLaunchKernel(batch ? (const void*)k_part_link<true> : (const void*)k_part_link<false>, dim3(L.num_sms),
                            dim3(AP_THREADS), largs, (size_t)nq * 4, st);
}

cudaError_t part_insert(const uint32_t* d_keys, uint64_t n, const MswsDev& D, const PartDev& part, const PartLaunch& L,
                        int hot, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    PartDev Q = part;
    // small tiles while large ones would leave more than half of the SMs idle
    Q.tile = n < PART_SMALL_MAX ? PART_TILE_SMALL : PART_TILE;
    Q.tiles = (uint32_t)((n + Q.tile - 1) / Q.tile);
    return part_steps(d_keys, n, D, Q, BatchDev{}, L, hot, Q.parts, st);
}

cudaError_t part_hot_batch(const uint32_t* d_keys, const BatchDev& B, uint64_t first, uint64_t fold, cudaStream_t st) {
    k_part_hot_batch<<<B.n_streams, 256, 0, st>>>(d_keys, B, first, fold);
    return cudaGetLastError();
}

cudaError_t part_insert_batch(const uint32_t* d_keys, const MswsDev& D, const PartDev& part, const BatchDev& B,
                              const PartLaunch& L, const BatchWindow& W, uint32_t tiles, uint32_t parts, bool hot,
                              cudaStream_t st) {
    if (tiles == 0) return cudaSuccess;
    PartDev Q = part;
    Q.tile = hot ? PART_TILE : PART_TILE_SMALL;
    Q.tiles = tiles;
    k_part_plan<<<1, 1024, 0, st>>>(B, W, Q.tile, D.ctl);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return part_steps(d_keys, 0, D, Q, B, L, hot, parts, st);
}

}  // namespace qsb
