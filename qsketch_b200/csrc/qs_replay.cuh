// qs_replay.cuh — the order-dependent arithmetic of one bucket, shared by the two insert paths
// (pass 1 + grid-wide ordered replay in qs_msws.cu, partitioned insert in qs_part.cu): does an
// addition cross the 8-bit threshold, where does a bucket's key sequence switch levels, and
// what the new high bucket then holds (device_sketch_v3.h:88-191).
#pragma once
#include "qs_device.cuh"

namespace qsb {

constexpr uint32_t NONE = 0xffffffffu;

__device__ __forceinline__ bool is_linked(const MswsDev& D, uint32_t w7) {
    return w7 > START && (uint64_t)(w7 - START) < D.n_high;
}

// A mask table of three counters per mask (the default) is kept as the counters' numbers, 5 bits
// each; any other (WIDE) as the masks.  Computed once, at create: recoding the table in every block of
// a query cost 0.2 us of the 3.5 that 10,007 keys take.
template <bool WIDE>
__device__ __forceinline__ const uint32_t* mask_codes(const MswsDev& D) {
    return WIDE ? D.masks : D.codes;
}
template <bool WIDE>
__device__ __forceinline__ uint32_t code_mask(uint32_t q) {
    return WIDE ? q : (1u << (q & 31u)) | (1u << ((q >> 5) & 31u)) | (1u << (q >> 10));
}

// Does a selected byte (nibble bit k selects byte k) of the pre-add word `old` reach CROSS
// once c is added: byte + c >= CROSS, i.e. byte >= CROSS - c, four bytes at a time.
// Selected bytes all below 64 with c below 64 cannot reach CROSS: a two-operation test
// settles the common case before the four-byte comparison.
__device__ __forceinline__ bool crosses(uint32_t old, uint32_t nib, uint32_t c) {
    if (!nib) return false;
    if (c >= CROSS) return true;
    const uint32_t sel = expand_nibble(nib) * 0xffu;
    if (c < 64u && !(old & sel & 0xC0C0C0C0u)) return false;
    return (__vcmpgeu4(old, (CROSS - c) * 0x01010101u) & sel) != 0u;
}

// Occurrences of counter c (lane c) among the 32 masks of the warp: seven warp sums of the
// masks expanded to one byte per counter (a byte counts at most 32, so no carries).
__device__ __forceinline__ uint32_t group_counts(uint32_t m) {
    const int lane = threadIdx.x & 31;
    uint32_t mine = 0;
#pragma unroll
    for (int w = 0; w < 7; ++w) {
        const uint32_t t = __reduce_add_sync(0xffffffffu, expand_nibble((m >> (4 * w)) & 0xfu));
        if ((lane >> 2) == w) mine = t;
    }
    return lane < LOW_COUNTERS ? (mine >> (8 * (lane & 3))) & 0xffu : 0u;
}

// 32 consecutive records (mask m, 0 for lanes that are not this bucket's): returns the lane
// of the first record that sees a selected counter above LIMIT, or -1; `cur` advances over
// the records before it (all 32 when none triggers).
__device__ __forceinline__ int link_step(uint32_t m, uint32_t& cur) {
    const int lane = threadIdx.x & 31;
    // The last record with counter c sees cur + (occurrences - 1): when that stays within
    // LIMIT for every counter, no record of the group switches.
    const uint32_t tot = group_counts(m);
    if (!__any_sync(0xffffffffu, tot && cur + tot > LIMIT + 1)) {
        cur += tot;
        return -1;
    }
    const uint32_t lt = lanemask_lt();
    bool trig = false;
    uint32_t inc = 0;
#pragma unroll
    for (int c = 0; c < LOW_COUNTERS; ++c) {
        const uint32_t bal = __ballot_sync(0xffffffffu, (m >> c) & 1u);
        const uint32_t cc = __shfl_sync(0xffffffffu, cur, c);
        if (((m >> c) & 1u) && cc + __popc(bal & lt) > LIMIT) trig = true;
        if (lane == c) inc = __popc(bal);
    }
    const uint32_t tb = __ballot_sync(0xffffffffu, trig);
    if (!tb) {
        cur += inc;
        return -1;
    }
    const int j = __ffs(tb) - 1;
    const uint32_t before = (1u << j) - 1u;
#pragma unroll
    for (int c = 0; c < LOW_COUNTERS; ++c) {
        const uint32_t bal = __ballot_sync(0xffffffffu, (m >> c) & 1u);
        if (lane == c) cur += __popc(bal & before);
    }
    return j;
}

// Where the replay of one flagged bucket ended (per lane c: counter c).
struct ReplayOut {
    bool found;        // a key switched the bucket to the high level
    uint32_t L;        // that key's record: index into the records the replay read
    uint32_t n_after;  // the bucket's keys at or after the switch
    uint32_t n_total;  // the bucket's keys in the chunk
    uint32_t T;        // the chunk's increments of counter c
    uint32_t P;        // counter c before the chunk
    uint32_t cur;      // counter c when the switch happens (final low value)
    uint32_t mL;       // the switching key's mask
};

// Increments of high counter `lane` in the new high bucket: the switching key's and all
// later keys'.
__device__ __forceinline__ uint32_t high_increments(const MswsDev& D, const ReplayOut& o) {
    const int lane = threadIdx.x & 31;
    uint32_t H = o.T - (o.cur - o.P);
    if (D.compat_v3) {  // device_sketch_v3.h:187: the switching key lands on bit % 8
        if (lane < LOW_COUNTERS && ((o.mL >> lane) & 1u)) H -= 1u;
        if (lane < 8) H += __popc(o.mL & (0x01010101u << lane));
    }
    return H;
}

// Link bucket b to high id `id` (global; ok: inside the pool) with high increments H, or
// saturate it when the pool has run out (its n_after keys are dropped).
__device__ __forceinline__ void link_bucket(const MswsDev& D, uint32_t b, uint32_t id, bool ok, uint32_t H,
                                            uint32_t n_after) {
    const int lane = threadIdx.x & 31;
    if (ok) {
        __stcg(D.high + (uint64_t)(id - START) * HIGH_WORDS + lane, H);
    } else if (lane == 0) {
        atomicOr(&D.ctl->status, ST_POOL_FULL);
        atomicAdd(&D.ctl->dropped, (unsigned long long)n_after);
    }
    if (lane == 7) __stcg(D.low + (uint64_t)b * LOW_WORDS + 7, ok ? id : SATURATED);
}

// Rank of switch position p among all switch positions of the chunk (the result in every
// lane): the exclusive prefix `spre` of the per-SW_BLOCK counts, plus the set bits before p
// in its block of 128 words.
__device__ __forceinline__ uint32_t switch_rank(const MswsDev& D, const uint32_t* spre, uint32_t p) {
    const int lane = threadIdx.x & 31;
    const uint32_t q = p / SW_BLOCK, w = p >> 5;
    uint32_t c = 0;
#pragma unroll
    for (int k = 0; k < (int)(SW_BLOCK / 32 / 32); ++k) {
        const uint32_t wi = q * (SW_BLOCK / 32) + k * 32 + lane;
        if (wi < w) c += __popc(__ldcg(D.sw_bits + wi));
    }
    if (lane == 0) c += __popc(__ldcg(D.sw_bits + w) & ((1u << (p & 31)) - 1u));
    return spre[q] + __reduce_add_sync(0xffffffffu, c);
}

// ---- batched streams ----------------------------------------------------------------------

__device__ __forceinline__ bool in_window(const BatchDev& B, const BatchWindow& W, uint32_t s, uint64_t len) {
    if (W.which == STREAMS_ALL) return true;
    return batch_dense(len, B.desc[s].fm_low.d, B.desc[s].parts) == (W.which == STREAMS_DENSE);
}

// The stream whose bucket range holds global bucket g (bases strictly increase).
__device__ __forceinline__ uint32_t stream_of_bucket(const BatchDev& B, uint32_t g) {
    uint32_t lo = 0, hi = B.n_streams;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(&B.desc[mid].low_base) <= g)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// The stream of work item `it` (< item_off[n_streams]): the last s with item_off[s] <= it.
// Called by a whole warp: each step probes 32 evenly spaced offsets, so 512 streams take two
// dependent loads instead of nine.
__device__ __forceinline__ uint32_t stream_of_item_warp(const BatchDev& B, uint32_t it) {
    const int lane = threadIdx.x & 31;
    uint32_t lo = 0, hi = B.n_streams;  // item_off[lo] <= it; the answer lies in [lo, hi)
    while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t idx = lo + lane * step;
        const bool le = idx < hi && __ldcg(B.item_off + idx) <= it;
        const uint32_t bal = __ballot_sync(0xffffffffu, le);  // lane 0 always holds
        const uint32_t last = 31 - __clz(bal);
        lo += last * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

}  // namespace qsb
