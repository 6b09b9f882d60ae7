// qs_remove.cu — REMOVE: one occurrence of each key taken out of the sketch.
//
// The reference has no deletion code; its paper defines deletion as the insertion with a
// subtraction (doc/main.tex:232, "increase or decrease the count variables").  For the
// two-level MSWS the bucket's level decides where a removal lands: a linked bucket's selected
// high counters lose one, an unlinked bucket's selected 8-bit low counters lose one, each
// floored at 0; a saturated bucket drops the removal (counted).  Removals never link or
// unlink a bucket, so within one call the result per counter is max(0, value - removals)
// whatever the order of the keys: a saturating subtraction per word, applied by a CAS loop
// after equal keys of a warp are merged (one update of c removals instead of c updates).
// Count-min: each row's counter loses one, floored at 0.
//
// Contention decides the cost: with one update per warp and key, the hundreds of warps that
// hold a heavy key's occurrences retried their compare-and-swaps against each other (3 M keys of a
// power law of exponent 1, 130 ms).  So equal keys of a 2048-key tile merge in shared memory
// first, and a u32 counter takes a saturating subtraction in one atomic without retries:
//   old = atomicAdd(p, -c); if old < c, the deficit (c, or c - old when old >= 0) goes back.
// Let W be the counter plus the deficits still to go back.  The first subtraction below zero
// leaves W = 0, and while any deficit is out the counter is negative, so every later
// subtraction gives back all of its c: W stays 0, as max(0, value - removals) asks, and W is the
// counter when the kernel ends.  Needs counters and the call's keys below 2^31, so that negative is
// told from large: the caller knows how many keys were inserted (SIGNED); otherwise the
// compare-and-swap loop stays.
#include "qs_device.cuh"
#include "qs_kernels.h"

namespace qsb {

constexpr int RM_THREADS = 256;
constexpr uint32_t RM_TRIES = 1u << 22;  // CAS attempts per word before giving up (ST_TIMEOUT)

// Per-byte saturating subtraction of `dec` from *w; false if the CAS never won.
__device__ __forceinline__ bool sat_sub_bytes(uint32_t* w, uint32_t dec) {
    uint32_t old = __ldcg(w);
    for (uint32_t it = 0; it < RM_TRIES; ++it) {
        const uint32_t nw = __vsubus4(old, dec);
        if (nw == old) return true;  // every selected byte already 0
        const uint32_t prev = atomicCAS(w, old, nw);
        if (prev == old) return true;
        old = prev;
    }
    return false;
}

// Saturating subtraction of c from the u32 counter *p; false if the CAS never won.
__device__ __forceinline__ bool sat_sub_u32(uint32_t* p, uint32_t c) {
    uint32_t old = __ldcg(p);
    for (uint32_t it = 0; it < RM_TRIES; ++it) {
        const uint32_t nw = old > c ? old - c : 0u;
        if (nw == old) return true;
        const uint32_t prev = atomicCAS(p, old, nw);
        if (prev == old) return true;
        old = prev;
    }
    return false;
}

template <bool SIGNED>
__device__ __forceinline__ bool sub_u32(uint32_t* p, uint32_t c) {
    if (!SIGNED) return sat_sub_u32(p, c);
    const int32_t old = (int32_t)atomicAdd(p, 0u - c);
    if (old < (int32_t)c) atomicAdd(p, c - (uint32_t)max(old, 0));
    return true;
}

constexpr uint32_t RM_TILE = 2048, RM_SLOTS = 4096, RM_PROBES = 16;
constexpr uint32_t RM_EMPTY = 0xffffffffu;

struct RmTable {
    uint32_t key[RM_SLOTS], cnt[RM_SLOTS];
    uint32_t top;  // occurrences of the key that equals RM_EMPTY
};

// Tile by tile: equal keys merge in the table, then fn(key, count) once per distinct key (a key
// that finds no slot within RM_PROBES goes to fn at once).
template <class F>
__device__ __forceinline__ void merged_tiles(const uint32_t* __restrict__ keys, uint64_t n, RmTable& T, F fn) {
    const uint32_t tid = threadIdx.x;
    for (uint32_t i = tid; i < RM_SLOTS; i += RM_THREADS) T.key[i] = RM_EMPTY, T.cnt[i] = 0u;
    if (tid == 0) T.top = 0u;
    for (uint64_t t0 = (uint64_t)blockIdx.x * RM_TILE; t0 < n; t0 += (uint64_t)gridDim.x * RM_TILE) {
        uint32_t k[RM_TILE / RM_THREADS];
#pragma unroll
        for (uint32_t j = 0; j < RM_TILE / RM_THREADS; ++j) {
            const uint64_t i = t0 + j * RM_THREADS + tid;
            k[j] = i < n ? __ldcs(keys + i) : 0u;
        }
        __syncthreads();
#pragma unroll
        for (uint32_t j = 0; j < RM_TILE / RM_THREADS; ++j) {
            if (t0 + j * RM_THREADS + tid >= n) break;
            if (k[j] == RM_EMPTY) {
                atomicAdd(&T.top, 1u);
                continue;
            }
            const uint32_t h = k[j] * 0x9E3779B1u >> 20;
            uint32_t q = 0;
            for (; q < RM_PROBES; ++q) {
                const uint32_t s = (h + q) & (RM_SLOTS - 1);
                uint32_t seen = reinterpret_cast<volatile uint32_t*>(T.key)[s];
                if (seen == RM_EMPTY) seen = atomicCAS(T.key + s, RM_EMPTY, k[j]);
                if (seen == RM_EMPTY || seen == k[j]) {
                    atomicAdd(T.cnt + s, 1u);
                    break;
                }
            }
            if (q == RM_PROBES) fn(k[j], 1u);
        }
        __syncthreads();
        for (uint32_t i = tid; i < RM_SLOTS; i += RM_THREADS) {
            const uint32_t key = T.key[i], c = T.cnt[i];
            if (key == RM_EMPTY) continue;
            T.key[i] = RM_EMPTY;
            T.cnt[i] = 0u;
            fn(key, c);
        }
        if (tid == 0 && T.top) {
            fn(RM_EMPTY, T.top);
            T.top = 0u;
        }
    }
}
static_assert(RM_SLOTS == 1u << 12, "12 hash bits");

template <bool SIGNED>
__global__ void __launch_bounds__(RM_THREADS) k_msws_remove(const uint32_t* __restrict__ keys, uint64_t n, MswsDev D) {
    __shared__ RmTable T;
    bool ok = true;
    uint32_t dropped = 0;
    merged_tiles(keys, n, T, [&](uint32_t key, uint32_t c) {
        const uint32_t hv = key * D.seed;
        const uint32_t b = fast_mod(D.fm_low, hv);
        const uint32_t m = __ldg(D.masks + fast_mod(D.fm_mask, hv));
        uint32_t* wp = D.low + (uint64_t)b * LOW_WORDS;
        const uint32_t ptr = __ldcg(wp + 7);
        if (ptr == SATURATED) {
            dropped += c;
        } else if (ptr > START && (uint64_t)(ptr - START) < D.n_high) {
            uint32_t* hb = D.high + (uint64_t)(ptr - START) * HIGH_WORDS;
            for (uint32_t mm = m; mm; mm &= mm - 1) ok &= sub_u32<SIGNED>(hb + (__ffs(mm) - 1), c);
        } else {
            // bytes hold at most 129: more removals than that empty them
            const uint32_t cb = min(c, 255u);
#pragma unroll
            for (int w = 0; w < 7; ++w) {
                const uint32_t nib = (m >> (4 * w)) & 0xfu;
                if (nib) ok &= sat_sub_bytes(wp + w, expand_nibble(nib) * cb);
            }
        }
    });
    if (!ok) atomicOr(&D.ctl->status, ST_TIMEOUT);
    if (dropped) atomicAdd(&D.ctl->dropped, (unsigned long long)dropped);
}

template <bool SIGNED>
__global__ void __launch_bounds__(RM_THREADS) k_cm_remove(const uint32_t* __restrict__ keys, uint64_t n, CmDev D,
                                                          uint32_t* __restrict__ status) {
    __shared__ RmTable T;
    bool ok = true;
    merged_tiles(keys, n, T, [&](uint32_t key, uint32_t c) {
        if (D.masks) {  // one-level bucket sketch: the selected counters of the key's bucket
            const uint32_t hv = key * D.seeds[0];
            uint32_t* bucket = D.table + (uint64_t)fast_mod(D.fm, hv) * D.rows;
            for (uint32_t mm = __ldg(D.masks + fast_mod(D.fm_mask, hv)); mm; mm &= mm - 1)
                ok &= sub_u32<SIGNED>(bucket + (__ffs(mm) - 1), c);
            return;
        }
        for (uint32_t j = 0; j < D.rows; ++j)
            ok &= sub_u32<SIGNED>(D.table + (uint64_t)j * D.n + fast_mod(D.fm, key * D.seeds[j]), c);
    });
    if (!ok && status) atomicOr(status, ST_TIMEOUT);
}

// Persistent blocks of at least a tile each; 33 KB of shared memory leaves six to an SM.
static int rm_grid(uint64_t n, int blocks) {
    return (int)std::min<uint64_t>((uint64_t)blocks, (n + RM_TILE - 1) / RM_TILE);
}

cudaError_t msws_remove(const uint32_t* d_keys, uint64_t n, const MswsDev& D, const MswsLaunch& L, bool below_2_31,
                        cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const int grid = rm_grid(n, L.num_sms * 6);
    if (below_2_31)
        k_msws_remove<true><<<grid, RM_THREADS, 0, st>>>(d_keys, n, D);
    else
        k_msws_remove<false><<<grid, RM_THREADS, 0, st>>>(d_keys, n, D);
    return cudaGetLastError();
}

cudaError_t cm_remove(const uint32_t* d_keys, uint64_t n, const CmDev& D, int grid, bool below_2_31, uint32_t* d_status,
                      cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const int g = rm_grid(n, grid);
    if (below_2_31)
        k_cm_remove<true><<<g, RM_THREADS, 0, st>>>(d_keys, n, D, d_status);
    else
        k_cm_remove<false><<<g, RM_THREADS, 0, st>>>(d_keys, n, D, d_status);
    return cudaGetLastError();
}

}  // namespace qsb
