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
// What bounds it now: the two round trips to L2 per pair of distinct keys of a tile.  3 M keys of
// a power law (exponent 1) 130 ms -> 0.23 ms; 2^20 uniform keys out of 64 MB 74 us -> 53, out of 0.5 MB
// 84 -> 88 (the compare-and-swaps of words that keys share); 1,000 keys 13 -> 10 us.
#include "qs_device.cuh"
#include "qs_kernels.h"

namespace qsb {

constexpr int RM_THREADS = 256;
constexpr int RM_KEYS = 2;  // distinct keys a thread updates at a time
constexpr uint32_t RM_TRIES = 1u << 22;  // CAS attempts per word before giving up (ST_TIMEOUT)

// Per-byte saturating subtraction of `dec` from *w, last seen as `old`; false if the CAS never won.
__device__ __forceinline__ bool sat_sub_bytes(uint32_t* w, uint32_t old, uint32_t dec) {
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

// c less in each of the counters base[sel(i)], i < n <= 4: all atomics in flight before a result is
// looked at.
template <bool SIGNED, class Sel>
__device__ __forceinline__ bool sub_u32(uint32_t* base, int n, uint32_t c, Sel sel) {
    bool ok = true;
    if (!SIGNED) {
        for (int i = 0; i < n; ++i) ok &= sat_sub_u32(base + sel(i), c);
        return ok;
    }
    int32_t old[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) old[i] = i < n ? (int32_t)atomicAdd(base + sel(i), 0u - c) : (int32_t)c;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (old[i] < (int32_t)c) atomicAdd(base + sel(i), c - (uint32_t)max(old[i], 0));
    return ok;
}
// The selected counters of mask m, four at a time.
template <bool SIGNED>
__device__ __forceinline__ bool sub_mask(uint32_t* base, uint32_t m, uint32_t c) {
    bool ok = true;
    while (m) {
        uint32_t bit[4];
        int n = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            bit[i] = m ? __ffs(m) - 1 : 0u;
            n += m != 0;
            m &= m - 1;
        }
        ok &= sub_u32<SIGNED>(base, n, c, [&](int i) { return bit[i]; });
    }
    return ok;
}

constexpr uint32_t RM_TILE = 2048, RM_BITS = 12, RM_SLOTS = 1u << RM_BITS, RM_PROBES = 16;
constexpr uint32_t RM_EMPTY = 0xffffffffu;

constexpr uint32_t RM_KPT = RM_TILE / RM_THREADS;

struct RmTable {
    uint32_t key[RM_SLOTS], cnt[RM_SLOTS];
    uint32_t top;  // occurrences of the key that equals RM_EMPTY
};

// Tile by tile: equal keys merge in the table, then fn(keys, counts) over the distinct keys, RM_KEYS
// of a thread at a time, so that it waits one round trip for their loads (a key that finds no
// slot within RM_PROBES is taken by itself).  The table has 2^bits slots, at least two per key of the
// tile: small tiles clear and walk no more than they fill (walking all 4096 slots for 1,000 uniform
// keys 18 us, so 10).  Who takes a distinct key:
//   OWN   the thread that brought it first, from its registers: 2^18 uniform keys 23 -> 21 us
//   else  the threads walk the slots, which spreads the distinct keys of skewed tiles evenly:
//         full tiles, 2^21 keys of a power law 0.6 172 us against 203, uniform 98 against 113; and
//         tables of a few buckets, 2^18 keys into 509 91 us against 98
template <bool OWN, class F>
__device__ __forceinline__ void merged_tiles(const uint32_t* __restrict__ keys, uint64_t n, uint32_t tile, uint32_t bits,
                                             RmTable& T, F fn) {
    const uint32_t tid = threadIdx.x, slots = 1u << bits;
    for (uint32_t i = tid; i < slots; i += RM_THREADS) T.key[i] = RM_EMPTY, T.cnt[i] = 0u;
    if (tid == 0) T.top = 0u;
    for (uint64_t t0 = (uint64_t)blockIdx.x * tile; t0 < n; t0 += (uint64_t)gridDim.x * tile) {
        const uint64_t t1 = umin64(n, t0 + tile);
        uint32_t k[RM_KPT], slot[RM_KPT];  // slot: NONE another thread's, LONE without one
        constexpr uint32_t NONE = 0xffffffffu, LONE = 0xfffffffeu;
#pragma unroll
        for (uint32_t j = 0; j < RM_KPT; ++j) {
            const uint64_t i = t0 + j * RM_THREADS + tid;
            k[j] = i < t1 ? __ldcs(keys + i) : 0u;
            slot[j] = NONE;
        }
        __syncthreads();
#pragma unroll
        for (uint32_t j = 0; j < RM_KPT; ++j) {
            if (t0 + j * RM_THREADS + tid >= t1) break;
            if (k[j] == RM_EMPTY) {
                atomicAdd(&T.top, 1u);
                continue;
            }
            const uint32_t h = k[j] * 0x9E3779B1u >> (32u - bits);
            slot[j] = LONE;
            for (uint32_t q = 0; q < RM_PROBES; ++q) {
                const uint32_t s = (h + q) & (slots - 1u);
                uint32_t seen = reinterpret_cast<volatile uint32_t*>(T.key)[s];
                if (seen == RM_EMPTY) seen = atomicCAS(T.key + s, RM_EMPTY, k[j]);
                if (seen == RM_EMPTY || seen == k[j]) {
                    atomicAdd(T.cnt + s, 1u);
                    slot[j] = OWN && seen == RM_EMPTY ? s : NONE;
                    break;
                }
            }
            if (!OWN && slot[j] == LONE) {
                const uint32_t one[RM_KEYS] = {k[j]}, c[RM_KEYS] = {1u};
                fn(one, c);
            }
        }
        __syncthreads();
        if (OWN) {
#pragma unroll
            for (uint32_t j0 = 0; j0 < RM_KPT; j0 += RM_KEYS) {
                if (t0 + j0 * RM_THREADS >= t1) break;  // uniform over the block
                uint32_t key[RM_KEYS], c[RM_KEYS];
#pragma unroll
                for (int u = 0; u < RM_KEYS; ++u) {
                    const uint32_t s = slot[j0 + u];
                    key[u] = k[j0 + u];
                    c[u] = s == NONE ? 0u : 1u;
                    if (s < slots) {
                        c[u] = T.cnt[s];
                        T.key[s] = RM_EMPTY;
                        T.cnt[s] = 0u;
                    }
                }
                fn(key, c);
            }
        } else {
            for (uint32_t i0 = tid; i0 < slots; i0 += RM_KEYS * RM_THREADS) {
                uint32_t key[RM_KEYS], c[RM_KEYS];
#pragma unroll
                for (int u = 0; u < RM_KEYS; ++u) {
                    const uint32_t i = i0 + u * RM_THREADS;
                    key[u] = T.key[i];
                    c[u] = key[u] == RM_EMPTY ? 0u : T.cnt[i];
                    T.key[i] = RM_EMPTY;
                    T.cnt[i] = 0u;
                }
                fn(key, c);
            }
        }
        if (tid == 0 && T.top) {
            const uint32_t one[RM_KEYS] = {RM_EMPTY}, c[RM_KEYS] = {T.top};
            fn(one, c);
            T.top = 0u;
        }
    }
}
static_assert(RM_SLOTS == 1u << RM_BITS && RM_SLOTS == 2 * RM_TILE, "two slots per key of a full tile");
constexpr uint32_t RM_MIN_BITS = 9;
static_assert((1u << RM_MIN_BITS) % (RM_KEYS * RM_THREADS) == 0 && RM_TILE % RM_THREADS == 0 && RM_KPT % RM_KEYS == 0, "whole rounds");

// SERIAL: the words of an unlinked bucket one after the other, each loaded just before its
// compare-and-swap, for tables whose words many keys in flight share (all words at once, with the
// values the bucket was read with, mostly retry: 2^21 uniform keys, 16,381 buckets 234 us against
// 174, 65,521 150 against 139; 131,071 125 against 134).
template <bool SIGNED, bool OWN, bool SERIAL>
__global__ void __launch_bounds__(RM_THREADS, 4) k_msws_remove(const uint32_t* __restrict__ keys, uint64_t n, uint32_t tile,
                                                               uint32_t bits, MswsDev D) {
    __shared__ RmTable T;
    bool ok = true;
    uint32_t dropped = 0;
    merged_tiles<OWN>(keys, n, tile, bits, T, [&](const uint32_t (&key)[RM_KEYS], const uint32_t (&c)[RM_KEYS]) {
        uint32_t m[RM_KEYS];
        uint32_t* wp[RM_KEYS];
        uint4 lo[RM_KEYS], hi[RM_KEYS];
#pragma unroll
        for (int u = 0; u < RM_KEYS; ++u) {  // c = 0: no key
            const uint32_t hv = key[u] * D.seed;
            wp[u] = D.low + (uint64_t)fast_mod(D.fm_low, hv) * LOW_WORDS;
            m[u] = c[u] ? __ldg(D.masks + fast_mod(D.fm_mask, hv)) : 0u;
            lo[u] = c[u] ? __ldcg(reinterpret_cast<const uint4*>(wp[u])) : make_uint4(0, 0, 0, 0);
            hi[u] = c[u] ? __ldcg(reinterpret_cast<const uint4*>(wp[u]) + 1) : make_uint4(0, 0, 0, 0);
        }
        if (SERIAL) {
            uint32_t left[RM_KEYS];  // the next selected word of each key at a time
#pragma unroll
            for (int u = 0; u < RM_KEYS; ++u) {
                const uint32_t ptr = hi[u].w;
                left[u] = ptr == SATURATED || (ptr > START && (uint64_t)(ptr - START) < D.n_high) ? 0u : m[u];
            }
            for (;;) {
                uint32_t any = 0;
#pragma unroll
                for (int u = 0; u < RM_KEYS; ++u) any |= left[u];
                if (!any) break;
                uint32_t old[RM_KEYS], dec[RM_KEYS];
                uint32_t* p[RM_KEYS];
#pragma unroll
                for (int u = 0; u < RM_KEYS; ++u) {
                    dec[u] = 0;
                    if (!left[u]) continue;
                    const uint32_t i = (uint32_t)(__ffs(left[u]) - 1) >> 2, nib = (left[u] >> (4 * i)) & 0xfu;
                    left[u] &= ~(0xfu << (4 * i));
                    p[u] = wp[u] + i;
                    dec[u] = expand_nibble(nib) * min(c[u], 255u);
                    old[u] = __ldcg(p[u]);
                }
#pragma unroll
                for (int u = 0; u < RM_KEYS; ++u)
                    if (dec[u]) ok &= sat_sub_bytes(p[u], old[u], dec[u]);
            }
#pragma unroll
            for (int u = 0; u < RM_KEYS; ++u) {
                if (!c[u]) continue;
                const uint32_t ptr = hi[u].w;
                if (ptr == SATURATED)
                    dropped += c[u];
                else if (ptr > START && (uint64_t)(ptr - START) < D.n_high)
                    ok &= sub_mask<SIGNED>(D.high + (uint64_t)(ptr - START) * HIGH_WORDS, m[u], c[u]);
            }
            return;
        }
        uint32_t prev[RM_KEYS][7];  // low level: the words' compare-and-swaps, all in flight
#pragma unroll
        for (int u = 0; u < RM_KEYS; ++u) {
            if (!c[u]) continue;
            const uint32_t ptr = hi[u].w;
            if (ptr == SATURATED || (ptr > START && (uint64_t)(ptr - START) < D.n_high)) continue;
            const uint32_t w[7] = {lo[u].x, lo[u].y, lo[u].z, lo[u].w, hi[u].x, hi[u].y, hi[u].z};
            const uint32_t cb = min(c[u], 255u);  // bytes hold at most 129: more removals empty them
#pragma unroll
            for (int i = 0; i < 7; ++i) {
                const uint32_t dec = expand_nibble((m[u] >> (4 * i)) & 0xfu) * cb, nw = __vsubus4(w[i], dec);
                prev[u][i] = nw != w[i] ? atomicCAS(wp[u] + i, w[i], nw) : w[i];
            }
        }
#pragma unroll
        for (int u = 0; u < RM_KEYS; ++u) {
            if (!c[u]) continue;
            const uint32_t ptr = hi[u].w;
            if (ptr == SATURATED) {
                dropped += c[u];
            } else if (ptr > START && (uint64_t)(ptr - START) < D.n_high) {
                ok &= sub_mask<SIGNED>(D.high + (uint64_t)(ptr - START) * HIGH_WORDS, m[u], c[u]);
            } else {
                const uint32_t w[7] = {lo[u].x, lo[u].y, lo[u].z, lo[u].w, hi[u].x, hi[u].y, hi[u].z};
                const uint32_t cb = min(c[u], 255u);
#pragma unroll
                for (int i = 0; i < 7; ++i)
                    if (prev[u][i] != w[i])
                        ok &= sat_sub_bytes(wp[u] + i, prev[u][i], expand_nibble((m[u] >> (4 * i)) & 0xfu) * cb);
            }
        }
    });
    if (!ok) atomicOr(&D.ctl->status, ST_TIMEOUT);
    if (dropped) atomicAdd(&D.ctl->dropped, (unsigned long long)dropped);
}

template <bool SIGNED>
__global__ void __launch_bounds__(RM_THREADS, 4) k_cm_remove(const uint32_t* __restrict__ keys, uint64_t n, uint32_t tile,
                                                          uint32_t bits, CmDev D, uint32_t* __restrict__ status) {
    __shared__ RmTable T;
    bool ok = true;
    merged_tiles<true>(keys, n, tile, bits, T, [&](const uint32_t (&key)[RM_KEYS], const uint32_t (&c)[RM_KEYS]) {
#pragma unroll
        for (int u = 0; u < RM_KEYS; ++u) {
            if (!c[u]) continue;
            if (D.masks) {  // one-level bucket sketch: the selected counters of the key's bucket
                const uint32_t hv = key[u] * D.seeds[0];
                ok &= sub_mask<SIGNED>(D.table + (uint64_t)fast_mod(D.fm, hv) * D.rows,
                                       __ldg(D.masks + fast_mod(D.fm_mask, hv)), c[u]);
                continue;
            }
            for (uint32_t j0 = 0; j0 < D.rows; j0 += 4) {
                const uint32_t nj = min(4u, D.rows - j0);
                uint64_t at[4];
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j)
                    at[j] = j < nj ? (uint64_t)(j0 + j) * D.n + fast_mod(D.fm, key[u] * D.seeds[j0 + j]) : 0u;
                ok &= sub_u32<SIGNED>(D.table, (int)nj, c[u], [&](int i) { return at[i]; });
            }
        }
    });
    if (!ok && status) atomicOr(status, ST_TIMEOUT);
}

// Persistent blocks of a tile each (64 registers leave four to an SM); small calls take smaller
// tiles, so that they spread over the chip: a thread waits two round trips per two keys.
static uint32_t rm_tile(uint64_t n, int blocks) {
    const uint64_t even = (n + blocks - 1) / blocks;
    return (uint32_t)std::min<uint64_t>(RM_TILE, std::max<uint64_t>(RM_THREADS, even));
}

static uint32_t rm_bits(uint32_t tile) {
    uint32_t bits = RM_MIN_BITS;
    while ((1u << bits) < 2 * tile) ++bits;
    return bits;
}

cudaError_t msws_remove(const uint32_t* d_keys, uint64_t n, const MswsDev& D, const MswsLaunch& L, bool below_2_31,
                        cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    uint32_t tile = rm_tile(n, L.num_sms * 4), bits = rm_bits(tile);
    const int grid = (int)std::min<uint64_t>((uint64_t)L.num_sms * 4, (n + tile - 1) / tile);
    // below 4,096 buckets nearly all are linked by the time words are shared; walked slots beside
    // SERIAL took 358 us where the 2^21 keys into 16,381 buckets take 174
    const bool few = D.n_low < (1u << 12), serial = !few && D.n_low < 3u << 15;
    const bool own = serial || (!few && tile <= RM_TILE / 2);
    const void* fn = below_2_31 ? (serial ? (const void*)k_msws_remove<true, true, true>
                                   : own  ? (const void*)k_msws_remove<true, true, false>
                                          : (const void*)k_msws_remove<true, false, false>)
                                : (serial ? (const void*)k_msws_remove<false, true, true>
                                   : own  ? (const void*)k_msws_remove<false, true, false>
                                          : (const void*)k_msws_remove<false, false, false>);
    MswsDev Dc = D;
    void* args[] = {(void*)&d_keys, (void*)&n, (void*)&tile, (void*)&bits, (void*)&Dc};
    return cudaLaunchKernel(fn, dim3(grid), dim3(RM_THREADS), args, 0, st);
}

cudaError_t cm_remove(const uint32_t* d_keys, uint64_t n, const CmDev& D, int grid, bool below_2_31, uint32_t* d_status,
                      cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const uint32_t tile = rm_tile(n, grid / 2);  // grid: eight blocks an SM
    const int g = (int)std::min<uint64_t>((uint64_t)grid / 2, (n + tile - 1) / tile);
    if (below_2_31)
        k_cm_remove<true><<<g, RM_THREADS, 0, st>>>(d_keys, n, tile, rm_bits(tile), D, d_status);
    else
        k_cm_remove<false><<<g, RM_THREADS, 0, st>>>(d_keys, n, tile, rm_bits(tile), D, d_status);
    return cudaGetLastError();
}

}  // namespace qsb
