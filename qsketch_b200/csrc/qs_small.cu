// qs_small.cu — the MSWS insert of few keys: one block per sketch, start to end.
//
// A call of a thousand keys through pass 1 and the grid-wide replay is all latency: two launches, a
// 296-block replay with four grid barriers (31 us when a bucket crosses).  Here one block
// applies up to SMALL_CHUNK keys at a time with the same returning atomics on the tables in L2, and
// if a bucket crossed, replays it on the spot: the block holds all of the chunk's keys in array
// order, so the record that takes a counter past the threshold is the switching key, and the
// order of the switching keys gives the high ids.  Longer key runs go chunk after chunk.  A batch
// runs one block per short stream.  Nothing waits across blocks.
//
// What bounds it: a chunk's three dependent trips to L2 (index words, counter atomics, link), then
// the replay where a bucket crossed.  1,000 keys, clear + insert + query 46 -> 25 us; 512 slices of
// 1,000 keys, pass 1 + replay 118 us -> 37 us.  256 threads a block measured the same as 512.  The
// limit of SMALL_STREAM keys: two chunks; beyond it pass 1 spreads the keys over more SMs.  Against pass 1
// and the replay, cleared / warm, at 4,096 keys: Zipf 1.4 120 -> 51 / 34 -> 21 us, Zipf 1.1 69 -> 35 /
// 34 -> 28, exponent 0.7 17 -> 21 / 34 -> 29, uniform 15 -> 21 / 15 -> 21 (3,000 keys: 15 -> 17).  One
// chunk of 1,024 threads instead of two: uniform 18, but Zipf 1.4 64.
#include "qs_kernels.h"
#include "qs_replay.cuh"

namespace qsb {

constexpr int SM_THREADS = 512, SM_WARPS = SM_THREADS / 32;
constexpr uint32_t SMALL_CHUNK = 2048;
constexpr int SM_KPT = SMALL_CHUNK / SM_THREADS;
constexpr int SM_PER = SMALL_CHUNK / 32 / 32;  // warp counts per lane of the scan

// c = 1 occurrence to the selected low counters of bucket words bw: all atomics in flight.
__device__ __forceinline__ bool small_low_add(uint32_t* bw, uint32_t m) {
    uint32_t old[7];
#pragma unroll
    for (int w = 0; w < 7; ++w) {
        const uint32_t nib = (m >> (4 * w)) & 0xfu;
        old[w] = nib ? atomicAdd(bw + w, expand_nibble(nib)) : 0u;
    }
    bool cross = false;
#pragma unroll
    for (int w = 0; w < 7; ++w) cross |= crosses(old[w], (m >> (4 * w)) & 0xfu, 1u);
    return cross;
}

template <bool BATCH>
__global__ void __launch_bounds__(SM_THREADS) k_msws_small(const uint32_t* __restrict__ keys, uint64_t n, MswsDev D,
                                                           BatchDev B) {
    // record: slot << 40 | key of the chunk << 28 | mask
    __shared__ unsigned long long s_rec[SMALL_CHUNK];
    __shared__ uint32_t s_fl[SMALL_CHUNK];             // flagged buckets by slot
    __shared__ uint16_t s_pos[SMALL_CHUNK];            // their switching keys (0xffff: none)
    __shared__ uint32_t s_wcnt[SMALL_CHUNK / 32], s_cnt[SM_WARPS][32];
    __shared__ uint32_t s_nflag, s_nrec, s_drop, s_rb, s_rk, s_base, s_found;
    const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    Ctl* ctl = D.ctl;
    uint32_t seed = D.seed, low_base = 0, high_base = 0;
    uint64_t n_high = D.n_high, k0 = 0, k1 = n;
    FastMod fm = D.fm_low;
    uint32_t* next_id = &ctl->next_id;
    if (BATCH) {
        const uint32_t s = blockIdx.x;
        k0 = __ldcg(B.lo + s), k1 = __ldcg(B.hi + s);
        if (k0 >= k1 || k1 - k0 > SMALL_STREAM) return;  // the plan leaves these to the other kernels
        const StreamDesc* sd = B.desc + s;
        fm = FastMod{__ldg(&sd->fm_low.M), __ldg(&sd->fm_low.d)};
        seed = __ldg(&sd->seed), low_base = __ldg(&sd->low_base), high_base = __ldg(&sd->high_base);
        n_high = __ldg(&sd->n_high);
        next_id = B.next_id + s;
    } else {
        griddep_launch_dependents();
        griddep_wait();
    }
    if (tid == 0) s_nflag = s_drop = s_rb = s_rk = 0;
    for (; k0 < k1; k0 += SMALL_CHUNK) {
        const uint32_t cnt = (uint32_t)umin64(SMALL_CHUNK, k1 - k0);
        uint32_t b[SM_KPT], m[SM_KPT], w7[SM_KPT];
#pragma unroll
        for (int u = 0; u < SM_KPT; ++u) {
            const uint32_t i = u * SM_THREADS + tid;
            const uint32_t hv = (i < cnt ? __ldg(keys + k0 + i) : 0u) * seed;
            b[u] = low_base + fast_mod(fm, hv);
            m[u] = i < cnt ? __ldg(D.masks + fast_mod(D.fm_mask, hv)) : 0u;  // 0: no key
        }
#pragma unroll
        for (int u = 0; u < SM_KPT; ++u) w7[u] = m[u] ? __ldcg(D.low + (uint64_t)b[u] * LOW_WORDS + 7) : SATURATED;
        if (tid == 0) {
            s_nrec = s_found = 0;
            s_base = __ldcg(next_id);
        }
        __syncthreads();
        // every index word is read before any is flagged
        uint32_t act = 0;  // bit u: key u was added to an unlinked bucket
#pragma unroll
        for (int u = 0; u < SM_KPT; ++u) {
            if (!m[u]) continue;
            if (w7[u] == SATURATED) {
                atomicAdd(&s_drop, 1u);
            } else if (is_linked(D, w7[u])) {
                uint32_t* hb = D.high + (uint64_t)(w7[u] - START) * HIGH_WORDS;
                for (uint32_t mm = m[u]; mm; mm &= mm - 1) atomicAdd(hb + (__ffs(mm) - 1), 1u);
            } else {
                act |= 1u << u;
                uint32_t* bw = D.low + (uint64_t)b[u] * LOW_WORDS;
                if (small_low_add(bw, m[u]) && !(atomicOr(bw + 7, FLAG) & FLAG)) {
                    const uint32_t slot = atomicAdd(&s_nflag, 1u);
                    s_fl[slot] = b[u];
                    atomicExch(bw + 7, FLAG | slot);
                }
            }
        }
        __syncthreads();
        const uint32_t F = s_nflag;
        if (F == 0) continue;
        // the flagged buckets' keys, in array order
        uint32_t slot[SM_KPT];
#pragma unroll
        for (int u = 0; u < SM_KPT; ++u) {
            const uint32_t w = (act >> u) & 1u ? __ldcg(D.low + (uint64_t)b[u] * LOW_WORDS + 7) : 0u;
            slot[u] = w & FLAG ? w & ~FLAG : NONE;
            const uint32_t bal = __ballot_sync(0xffffffffu, slot[u] != NONE);
            if (lane == 0) s_wcnt[u * SM_WARPS + wid] = __popc(bal);
        }
        __syncthreads();
        if (wid == 0) {
            uint32_t c[SM_PER], sum = 0;
#pragma unroll
            for (int i = 0; i < SM_PER; ++i) sum += c[i] = s_wcnt[SM_PER * lane + i];
            uint32_t v = sum;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, v, d);
                if (lane >= d) v += y;
            }
            if (lane == 31) s_nrec = v;
            v -= sum;
#pragma unroll
            for (int i = 0; i < SM_PER; ++i) {
                s_wcnt[SM_PER * lane + i] = v;
                v += c[i];
            }
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < SM_KPT; ++u) {
            const uint32_t bal = __ballot_sync(0xffffffffu, slot[u] != NONE);
            if (slot[u] != NONE)
                s_rec[s_wcnt[u * SM_WARPS + wid] + __popc(bal & lanemask_lt())] =
                    (unsigned long long)slot[u] << 40 | (unsigned long long)(u * SM_THREADS + tid) << 28 | m[u];
        }
        __syncthreads();
        const uint32_t K = s_nrec;
        uint32_t* rc = s_cnt[wid];
        constexpr uint32_t MASK = (1u << 28) - 1u;
        // adds the masks of slot s's records from key `from` on to rc; their number
        auto total = [&](uint32_t s, uint32_t from) {
            uint32_t keys_n = 0;
            __syncwarp();
            rc[lane] = 0u;
            __syncwarp();
            for (uint32_t q = 0; q < K; q += 32) {
                const unsigned long long r = q + lane < K ? s_rec[q + lane] : ~0ull;
                const bool mine = (uint32_t)(r >> 40) == s && ((uint32_t)(r >> 28) & 0xfffu) >= from;
                keys_n += __popc(__ballot_sync(0xffffffffu, mine));
                if (mine)
                    for (uint32_t mm = (uint32_t)r & MASK; mm; mm &= mm - 1) atomicAdd(rc + (__ffs(mm) - 1), 1u);
            }
            __syncwarp();
            return keys_n;
        };
        for (uint32_t s = wid; s < F; s += SM_WARPS) {
            uint32_t* bw = D.low + (uint64_t)s_fl[s] * LOW_WORDS;
            const uint32_t keys_n = total(s, 0u);
            const uint32_t T = lane < LOW_COUNTERS ? rc[lane] : 0u;
            // the counters before the chunk: final words minus the chunk's additions
            uint32_t sum = 0;
            const uint32_t fw = lane < 7 ? __ldcg(bw + lane) : 0u;
#pragma unroll
            for (int k = 0; k < 4; ++k) sum += __shfl_sync(0xffffffffu, T, (4 * (lane & 7) + k) & 31) << (8 * k);
            const uint32_t pw = __shfl_sync(0xffffffffu, fw - sum, (lane >> 2) & 7);
            uint32_t cur = lane < LOW_COUNTERS ? (pw >> (8 * (lane & 3))) & 0xffu : 0u, at = 0xffffu;
            __syncwarp();
            rc[lane] = cur;
            __syncwarp();
            for (uint32_t q = 0; q < K; q += 32) {
                const unsigned long long r = q + lane < K ? s_rec[q + lane] : ~0ull;
                const bool mine = (uint32_t)(r >> 40) == s;
                if (!__any_sync(0xffffffffu, mine)) continue;
                const uint32_t mk = mine ? (uint32_t)r & MASK : 0u;
                for (uint32_t mm = mk; mm; mm &= mm - 1) atomicAdd(rc + (__ffs(mm) - 1), 1u);
                __syncwarp();
                const uint32_t now = reinterpret_cast<volatile uint32_t*>(rc)[lane];
                const bool over = lane < LOW_COUNTERS && now != cur && now > LIMIT + 1;
                if (!__any_sync(0xffffffffu, over)) {
                    cur = now;
                    continue;
                }
                uint32_t occ = 0;
#pragma unroll
                for (uint32_t c = 0; c < LOW_COUNTERS; ++c) {
                    const uint32_t bal = __ballot_sync(0xffffffffu, (mk >> c) & 1u);
                    if (lane == c) occ = bal;
                }
                // the record that takes a counter to LIMIT + 2 saw LIMIT + 1: the switching key
                const uint32_t j = __reduce_min_sync(0xffffffffu, over ? __fns(occ, 0, LIMIT + 2 - cur) : 32u);
                cur += __popc(occ & ((1u << j) - 1u));
                at = __shfl_sync(0xffffffffu, (uint32_t)(r >> 28) & 0xfffu, j);
                break;
            }
            if (at != 0xffffu) {
                uint32_t word = 0;
#pragma unroll
                for (int k = 0; k < 4; ++k) word |= __shfl_sync(0xffffffffu, cur, (4 * (lane & 7) + k) & 31) << (8 * k);
                if (lane < 7) __stcg(bw + lane, word);
            } else if (lane == 7) {
                __stcg(bw + 7, 0u);  // every key added low
            }
            if (lane == 0) {
                s_pos[s] = (uint16_t)at;
                if (at != 0xffffu) atomicAdd(&s_found, 1u);
                atomicAdd(&s_rb, 1u);
                atomicAdd(&s_rk, keys_n);
            }
        }
        __syncthreads();
        // high ids in the order of the switching keys
        for (uint32_t s = wid; s < F; s += SM_WARPS) {
            const uint32_t at = s_pos[s];
            if (at == 0xffffu) continue;  // warp-uniform
            uint32_t rank = 0;
            for (uint32_t q = lane; q < F; q += 32) rank += s_pos[q] < at;
            rank = __reduce_add_sync(0xffffffffu, rank);
            const uint32_t own = s_base + rank;
            const bool ok = (uint64_t)(own - START) < n_high;
            const uint32_t n_after = total(s, at);
            ReplayOut o;
            o.T = lane < LOW_COUNTERS ? rc[lane] : 0u;  // the switching key's and all later ones'
            o.cur = o.P = 0;
            o.mL = 0;
            if (D.compat_v3) {
                for (uint32_t q = 0; q < K; q += 32) {
                    const unsigned long long r = q + lane < K ? s_rec[q + lane] : ~0ull;
                    const uint32_t hit = __ballot_sync(0xffffffffu, (uint32_t)(r >> 40) == s && ((uint32_t)(r >> 28) & 0xfffu) == at);
                    if (hit) o.mL = __shfl_sync(0xffffffffu, (uint32_t)r & MASK, __ffs(hit) - 1);
                }
            }
            link_bucket(D, s_fl[s], own + high_base, ok, high_increments(D, o), n_after);
            if (BATCH && lane == 0 && !ok) atomicOr(B.status + blockIdx.x, ST_POOL_FULL);
        }
        __syncthreads();
        if (tid == 0) {
            if (s_found) *next_id = (uint32_t)min((unsigned long long)s_base + s_found, (unsigned long long)START + n_high);
            s_nflag = 0;
        }
        __syncthreads();
    }
    __syncthreads();
    if (tid == 0) {
        if (s_drop) atomicAdd(&ctl->dropped, (unsigned long long)s_drop);
        if (s_rb) {
            atomicAdd(&ctl->repaired_buckets, (unsigned long long)s_rb);
            atomicAdd(&ctl->repaired_keys, (unsigned long long)s_rk);
        }
    }
}

// A cleared sketch in one launch (two memsets and a copy before, three more copies and memsets and a
// host wait for a batch): tables to zero with 16-byte stores, the control block and the batch's
// per-stream state to their initial values.  Bound by the stores; short-lived blocks of four stores a
// thread, handed out in order, keep them to few DRAM pages at a time: 512 MB 90 us in four persistent
// blocks an SM (80 by two memsets and a copy), so 78; 1.2 GB 199 (172), 165; 80 MB 15.1 (21.1), 14.6.
__global__ void __launch_bounds__(512) k_msws_clear(MswsDev D, Ctl init, BatchDev B) {
    const uint64_t gtid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, all = (uint64_t)gridDim.x * blockDim.x;
    const uint4 zero = make_uint4(0, 0, 0, 0);
    uint4* low = reinterpret_cast<uint4*>(D.low);
    uint4* high = reinterpret_cast<uint4*>(D.high);
    const uint64_t nl = D.n_low * (LOW_WORDS / 4), nh = D.n_high * (HIGH_WORDS / 4);
    for (uint64_t i = gtid; i < nl; i += all) low[i] = zero;
    for (uint64_t i = gtid; i < nh; i += all) high[i] = zero;
    if (gtid == 0) *D.ctl = init;
    for (uint64_t s = gtid; s < B.n_streams; s += all) {
        B.next_id[s] = FIRST_ID;
        B.status[s] = 0u;
        B.first[s] = 0ull;  // the control block's link generation, which tags these, restarts
    }
}

cudaError_t msws_clear(const MswsDev& D, const Ctl& init, const BatchDev& B, cudaStream_t st) {
    const uint64_t words = std::max<uint64_t>(D.n_low * (LOW_WORDS / 4), D.n_high * (HIGH_WORDS / 4));
    const int grid = (int)std::min<uint64_t>(1ull << 20, (words + 2047) / 2048);
    k_msws_clear<<<grid, 512, 0, st>>>(D, init, B);
    return cudaGetLastError();
}

cudaError_t small_insert(const uint32_t* d_keys, uint64_t n, const MswsDev& D, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    MswsDev Dc = D;
    BatchDev B{};
    void* args[] = {(void*)&d_keys, (void*)&n, (void*)&Dc, (void*)&B};
    return launch_pdl((const void*)k_msws_small<false>, dim3(1), dim3(SM_THREADS), 0, st, args, false);
}

cudaError_t small_insert_batch(const uint32_t* d_keys, const MswsDev& D, const BatchDev& B, cudaStream_t st) {
    k_msws_small<true><<<B.n_streams, SM_THREADS, 0, st>>>(d_keys, 0, D, B);
    return cudaGetLastError();
}

}  // namespace qsb
