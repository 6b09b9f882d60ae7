#!/usr/bin/env python
"""QSketch insert/query throughput on B200 — one JSON line on rank 0.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                    [--config zipf|uniform|mixed|cm|ablation|learned|batched|zipf_prof|batched_prof]

A step is one pass of the hot path over one batch of synthetic input: clear the sketch,
insert the whole key stream, query the distinct keys.  The default workload is the
Zipf-skewed stream (2^27 keys, Zipf s=1.1 over 2^24 ranks, 64 MB low table, 16 MB high
pool, query the 2^24 distinct keys); `--config uniform` is the 2^24-key uniform case,
`--config mixed` the HBM-bound interleaved insert/query stream, `--config learned` the
learned heavy-hitter split against the plain sketch at equal bytes (relative error of both,
throughput with and without the warm-up/training phase), `--config batched` 512 uneven
streams with one sketch each, inserted and queried as one batch, and `--config cm` the plain
count-min (the in-GPU baseline) on the uniform stream at the uniform configuration's bytes,
with the MSWS sketch of those bytes timed beside it.
For N > 1 (one process per GPU; without torchrun's environment, `--gpus N` starts the N
ranks itself) every rank runs its own sketch over its own seeded stream: the path has no
data exchange, so this is weak scaling with no collective on the data path.
`--impl reference` times the CPU restatement of the reference path (oracle/, one pass that
partitions the keys by bucket over all host threads, then each thread applies its part in
array order) on the host cores, rank 0 only, over the same key stream as the GPU arm.
"""
import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "insert/query Gkeys/s on 1 B200; avg rel. error learned vs plain at equal bytes"
SEED = 2654435769  # odd multiplier in the reference's seed range [1, 2^32-1]

CONFIGS = {
    "zipf": dict(workload="zipf1.1_2^27keys_2^24ranks_low64MB_high16MB_query2^24", kind=1, n_keys=1 << 27,
                 n_ranks=1 << 24, s=1.1, n_low=2097143, n_high=1 << 17, n_query=1 << 24),
    "uniform": dict(workload="uniform_2^24keys_nlow262139_high8MB_query2^24", kind=0, n_keys=1 << 24, n_ranks=0,
                    s=0.0, n_low=262139, n_high=1 << 16, n_query=1 << 24),
    # HBM-bound mixed workload: 2^28 operations in 2^20-key batches, each batch 90 % inserts
    # then 10 % queries; Zipf 0.8 over 2^26 ranks; 256 MB low table (> L2), 64 MB high pool
    "mixed": dict(workload="mixed_2^28ops_batch2^20_90ins10qry_zipf0.8_2^26ranks_low256MB_high64MB", kind=2,
                  n_keys=1 << 28, n_ranks=1 << 26, s=0.8, n_low=8388593, n_high=1 << 19, n_query=0,
                  batch=1 << 20, insert_frac=0.9),
    # learned heavy-hitter split vs the plain sketch at equal bytes: 2^28 keys (class<<16)|suffix,
    # class Zipf 1.0 over 2^16, suffix Zipf 1.2 over 2^16 permuted per class; 64 MB each form
    "learned": dict(workload="class_keys_2^28_classZipf1.0_suffixZipf1.2_64MB_learned_vs_plain", kind=3,
                    n_keys=1 << 28, n_ranks=0, s=0.0, budget=64 << 20, warmup=1 << 24, table_slots=1 << 17,
                    n_low=0, n_high=0, n_query=0),
    # batched uneven streams: 512 per-stream sketches, lengths log-uniform in [2^10, 2^22],
    # Zipf s ~ U[0.6, 1.4] over 2^20 ranks, sketch sizes log-uniform in [32 KB, 16 MB],
    # n_low = prime <= bytes/32, high pool bytes/4; inserted and queried in one batch each
    "batched": dict(workload="512_streams_len_2^10..2^22_zipf0.6..1.4_2^20ranks_sketch32KB..16MB_pool_bytes/4",
                    kind=4, n_streams=512, n_keys=0, n_ranks=1 << 20, s=0.0, n_low=0, n_high=0, n_query=0),
    # a smaller batch for Nsight Compute captures: 64 streams of 2^10..2^21 keys (key stream
    # and tables still larger than L2)
    "batched_prof": dict(workload="64_streams_len_2^10..2^21_zipf0.6..1.4_2^20ranks_sketch32KB..16MB_pool_bytes/4",
                         kind=4, n_streams=64, max_len=1 << 21, n_keys=0, n_ranks=1 << 20, s=0.0, n_low=0, n_high=0,
                         n_query=0),
    # plain count-min (device_sketch_v0.h), m = 3 rows, n = find_greatest_prime(8 MB / 4 / 3):
    # the uniform configuration's 2^24 keys at (no more than) its 8 MB, queried for every key
    "cm": dict(workload="countmin_m3_n524287_uniform_2^24keys_query2^24", kind=5, n_keys=1 << 24, n_ranks=0,
               s=0.0, n_low=524287, rows=3, n_high=0, n_query=1 << 24),
    # ablation: the two-level MSWS against the one-level sketches the reference also ships — the
    # count-min (m = 3 rows), the warp sketch (32 counters per bucket) and the sub-warp sketches
    # (8 and 16) — at no more than the uniform configuration's 8 MB of low table, on 2^24 uniform
    # keys and 2^24 Zipf(1.1) keys over 2^22 ranks
    "ablation": dict(workload="msws_vs_countmin_warp_subwarp_8MB_uniform_and_zipf1.1_2^24keys", kind=6,
                     n_keys=1 << 24, n_ranks=1 << 22, s=1.1, n_low=262139, n_high=1 << 16, n_query=0),
    # a smaller skewed case for Nsight Compute captures (key stream still larger than L2)
    "zipf_prof": dict(workload="zipf1.1_2^25keys_2^22ranks_low16MB_high4MB_query2^22", kind=1, n_keys=1 << 25,
                      n_ranks=1 << 22, s=1.1, n_low=524287, n_high=1 << 15, n_query=1 << 22),
}
INSERT_BYTES_PER_KEY = 68  # pass 1: 4 B key + 32 B bucket sector read + 32 B write-back
PART_BYTES_PER_KEY = 16    # partitioned: 4 B key + its 6 B entry written and read (the table streams once a chunk)
L2_BYTES = 126 << 20      # B200 L2: tables above this live in HBM
QUERY_BYTES_PER_KEY = 40   # 4 B key + 32 B bucket sector + 4 B result


def peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        with open(p) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


def traffic_per_unit(config, kernel):
    """DRAM bytes per key of `kernel` from one ncu capture (profiles/traffic.json), or None."""
    tfile = os.path.join(ROOT, "profiles", "traffic.json")
    if not os.path.exists(tfile):
        return None
    with open(tfile) as f:
        k = json.load(f).get(f"{config}:{kernel}")
    return k["dram_bytes_per_unit"] if k else None


# Three distinct counters of 28, four to a 32-bit word: the expected number of distinct words
# a key's increments touch is 3 P(all apart) + 2 P(one pair shares) + 1 P(all share).
MSWS_WORD_OPS_PER_KEY = 3 * (24 / 27) * (20 / 26) + 2 * (1 - (24 / 27) * (20 / 26) - (3 / 27) * (2 / 26)) + \
    (3 / 27) * (2 / 26)


def l2_atomic_roofline(probes, units_per_s, word_ops_per_unit, kernel, what):
    """Roofline against the L2's atomic units.  Their ceiling is a rate of 32-bit word
    operations: the random-sector probes reach about the same word rate whether each sector
    takes 3 words from 3 lanes (kind 0) or 1 word from every lane (kind 7), while their sector
    rates differ threefold.  achieved = units/s x word operations per unit; the sector view
    (one sector per unit against the best sector rate) is given beside it."""
    if not probes:
        return {"bound": "l2_atomic", "kernel": kernel, "achieved": None, "peak": None, "frac": None}
    word_rates = {"red_3word_subwarp": 3 * probes["red_3word_subwarp"],
                  "red_1word_per_lane": probes["red_1word_per_lane"]}
    peak = max(word_rates.values())
    sect = max(probes.values())
    ach = units_per_s * word_ops_per_unit
    return {"bound": "l2_atomic", "kernel": kernel, "achieved": round(ach / 1e9, 3), "peak": round(peak / 1e9, 3),
            "unit": "G atomic word-ops/s", "frac": round(ach / peak, 4),
            "peak_source": "live probes on a table of this size (qs_probe kind 0: 3 words per random sector from "
                           "a sub-warp of 8; kind 7: one word per lane, every lane its own random sector), "
                           "G word-ops/s: " + ", ".join(f"{k} {v / 1e9:.2f}" for k, v in word_rates.items()),
            "word_ops_per_unit": round(word_ops_per_unit, 4), "units_per_s": round(units_per_s / 1e9, 4),
            "units": what,
            "sector_view": {"achieved_gsectors": round(units_per_s / 1e9, 3), "peak_gsectors": round(sect / 1e9, 3),
                            "frac": round(units_per_s / sect, 4),
                            "note": "one 32 B bucket sector per unit against the best probe sector rate"}}


def atomic_probes(table_bytes):
    """Random-sector red rates (sectors/s) on a table of `table_bytes`: 3 words per sector from
    a sub-warp of 8 lanes (kind 0), and one word per lane, every lane its own sector (kind 7)."""
    from qsketch_b200 import data
    return {"red_3word_subwarp": data.probe(0, table_bytes, 1 << 26),
            "red_1word_per_lane": data.probe(7, table_bytes, 1 << 26)}


class Clocks:
    """Samples SM clock and throttle reasons during the timed region: NVML every 5 ms in a
    thread (nvidia-smi's 100 ms loop can miss a short region), else nvidia-smi."""

    REASONS = {"hw_slowdown": 0x8, "sw_thermal_slowdown": 0x20, "hw_thermal_slowdown": 0x40, "sw_power_cap": 0x4}

    def __init__(self, index):
        self.index = index
        self.samples = []
        self.reasons = set()
        self.max_mhz = None
        self.stop = threading.Event()
        self.nvml = None

    def __enter__(self):
        try:
            import pynvml
            pynvml.nvmlInit()
            self.nvml = pynvml
            self.h = pynvml.nvmlDeviceGetHandleByIndex(self.index)
            self.max_mhz = pynvml.nvmlDeviceGetMaxClockInfo(self.h, pynvml.NVML_CLOCK_SM)
        except Exception:
            self.nvml = None
        self.t = threading.Thread(target=self._run, daemon=True)
        self.t.start()
        return self

    def _sample_nvml(self):
        n = self.nvml
        self.samples.append(n.nvmlDeviceGetClockInfo(self.h, n.NVML_CLOCK_SM))
        r = n.nvmlDeviceGetCurrentClocksEventReasons(self.h)
        for name, bit in self.REASONS.items():
            if r & bit:
                self.reasons.add(name)

    def _run(self):
        if self.nvml:
            while True:
                try:
                    self._sample_nvml()
                except Exception:
                    break
                if self.stop.wait(0.005):
                    break
            return
        fields = ("clocks.sm,clocks.max.sm,clocks_event_reasons.hw_slowdown,"
                  "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
                  "clocks_event_reasons.sw_power_cap")
        while not self.stop.is_set():
            try:
                out = subprocess.run(["nvidia-smi", "-i", str(self.index), f"--query-gpu={fields}",
                                      "--format=csv,noheader,nounits"], capture_output=True, text=True,
                                     timeout=5).stdout.strip().split(",")
                self.samples.append(float(out[0]))
                self.max_mhz = float(out[1])
                for name, v in zip(["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"],
                                   out[2:6]):
                    if v.strip().lower() == "active":
                        self.reasons.add(name)
            except Exception:
                break

    def __exit__(self, *exc):
        self.stop.set()
        self.t.join(timeout=10)
        if self.nvml and not self.samples:
            try:
                self._sample_nvml()
            except Exception:
                pass

    def summary(self):
        if not self.samples:
            return {"sm_mhz": None, "sm_max_mhz": self.max_mhz, "reasons": sorted(self.reasons), "samples": 0}
        return {"sm_mhz": statistics.median(self.samples), "sm_max_mhz": self.max_mhz,
                "reasons": sorted(self.reasons), "samples": len(self.samples)}


# ---------------------------------------------------------------------------------------
def dist_setup(gpus):
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world != gpus and world > 1:
        raise SystemExit(f"--gpus {gpus} but WORLD_SIZE={world}")
    return world, rank, local


def init_ranks(args):
    """One process per GPU; returns (world, rank, local, barrier, max_over_ranks)."""
    from qsketch_b200.replicas import Ranks

    dist_setup(args.gpus)
    r = Ranks(backend="nccl")
    return r.world, r.rank, r.local, r.barrier, r.max


def run_ours(args, cfg):
    import torch
    import torch.distributed as dist

    import qsketch_b200 as qs
    from qsketch_b200 import data

    if cfg["kind"] == 3:
        return run_learned(args, cfg)
    if cfg["kind"] == 4:
        return run_batched(args, cfg)
    if cfg["kind"] == 5:
        return run_cm(args, cfg)
    if cfg["kind"] == 6:
        return run_ablation(args, cfg)
    if args.shard:
        return run_sharded(args, cfg)
    world, rank, local, barrier, max_over_ranks = init_ranks(args)

    stream = torch.cuda.current_stream()
    seed = 1000 + rank
    perm_seed = 99 + 7919 * rank
    if cfg["kind"] == 1:
        keys, ranks = data.zipf_keys(cfg["n_keys"], cfg["n_ranks"], cfg["s"], seed=seed, perm_seed=perm_seed,
                                     with_ranks=True)
        queries = data.rank_keys(perm_seed, 0, cfg["n_query"])
        exact = data.rank_histogram(ranks, cfg["n_ranks"])[:cfg["n_query"]].contiguous()
        del ranks
    elif cfg["kind"] == 2:
        keys = data.zipf_keys(cfg["n_keys"], cfg["n_ranks"], cfg["s"], seed=seed, perm_seed=perm_seed)
        exact = None
    else:
        keys = data.uniform_keys(cfg["n_keys"], seed=seed)
        queries = keys[:cfg["n_query"]]
        exact = None
    if cfg["kind"] == 2:  # per batch: the first 90 % insert, the rest query
        B = cfg["batch"]
        ni_b = int(B * cfg["insert_frac"])
        nbat = cfg["n_keys"] // B
        ins_views = [keys[b * B:b * B + ni_b] for b in range(nbat)]
        q_views = [keys[b * B + ni_b:(b + 1) * B] for b in range(nbat)]
        queries = torch.cat(q_views)
        cfg = dict(cfg, n_query=queries.numel())
    out = torch.empty(cfg["n_query"], dtype=torch.uint32, device="cuda")
    # the library's autotuner picks the pass-1 knobs (outside the timed region; no knob changes
    # any result) on another stream of the same configuration — another seed — so the setting
    # is not fitted to the timed data; the sketch below takes them from its table
    from qsketch_b200 import autotune
    autotune.reset()
    if not args.autotune:
        tune_keys = None
    elif cfg["kind"] == 1:
        tune_keys = data.zipf_keys(cfg["n_keys"], cfg["n_ranks"], cfg["s"], seed=seed + 7777,
                                   perm_seed=perm_seed + 7777)
    elif cfg["kind"] == 2:
        tune_keys = data.zipf_keys(16 * cfg["batch"], cfg["n_ranks"], cfg["s"], seed=seed + 7777,
                                   perm_seed=perm_seed + 7777)
    else:
        tune_keys = data.uniform_keys(cfg["n_keys"], seed=seed + 7777)
    # (the mixed workload inserts one batch per call: tune on 16 batches' inserts in chunks of
    # one batch, so the tuner sees the real chunk size and a sketch that fills)
    if tune_keys is None:
        tuned = {k: 0 for k in ("lanes_per_key", "aggregate", "route", "ctas_per_sm", "max_batch", "first_chunk",
                                "keys_per_tile")}
    elif cfg["kind"] == 2:
        sample = torch.cat([tune_keys[b * cfg["batch"]:b * cfg["batch"] + ni_b] for b in range(16)])
        tuned, _ = autotune.autotune(cfg["n_low"], cfg["n_high"], sample, reps=3, hash_seed=SEED, mask_rng=1,
                                     max_batch=(ni_b + 31) // 32 * 32)
        del sample
    else:
        # (whole-stream samples take a few ms each: 8 repetitions per setting keep the
        # search's picks from following run-to-run noise of a few percent)
        tuned, _ = autotune.autotune(cfg["n_low"], cfg["n_high"], tune_keys, reps=8, hash_seed=SEED, mask_rng=1)
    del tune_keys
    sk = qs.Sketch_GPU_Sub_Warp_Level(cfg["n_low"], 8, cfg["n_high"], 32, hash_seed=SEED, mask_rng=1)
    n_ins, n_q = cfg["n_keys"], cfg["n_query"]
    if cfg["kind"] == 2:
        n_ins = n_ins - n_q
        out_views = list(torch.split(out, [v.numel() for v in q_views]))

    def step_mixed(ev=None):
        sk.clear()
        if ev:
            ev[0].record(stream)
        for iv, qv, ov in zip(ins_views, q_views, out_views):
            sk.insert(iv)
            sk.search(qv, counts=ov)
        if ev:
            ev[1].record(stream)
            ev[2].record(stream)

    def step(ev=None):
        if cfg["kind"] == 2:
            return step_mixed(ev)
        sk.clear()
        if ev:
            ev[0].record(stream)
        sk.insert(keys)
        if ev:
            ev[1].record(stream)
        sk.search(queries, counts=out)
        if ev:
            ev[2].record(stream)

    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()
    sk.sync()
    prof0 = sk.profile()
    launches0 = prof0["insert_launches"] + prof0["repair_launches"] + prof0["query_launches"]

    evs = [[torch.cuda.Event(enable_timing=True) for _ in range(3)] for _ in range(args.steps)]
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with Clocks(local) as clk:
        barrier()
        torch.cuda.synchronize()
        torch.cuda.nvtx.range_push("timed")  # lets a profiler capture the timed steps only
        t0.record(stream)
        for i in range(args.steps):
            step(evs[i])
        t1.record(stream)
        torch.cuda.synchronize()
        torch.cuda.nvtx.range_pop()
        barrier()
    total_ms = max_over_ranks(t0.elapsed_time(t1))
    ins_ms = max_over_ranks(sum(e[0].elapsed_time(e[1]) for e in evs) / args.steps)
    q_ms = max_over_ranks(sum(e[1].elapsed_time(e[2]) for e in evs) / args.steps)
    sk.sync()
    prof1 = sk.profile()
    launches = prof1["insert_launches"] + prof1["repair_launches"] + prof1["query_launches"] - launches0
    ms_per_step = total_ms / args.steps
    value = world * (n_ins + n_q) / (ms_per_step * 1e6)

    # accuracy of the plain sketch against exact counts
    rel = ratio = None
    if exact is not None:
        rel, ratio = data.error_metrics(out, exact)

    # one instrumented step: per-launch CUDA events inside the library, for the roofline
    sk.set_profiling(True)
    step()
    torch.cuda.synchronize()
    prof = sk.profile()
    sk.set_profiling(False)
    hbm, peak_kind = peaks()
    # large calls with default knobs are partitioned: no replay launches
    parted = prof["repair_launches"] == 0
    insert_bytes = PART_BYTES_PER_KEY if parted else INSERT_BYTES_PER_KEY
    kern = {"insert": (prof["insert_ms"], prof["insert_timed"], n_ins, insert_bytes),
            "query": (prof["query_ms"], prof["query_timed"], n_q, QUERY_BYTES_PER_KEY)}
    dom = max(kern, key=lambda k: kern[k][0])
    ms_k, launches_k, units, bpu = kern[dom]
    per_launch_units = units / max(1, launches_k)
    avg_ms = ms_k / max(1, launches_k)
    achieved = per_launch_units * bpu / (avg_ms * 1e-3) / 1e9
    dram_per_key = traffic_per_unit(args.config, dom)
    table_bytes = cfg["n_low"] * 32 + cfg["n_high"] * 128
    # the L2 atomic ceiling: the best of the random-sector red probes on a table of this size
    probes = atomic_probes(max(64 << 20, cfg["n_low"] * 32)) if rank == 0 else {}
    if cfg["kind"] == 2:  # inserts and queries interleave: split their rates by kernel time
        ins_ms = prof["insert_ms"] + prof["repair_ms"]
        q_ms = prof["query_ms"]
    insert_step_ms = prof["insert_ms"] + prof["repair_ms"]  # pass 1 + ordered replay of the step
    keys_per_s = n_ins / (insert_step_ms * 1e-3)
    ins_kernel = "k_part_split + k_part_apply + k_part_link" if parted else "k_msws_insert"
    hbm_line = {"bound": "hbm", "kernel": ins_kernel if dom == "insert" else "k_msws_query",
                "achieved": round(achieved, 1), "peak": hbm, "unit": "GB/s", "frac": round(achieved / hbm, 4),
                "traffic": dram_per_key * per_launch_units if dram_per_key else None, "peak_source": peak_kind,
                "bytes_per_unit": bpu, "units_per_launch": per_launch_units, "avg_launch_ms": round(avg_ms, 5)}
    if parted:  # counters live in shared memory: no L2 atomics, and far from DRAM
        roofline = dict(hbm_line, note="against DRAM; the kernels are bound by instruction issue and the shared-memory "
                                       "pipe, each about half busy between block barriers (profiles/k_part_insert_2^24.md)")
    elif table_bytes > L2_BYTES:  # the tables live in HBM: bucket sectors cost DRAM traffic
        roofline = hbm_line
    else:  # L2-resident tables: the L2's atomic units bound the insert
        roofline = l2_atomic_roofline(probes, keys_per_s, MSWS_WORD_OPS_PER_KEY,
                                      "k_msws_insert + k_msws_repair (pass 1 + ordered replay)",
                                      "each key adds 1 to 3 of its bucket's 28 packed 8-bit counters: "
                                      f"{MSWS_WORD_OPS_PER_KEY:.4f} 32-bit words on average (the expected number "
                                      "of distinct words holding 3 distinct counters of 28, 4 per word)")
        roofline.update({"traffic": round(dram_per_key * n_ins) if dram_per_key else None,
                         "traffic_unit": "DRAM bytes per step of the insert kernels (ncu dram__bytes per key x keys)",
                         "algorithmic_dram_bytes": n_ins * 4, "insert_ms_per_step": round(insert_step_ms, 4)})
    ins_rate = per_launch_units / (avg_ms * 1e-3) if dom == "insert" else n_ins / (prof["insert_ms"] * 1e-3)
    atomic_peak = probes.get("red_3word_subwarp")

    # end to end through the host-buffer C ABI calls: pinned keys in, counts out
    hk = keys.cpu().pin_memory()
    hq = queries.cpu().pin_memory()
    ho = torch.empty(n_q, dtype=torch.uint32).pin_memory()
    e2e_steps = max(1, min(args.steps, 5))

    def e2e_step():
        sk.clear()
        if cfg["kind"] == 2:
            B, qo = cfg["batch"], 0
            for b in range(len(ins_views)):
                sk.insert_host(hk[b * B:b * B + ni_b])
                nq_b = B - ni_b
                sk.search_host(hk[b * B + ni_b:(b + 1) * B], ho[qo:qo + nq_b])
                qo += nq_b
        else:
            sk.insert_host(hk)
            sk.search_host(hq, ho)

    e2e_step()
    torch.cuda.synchronize()
    barrier()
    w0 = time.perf_counter()
    for _ in range(e2e_steps):
        e2e_step()
    torch.cuda.synchronize()
    e2e_ms = max_over_ranks((time.perf_counter() - w0) * 1e3 / e2e_steps)
    barrier()
    assert torch.equal(ho.cuda(), out), "host-buffer query results differ from the device path"

    if rank == 0:
        line = {
            "metric": METRIC, "value": round(value, 4), "unit": "Gkeys/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": round(ms_per_step, 4), "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "u32",
            "data": "synthetic: seeded Zipf(s) ranks by rejection-inversion mapped to distinct u32 keys"
                    if cfg["kind"] == 1 else "synthetic: seeded xorshift64* uniform u32 keys",
            "config": {"workload": cfg["workload"], "n_keys": n_ins, "n_query": n_q, "n_low": cfg["n_low"],
                       "n_high": cfg["n_high"], "hash_mask_ones": 3, "hash_mask_table_sz": 1021,
                       "l2": "key stream of %d MB per step > 126 MB L2" % (n_ins * 4 >> 20),
                       "parallelism": "independent sketch per GPU" if world > 1 else "single GPU",
                       "insert_knobs": {k: tuned[k] for k in ("lanes_per_key", "aggregate", "route", "ctas_per_sm",
                                                              "max_batch", "first_chunk", "keys_per_tile")}},
            "insert_gkeys_per_s": round(world * n_ins / (ins_ms * 1e6), 4),
            "query_gkeys_per_s": round(world * n_q / (q_ms * 1e6), 4),
            "avg_rel_error": rel, "mean_est_over_exact": ratio,
            "hbm_gbs_algorithmic": round((n_ins * insert_bytes + n_q * QUERY_BYTES_PER_KEY) /
                                         (ms_per_step * 1e-3) / 1e9, 1),
            "e2e": {"value": round(world * (n_ins + n_q) / (e2e_ms * 1e6), 4), "unit": "Gkeys/s",
                    "h2d_bytes_per_step": (n_ins + n_q) * 4, "d2h_bytes_per_step": n_q * 4,
                    "ms_per_step": round(e2e_ms, 3), "api": "qs_insert_host + qs_query_host"},
            "gpu_launches": int(launches),
            "roofline": roofline,
            "hbm_roofline": hbm_line,
            "pass1_atomic_roofline": None if parted else {
                                      "kernel": ins_kernel + " alone", "achieved_gsectors": round(ins_rate / 1e9, 3),
                                      "peak_gsectors": round(atomic_peak / 1e9, 3) if atomic_peak else None,
                                      "frac": round(ins_rate / atomic_peak, 4) if atomic_peak else None,
                                      "probe": "random 32 B sectors, 3 red.add.u32 words per sector, sub-warp "
                                               "of 8"},
            "kernel_ms_per_step": {"insert": round(prof["insert_ms"], 4), "repair": round(prof["repair_ms"], 4),
                                   "query": round(prof["query_ms"], 4)},
            # the instrumented step's repair by phase (indices as qs_profile documents them)
            "repair_phase_ms": [round(x, 3) for x in prof["repair_phase_ms"]],
            "repairs_active": int(prof["repairs_active"]),
            "clocks": clk.summary(),
        }
        if args.cpu_baseline:
            line["cpu_baseline"] = cpu_baseline(cfg, keys.cpu().numpy(), queries.cpu().numpy())
        print(json.dumps(line), flush=True)
    sk.close()
    if world > 1:
        dist.destroy_process_group()


def run_sharded(args, cfg):
    """`--shard`: one sketch sharded by bucket over the N ranks (qsketch_b200/sharded.py),
    strong scaling: the configuration's stream is split into N consecutive parts, rank r
    inserting part r and querying part r of the distinct keys; every insert and query routes
    the keys to their owner shards with an all-to-all (NCCL).  The estimates equal one sketch
    fed the whole stream in order."""
    import torch
    import torch.distributed as dist

    from qsketch_b200 import data
    from qsketch_b200.sharded import ShardedSketch

    if cfg["kind"] not in (0, 1):
        raise SystemExit("--shard runs the zipf, zipf_prof and uniform configurations")
    world, rank, local, barrier, max_over_ranks = init_ranks(args)
    stream = torch.cuda.current_stream()
    n, nq = cfg["n_keys"], cfg["n_query"]
    lo, hi = n * rank // world, n * (rank + 1) // world
    qlo, qhi = nq * rank // world, nq * (rank + 1) // world
    if cfg["kind"] == 1:
        keys = data.zipf_keys(n, cfg["n_ranks"], cfg["s"], seed=1000, perm_seed=99)[lo:hi].clone()
        queries = data.rank_keys(99, qlo, qhi - qlo)
    else:
        keys = data.uniform_keys(n, seed=1000)[lo:hi].clone()
        queries = keys[qlo - lo:qhi - lo].clone() if qhi <= hi else data.uniform_keys(n, seed=1000)[qlo:qhi].clone()
    torch.cuda.empty_cache()
    ss = ShardedSketch(cfg["n_low"], cfg["n_high"], hash_seed=SEED, mask_rng=1)

    def step():
        ss.local.clear()
        ss.insert(keys)
        return ss.search(queries)

    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    def local_launches():
        p = ss.local.profile()
        return p["insert_launches"] + p["repair_launches"] + p["query_launches"]

    with Clocks(local) as clk:
        barrier()
        torch.cuda.synchronize()
        launches0 = local_launches()
        t0.record(stream)
        for _ in range(args.steps):
            out = step()
        t1.record(stream)
        torch.cuda.synchronize()
        barrier()
    # the local sketch's kernels, plus per step with several ranks the routing kernels: count,
    # scan and scatter per partition (insert and query) and the query's unpartition
    launches = local_launches() - launches0 + (7 * args.steps if world > 1 else 0)
    ms_per_step = max_over_ranks(t0.elapsed_time(t1)) / args.steps
    hk, hq = keys.cpu().pin_memory(), queries.cpu().pin_memory()
    ho = torch.empty(queries.numel(), dtype=torch.uint32).pin_memory()
    dk, dq = torch.empty_like(keys), torch.empty_like(queries)
    ss.local.clear()
    torch.cuda.synchronize()
    barrier()
    w0 = time.perf_counter()
    dk.copy_(hk, non_blocking=True)
    ss.insert(dk)
    dq.copy_(hq, non_blocking=True)
    ho.copy_(ss.search(dq), non_blocking=True)
    torch.cuda.synchronize()
    e2e_ms = max_over_ranks((time.perf_counter() - w0) * 1e3)
    assert torch.equal(ho.cuda(), out), "host-buffer estimates differ from the device path"
    if rank == 0:
        print(json.dumps({
            "metric": METRIC, "value": round((n + nq) / (ms_per_step * 1e6), 4), "unit": "Gkeys/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms_per_step, 4),
            "higher_is_better": True, "scaling": "strong", "vs_baseline": None, "dtype": "u32",
            "data": "synthetic: the configuration's seeded stream, split into one consecutive part per rank",
            "config": {"workload": cfg["workload"], "n_keys": n, "n_query": nq, "n_low": cfg["n_low"],
                       "n_high_per_shard": cfg["n_high"], "parallelism": f"bucket-sharded over {world} GPU(s), "
                       "keys routed by one all-to-all per insert and two per query (NCCL)"},
            "e2e": {"value": round((n + nq) / (e2e_ms * 1e6), 4), "unit": "Gkeys/s",
                    "h2d_bytes_per_step": (n + nq) * 4, "d2h_bytes_per_step": nq * 4, "ms_per_step": round(e2e_ms, 3),
                    "api": "ShardedSketch.insert + search"},
            "gpu_launches": int(launches),
            "clocks": clk.summary(),
        }), flush=True)
    ss.local.close()
    if world > 1:
        dist.destroy_process_group()


def run_ablation(args, cfg):
    """The MSWS against the one-level sketches at equal bytes: insert and query Gkeys/s (CUDA
    events, mean over the steps) and, on the Zipf stream, the average relative error against
    exact counts of its distinct keys."""
    import torch
    import torch.distributed as dist

    import qsketch_b200 as qs
    from qsketch_b200 import data

    world, rank, local, barrier, max_over_ranks = init_ranks(args)
    stream = torch.cuda.current_stream()
    n = cfg["n_keys"]
    budget = cfg["n_low"] * 32  # the MSWS low table's bytes
    streams = {"uniform": data.uniform_keys(n, seed=1000 + rank)}
    zk, zr = data.zipf_keys(n, cfg["n_ranks"], cfg["s"], seed=1000 + rank, perm_seed=99 + rank, with_ranks=True)
    streams["zipf"] = zk
    zq = data.rank_keys(99 + rank, 0, cfg["n_ranks"])
    zexact = data.rank_histogram(zr, cfg["n_ranks"])
    del zr
    keep = zexact.view(torch.int32) > 0  # (uint32 tensors index through an int32 view)
    zq = zq.view(torch.int32)[keep].view(torch.uint32).contiguous()
    zexact = zexact.view(torch.int32)[keep].view(torch.uint32).contiguous()
    prime = qs.find_greatest_prime
    makers = {
        "msws": lambda: qs.Sketch_GPU_Sub_Warp_Level(cfg["n_low"], 8, cfg["n_high"], 32, hash_seed=SEED, mask_rng=1),
        "countmin_m3": lambda: qs.Sketch_GPU_Thread(prime(budget // 12), 3, seed_rng=1),
        "warp_m32": lambda: qs.Sketch_GPU_Warp(prime(budget // 128), 32, hash_seed=SEED, mask_rng=1),
        "subwarp_m16": lambda: qs.Sketch_GPU_Sub_Warp(prime(budget // 64), 16, hash_seed=SEED, mask_rng=1),
        "subwarp_m8": lambda: qs.Sketch_GPU_Sub_Warp(prime(budget // 32), 8, hash_seed=SEED, mask_rng=1),
    }
    rows = {}
    launches = 0  # every sketch's kernels inside the timed loops
    with Clocks(local) as clk:
        for name, make in makers.items():
            sk = make()
            row = {"table_bytes": int(sk.info()["n_low"]) * int(sk.info()["m_low"]) * 4}
            for sname, keys in streams.items():
                out = torch.empty(n, dtype=torch.uint32, device="cuda")
                for _ in range(args.warmup):
                    sk.clear()
                    sk.insert(keys)
                    sk.search(keys, counts=out)
                ev = [[torch.cuda.Event(enable_timing=True) for _ in range(3)] for _ in range(args.steps)]
                barrier()
                p0 = sk.profile()
                for e in ev:
                    sk.clear()
                    e[0].record(stream)
                    sk.insert(keys)
                    e[1].record(stream)
                    sk.search(keys, counts=out)
                    e[2].record(stream)
                torch.cuda.synchronize()
                p1 = sk.profile()
                launches += sum(p1[k] - p0[k] for k in ("insert_launches", "repair_launches", "query_launches"))
                ins = max_over_ranks(sum(e[0].elapsed_time(e[1]) for e in ev) / args.steps)
                qry = max_over_ranks(sum(e[1].elapsed_time(e[2]) for e in ev) / args.steps)
                row[sname] = {"insert_gkeys_per_s": round(n / (ins * 1e6), 3),
                              "query_gkeys_per_s": round(n / (qry * 1e6), 3)}
                if sname == "zipf":
                    rel, _ = data.error_metrics(sk.search(zq), zexact)
                    row[sname]["avg_rel_error"] = rel
            rows[name] = row
            sk.close()
    if rank == 0:
        m = rows["msws"]["uniform"]
        print(json.dumps({
            "metric": METRIC, "value": round(2 / (1 / m["insert_gkeys_per_s"] + 1 / m["query_gkeys_per_s"]), 4),
            "unit": "Gkeys/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": round(2 * n / (2 / (1 / m["insert_gkeys_per_s"] + 1 / m["query_gkeys_per_s"])) / 1e6, 4),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u32",
            "data": "synthetic: seeded uniform and Zipf(1.1) u32 keys",
            "config": {"workload": cfg["workload"], "n_keys": n, "budget_bytes": budget,
                       "note": "value: the MSWS on the uniform stream (insert + query of every key); the table "
                               "compares every sketch on both streams"},
            "ablation": rows, "gpu_launches": int(launches), "clocks": clk.summary(),
        }), flush=True)
    if world > 1:
        dist.destroy_process_group()


def run_cm(args, cfg):
    """Plain count-min (Sketch_GPU_Thread, device_sketch_v0.h:105-191), the in-GPU baseline: a
    step is clear + insert the 2^24 uniform keys + query every key.  Beside it, the MSWS sketch
    of the uniform configuration (8 MB low table) runs the same step, for the count-min vs
    MSWS comparison the reference publishes."""
    import torch
    import torch.distributed as dist

    import qsketch_b200 as qs
    from qsketch_b200 import data

    world, rank, local, barrier, max_over_ranks = init_ranks(args)
    stream = torch.cuda.current_stream()
    n, rows = cfg["n_keys"], cfg["rows"]
    keys = data.uniform_keys(n, seed=1000 + rank)
    out = torch.empty(n, dtype=torch.uint32, device="cuda")
    out_m = torch.empty_like(out)
    cm = qs.Sketch_GPU_Thread(cfg["n_low"], rows, seed_rng=1 + rank)
    ms_cfg = CONFIGS["uniform"]
    msws = qs.Sketch_GPU_Sub_Warp_Level(ms_cfg["n_low"], 8, ms_cfg["n_high"], 32, hash_seed=SEED, mask_rng=1)

    def step(sk, ev=None):
        sk.clear()
        if ev:
            ev[0].record(stream)
        sk.insert(keys)
        if ev:
            ev[1].record(stream)
        sk.search(keys, counts=out if sk is cm else out_m)
        if ev:
            ev[2].record(stream)

    for _ in range(args.warmup):
        step(cm)
        step(msws)
    torch.cuda.synchronize()
    cm.profile()
    K = args.steps
    evs = [[torch.cuda.Event(enable_timing=True) for _ in range(3)] for _ in range(K)]
    mevs = [[torch.cuda.Event(enable_timing=True) for _ in range(3)] for _ in range(K)]
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with Clocks(local) as clk:
        barrier()
        torch.cuda.synchronize()
        t0.record(stream)
        for i in range(K):
            step(cm, evs[i])
        t1.record(stream)
        torch.cuda.synchronize()
        barrier()
    ms_per_step = max_over_ranks(t0.elapsed_time(t1)) / K
    ins_ms = max_over_ranks(sum(e[0].elapsed_time(e[1]) for e in evs) / K)
    q_ms = max_over_ranks(sum(e[1].elapsed_time(e[2]) for e in evs) / K)
    launches = cm.profile()
    launches = launches["insert_launches"] + launches["query_launches"]
    for i in range(K):  # the MSWS sketch of the uniform configuration, same keys, same step
        step(msws, mevs[i])
    torch.cuda.synchronize()
    m_ins = sum(e[0].elapsed_time(e[1]) for e in mevs) / K
    m_q = sum(e[1].elapsed_time(e[2]) for e in mevs) / K
    probes = atomic_probes(max(64 << 20, cfg["n_low"] * rows * 4)) if rank == 0 else {}

    hk = keys.cpu().pin_memory()
    ho = torch.empty(n, dtype=torch.uint32).pin_memory()
    e2e_steps = max(1, min(K, 5))

    def e2e_step():
        cm.clear()
        cm.insert_host(hk)
        cm.search_host(hk, ho)

    e2e_step()
    torch.cuda.synchronize()
    barrier()
    w0 = time.perf_counter()
    for _ in range(e2e_steps):
        e2e_step()
    torch.cuda.synchronize()
    e2e_ms = max_over_ranks((time.perf_counter() - w0) * 1e3 / e2e_steps)
    assert torch.equal(ho.cuda(), out), "host-buffer count-min estimates differ from the device path"
    if rank == 0:
        line = {
            "metric": METRIC, "value": round(world * 2 * n / (ms_per_step * 1e6), 4), "unit": "Gkeys/s",
            "n_gpus": world, "steps": K, "warmup": args.warmup, "ms_per_step": round(ms_per_step, 4),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u32",
            "data": "synthetic: seeded xorshift64* uniform u32 keys",
            "config": {"workload": cfg["workload"], "n_keys": n, "n_query": n, "n": cfg["n_low"], "rows": rows,
                       "table_bytes": cfg["n_low"] * rows * 4,
                       "l2": "key stream of %d MB per step > 126 MB L2" % (n * 4 >> 20),
                       "parallelism": "independent sketch per GPU" if world > 1 else "single GPU"},
            "insert_gkeys_per_s": round(world * n / (ins_ms * 1e6), 4),
            "query_gkeys_per_s": round(world * n / (q_ms * 1e6), 4),
            "msws_same_keys": {"workload": ms_cfg["workload"],
                               "insert_gkeys_per_s": round(n / (m_ins * 1e6), 4),
                               "query_gkeys_per_s": round(n / (m_q * 1e6), 4),
                               "value": round(2 * n / ((m_ins + m_q) * 1e6), 4),
                               "note": "MSWS at 8 MB low + 8 MB high on the same keys; the reference's own "
                                       "count-min vs MSWS insert ratio is 0.42 vs 1.22 Gkeys/s on an RTX 2080 Ti "
                                       "(doc/data/qsketch/perf_2080ti_1.0.dat)"},
            "e2e": {"value": round(world * 2 * n / (e2e_ms * 1e6), 4), "unit": "Gkeys/s",
                    "h2d_bytes_per_step": 2 * n * 4, "d2h_bytes_per_step": n * 4,
                    "ms_per_step": round(e2e_ms, 3), "api": "qs_insert_host + qs_query_host"},
            "gpu_launches": int(launches),
            "roofline": dict(l2_atomic_roofline(probes, n / (ins_ms * 1e-3), rows, "k_cm_insert",
                                                f"each key adds 1 to one 32-bit counter in each of the {rows} rows"),
                             traffic=(round(traffic_per_unit("cm", "insert") * n)
                                      if traffic_per_unit("cm", "insert") else None),
                             traffic_unit="DRAM bytes per insert launch (ncu dram__bytes per key x keys)",
                             algorithmic_dram_bytes=n * 4),
            "clocks": clk.summary(),
        }
        if args.cpu_baseline:
            line["cpu_baseline"] = cpu_baseline(cfg, keys.cpu().numpy(), keys.cpu().numpy())
        print(json.dumps(line), flush=True)
    cm.close()
    msws.close()
    if world > 1:
        dist.destroy_process_group()


def run_learned(args, cfg):
    """Learned split vs plain MSWS at equal bytes.  A step is: a fresh learned sketch (created
    outside the timed events) takes the whole stream — warm-up inserts, training, routed
    inserts — then answers the distinct keys.  The plain sketch with the same budget runs the
    same step beside it."""
    import torch
    import torch.distributed as dist

    from qsketch_b200 import data
    from qsketch_b200.learned import LearnedSketch, plain_equal_bytes

    world, rank, local, barrier, max_over_ranks = init_ranks(args)
    stream = torch.cuda.current_stream()
    n, warm = cfg["n_keys"], cfg["warmup"]
    keys = data.class_keys(n, seed=5 + rank, perm_seed=11 + 7919 * rank)
    uniq, exact = data.exact_counts(keys)
    n_q = uniq.numel()
    out_l = torch.empty(n_q, dtype=torch.uint32, device="cuda")
    out_p = torch.empty_like(out_l)
    params = dict(budget_bytes=cfg["budget"], warmup_keys=warm, table_slots=cfg["table_slots"], hash_seed=SEED)
    plain = plain_equal_bytes(cfg["budget"], hash_seed=SEED)

    def ev():
        return torch.cuda.Event(enable_timing=True)

    def learned_step(e):
        lk = LearnedSketch(**params)
        torch.cuda.synchronize()
        e[0].record(stream)
        lk.insert(keys[:warm])
        e[1].record(stream)
        lk.insert(keys[warm:])
        e[2].record(stream)
        lk.search(uniq, counts=out_l)
        e[3].record(stream)
        torch.cuda.synchronize()
        return lk

    def plain_step(e):
        plain.clear()
        e[0].record(stream)
        plain.insert(keys)
        e[1].record(stream)
        plain.search(uniq, counts=out_p)
        e[2].record(stream)

    for _ in range(args.warmup):
        learned_step([ev() for _ in range(4)]).close()
        plain_step([ev() for _ in range(3)])
    torch.cuda.synchronize()
    le = [[ev() for _ in range(4)] for _ in range(args.steps)]
    pe = [[ev() for _ in range(3)] for _ in range(args.steps)]
    lk = None
    with Clocks(local) as clk:
        barrier()
        torch.cuda.synchronize()
        for i in range(args.steps):
            if lk is not None:
                lk.close()
            lk = learned_step(le[i])
        for i in range(args.steps):
            plain_step(pe[i])
        torch.cuda.synchronize()
        barrier()
    K = args.steps
    warm_ms = max_over_ranks(sum(e[0].elapsed_time(e[1]) for e in le) / K)
    rest_ms = max_over_ranks(sum(e[1].elapsed_time(e[2]) for e in le) / K)
    lq_ms = max_over_ranks(sum(e[2].elapsed_time(e[3]) for e in le) / K)
    p_ins_ms = max_over_ranks(sum(e[0].elapsed_time(e[1]) for e in pe) / K)
    p_q_ms = max_over_ranks(sum(e[1].elapsed_time(e[2]) for e in pe) / K)
    ms_per_step = warm_ms + rest_ms + lq_ms
    info = lk.info()
    re_l, ratio_l = data.error_metrics(out_l, exact)
    re_p, ratio_p = data.error_metrics(out_p, exact)

    # end to end: keys from pinned host memory, counts back to the host, inside the timed region
    hk = keys.cpu().pin_memory()
    hu = uniq.cpu().pin_memory()
    ho = torch.empty(n_q, dtype=torch.uint32).pin_memory()
    dk = torch.empty_like(keys)
    du = torch.empty_like(uniq)
    lk.close()
    lk2 = LearnedSketch(**params)
    torch.cuda.synchronize()
    barrier()
    w0 = time.perf_counter()
    dk.copy_(hk, non_blocking=True)
    lk2.insert(dk)
    du.copy_(hu, non_blocking=True)
    lk2.search(du, counts=out_l)
    ho.copy_(out_l, non_blocking=True)
    torch.cuda.synchronize()
    e2e_ms = max_over_ranks((time.perf_counter() - w0) * 1e3)
    lk2.close()

    # diagnostic bound: the stream's true heaviest keys (exact counts) admitted before the first
    # key, no training — what any classifier could gain with this table
    order = torch.argsort(exact.to(torch.int64), descending=True)[:int(0.75 * cfg["table_slots"])]
    top = uniq.view(torch.int32)[order].cpu().numpy().view(np.uint32)
    lo = LearnedSketch(**params)
    lo.admit_keys(top)
    lo.insert(keys)
    out_o = lo.search(uniq)
    re_o, _ = data.error_metrics(out_o, exact)
    lo.close()

    rest_keys = n - warm
    achieved = rest_keys * PART_BYTES_PER_KEY / (rest_ms * 1e-3) / 1e9
    hbm, peak_kind = peaks()
    if rank == 0:
        line = {
            "metric": METRIC, "value": round(world * (n + n_q) / (ms_per_step * 1e6), 4), "unit": "Gkeys/s",
            "n_gpus": world, "steps": K, "warmup": args.warmup, "ms_per_step": round(ms_per_step, 3),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u32 sketch, bf16/fp32 MLP",
            "data": "synthetic: seeded (class<<16)|suffix keys, class Zipf 1.0, suffix Zipf 1.2 permuted per class",
            "config": {"workload": cfg["workload"], "n_keys": n, "n_query": n_q, "budget_bytes": cfg["budget"],
                       "warmup_keys": warm, "table_slots": cfg["table_slots"],
                       "l2": "key stream of %d MB per step > 126 MB L2" % (n * 4 >> 20),
                       "parallelism": "independent sketch per GPU" if world > 1 else "single GPU"},
            "avg_rel_error": re_l, "avg_rel_error_plain": re_p, "re_ratio_learned_over_plain": re_l / re_p,
            "avg_rel_error_true_top_admitted": re_o, "re_ratio_true_top_over_plain": re_o / re_p,
            "mean_est_over_exact": ratio_l, "mean_est_over_exact_plain": ratio_p,
            "learned": {"warmup_and_train_ms": round(warm_ms, 3), "routed_insert_ms": round(rest_ms, 3),
                        "routed_insert_gkeys_per_s": round(world * rest_keys / (rest_ms * 1e6), 4),
                        "whole_stream_insert_gkeys_per_s": round(world * n / ((warm_ms + rest_ms) * 1e6), 4),
                        "query_gkeys_per_s": round(world * n_q / (lq_ms * 1e6), 4),
                        "train_ms": round(info["train_ms"], 2), "table_fill": info["table_fill"],
                        "train_examples": info["train_examples"], "adam_steps": info["steps"],
                        "warmup_replayed": info["warmup_replayed"],
                        "train_phase_ms": dict(zip(["distinct", "labels_and_set", "epochs", "admission", "replay"],
                                                   [round(x, 2) for x in info["train_phase_ms"]])),
                        "train_precision": info["train_precision"], "train_recall": info["train_recall"],
                        "sketch_bytes": info["sketch_bytes"], "table_bytes": info["table_bytes"],
                        "mlp_bytes": info["mlp_bytes"]},
            "plain": {"insert_gkeys_per_s": round(world * n / (p_ins_ms * 1e6), 4),
                      "query_gkeys_per_s": round(world * n_q / (p_q_ms * 1e6), 4),
                      "value": round(world * (n + n_q) / ((p_ins_ms + p_q_ms) * 1e6), 4)},
            "e2e": {"value": round(world * (n + n_q) / (e2e_ms * 1e6), 4), "unit": "Gkeys/s",
                    "h2d_bytes_per_step": (n + n_q) * 4, "d2h_bytes_per_step": n_q * 4,
                    "ms_per_step": round(e2e_ms, 3), "api": "qs_learned_insert + qs_learned_query"},
            "gpu_launches": None,
            "roofline": {"bound": "hbm", "kernel": "routed insert (k_route, k_part_split + k_part_apply + k_part_link)",
                         "achieved": round(achieved, 1), "peak": hbm, "unit": "GB/s",
                         "frac": round(achieved / hbm, 4), "traffic": None, "peak_source": peak_kind,
                         "bytes_per_unit": PART_BYTES_PER_KEY, "units": rest_keys},
            "clocks": clk.summary(),
        }
        print(json.dumps(line), flush=True)
    plain.close()
    if world > 1:
        dist.destroy_process_group()


def run_batched(args, cfg):
    """512 uneven streams, each with its own sketch, in one batch (qs_batch_*).  A step is:
    clear every sketch, insert every stream, query every stream's keys.  Beside it: the same
    streams through as many separate sketches one call after another, and the latency of a small
    serving batch eager vs replayed from a CUDA graph."""
    import torch
    import torch.distributed as dist

    import qsketch_b200 as qs
    from qsketch_b200 import data
    from qsketch_b200.batch import BatchedSketches

    world, rank, local, barrier, max_over_ranks = init_ranks(args)
    stream = torch.cuda.current_stream()
    S = cfg["n_streams"]
    w = data.uneven_streams(S, seed=1000 + rank, n_ranks=cfg["n_ranks"], max_len=cfg.get("max_len", 1 << 22))
    keys, offs = w["keys"], w["offsets"]
    total = keys.numel()
    out = torch.empty(total, dtype=torch.uint32, device="cuda")
    b = BatchedSketches(w["n_low"], w["n_high"], seed_rng=1 + rank, max_batch=1 << 22)
    # lanes per key per sketch-size class, timed on other keys of the same stream shapes
    cls_lpk = {}
    if args.autotune:
        tw = data.uneven_streams(S, seed=1000 + rank, n_ranks=cfg["n_ranks"], max_len=cfg.get("max_len", 1 << 22),
                                 key_seed=5000 + rank)
        cls_lpk = b.autotune(tw["keys"], tw["offsets"], reps=2)
        del tw
        torch.cuda.empty_cache()

    def step(ev=None):
        b.clear()
        if ev:
            ev[0].record(stream)
        b.insert(keys, offs, total)
        if ev:
            ev[1].record(stream)
        b.search(keys, offs, total, counts=out)
        if ev:
            ev[2].record(stream)

    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()
    launches0 = b.info()["launches"]
    evs = [[torch.cuda.Event(enable_timing=True) for _ in range(3)] for _ in range(args.steps)]
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with Clocks(local) as clk:
        barrier()
        torch.cuda.synchronize()
        torch.cuda.nvtx.range_push("timed")  # lets a profiler capture the timed steps only
        t0.record(stream)
        for i in range(args.steps):
            step(evs[i])
        t1.record(stream)
        torch.cuda.synchronize()
        torch.cuda.nvtx.range_pop()
        barrier()
    K = args.steps
    ms_per_step = max_over_ranks(t0.elapsed_time(t1)) / K
    ins_ms = max_over_ranks(sum(e[0].elapsed_time(e[1]) for e in evs) / K)
    q_ms = max_over_ranks(sum(e[1].elapsed_time(e[2]) for e in evs) / K)
    launches = b.info()["launches"] - launches0
    info = b.info()

    # per-kernel times of one instrumented step
    b.set_profiling(True)
    step()
    torch.cuda.synchronize()
    prof = b.profile()
    b.set_profiling(False)
    hbm, peak_kind = peaks()
    avg_ins = prof["insert_ms"] / max(1, prof["insert_timed"])
    per_launch = total / max(1, prof["insert_timed"])
    achieved = per_launch * PART_BYTES_PER_KEY / (avg_ins * 1e-3) / 1e9

    # the same streams through separate sketches, one call after another (one pass)
    alone = [qs.Sketch_GPU_Sub_Warp_Level(int(w["n_low"][s]), 8, int(w["n_high"][s]), 32,
                                          hash_seed=int(sd), max_batch=1 << 20)
             for s, sd in enumerate(b.seeds())]
    off = offs.cpu().numpy()
    out2 = torch.empty_like(out)

    def alone_pass():
        for s in range(S):
            alone[s].clear()
            alone[s].insert(keys[off[s]:off[s + 1]])
            alone[s].search(keys[off[s]:off[s + 1]], counts=out2[off[s]:off[s + 1]])

    alone_pass()
    torch.cuda.synchronize()
    a0, a1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a0.record(stream)
    alone_pass()
    a1.record(stream)
    torch.cuda.synchronize()
    alone_ms = a0.elapsed_time(a1)
    for sk in alone:
        sk.close()

    # serving latency: the first 1024 keys of every stream (2^19 keys), eager vs graph replay
    nsv = np.minimum(w["lengths"], 1024)
    sv_keys = torch.cat([keys[off[s]:off[s] + nsv[s]] for s in range(S)])
    sv_offs = torch.tensor(np.concatenate([[0], np.cumsum(nsv)]), dtype=torch.int64, device="cuda")
    sv_out = torch.empty_like(sv_keys)
    bs = BatchedSketches(w["n_low"], w["n_high"], seed_rng=1 + rank, max_batch=1 << 20)

    def serve(graph):
        if graph:
            bs.insert_graph(sv_keys, sv_offs)
            bs.search_graph(sv_keys, sv_offs, sv_out)
        else:
            bs.insert(sv_keys, sv_offs, sv_keys.numel())
            bs.search(sv_keys, sv_offs, sv_keys.numel(), counts=sv_out)

    lat = {}
    for graph in (False, True):
        for _ in range(3):
            serve(graph)
        torch.cuda.synchronize()
        reps = 20
        h0 = time.perf_counter()
        for _ in range(reps):
            serve(graph)
        torch.cuda.synchronize()
        lat["graph" if graph else "eager"] = (time.perf_counter() - h0) * 1e3 / reps
    graph_ok = bs.info()["graph_capture"]
    bs.close()

    # end to end: keys and offsets from pinned host memory, counts back, inside the timed region
    hk = keys.cpu().pin_memory()
    ho_offs = offs.cpu().pin_memory()
    hout = torch.empty(total, dtype=torch.uint32).pin_memory()
    dk = torch.empty_like(keys)
    do = torch.empty_like(offs)
    b.clear()
    torch.cuda.synchronize()
    barrier()
    w0 = time.perf_counter()
    dk.copy_(hk, non_blocking=True)
    do.copy_(ho_offs, non_blocking=True)
    b.insert(dk, do, total)
    b.search(dk, do, total, counts=out)
    hout.copy_(out, non_blocking=True)
    torch.cuda.synchronize()
    e2e_ms = max_over_ranks((time.perf_counter() - w0) * 1e3)
    status = b.status()
    if rank == 0:
        line = {
            "metric": METRIC, "value": round(world * 2 * total / (ms_per_step * 1e6), 4), "unit": "Gkeys/s",
            "n_gpus": world, "steps": K, "warmup": args.warmup, "ms_per_step": round(ms_per_step, 4),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u32",
            "data": "synthetic: per stream seeded Zipf(s) ranks by rejection-inversion mapped to distinct u32 keys",
            "config": {"workload": cfg["workload"], "n_streams": S, "n_keys": total, "n_query": total,
                       "table_bytes": int(info["table_bytes"]), "streams_pool_full": int(info["streams_pool_full"]),
                       "l2": "key stream of %d MB and tables of %d MB per step > 126 MB L2"
                             % (total * 4 >> 20, info["table_bytes"] >> 20),
                       "parallelism": "independent batch per GPU" if world > 1 else "single GPU",
                       "class_lanes_per_key": {str(k): v for k, v in cls_lpk.items()}},
            "insert_gkeys_per_s": round(world * total / (ins_ms * 1e6), 4),
            "query_gkeys_per_s": round(world * total / (q_ms * 1e6), 4),
            "repair_phase_ms": [round(x, 3) for x in prof["repair_phase_ms"]],
            "alone": {"ms": round(alone_ms, 3), "gkeys_per_s": round(2 * total / (alone_ms * 1e6), 4),
                      "note": "the same streams through %d separate sketches, one insert + one query call each" % S},
            "serving_batch": {"keys": int(sv_keys.numel()), "eager_ms": round(lat["eager"], 4),
                              "graph_ms": round(lat["graph"], 4), "graph_capture": int(graph_ok),
                              "note": "insert + query of the first 1024 keys of every stream, host wall time"},
            "status": int(status),
            "e2e": {"value": round(world * 2 * total / (e2e_ms * 1e6), 4), "unit": "Gkeys/s",
                    "h2d_bytes_per_step": total * 4 + (S + 1) * 8, "d2h_bytes_per_step": total * 4,
                    "ms_per_step": round(e2e_ms, 3), "api": "qs_batch_insert + qs_batch_query"},
            "gpu_launches": int(launches),
            "roofline": {"bound": "hbm",
                         "kernel": "k_part_split + k_part_apply + k_part_link (dense streams), k_batch_insert (the rest)",
                         "achieved": round(achieved, 1), "peak": hbm,
                         "unit": "GB/s", "frac": round(achieved / hbm, 4), "traffic": None,
                         "peak_source": peak_kind, "bytes_per_unit": PART_BYTES_PER_KEY,
                         "units_per_launch": per_launch, "avg_launch_ms": round(avg_ins, 5)},
            "kernel_ms_per_step": {"insert": round(prof["insert_ms"], 4), "repair": round(prof["repair_ms"], 4),
                                   "query": round(prof["query_ms"], 4)},
            "clocks": clk.summary(),
        }
        print(json.dumps(line), flush=True)
    b.close()
    if world > 1:
        dist.destroy_process_group()


# ---------------------------------------------------------------------------------------
def host_zipf_keys(n, n_ranks, s, seed):
    """Bounded Zipf(s) over n_ranks by inverse CDF (numpy), ranks mapped by a seeded bijection."""
    rng = np.random.default_rng(seed)
    w = np.arange(1, n_ranks + 1, dtype=np.float64) ** (-s)
    cdf = np.cumsum(w)
    cdf /= cdf[-1]
    r = np.searchsorted(cdf, rng.random(n)).astype(np.uint32)
    return r * np.uint32(2654435761) ^ np.uint32(0x5bd1e995), np.arange(n_ranks, dtype=np.uint32) * \
        np.uint32(2654435761) ^ np.uint32(0x5bd1e995)


def cpu_baseline(cfg, keys, queries):
    """The CPU path (the oracle, all host threads) on a bounded prefix of this run's own
    stream: about 10-30 s of CPU work."""
    threads = os.cpu_count() or 1
    ni = min(keys.size, 1 << 25)
    if cfg["kind"] == 2:
        ni -= ni % cfg["batch"]
        q = None
    else:
        q = queries[:min(queries.size, 1 << 22)]
    ti, tq, n_ins, n_q = reference_step(cfg, keys[:ni], q, threads)
    return {"value": round((n_ins + n_q) / (ti + tq) / 1e9, 5), "unit": "Gkeys/s", "cores": threads, "kind": "port",
            "sample": f"first {ni} keys of this run's stream ({n_ins} inserted, {n_q} queried) into a sketch of the "
                      "same size (oracle/oracle.cpp, keys partitioned by bucket over the threads, array order per "
                      "bucket)",
            "insert_gkeys_per_s": round(n_ins / ti / 1e9, 5), "query_gkeys_per_s": round(n_q / tq / 1e9, 5)}


def reference_inputs(cfg):
    """The GPU arm's rank-0 key stream (same generator, seeds and sizes) as host arrays.  On a
    machine with a GPU it is generated once by libqsketch's generator and copied to the host
    (input preparation, outside any timing; the timed work is the CPU path alone).  Without a
    GPU a numpy stand-in of the same shape is used, and the line says it is not the same
    stream.  Returns (keys, queries, same_stream)."""
    kind = cfg["kind"]
    try:
        import torch
        gpu = torch.cuda.is_available()
    except Exception:  # pragma: no cover
        gpu = False
    if gpu:
        from qsketch_b200 import data
        if kind in (1, 2):
            keys = data.zipf_keys(cfg["n_keys"], cfg["n_ranks"], cfg["s"], seed=1000, perm_seed=99).cpu().numpy()
            queries = data.rank_keys(99, 0, cfg["n_query"]).cpu().numpy() if kind == 1 else None
        else:
            keys = data.uniform_keys(cfg["n_keys"], seed=1000).cpu().numpy()
            queries = keys[:cfg["n_query"]]
        return keys, queries, True
    if kind in (1, 2):
        keys, distinct = host_zipf_keys(cfg["n_keys"], cfg["n_ranks"], cfg["s"], 1000)
        queries = distinct[:cfg["n_query"]] if kind == 1 else None
    else:
        keys = np.random.default_rng(1000).integers(0, 1 << 32, cfg["n_keys"], dtype=np.uint64).astype(np.uint32)
        queries = keys[:cfg["n_query"]]
    return keys, queries, False


def threaded_query(sketch, queries, threads):
    """Query with `threads` host threads over contiguous parts (ctypes releases the GIL)."""
    parts = np.array_split(queries, threads)
    outs = [None] * threads

    def q(i):
        outs[i] = sketch.query(parts[i])

    th = [threading.Thread(target=q, args=(i,)) for i in range(threads)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    return np.concatenate(outs)


def reference_step(cfg, keys, queries, threads):
    """One step of the CPU path on a fresh sketch; returns (insert s, query s, keys inserted,
    keys queried)."""
    import oracle
    kind = cfg["kind"]
    if kind == 5:
        sk = oracle.CountMin(cfg["n_low"], oracle.draw_seeds(1, cfg["rows"]))
    else:
        sk = oracle.Msws(cfg["n_low"], cfg["n_high"], SEED, oracle.generate_hashmask(1))
    ti = tq = 0.0
    if kind == 2:  # per batch: insert its first 90 %, then query the rest
        B = cfg["batch"]
        ni_b = int(B * cfg["insert_frac"])
        n_ins = n_q = 0
        for b0 in range(0, keys.size - B + 1, B):
            t0 = time.perf_counter()
            sk.insert(keys[b0:b0 + ni_b], threads=threads)
            t1 = time.perf_counter()
            threaded_query(sk, keys[b0 + ni_b:b0 + B], threads)
            t2 = time.perf_counter()
            ti += t1 - t0
            tq += t2 - t1
            n_ins += ni_b
            n_q += B - ni_b
        return ti, tq, n_ins, n_q
    t0 = time.perf_counter()
    sk.insert(keys, threads=threads)
    t1 = time.perf_counter()
    threaded_query(sk, queries, threads)
    t2 = time.perf_counter()
    return t1 - t0, t2 - t1, keys.size, queries.size


def run_reference(args, cfg):
    world, rank, _ = dist_setup(args.gpus)
    if rank != 0:
        return
    if cfg["kind"] in (3, 4, 6):
        print(json.dumps({"impl": "reference", "unavailable": "the reference has no learned heavy-hitter split, "
                          "no batched multi-sketch path and no CPU one-level bucket sketches; its plain path is "
                          "timed under --config zipf, uniform, mixed and cm"}), flush=True)
        return
    threads = os.cpu_count() or 1
    keys, queries, same = reference_inputs(cfg)
    for _ in range(args.warmup):
        reference_step(cfg, keys, queries, threads)
    tot, ti_s, tq_s = 0.0, 0.0, 0.0
    for _ in range(args.steps):
        ti, tq, ni, nq = reference_step(cfg, keys, queries, threads)
        tot += ti + tq
        ti_s += ti
        tq_s += tq
    ms = tot * 1e3 / args.steps
    v = (ni + nq) / (ms * 1e6)
    path = ("count-min (oracle/oracle.cpp or_cm_insert_mt, relaxed atomic adds)" if cfg["kind"] == 5 else
            "MSWS (oracle/oracle.cpp or_msws_insert_mt: one pass partitions the keys by bucket, then each "
            "thread applies its part in array order)")
    sample = (f"per step: a fresh sketch, insert {ni} keys, query {nq} keys of the {cfg['workload']} stream "
              f"(the whole workload); CPU restatement of the reference path, {path}, queries split over the "
              "threads")
    print(json.dumps({
        "metric": METRIC, "value": round(v, 5), "unit": "Gkeys/s", "n_gpus": args.gpus, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": round(ms, 3), "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "u32",
        "data": ("synthetic: the GPU arm's rank-0 stream (libqsketch's seeded generator), copied to the host"
                 if same else "synthetic: numpy stand-in of the stream's shape (no GPU to generate the same one)"),
        "config": {"workload": cfg["workload"], "n_keys": int(ni), "n_query": int(nq), "n_low": cfg["n_low"],
                   "n_high": cfg["n_high"], "same_config": bool(same)},
        "impl": "reference",
        "insert_gkeys_per_s": round(ni * args.steps / ti_s / 1e9, 5),
        "query_gkeys_per_s": round(nq * args.steps / tq_s / 1e9, 5),
        "cpu_baseline": {"value": round(v, 5), "unit": "Gkeys/s", "cores": threads, "kind": "port",
                         "sample": sample},
        "e2e": {"value": round(v, 5), "unit": "Gkeys/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }), flush=True)


def relaunch_ranks(n):
    """`--gpus N` outside torchrun: start the N ranks (one process per GPU) through
    torch.distributed.run on this node and wait for them."""
    import socket
    with socket.socket() as so:
        so.bind(("127.0.0.1", 0))
        port = so.getsockname()[1]
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", f"--nproc-per-node={n}",
           "--master-addr", "127.0.0.1", "--master-port", str(port), os.path.abspath(__file__)] + sys.argv[1:]
    return subprocess.run(cmd).returncode


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=30)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--config", choices=sorted(CONFIGS), default="zipf")
    ap.add_argument("--no-cpu-baseline", dest="cpu_baseline", action="store_false")
    ap.add_argument("--shard", action="store_true",
                    help="one sketch sharded by bucket over the N GPUs (strong scaling) instead of N replicas")
    ap.add_argument("--no-autotune", dest="autotune", action="store_false",
                    help="the library's default insert knobs instead of the autotuner's (profiling runs)")
    args = ap.parse_args()
    if args.warmup < 3:
        ap.error("--warmup must be >= 3")
    cfg = CONFIGS[args.config]
    if args.gpus > 1 and "WORLD_SIZE" not in os.environ:
        sys.exit(relaunch_ranks(args.gpus))
    if args.impl == "reference":
        run_reference(args, cfg)
    else:
        run_ours(args, cfg)


if __name__ == "__main__":
    main()
