#!/usr/bin/env python
"""Benchmark: Mpixel/s of JPEG 2000 decode on B200.

Workload (one step): decode of one 4096x4096 3-component 8-bit image coded
with the forward ICT, a 6-level 9/7 DWT, deadzone quantisation with base step
1/128 scaled by the 9/7 synthesis L2 norms, and 64x64 code-blocks with all
passes (12,288 code-blocks).  Synthetic seeded input (bilinear gradients plus
N(0, 8^2) noise), coded by the project's harness encoder at start-up.

  value   device-resident: Tier-1 + fused dequantisation, reverse DWT and fused
          inverse ICT/DC shift from a codestream already in HBM, timed with CUDA
          events per step; L2 is flushed (a 256 MiB write) between steps,
          outside the timed events.
  e2e     the public C-ABI call tc_decode_j2k (Decoder.decode): codestream in
          pinned host memory in, samples out to pinned host memory, parse + H2D
          + kernels + D2H inside the timer.

Multi-GPU: the path does not shard (one image per decode); --gpus N runs N
independent replicas (no collective), value = total pixels / max-over-ranks time.

--impl reference: the reference's CPU path on the host cores (the oracle port
of its algorithm), on a bounded sample of the same workload.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import threading
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "Mpixel/s decode, batched vs per-image, 1 B200; p50/p99 latency; DWT % HBM peak"
WORKLOAD = dict(workload="lossy_decode_4096x4096x3_8bit_ict_97_6lvl_step1/128_cblk64", width=4096, height=4096,
                ncomp=3, bits=8, levels=6, base_step=1.0 / 128, cblk=64, seed=2)
E2E_THREADS = 3   # host threads of the end-to-end stream
SAMPLE = dict(width=1024, height=1024)   # CPU baseline sample (1/16 of the pixels)


def log(*a):
    print(*a, file=sys.stderr, flush=True)


def make_workload(w, h, seed):
    from thousandthchicken_b200 import codec
    from thousandthchicken_b200.synth import gradient_noise_image
    img = gradient_noise_image(w, h, WORKLOAD["ncomp"], WORKLOAD["bits"], seed)
    cs = codec.encode(img, WORKLOAD["bits"], levels=WORKLOAD["levels"], reversible=False, mct=True,
                      base_step=WORKLOAD["base_step"])
    return img, cs


SERVE_RATES = "50,100,200,500,1000,2000"
SERVE_BUDGET = 40 << 30
SERVE_BACKLOG_S = 2.0    # a rate is not sustained once a request waits this long unbatched
SERVE_BATCH_SAMPLES = 128 << 20   # samples per batch (about 50 ms of decode)


def serve_section(args, specs, streams, device):
    """Served decode: Poisson arrivals of requests drawn from the mixed-size
    batch's 256 codestreams plus 20% single-component 16-bit 2048x2048
    lossless images (radial field + N(0, 40^2) noise), device-memory budget
    40 GB.  First the capacity of each path (every request available at
    once).  Then, for each rate of --serve-rates and at 80% of the
    continuous-batching capacity, min(1000, 5 s x rate) arrivals (the first
    requests of one fixed sequence) served by the continuous-batching server
    (batches of up to 16 requests and 128 Mi samples, two in flight) and by
    the per-image path (one request per batch, one in flight) on the same
    arrivals.  A rate is sustained when no request waits more than 2 s
    before its batch starts; otherwise the run stops admitting there and the
    rate is reported as overloaded with the throughput reached.  p50/p99 are
    over the requests served."""
    from thousandthchicken_b200 import codec
    from thousandthchicken_b200.serve import Request, Server, latency_stats, poisson_arrivals
    from thousandthchicken_b200.synth import radial_noise_image
    rng = np.random.default_rng(5)
    radial = [codec.encode(radial_noise_image(2048, 2048, 16, seed=50 + i), 16, levels=5, reversible=True,
                           mct=False) for i in range(4)]
    pool = [(cs_, sp["w"] * sp["h"]) for sp, cs_ in zip(specs, streams)] + [(cs_, 2048 * 2048) for cs_ in radial]
    nmix = len(streams)

    def picks(n, seed):
        r = np.random.default_rng(seed)
        return [nmix + int(r.integers(len(radial))) if r.random() < 0.2 else int(r.integers(nmix))
                for _ in range(n)]

    paths = {"continuous_batching": dict(max_batch=16, inflight=2, max_batch_samples=SERVE_BATCH_SAMPLES),
             "per_image": dict(max_batch=1, inflight=1)}
    servers = {k: Server(device, budget_bytes=SERVE_BUDGET, **kw) for k, kw in paths.items()}
    # warm-up: the largest requests once, so plan buffers and pinned staging
    # reach their working size before any timed run
    big = sorted(range(len(pool)), key=lambda i: -len(pool[i][0]))[:16]
    for srv in servers.values():
        srv.run([Request(k, pool[i][0], 0.0) for k, i in enumerate(big)], realtime=False)
    out = {"budget_bytes": SERVE_BUDGET, "batch_samples_cap": SERVE_BATCH_SAMPLES, "pool_images": len(pool),
           "radial_share": 0.2, "capacity": {}, "by_rate": []}
    cap_ids = picks(48, 7)
    mpx = sum(pool[i][1] for i in cap_ids) / 1e6
    for name, srv in servers.items():
        done, wall = srv.run([Request(k, pool[i][0], 0.0) for k, i in enumerate(cap_ids)], realtime=False)
        out["capacity"][name] = {"requests": len(cap_ids), "mpix_s": round(mpx / wall, 2),
                                 "req_s": round(len(cap_ids) / wall, 2)}
    rates = [float(r) for r in str(args.serve_rates).split(",") if r]
    sustained_rate = round(0.8 * out["capacity"]["continuous_batching"]["req_s"], 1)
    seq = picks(1000, 13)   # one request sequence for every rate (its first n)
    for rate in sorted(set(rates + [sustained_rate])):
        n = int(min(1000, max(20, 5 * rate)))
        ids = seq[:n]
        arr = poisson_arrivals(n, rate, seed=9)
        row = {"rate_per_s": rate, "requests": n, "arrival_span_s": round(float(arr[-1]), 3)}
        for name, srv in servers.items():
            reqs = [Request(k, pool[i][0], float(a)) for k, (i, a) in enumerate(zip(ids, arr))]
            done, wall = srv.run(reqs, realtime=True, stop_backlog_s=SERVE_BACKLOG_S)
            ok = [r for r in done if not r.error]
            served_mpx = sum(pool[ids[r.rid]][1] for r in ok) / 1e6
            st = latency_stats(ok)
            row[name] = {"sustained": srv.stats["stopped_at_s"] is None, "served": len(ok),
                         "failed": srv.stats["failed"], "unserved": srv.stats["unserved"],
                         "mpix_s": round(served_mpx / wall, 2), "wall_s": round(wall, 3),
                         "p50_ms": round(st["p50_ms"], 2), "p99_ms": round(st["p99_ms"], 2),
                         "peak_admitted_bytes": srv.stats["peak_admitted_bytes"],
                         "peak_device_bytes": srv.stats["peak_device_bytes"]}
        out["by_rate"].append(row)
    for srv in servers.values():
        srv.close()
    for name in paths:
        ok = [r for r in out["by_rate"] if r[name]["sustained"]]
        best = max(ok, key=lambda r: r["rate_per_s"]) if ok else None
        out[name] = {"max_sustained_rate": best["rate_per_s"] if best else None,
                     "p50_ms": best[name]["p50_ms"] if best else None,
                     "p99_ms": best[name]["p99_ms"] if best else None,
                     "mpix_s": best[name]["mpix_s"] if best else None}
    out["budget_respected"] = all(r[n]["peak_device_bytes"] <= SERVE_BUDGET for r in out["by_rate"] for n in paths)
    return out


def measured_peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return float(d["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


class ClockSampler:
    """nvidia-smi clock/throttle samples during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.idx = gpu_index
        self.proc = None
        self.file = None

    def start(self):
        try:
            self.file = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.idx}", f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=self.file, stderr=subprocess.DEVNULL)
        except (OSError, FileNotFoundError):
            self.proc = None

    def stop(self):
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        self.file.flush()
        rows = []
        for line in Path(self.file.name).read_text().splitlines():
            f = [x.strip() for x in line.split(",")]
            if len(f) >= 9:
                rows.append(f)
        os.unlink(self.file.name)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}

        def num(x):
            try:
                return float(x)
            except ValueError:
                return None
        sm = [num(r[1]) for r in rows if num(r[1])]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[k] for r in rows for k in range(4) if r[5 + k].lower() == "active"})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": num(rows[0][2]),
                "reasons": reasons, "samples": len(rows)}


def dwt_bytes(w, h, c, levels):
    """Algorithmic HBM bytes of the reverse DWT stage: every level reads its
    four subbands (4 B each) and writes its output once (4 B; the last level
    writes 1 B 8-bit samples after the fused colour transform)."""
    ws, hs = [w], [h]
    for _ in range(levels):
        ws.append((ws[-1] + 1) // 2)
        hs.append((hs[-1] + 1) // 2)
    b = 0
    for lvl in range(levels, 0, -1):
        n = ws[lvl - 1] * hs[lvl - 1] * c
        b += 4 * n + (1 * n if lvl == 1 else 4 * n)
    return b


def max_over_ranks(x: float, dist, device) -> float:
    """The largest of the ranks' values of x (x itself without a process
    group).  Every rank must call it at the same point."""
    if dist is None:
        return float(x)
    import torch
    t = torch.tensor([float(x)], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def _oracle():
    sys.path.insert(0, str(ROOT / "oracle"))
    import oracle as O
    O.build()
    return O


def run_reference(args, rank):
    """The reference arm: the reference's CPU implementation of the path (the
    oracle port of its algorithm) on all host cores, decoding the workload
    image itself.  The image is generated and coded here by the oracle's own
    encoder (byte-identical code-blocks to the harness encoder's, which a
    CPU test checks), so this process never loads libtc_j2k.so.  A step is
    one full decode: Tier-1 with dequantisation, reverse 9/7, inverse ICT and
    DC shift.  When oracle/_ref holds the reference's own Tier-1 kernel
    (compiled from its OpenCL C, D1/D2 fixed), it is also timed on the same
    code-blocks."""
    if rank != 0:
        return
    O = _oracle()
    from thousandthchicken_b200.synth import gradient_noise_image   # numpy only
    W, H, Cn = WORKLOAD["width"], WORKLOAD["height"], WORKLOAD["ncomp"]
    cores = os.cpu_count() or 1
    img = gradient_noise_image(W, H, Cn, WORKLOAD["bits"], WORKLOAD["seed"])
    t0 = time.perf_counter()
    et = O.encode_tile(img, WORKLOAD["bits"], WORKLOAD["levels"], False, True, WORKLOAD["base_step"],
                       cblk=WORKLOAD["cblk"], threads=cores)
    log(f"[reference] oracle encode: {et.n} code-blocks in {time.perf_counter() - t0:.1f}s")
    for _ in range(args.warmup):
        out, _f = et.decode(r=0.5, threads=cores)
    times = []
    for _ in range(args.steps):
        t0 = time.perf_counter()
        out, _f = et.decode(r=0.5, threads=cores)
        times.append(time.perf_counter() - t0)
    total = sum(times)
    mpx = W * H * args.steps / total / 1e6
    sample = f"the full {W}x{H}x{Cn} workload image, one oracle decode per step"
    line = {"impl": "reference", "metric": METRIC, "value": round(mpx, 3), "unit": "Mpixel/s", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(1000 * total / args.steps, 3),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic", "config": workload_config(et.n),
            "cpu_baseline": {"value": round(mpx, 3), "unit": "Mpixel/s", "cores": cores, "kind": "port",
                             "sample": sample},
            "e2e": {"value": round(mpx, 3), "unit": "Mpixel/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
            "psnr_db": round(_psnr(out, img), 2),
            "input": "coded by the oracle's encoder (ISO C.2/D.3 restatement), code-blocks byte-identical to the "
                     "harness encoder's"}
    rk = reference_kernel_tier1(et, cores)
    if rk:
        line["reference_kernel_tier1"] = rk
    line["repo_libraries_mapped"] = repo_libraries_mapped()
    print(json.dumps(line), flush=True)


def repo_libraries_mapped():
    """Shared libraries of this repository mapped into this process."""
    try:
        maps = Path("/proc/self/maps").read_text()
    except OSError:
        return None
    root = str(ROOT)
    return sorted({ln.split()[-1][len(root) + 1:] for ln in maps.splitlines()
                   if ln.split() and ln.split()[-1].startswith(root) and ".so" in ln.split()[-1]})


def reference_kernel_tier1(et, cores):
    """The reference's own Tier-1 kernel g_decode (coefficient_coder.cl,
    compiled as host code with its D1/D2 state bugs fixed) on the workload's
    code-blocks, one work-item per block over all cores: code-blocks/s of
    one timed run after one warm-up.  None when oracle/_ref is not built."""
    import ref as R
    if not R.available():
        return None
    blocks = []
    for i in range(et.n):
        c = et.arr[i]
        seg = et.pool[c.seg_off:c.seg_off + c.seg_len].tobytes() + b"\xff"   # D22: one byte read early
        blocks.append((seg, c.w, c.h, c.orient, c.mb, c.mb - c.zero_bitplanes))
    R.t1_decode(blocks, patched=True, threads=cores)
    t0 = time.perf_counter()
    _, skipped = R.t1_decode(blocks, patched=True, threads=cores)
    dt = time.perf_counter() - t0
    return {"cblk_per_s": round(len(blocks) / dt, 1), "ms": round(dt * 1e3, 1), "blocks": len(blocks),
            "skipped_over_16KiB": int(skipped), "cores": cores,
            "what": "reference g_decode (coefficient_coder.cl:778-819, D1/D2 fixed) on the workload's code-blocks"}


def workload_config(ncblk):
    """The config object both arms print: the workload and its code-block
    count, nothing about how either arm times it."""
    return {**WORKLOAD, "code_blocks": int(ncblk)}


def _psnr(a, b):
    d = a.astype(np.float64) - b.astype(np.float64)
    mse = float(np.mean(d * d))
    return 99.0 if mse == 0 else 10 * np.log10(255.0 ** 2 / mse)


def oracle_check(O, cs, got, img, cores):
    """The GPU's decode of the workload image against the FP64 oracle: the
    oracle decodes the same codestream's code-blocks (Tier-1, dequantisation,
    9/7 in FP64, ISO inverse ICT, DC shift) on all host cores.  Returns
    (parity, cpu_baseline): the GPU output's difference from the oracle's
    rounded samples (max, share of samples differing, PSNR) and from its
    unrounded FP64 samples clamped to the sample range (max and PSNR), the
    PSNR of both against the original; and the oracle decode's own rate."""
    from thousandthchicken_b200 import codec
    W, H, Cn, bits = WORKLOAD["width"], WORKLOAD["height"], WORKLOAD["ncomp"], WORKLOAD["bits"]
    info, desc, pool = codec.parse(cs)
    arr = O.cblk_array(desc, W, H)
    args = (arr, len(desc), pool, W, H, Cn, bits, WORKLOAD["levels"], False, True)
    t0 = time.perf_counter()
    O.decode_cblks(*args, r=0.5, threads=cores)
    dt = time.perf_counter() - t0
    want, f64 = O.decode_cblks(*args, r=0.5, threads=cores, f64=True)
    mx = float((1 << bits) - 1)
    g = got.astype(np.float64)
    d = np.abs(g - want.astype(np.float64))
    e = np.abs(g - np.clip(f64, 0.0, mx))

    def psnr(err):
        mse = float(np.mean(err * err))
        return 99.0 if mse == 0 else round(10 * np.log10(mx * mx / mse), 2)
    parity = {"max_abs": int(d.max()), "frac_differing": round(float((d > 0).mean()), 6),
              "psnr_vs_oracle_db": psnr(d), "max_abs_vs_fp64": round(float(e.max()), 4),
              "psnr_vs_fp64_db": psnr(e), "psnr_vs_original_db": psnr(g - img.astype(np.float64)),
              "oracle_psnr_vs_original_db": psnr(want.astype(np.float64) - img.astype(np.float64)),
              "ok": bool(d.max() <= 1),
              "what": f"full {W}x{H}x{Cn} GPU decode vs the FP64 oracle decode of the same code-blocks "
                      "(max_abs in LSB of the 8-bit output)"}
    cpu = {"value": round(W * H / dt / 1e6, 3), "unit": "Mpixel/s", "cores": cores, "kind": "port",
           "sample": f"the full {W}x{H}x{Cn} workload image, one oracle decode (Tier-1, dequantisation, FP64 9/7, "
                     "inverse ICT, DC shift)"}
    return parity, cpu


def encode_section(ctx, img):
    """The forward pipeline: the workload image encoded on the GPU
    (tc_encode_j2k_gpu: colour, DWT, quantisation and Tier-1 as kernels,
    packets on the host; host samples in, codestream out, median of 3)
    against the host encoder on all cores, and a lossless 1024^2 check that
    both write the same bytes."""
    from thousandthchicken_b200 import codec
    kw = dict(levels=WORKLOAD["levels"], reversible=False, mct=True, base_step=WORKLOAD["base_step"])
    bits = WORKLOAD["bits"]
    mpx = img.shape[1] * img.shape[2] / 1e6
    codec.encode_gpu(ctx, img, bits, **kw)
    ts = []
    for _ in range(3):
        t0 = time.perf_counter()
        codec.encode_gpu(ctx, img, bits, **kw)
        ts.append(time.perf_counter() - t0)
    gpu_s = sorted(ts)[1]
    t0 = time.perf_counter()
    codec.encode(img, bits, **kw)
    host_s = time.perf_counter() - t0
    small = np.ascontiguousarray(img[:, :1024, :1024])
    same = codec.encode_gpu(ctx, small, bits, levels=5, reversible=True) == codec.encode(small, bits, levels=5,
                                                                                           reversible=True)
    return {"gpu_mpix_s": round(mpx / gpu_s, 1), "gpu_ms": round(gpu_s * 1e3, 2),
            "host_mpix_s": round(mpx / host_s, 1), "host_ms": round(host_s * 1e3, 1),
            "host_threads": os.cpu_count() or 1, "lossless_1024_identical": bool(same),
            "what": "encode of the workload image (ICT, 6-level 9/7, step 1/128, 64x64 blocks), host samples in, "
                    "codestream out"}


def tier1_batched_section(ctx, stream, flush, cores):
    """The batched Tier-1 workload: 200,000 code-blocks (60% 64x64, 30%
    32x32, 10% edge blocks 1-64 wide and tall; Laplacian coefficients with
    4-14 bit-planes and about 15% zeros), each truncated at a seeded pass
    count, coded by the GPU Tier-1 encoder outside timing.  Decoded in one
    persistent launch and with one launch per image (groups of 64-4096
    blocks), each timed with CUDA events (median of 5, L2 flushed before
    each).  Checked bit for bit against the truncated coefficients (the
    oracle's ISO D.3 rule on the source coefficients, every block), against
    the oracle's decode of 5,000 sampled codewords and against the
    reference's own Tier-1 kernel on the sampled blocks that kept every
    pass."""
    import torch
    from thousandthchicken_b200.blockbatch import BlockBatch
    from thousandthchicken_b200.synth import c3_coefficients, c3_geometry
    O = _oracle()
    dev = torch.device("cuda", ctx.device)
    t0 = time.perf_counter()
    geom = c3_geometry(200_000, seed=3)
    coef = c3_coefficients(geom, dev, seed=3)
    bb = BlockBatch(ctx, geom, coef)
    torch.cuda.synchronize()
    prep_s = time.perf_counter() - t0

    def timed(fn, reps=5):
        ms = []
        with torch.cuda.stream(stream):
            fn()
            for k in range(reps):
                flush.fill_(k & 0xFF)
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record(stream)
                fn()
                b.record(stream)
                b.synchronize()
                ms.append(a.elapsed_time(b))
        return sorted(ms)[reps // 2]

    per_ms = timed(bb.decode_per_image)
    per_out = bb.out.cpu().numpy()
    bat_ms = timed(bb.decode_batched)
    ctx.synchronize()
    got = bb.out.cpu().numpy()
    d = bb.desc
    want = O.t1_truncate_batch(coef.cpu().numpy(), geom["off"], geom["w"], geom["h"], d["passes"], threads=cores)
    exact = bool(np.array_equal(got, want))
    pool = bb.pool.cpu().numpy()
    rng = np.random.default_rng(6)
    sample = rng.choice(bb.n, 5000, replace=False)
    oracle_ok, full = True, []
    for i in sample:
        w, h, off = int(d["w"][i]), int(d["h"][i]), int(geom["off"][i])
        seg = pool[i * bb.cap: i * bb.cap + int(d["seg_len"][i])].tobytes()
        nbp = int(d["mb"][i]) - int(d["zero_bitplanes"][i])
        mine = got[off: off + w * h].reshape(h, w)
        q, _ = O.t1_decode(seg, w, h, int(d["orient"][i]), nbp if d["passes"][i] else 0, int(d["passes"][i]))
        oracle_ok &= bool(np.array_equal(mine, q))
        if d["passes"][i] and d["passes"][i] == 3 * nbp - 2 and w >= 2:
            full.append((i, seg + b"\xff", mine))   # the reference kernel reads one byte early (D22)
    ref_check = None
    import ref as R
    if R.available() and full:
        blocks = [(seg, int(d["w"][i]), int(d["h"][i]), int(d["orient"][i]), int(d["mb"][i]),
                   int(d["mb"][i]) - int(d["zero_bitplanes"][i])) for i, seg, _ in full]
        ref_raw, skipped = R.t1_decode(blocks, patched=True, threads=cores)
        same = 0
        for k, (i, _, mine) in enumerate(full):
            h, w = mine.shape
            mb = int(d["mb"][i])
            raw = (np.abs(mine).astype(np.uint32) << np.uint32(31 - mb)) | \
                  ((mine < 0).astype(np.uint32) << np.uint32(31))
            same += bool(np.array_equal(ref_raw[k, :h, :w], raw))
        ref_check = {"blocks": len(full), "identical": same, "skipped_over_16KiB": int(skipped)}
    nbp = d["mb"].astype(int) - d["zero_bitplanes"].astype(int)
    out = {"blocks": bb.n, "images": len(geom["images"]), "coefficients": geom["elems"],
           "codeword_bytes": bb.codeword_bytes,
           "truncated_share": round(float(((d["passes"] > 0) & (d["passes"] < 3 * nbp - 2)).mean()), 4),
           "batched_ms": round(bat_ms, 3), "per_image_ms": round(per_ms, 3),
           "cblk_per_s": round(bb.n / (bat_ms / 1000.0), 1), "per_image_cblk_per_s": round(bb.n / (per_ms / 1000.0), 1),
           "speedup": round(per_ms / bat_ms, 3), "bit_exact": exact,
           "per_image_identical": bool(np.array_equal(per_out, got)),
           "oracle_sample": {"blocks": len(sample), "identical": oracle_ok},
           "reference_kernel_untruncated": ref_check, "prepare_s": round(prep_s, 1),
           "what": "200,000 uneven code-blocks truncated at seeded pass counts, one persistent Tier-1 launch vs one "
                   "launch per image; bit_exact against the truncated source coefficients"}
    bb.close()
    del coef
    torch.cuda.empty_cache()
    return out


WAVE_BYTES = 24 << 30   # device memory of one wave of the mixed batch (plans + outputs)


def encode_mixed(ctx, specs):
    """The mixed batch's codestreams: each image generated on the device
    (seeded), read back and coded by the GPU encoder (tc_encode_j2k_gpu),
    outside any timing."""
    import torch
    from thousandthchicken_b200 import codec
    from thousandthchicken_b200.synth import gradient_noise_image_device
    dev = torch.device("cuda", ctx.device)
    out = []
    for sp in specs:
        img = gradient_noise_image_device(sp["w"], sp["h"], sp["c"], sp["bits"], sp["seed"], dev).cpu().numpy()
        if img.dtype == np.int16:
            img = img.view(np.uint16)
        out.append(codec.encode_gpu(ctx, img, sp["bits"], levels=sp["levels"], reversible=sp["reversible"],
                                    mct=sp["c"] == 3, base_step=sp["base_step"]))
    return out


def mixed_waves(specs, streams, budget=WAVE_BYTES):
    """Consecutive images grouped so that each group's device memory
    (coefficients, DWT scratch, outputs, codestreams, descriptors) stays
    under the budget."""
    from thousandthchicken_b200.codec import read_header
    from thousandthchicken_b200.serve import request_device_bytes
    waves, cur, used = [], [], 0
    for i, cs in enumerate(streams):
        b = request_device_bytes(read_header(cs), len(cs))
        if cur and used + b > budget:
            waves.append(cur)
            cur, used = [], 0
        cur.append(i)
        used += b
    if cur:
        waves.append(cur)
    return waves


def mixed_section(ctx, stream, specs, streams, cores):
    """Mixed-size batch: 256 images of 256-8192 per side decoded in waves
    under a device-memory budget, (a) batched: one plan per wave (one Tier-1
    queue over all its code-blocks, DWT levels of all its images in shared
    launches) replayed as a CUDA graph per shape bucket, and (b) per image:
    one plan per image executed one after another, the plain per-image GPU
    path.  Each is timed with CUDA events on the context's stream over one
    execute of every image after one untimed execute (the waves are larger
    than L2).  Lossless outputs are compared with the source image
    regenerated on the device; lossy ones give their PSNR against it, and
    the two smallest lossy images are compared with the FP64 oracle."""
    import torch
    from thousandthchicken_b200 import codec
    from thousandthchicken_b200.stages import Plan
    from thousandthchicken_b200.synth import gradient_noise_image_device
    dev = torch.device("cuda", ctx.device)
    from thousandthchicken_b200 import autotune
    waves = mixed_waves(specs, streams)
    mpx = sum(sp["w"] * sp["h"] for sp in specs) / 1e6
    # autotune a few shape buckets on single images of the batch (smallest,
    # median and largest lossy RGB image, a median lossless RGB one); the
    # per-image path then applies each plan's bucket choice
    rgb_lossy = sorted([i for i, sp in enumerate(specs) if sp["c"] == 3 and not sp["reversible"]],
                       key=lambda i: specs[i]["w"] * specs[i]["h"])
    rgb_lossless = sorted([i for i, sp in enumerate(specs) if sp["c"] == 3 and sp["reversible"]],
                          key=lambda i: specs[i]["w"] * specs[i]["h"])
    tuned = {}
    for i in [rgb_lossy[0], rgb_lossy[len(rgb_lossy) // 2], rgb_lossy[-1], rgb_lossless[len(rgb_lossless) // 2]]:
        tp = Plan(ctx, [streams[i]])
        to = tp.alloc_outputs()
        with torch.cuda.stream(stream):
            r_ = autotune.tune_plan(tp, to, trials=2, use_cache=False)
        tuned[r_["bucket"]] = {k: r_[k] for k in ("lanes", "dwt", "tier1_ms", "dwt_ms")}
        tuned[r_["bucket"]]["image"] = f"{specs[i]['w']}x{specs[i]['h']}x{specs[i]['c']}"
        tp.close()
        del to
    autotune._set(ctx, 32, autotune.L.TC_DWT_TMA)
    lossy_small = sorted([i for i, sp in enumerate(specs) if not sp["reversible"]],
                         key=lambda i: specs[i]["w"] * specs[i]["h"])[:2]
    kept = {}
    res = {"per_image": 0.0, "batched": 0.0}
    exact, psnrs, graphs = True, [], {"captures": 0, "updates": 0, "replays": 0}
    for path in ("per_image", "batched"):
        for wave in waves:
            ws = [streams[i] for i in wave]
            plans = [Plan(ctx, ws)] if path == "batched" else [Plan(ctx, [s_]) for s_ in ws]
            if path == "batched":
                autotune._set(ctx, 32, autotune.L.TC_DWT_TMA)
                plans[0].set_graph(True)
            outs = [p_.alloc_outputs() for p_ in plans]
            with torch.cuda.stream(stream):
                for p_, o_ in zip(plans, outs):
                    if path == "per_image":
                        autotune.apply(p_, tuned)
                    p_.execute(o_)
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record(stream)
                for p_, o_ in zip(plans, outs):
                    if path == "per_image":
                        autotune.apply(p_, tuned)
                    p_.execute(o_)
                b.record(stream)
            b.synchronize()
            ctx.synchronize()
            res[path] += a.elapsed_time(b)
            if path == "batched":
                for k, v in plans[0].graph_stats().items():
                    graphs[k] += v
                for i, o_ in zip(wave, outs[0]):
                    sp = specs[i]
                    ref = gradient_noise_image_device(sp["w"], sp["h"], sp["c"], sp["bits"], sp["seed"], dev)
                    if sp["reversible"]:
                        exact &= bool(torch.equal(o_, ref))
                    else:
                        mx = float((1 << sp["bits"]) - 1)
                        d = o_.float() - ref.float()
                        mse = float((d * d).mean())
                        psnrs.append(99.0 if mse == 0 else 10 * np.log10(mx * mx / mse))
                    if i in lossy_small:
                        kept[i] = o_.cpu().numpy()
                    del ref
            for p_ in plans:
                p_.close()
            del outs, plans
            torch.cuda.empty_cache()
    # the two smallest lossy images against the FP64 oracle
    O = _oracle()
    orc = []
    for i in lossy_small:
        sp = specs[i]
        info, desc, pool = codec.parse(streams[i])
        want = O.decode_tile(desc, pool, sp["w"], sp["h"], sp["c"], sp["bits"], sp["levels"], False, sp["c"] == 3,
                             r=0.5, threads=cores)
        got = kept[i].view(np.uint16) if kept[i].dtype == np.int16 else kept[i]
        d = np.abs(got.astype(np.int64) - want.astype(np.int64))
        orc.append({"image": i, "size": f"{sp['w']}x{sp['h']}x{sp['c']}", "bits": sp["bits"],
                    "max_abs": int(d.max()), "frac_differing": round(float((d > 0).mean()), 6)})
    return {"images": len(specs), "mpixels": round(mpx, 1), "waves": len(waves),
            "wave_budget_bytes": WAVE_BYTES,
            "codestream_bytes": int(sum(len(s_) for s_ in streams)),
            "batched_ms": round(res["batched"], 2), "per_image_ms": round(res["per_image"], 2),
            "batched_mpix_s": round(mpx / (res["batched"] / 1000.0), 2),
            "per_image_mpix_s": round(mpx / (res["per_image"] / 1000.0), 2),
            "speedup": round(res["per_image"] / res["batched"], 3),
            "lossless_bit_exact": exact, "lossy_min_psnr_db": round(min(psnrs), 2), "graphs": graphs,
            "autotune": tuned,
            "oracle_sample": orc,
            "workload": "256 images, W and H uniform 256-8192 step 16, 1/3 comps, 8/12-bit, half RCT + 5-level 5/3, "
                        "half ICT + 5-level 9/7 step 1/64, 64x64 blocks"}


def kernels_section(ctx, stream, flush, cs, hbm):
    """The stand-alone stage kernels on device-resident 4096x4096 data, each
    timed with CUDA events on the context's stream (median of 5 runs, L2
    flushed before each): achieved GB/s of algorithmic bytes against the
    measured copy bandwidth."""
    import torch
    from thousandthchicken_b200 import codec
    from thousandthchicken_b200.stages import (CoefficientCoder, DWTForward53, DWTForward97, DWTReverse97,
                                               Preprocessor, Quantizer, _dev_bytes)
    dev = torch.device("cuda", ctx.device)
    W = H = 4096
    g = torch.Generator(device=dev).manual_seed(3)

    def timed(fn):
        ms = []
        with torch.cuda.stream(stream):
            fn()
            for k in range(5):
                flush.fill_(k & 0xFF)
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record(stream)
                fn()
                b.record(stream)
                b.synchronize()
                ms.append(a.elapsed_time(b))
        return sorted(ms)[2]

    def entry(ms, nbytes, what):
        gbs = nbytes / (ms / 1000.0) / 1e9
        return {"ms": round(ms, 4), "bytes": int(nbytes), "gbs": round(gbs, 1), "frac": round(gbs / hbm, 4),
                "what": what}

    out = {}
    lv = 6
    xf = torch.randn((H, W), generator=g, device=dev) * 64
    yf = torch.empty_like(xf)
    zf = torch.empty_like(xf)
    db = sum(8 * w_ * h_ for w_, h_ in _level_dims(W, H, lv))  # 4 B read + 4 B written per sample and level
    out["forward_97"] = entry(timed(lambda: DWTForward97(ctx).run(xf, yf, W, H, lv)), db,
                              "tc_dwt_forward97, one 4096^2 fp32 plane, 6 levels")
    out["reverse_97"] = entry(timed(lambda: DWTReverse97(ctx).run(yf, zf, W, H, lv)), db,
                              "tc_dwt_reverse97, one 4096^2 fp32 plane, 6 levels")
    xi = torch.randint(-128, 128, (H, W), generator=g, device=dev, dtype=torch.int32)
    yi = torch.empty_like(xi)
    out["forward_53"] = entry(timed(lambda: DWTForward53(ctx).run(xi, yi, W, H, 5)),
                              sum(8 * w_ * h_ for w_, h_ in _level_dims(W, H, 5)),
                              "tc_dwt_forward53, one 4096^2 int32 plane, 5 levels")
    planes = [torch.randn((H, W), generator=g, device=dev) * 40 for _ in range(3)]
    px8 = [torch.empty((H, W), dtype=torch.uint8, device=dev) for _ in range(3)]
    pre = Preprocessor(ctx)
    out["colour_inverse_ict"] = entry(timed(lambda: pre.color_decoder_lossy(planes, px8, 8)), 3 * W * H * 5,
                                      "tc_color_inverse ICT, 3 x 4096^2 fp32 in, 8-bit out")
    fl = [torch.empty((H, W), device=dev) for _ in range(3)]
    out["colour_forward_ict"] = entry(timed(lambda: pre.color_coder_lossy(px8, fl, 8)), 3 * W * H * 5,
                                      "tc_color_forward ICT, 3 x 4096^2 8-bit in, fp32 out")
    info, desc, pool = codec.parse(cs)
    n = info["ncomp"] * W * H
    cc = CoefficientCoder(ctx)
    raw = cc.decode_blocks(desc, pool, n, raw=True)
    deq = torch.empty(n, dtype=torch.float32, device=dev)
    d_desc = _dev_bytes(np.ascontiguousarray(desc, codec.DESC_DTYPE), dev)
    q = Quantizer(ctx)
    out["dequantize_raw"] = entry(timed(lambda: q.dequantize(d_desc, len(desc), raw, deq, 0.5)), 8 * n,
                                  "tc_dequantize_raw over the 4096^2 x 3 workload's 12288 blocks")
    out["reverse_97_levels"] = dwt_levels(ctx, stream, flush, W, lv, hbm)
    ctx.synchronize()
    return out


def dwt_levels(ctx, stream, flush, n, levels, hbm, reps=7):
    """Per level of tc_dwt_reverse97 on an n x n fp32 plane: the time of each
    level as the difference of reverses with k and k - 1 levels (CUDA events,
    median of reps, L2 flushed before each), the full-size level first, with
    its algorithmic bytes (4 B read + 4 B written per output sample)."""
    import torch
    from thousandthchicken_b200.stages import DWTReverse97
    dev = torch.device("cuda", ctx.device)
    g = torch.Generator(device=dev).manual_seed(5)
    x = torch.randn((n, n), generator=g, device=dev) * 30
    y = torch.empty_like(x)
    k = DWTReverse97(ctx)
    med = {}
    with torch.cuda.stream(stream):
        for _ in range(3):
            k.run(x, y, n, n, levels)
        for lv in range(1, levels + 1):
            ms = []
            for r in range(reps):
                flush.fill_(r & 0xFF)
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record(stream)
                k.run(x, y, n, n, lv)
                b.record(stream)
                b.synchronize()
                ms.append(a.elapsed_time(b))
            med[lv] = sorted(ms)[reps // 2]
    rows = []
    for lv, (w_, h_) in enumerate(_level_dims(n, n, levels), start=1):
        us = (med[lv] - med.get(lv - 1, 0.0)) * 1e3
        nbytes = 8 * w_ * h_
        gbs = nbytes / max(us, 1e-3) / 1e3
        rows.append({"size": w_, "us": round(us, 1), "gbs": round(gbs, 1), "frac": round(gbs / hbm, 4)})
    return {"plane": n, "levels": rows,
            "what": "tc_dwt_reverse97 level by level (reverses of k and k-1 levels differenced), full size first"}


def tier1_only(kind, n, reps=12):
    """Tier-1 time (CUDA events on the plan's stream, L2 flushed before each
    run; min and median of `reps`) of one n x n x 3 image: the bench's lossy
    coding, or 12-bit samples coded losslessly (RCT, 5-level 5/3), with a
    hash of the decoded samples."""
    import hashlib
    import torch
    from thousandthchicken_b200 import codec
    from thousandthchicken_b200.stages import Context, Plan
    from thousandthchicken_b200.synth import gradient_noise_image
    if kind == "lossy":
        _, cs = make_workload(n, n, WORKLOAD["seed"])
    else:
        img = gradient_noise_image(n, n, 3, 12, WORKLOAD["seed"])
        cs = codec.encode(img, 12, levels=5, reversible=True, mct=True)
    stream = torch.cuda.Stream(0)
    ctx = Context(0, stream)
    plan = Plan(ctx, [cs])
    outs = plan.alloc_outputs()
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda:0")
    with torch.cuda.stream(stream):
        for _ in range(3):
            plan.execute(outs)
    ctx.synchronize()
    digest = hashlib.sha1(outs[0].cpu().numpy().tobytes()).hexdigest()[:12]
    plan.set_profiling(True)
    t1 = []
    with torch.cuda.stream(stream):
        for k in range(reps):
            flush.fill_(k & 0xFF)
            plan.execute(outs)
            t1.append(plan.stage_ms()[0])
    plan.set_profiling(False)
    t1.sort()
    return {"tier1": kind, "size": n, "code_blocks": plan.infos[0]["ncblk"], "tier1_ms_min": round(t1[0], 3),
            "tier1_ms_median": round(t1[len(t1) // 2], 3), "samples_sha1": digest}


def _level_dims(w, h, levels):
    """(width, height) of each level's region, the full size first."""
    dims = []
    for _ in range(levels):
        dims.append((w, h))
        w, h = (w + 1) // 2, (h + 1) // 2
    return dims


def run_ours(args, rank, world, local_rank):
    import torch
    from thousandthchicken_b200.stages import Context, Decoder, Plan

    torch.cuda.set_device(local_rank)
    dist = None
    if world > 1:
        import torch.distributed as dist
        import datetime
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300))

    W, H, Cn = WORKLOAD["width"], WORKLOAD["height"], WORKLOAD["ncomp"]
    t0 = time.perf_counter()
    img, cs = make_workload(W, H, WORKLOAD["seed"])
    log(f"[rank {rank}] encoded workload: {len(cs)} bytes in {time.perf_counter() - t0:.1f}s")

    stream = torch.cuda.Stream(local_rank)
    ctx = Context(local_rank, stream)
    plan = Plan(ctx, [cs])
    outs = plan.alloc_outputs()
    ncblk = plan.infos[0]["ncblk"]
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=f"cuda:{local_rank}")

    with torch.cuda.stream(stream):
        for _ in range(args.warmup):
            plan.execute(outs)
    ctx.synchronize()
    decoded = outs[0].cpu().numpy()
    psnr = _psnr(decoded, img)

    # device-resident timed region
    evs = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    launches0 = ctx.launches
    if dist:
        dist.barrier()
    torch.cuda.synchronize()
    sampler = ClockSampler(local_rank)
    sampler.start()
    wall0 = time.perf_counter()
    with torch.cuda.stream(stream):
        for k in range(args.steps):
            flush.fill_(k & 0xFF)            # evict L2 between steps (not inside the events)
            evs[k][0].record(stream)
            plan.execute(outs)
            evs[k][1].record(stream)
    torch.cuda.synchronize()
    if dist:
        dist.barrier()
    wall = time.perf_counter() - wall0
    clocks = sampler.stop()
    launches = ctx.launches - launches0
    step_ms = [a.elapsed_time(b) for a, b in evs]
    total_ms = max_over_ranks(sum(step_ms), dist, f"cuda:{local_rank}")
    ctx.synchronize()

    # per-stage device times (CUDA events on the plan's stream)
    plan.set_profiling(True)
    t1_ms, dwt_ms = [], []
    with torch.cuda.stream(stream):
        for k in range(max(3, min(args.steps, 10))):
            flush.fill_(k & 0xFF)
            plan.execute(outs)
            a, b = plan.stage_ms()
            t1_ms.append(a)
            dwt_ms.append(b)
    plan.set_profiling(False)

    # end to end through the public C-ABI call (host in, host out), the
    # codestream and the samples in pinned host memory
    dec = Decoder(ctx)
    host_cs = torch.empty(len(cs), dtype=torch.uint8, pin_memory=True).numpy()
    host_cs[:] = np.frombuffer(cs, np.uint8)
    host_out = torch.empty((Cn, H, W), dtype=torch.uint8, pin_memory=True).numpy()
    dec.decode(host_cs, host_out)
    e2e_times = []
    e2e_steps = max(1, min(args.steps, 5))
    if dist:
        dist.barrier()
    for _ in range(e2e_steps):
        t0 = time.perf_counter()
        dec.decode(host_cs, host_out)
        e2e_times.append(time.perf_counter() - t0)
    e2e_seq_s = max_over_ranks(sum(e2e_times) / e2e_steps, dist, f"cuda:{local_rank}")
    # A stream of images through the same call: E2E_THREADS host threads,
    # each with its own context (stream and buffers) and pinned output, take
    # images in turn, so one image's parse, upload and read-back overlap the
    # others' kernels.  Every image still makes its own host->device and
    # device->host copies; wall time over all images.  Three threads: a
    # call returns only after its reverse DWT, which waits for SM room behind
    # the next image's persistent Tier-1 launch, so with two threads the GPU
    # idles while the blocked thread parses and launches its next image
    # (measured on this workload: 1073 Mpixel/s with two threads, 1109 with
    # three, 1104 with four).
    decs = [(dec, host_out)]
    for _ in range(E2E_THREADS - 1):
        d = Decoder(Context(local_rank, torch.cuda.Stream(local_rank)))
        o = torch.empty((Cn, H, W), dtype=torch.uint8, pin_memory=True).numpy()
        d.decode(host_cs, o)
        decs.append((d, o))
    n_pipe = E2E_THREADS * max(2, min(args.steps, 4))

    def worker(d, o, n):
        for _ in range(n):
            d.decode(host_cs, o)

    if dist:
        dist.barrier()
    t0 = time.perf_counter()
    th = [threading.Thread(target=worker, args=(d, o, n_pipe // E2E_THREADS)) for d, o in decs]
    for t in th:
        t.start()
    for t in th:
        t.join()
    e2e_s = max_over_ranks((time.perf_counter() - t0) / n_pipe, dist, f"cuda:{local_rank}")
    same_out = all(bool(np.array_equal(host_out, o)) for _, o in decs[1:])

    batched, served, kernels, encode, tier1_batched = None, None, None, None, None
    if not args.core_only:
        kernels = kernels_section(ctx, stream, flush, cs, measured_peaks()[0])
        tier1_batched = tier1_batched_section(ctx, stream, flush, os.cpu_count() or 1)
        encode = encode_section(ctx, img)
        # the mixed-size batch at its stated size: batched waves vs per-image plans
        from thousandthchicken_b200.synth import c4_specs
        t0 = time.perf_counter()
        specs = c4_specs()
        mixed_streams = encode_mixed(ctx, specs)
        log(f"[rank {rank}] mixed batch: {len(specs)} images, {sum(map(len, mixed_streams)) / 1e9:.2f} GB of "
            f"codestreams in {time.perf_counter() - t0:.1f}s")
        batched = mixed_section(ctx, stream, specs, mixed_streams, os.cpu_count() or 1)

        # served decode: Poisson arrivals, continuous batching vs the per-image path
        served = serve_section(args, specs, mixed_streams, local_rank)

    if rank == 0:
        px = W * H
        value = px * args.steps * world / (total_ms / 1000.0) / 1e6
        hbm, peak_kind = measured_peaks()
        t1_avg = statistics.mean(t1_ms)
        dwt_avg = statistics.mean(dwt_ms)
        pool_bytes = len(cs)
        t1_bytes = pool_bytes + 4 * px * Cn
        dw_bytes = dwt_bytes(W, H, Cn, WORKLOAD["levels"])
        t1_gbs = t1_bytes / (t1_avg / 1000.0) / 1e9
        dwt_gbs = dw_bytes / (dwt_avg / 1000.0) / 1e9
        prof = {}
        tf = ROOT / "profiles" / "ncu_traffic.json"
        if tf.exists():
            prof = json.loads(tf.read_text())
        traffic = prof.get("t1_decode_warp_kernel_bytes_per_launch")
        inst = prof.get("t1_decode_warp_kernel_inst_per_launch")
        if prof.get("inst_workload") != f"{W}x{H}x{Cn}":
            inst = None   # counted on another size
        # Tier-1 is bound by instruction issue: one warp instruction per
        # cycle per SM sub-partition (148 SMs x 4) at the sampled SM clock
        sm_mhz = clocks.get("sm_mhz") or clocks.get("sm_max_mhz") or 1965.0
        issue_peak = 148 * 4 * sm_mhz * 1e6 / 1e9          # G warp instructions / s
        issue_achieved = inst / (t1_avg / 1000.0) / 1e9 if inst else None
        srt = sorted(step_ms)
        line = {
            "metric": METRIC, "value": round(value, 2), "unit": "Mpixel/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": round(total_ms / args.steps, 3), "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "fp32", "data": "synthetic",
            "config": workload_config(ncblk),
            "timing": {"codestream_bytes": pool_bytes, "l2": "256 MiB flush between steps, outside the timed events",
                       "parallelism": f"replicas x{world} (no collective)"},
            "latency_ms": {"p50": round(srt[len(srt) // 2], 3), "p99": round(srt[min(len(srt) - 1,
                                                                                    int(0.99 * len(srt)))], 3)},
            "stages_ms": {"tier1_dequant": round(t1_avg, 3), "dwt_colour": round(dwt_avg, 3)},
            "code_blocks_per_s": round(ncblk / (t1_avg / 1000.0), 1),
            "roofline": {"bound": "issue", "kernel": "t1_decode_warp_kernel",
                         "achieved": round(issue_achieved, 1) if issue_achieved else None,
                         "peak": round(issue_peak, 1), "unit": "G warp-instructions/s",
                         "frac": round(issue_achieved / issue_peak, 4) if issue_achieved else None,
                         "traffic": traffic, "inst_per_launch": inst,
                         "hbm": {"achieved": round(t1_gbs, 2), "peak": hbm, "unit": "GB/s",
                                 "frac": round(t1_gbs / hbm, 4), "peak_kind": peak_kind,
                                 "bytes": "codestream + 4 B per coefficient written"},
                         "note": "Tier-1 decodes the serial MQ chain of each code-block and is bound by instruction "
                                 "issue, not by HBM: achieved = warp instructions per launch (ncu "
                                 "smsp__inst_executed.sum of this workload, profiles/) / the live CUDA-event Tier-1 "
                                 "time; peak = 148 SMs x 4 issue slots x the sampled SM clock"},
            "dwt_roofline": {"bound": "hbm", "kernel": "reverse 9/7 levels (idwt_rev_kernel plane levels, idwt97_ict_tma_kernel last level)",
                             "achieved": round(dwt_gbs, 2), "peak": hbm, "unit": "GB/s",
                             "frac": round(dwt_gbs / hbm, 4), "bytes_per_step": dw_bytes, "peak_kind": peak_kind},
            "e2e": {"value": round(W * H * world / e2e_s / 1e6, 2), "unit": "Mpixel/s",
                    "h2d_bytes_per_step": pool_bytes + 40 * ncblk + 4 * ncblk,
                    "d2h_bytes_per_step": int(host_out.nbytes), "api": "tc_decode_j2k",
                    "mode": f"{n_pipe} images, {E2E_THREADS} host threads with a context each (pinned codestream in, "
                            "pinned samples out per image)",
                    "sequential_value": round(W * H * world / e2e_seq_s / 1e6, 2),
                    "outputs_identical": same_out},
            "gpu_launches": int(launches), "clocks": clocks, "psnr_db": round(psnr, 2),
            "wall_s_timed_region": round(wall, 3),
        }
        if batched is not None:
            line["batched_vs_per_image"] = batched
            line["served"] = served
            line["kernels"] = kernels
            line["encode"] = encode
            line["tier1_batched"] = tier1_batched
        if world == 1 and not args.no_cpu_baseline:
            line["parity"], line["cpu_baseline"] = oracle_check(_oracle(), cs, decoded, img, os.cpu_count() or 1)
        print(json.dumps(line), flush=True)
    plan.close()
    ctx.close()
    if dist:
        dist.barrier()
        dist.destroy_process_group()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--core-only", action="store_true",
                    help="report the headline workload only (no batched or served sections)")
    ap.add_argument("--serve-rates", default=SERVE_RATES,
                    help="served decode: Poisson arrival rates per second, comma-separated")
    ap.add_argument("--size", type=int, default=0,
                    help="square image side for a smaller case of the same workload (profiling)")
    ap.add_argument("--dwt-levels", type=int, default=0, metavar="N",
                    help="only time tc_dwt_reverse97 level by level on an N x N plane (profiling)")
    ap.add_argument("--dwt-depth", type=int, default=6, help="levels for --dwt-levels")
    ap.add_argument("--dwt-reps", type=int, default=7, help="timed runs per level count for --dwt-levels")
    ap.add_argument("--tier1", choices=["lossy", "lossless12"], default=None,
                    help="only time Tier-1 of one image of --size (default 4096): the bench's lossy coding, or "
                         "12-bit RCT + 5-level 5/3 (profiling)")
    args = ap.parse_args()
    if args.tier1:
        print(json.dumps(tier1_only(args.tier1, args.size or 4096)))
        return
    if args.dwt_levels:
        import torch
        from thousandthchicken_b200.stages import Context
        ctx = Context(0)
        flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
        res = dwt_levels(ctx, torch.cuda.current_stream(), flush, args.dwt_levels, args.dwt_depth,
                         measured_peaks()[0], reps=args.dwt_reps)
        print(json.dumps(res))
        return
    if args.size:
        WORKLOAD["width"] = WORKLOAD["height"] = args.size
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        run_reference(args, rank)
        return
    run_ours(args, rank, world, local_rank)


if __name__ == "__main__":
    main()
