#!/usr/bin/env python
"""Headline benchmark: batched greedy decode tok/s of the stories110M architecture (fp32) on
N B200s, sequences sharded over GPUs (replicated weights, no collective) -- the reference's headline
workload -- with the HBM roofline of the decode step and the reference's CPU path beside it.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--batch B] [--model s110m|7b] [--quant f32|q8]
    python bench.py --impl reference ...     # the reference's own CPU code (oracle/_ref) on the host cores

One "step" = one decode position for every one of the B slots of a GPU (one call of
thaDNN_s_forward_batch in the reference, src/thaDNN.cpp:13-81).

  value      tokens/s, everything resident in HBM: token/pos on the device, greedy argmax and
             slot bookkeeping on the device, one CUDA-graph replay per step.
  e2e        tokens/s through the reference-facing call (tha_forward_batch_*: HOST token[] /
             pos[] in, [B, vocab] logits into pinned HOST memory, host argmax), copies inside
             the timed region.
  roofline   algorithmic bytes of a decode step (weights once + KV rows read +
             KV rows written + embedding rows + logits) / measured step time, against the
             measured HBM copy bandwidth in MEASURED_PEAKS.json.
  cpu_baseline  oracle/_ref (the reference's run.cc / runq.c compiled unmodified) on the
             box's host cores, bounded sample.
Data is synthetic: seeded random-init weights of the named architecture (no network, no
checkpoint on the box), random prompt tokens.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import tempfile
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(ROOT, "tests"))

METRIC = "decode_tok_per_s"
UNIT = "tok/s"


def parse_args():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=256)
    ap.add_argument("--warmup", type=int, default=8)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--batch", type=int, default=int(os.environ.get("THA_BENCH_BATCH", "256")), help="slots per GPU")
    ap.add_argument("--model", default="s110m", choices=["s110m", "s15m", "7b"])
    ap.add_argument("--quant", default="f32", choices=["f32", "q8"])
    ap.add_argument("--seq-len", type=int, default=0, help="override the context length (KV slab size) of the architecture")
    ap.add_argument("--tp", type=int, default=1, help="tensor-parallel width (= WORLD_SIZE under torchrun): ONE replica split "
                    "over the GPUs, all-reduce fused into its consumer over NVLink peer memory (strong scaling)")
    ap.add_argument("--pos0", type=int, default=0, help="profiling aid: slots start at this position over a zero-filled KV cache "
                    "(same bytes and time per step as a real context of that length); the default 0 is the benchmark")
    ap.add_argument("--design", default="", choices=["", "timerax", "numizen", "bozovik", "mozetar", "logulix", "gavodra"], help="instead of the default workload: prompt and decode throughput of "
                    "this layer-program design at a few realistic layer sizes (random weights), beside the llama2 bf16 path at equal size")
    ap.add_argument("--design-sizes", default="w1024,w2048")
    ap.add_argument("--design-prompt", type=int, default=4096)
    ap.add_argument("--design-batch", type=int, default=64)
    ap.add_argument("--design-only", action="store_true", help="with --design: skip the llama2 arm")
    ap.add_argument("--kernels", action="store_true", help="with --design: print the per-kernel timeline of one prompt step and one "
                    "decode step (slower: an event after every launch) and skip the llama2 arm")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-extra", action="store_true", help="skip the bounded sub-records of the other configurations (extra.*)")
    ap.add_argument("--no-shares", action="store_true", help="skip the live-share measurement (roofline.live_shares_us)")
    ap.add_argument("--cpu-seconds", type=float, default=12.0, help="budget of the cpu_baseline sample")
    return ap.parse_args()


def model_config(name):
    from pkgload import load_pkg
    ck = load_pkg("checkpoint")
    return {"s110m": ck.STORIES110M, "s15m": ck.STORIES15M, "7b": ck.LLAMA2_7B}[name], ck


def model_label(name):
    return {"s110m": "stories110M", "s15m": "stories15M", "7b": "Llama-2-7B"}[name]


def measured_peak():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        return float(json.load(open(p))["hbm_gbs"]), "measured (MEASURED_PEAKS.json hbm_gbs)"
    except Exception:
        return 6650.0, "fallback (B200_PROFILING.md 6.65 TB/s)"


def measured_traffic(args):
    """dram__bytes_read.sum + dram__bytes_write.sum per decode step, from the committed ncu launch list of THIS
    configuration and THESE positions (profiles/traffic.json, keyed model/quant/B<slots>/pos<first>-<last>); None when
    that exact range was not captured (a capture at other positions says nothing about this step: the KV share differs)."""
    try:
        with open(os.path.join(ROOT, "profiles", "traffic.json")) as f:
            t = json.load(f)
        p0 = args.pos0 + args.warmup
        return t.get(f"{args.model}/{args.quant}/B{args.batch}/pos{p0}-{p0 + args.steps - 1}", {}).get("bytes_per_step")
    except OSError:
        return None


def step_bytes(cfg, weight_bytes, pos, B, elem_bytes_emb=4, write_logits=True):
    """ALGORITHMIC bytes of one decode step with every slot at position `pos`."""
    kv = 2 * cfg.n_layers * cfg.kv_dim * 4
    b = weight_bytes + B * (kv * (pos + 1) + kv) + B * cfg.dim * elem_bytes_emb
    if write_logits:
        b += B * cfg.vocab_size * 4
    return b


class ClockSampler:
    """nvidia-smi clocks / throttle reasons sampled DURING the timed region."""
    Q = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index=0):
        self.index, self.proc, self.lines = index, None, []

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "100"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except OSError:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self):
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        time.sleep(0.15)
        self.proc.terminate()
        try:
            self.proc.wait(timeout=2)
        except Exception:
            self.proc.kill()
        sm, mx, reasons, pw = [], [], set(), []
        for l in self.lines:
            f = [x.strip() for x in l.split(",")]
            if len(f) < 7:
                continue
            try:
                sm.append(float(f[0])); mx.append(float(f[1])); pw.append(float(f[2]))
            except ValueError:
                continue
            for name, v in zip(("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"), f[3:7]):
                if v.lower().startswith("active"):
                    reasons.add(name)
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "power_w_max": max(pw) if pw else None, "samples": len(sm), "reasons": sorted(reasons)}


# ------------------------------------------------------------------ model on the device ----
def build_weights(args, device):
    """Seeded random-init weights of the named architecture, resident in HBM.
    Returns (cfg, device weights, host weight dict or None)."""
    from pkgload import load_pkg
    import torch
    cfg, ck = model_config(args.model)
    eng = load_pkg("engine")
    if args.seq_len:
        import dataclasses
        cfg = dataclasses.replace(cfg, seq_len=args.seq_len)
    if args.model == "7b":
        # 26 GB of fp32 host RNG is too slow for a bench; fill on the device (same N(0, 0.02) law)
        return cfg, eng.device_random_weights(cfg, q8=(args.quant == "q8"), seed=1337, device=device), None
    w = ck.random_weights(cfg, seed=1337, std=0.02)
    if args.quant == "q8":
        gs = ck.v2_group_size(cfg)
        qt = {}
        for n in ck.V2_QORDER:
            t = w[n]
            if n == "tok_emb":
                q, s = ck.quantize_q80(t, gs)
                qt[n] = (q.reshape(t.shape), s)
            else:
                qs, ss = zip(*[ck.quantize_q80(t[l], gs) for l in range(cfg.n_layers)])
                qt[n] = (np.stack(qs).reshape(t.shape), np.stack(ss))
        qt["wcls"] = qt["tok_emb"]
        norms = {k: w[k] for k in ("rms_att", "rms_ffn", "rms_final")}
        return cfg, eng.DeviceWeightsQ8(cfg, gs, norms, qt, device=device), w
    return cfg, eng.DeviceWeights(cfg, w, device=device), w


def build_tp_rank(args, device, rank, tp):
    """This rank's shard of ONE replica split `tp` ways (hip_llama.cpp_b200/tp.py)."""
    from pkgload import load_pkg
    import dataclasses
    cfg, ck = model_config(args.model)
    eng, tpm = load_pkg("engine"), load_pkg("tp")
    if args.seq_len:
        cfg = dataclasses.replace(cfg, seq_len=args.seq_len)
    q8 = args.quant == "q8"
    host_w = None
    if args.model == "7b":
        dw = tpm.device_random_shard(cfg, tp, rank, q8, seed=1337, device=device)
    else:
        host_w = ck.random_weights(cfg, seed=1337, std=0.02)
        if q8:
            gs = ck.v2_group_size(cfg)
            qt = {}
            for n in ck.V2_QORDER:
                t = host_w[n]
                if n == "tok_emb":
                    q, s = ck.quantize_q80(t, gs)
                    qt[n] = (q.reshape(t.shape), s)
                else:
                    qs, ss = zip(*[ck.quantize_q80(t[l], gs) for l in range(cfg.n_layers)])
                    qt[n] = (np.stack(qs).reshape(t.shape), np.stack(ss))
            qt["wcls"] = qt["tok_emb"]
            lcfg, lqt = tpm.shard_q8(cfg, gs, qt, tp, rank)
            dw = eng.DeviceWeightsQ8(lcfg, gs, {k: host_w[k] for k in ("rms_att", "rms_ffn", "rms_final")}, lqt, device=device)
        else:
            lcfg, lw = tpm.shard_f32(cfg, host_w, tp, rank)
            dw = eng.DeviceWeights(lcfg, lw, device=device)
    e = tpm.TpRank(cfg, dw, tp, rank, args.batch, device=device)
    # for the byte count: a config whose kv_dim is this rank's share
    e.cfg_bytes = dataclasses.replace(cfg, n_kv_heads=cfg.n_kv_heads // tp)
    return cfg, dw, host_w, e


def run_ours(args, rank, world, local_rank):
    import torch
    import torch.distributed as dist
    from pkgload import load_pkg
    assert torch.cuda.is_available(), "bench.py needs a GPU (there is no CPU fallback)"
    torch.cuda.set_device(local_rank)
    device = f"cuda:{local_rank}"
    eng = load_pkg("engine")
    B, K, W = args.batch, args.steps, args.warmup
    tp = args.tp
    if tp > 1:
        if world != tp:
            raise SystemExit(f"--tp {tp} needs WORLD_SIZE == {tp} (torchrun --nproc-per-node {tp})")
        cfg, dw, host_w, e = build_tp_rank(args, device, rank, tp)
        e.connect_distributed()
    else:
        cfg, dw, host_w = build_weights(args, device)
    if args.pos0 + W + K + 1 > cfg.seq_len:
        raise SystemExit(f"pos0+warmup+steps must stay below seq_len={cfg.seq_len}")
    if tp == 1:
        e = eng.Engine(dw, B, device=device, with_att=False)
    wbytes = dw.nbytes()
    if tp > 1 and not e.q8:
        wbytes = sum(t.numel() * 4 for n, t in dw.t.items() if n not in ("wcls",))   # classifier == embedding table
    rng = np.random.default_rng(1234 + rank)
    tok0 = rng.integers(3, cfg.vocab_size, size=B).astype(np.int32)

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    # ---------------- resident loop: value + roofline ----------------
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        tok = torch.from_numpy(tok0).to(device)
        pos = torch.full((B,), args.pos0, dtype=torch.int32, device=device)
        nxt = torch.zeros(B, dtype=torch.int32, device=device)
        logits = torch.zeros(B, cfg.vocab_size, dtype=torch.float32, device=device)

        def step():
            if tp > 1:
                e.decode_step(tok, pos, logits, nxt, advance=True, stream=stream)
            else:
                e.decode_greedy(tok, pos, nxt, logits, stream=stream)

        for _ in range(W):
            step()
        stream.synchronize()
        launches_per_step = e.last_step_launches() + (1 if (e.q8 and tp == 1) else 0)
        sampler = ClockSampler(local_rank)
        barrier()
        if rank == 0:
            sampler.start()
        ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        ev0.record(stream)
        for _ in range(K):
            step()
        ev1.record(stream)
        stream.synchronize()
        barrier()
        clocks = sampler.stop() if rank == 0 else None
        ms = ev0.elapsed_time(ev1)
    ms_max = load_pkg("dp").max_over_ranks(ms, device)   # the job runs at the pace of its slowest rank
    value = (1 if tp > 1 else world) * B * K / (ms_max * 1e-3)
    if tp > 1 and e.check_error():
        raise SystemExit("tensor-parallel exchange: a wait on a peer timed out")
    # algorithmic bytes of the timed steps on this rank (positions W .. W+K-1); under --tp: this rank's shard
    # (its weights, the KV rows of its heads; embedding row, logits and classifier are replicated)
    cfg_b = e.cfg_bytes if tp > 1 else cfg
    total_bytes = sum(step_bytes(cfg_b, wbytes, p, B) for p in range(args.pos0 + W, args.pos0 + W + K))
    achieved = total_bytes / (ms * 1e-3) / 1e9
    peak, peak_src = measured_peak()

    # ---------------- where the timed step's time goes, live ----------------
    # One kernel class at a time is left out of the step (tha_set_option("skip", mask); graph + PDL stay on) over the
    # SAME positions; the difference to the full step is that class's live share.  The dominant class gets its own
    # roofline figures: algorithmic bytes per launch / live time per launch, and useful flops against the tensor peak.
    shares = None
    dominant = None
    if tp == 1 and not args.no_shares and launches_per_step > 1:
        try:
            lib = e.lib
            def timed(mask):
                lib.check(lib.c.tha_set_option(b"skip", mask), "skip")
                with torch.cuda.stream(stream):
                    pos.fill_(args.pos0); tok.copy_(torch.from_numpy(tok0).to(device))
                    for _ in range(W):
                        step()
                    a0, a1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                    a0.record(stream)
                    for _ in range(K):
                        step()
                    a1.record(stream)
                    stream.synchronize()
                return a0.elapsed_time(a1) * 1e3 / K
            full = timed(0)
            classes = (("layer_matmuls", 1), ("attention", 2), ("prep", 4), ("rope_scatter", 8), ("swiglu_or_quantise", 16),
                       ("classifier", 32), ("argmax", 64))
            shares = {"full_step": full}
            for name, mask in classes:
                shares[name] = max(0.0, full - timed(mask))
            lib.check(lib.c.tha_set_option(b"skip", 0), "skip")
            top = max((n for n, _ in classes), key=lambda n: shares[n])
            L, d, hd, kvd = cfg.n_layers, cfg.dim, cfg.hidden_dim, cfg.kv_dim
            elem = 1.0 + 4.0 / dw.gs if e.q8 else 4.0          # bytes per weight (Q8_0: int8 + one fp32 scale per group)
            layer_w = L * (2 * d * d + 2 * d * kvd + 3 * d * hd)
            mid = args.pos0 + W + K / 2.0
            # from 256 slots on the step runs as two concurrent half-batch branches: every kernel class launches twice
            # (the weights are still counted once: the second branch's read is an L2 hit)
            nb = 2 if launches_per_step > 12 * L else 1
            per = {"layer_matmuls": (4 * L * nb, layer_w * elem, 2.0 * B * layer_w),
                   "classifier": (nb, cfg.vocab_size * d * elem + B * cfg.vocab_size * 4, 2.0 * B * cfg.vocab_size * d),
                   "attention": (L * nb, B * 2 * kvd * 4 * (mid + 1) * L, 4.0 * B * d * (mid + 1) * L)}
            if top in per:
                n_launch, nbytes, flops = per[top]
                us = shares[top]
                try:
                    tf_peak = float(json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))["bf16_tflops_sustained"])
                except Exception:
                    tf_peak = 1381.0
                dominant = {"class": top, "launches_per_step": n_launch, "concurrent_branches": nb, "live_us_per_step": us,
                            "live_us_per_launch": us / n_launch * nb,   # two branches run side by side: a launch lasts twice its share
                            "algorithmic_bytes_per_step": nbytes, "achieved_gbs": nbytes / us / 1e3, "hbm_frac": nbytes / us / 1e3 / peak,
                            "useful_tflops": flops / us / 1e6, "tensor_frac_of_sustained_bf16": flops / us / 1e6 / tf_peak,
                            "note": "live = step time with this class minus step time without it, same positions, graph + PDL on"}
        except Exception as ex:   # a diagnostic, never the reason a bench line is missing
            shares = {"error": str(ex)}
    attn = {"live_shares_us": shares, "dominant_kernel": dominant}

    # ---------------- e2e: the driver's step with HOST buffers ----------------
    # Headline: the call the shipped driver makes every step in the reference's DEFAULT mode (temperature 1.0, top-p 0.9,
    # src/llama.cpp:897-900): tha_forward_sample_* = thaDNN_s_forward_batch + sample() per slot, HOST token / pos / forced
    # token / reseed in, HOST next tokens out, sampler on the device.  Beside it: the greedy form (-t 0), and the reference's
    # own signature (B * vocab logits into pinned host memory + host argmax), which is PCIe-bound by construction
    # (32.8 MB per step at 256 slots).
    e2e = None
    if not args.no_e2e and tp == 1:
        torch.set_num_threads(max(1, host_cores() // max(world, 1)))
        Ke = min(K, 128)
        tok_h = tok0.copy()
        pos_h = np.zeros(B, np.int32)
        nx_h = np.zeros(B, np.int32)
        force_h = np.full(B, -1, np.int32)
        seeds = np.full(B, 314028, np.uint64)

        def loop(fn):
            tok_h[:] = tok0
            pos_h[:] = 0
            for i in range(W):
                fn(i)
            barrier()
            t0 = time.perf_counter()
            for i in range(Ke):
                fn(W + i)
            torch.cuda.synchronize()
            return load_pkg("dp").max_over_ranks(time.perf_counter() - t0, device)

        def sstep(i):
            e.forward_sample(tok_h, pos_h, force_h, seeds if i == 0 else None, 1.0, 0.9, nx_h, stream=stream)
            tok_h[:] = nx_h
            pos_h[:] += 1

        dts = loop(sstep)
        e2e = {"value": world * B * Ke / dts, "unit": UNIT, "h2d_bytes_per_step": int((3 * 4 + 8) * B),
               "d2h_bytes_per_step": int(4 * B), "steps": Ke,
               "api": "tha_forward_sample_%s (thaDNN_s_forward_batch + sample(): temperature 1.0, top-p 0.9, one xorshift* "
                      "stream per slot; softmax / top-p / coin on the device)" % args.quant}

        def gstep(i):
            e.forward_greedy(tok_h, pos_h, nx_h, stream=stream)
            tok_h[:] = nx_h
            pos_h[:] += 1

        dtg = loop(gstep)
        e2e["greedy_call"] = {"value": world * B * Ke / dtg, "unit": UNIT, "h2d_bytes_per_step": int(2 * 4 * B),
                              "d2h_bytes_per_step": int(4 * B), "api": "tha_forward_greedy_%s (forward + sample_argmax, -t 0)" % args.quant}
        lg_host = torch.empty(B, cfg.vocab_size, dtype=torch.float32).pin_memory()

        def estep(i):
            e.forward_batch(tok_h, pos_h, lg_host, stream=stream)   # H2D token/pos, step, D2H logits, sync
            tok_h[:] = lg_host.argmax(dim=1).numpy()                # greedy sampler on the host cores
            pos_h[:] += 1

        Kl, Ke = min(Ke, 32), min(Ke, 32)
        dtl = loop(estep)
        e2e["logits_call"] = {"value": world * B * Kl / dtl, "unit": UNIT, "h2d_bytes_per_step": int(2 * 4 * B),
                              "d2h_bytes_per_step": int(B * cfg.vocab_size * 4), "steps": Kl,
                              "api": "tha_forward_batch_%s (thaDNN_s_forward_batch: [B, vocab] logits to pinned host memory) + host argmax" % args.quant}
        del lg_host

    # ---------------- parity sample: the benchmarked engine against the reference's own code ----------------
    parity = None
    if tp == 1 and rank == 0 and host_w is not None and not args.no_cpu_baseline:
        try:
            parity = parity_sample(args, cfg, host_w, e, B)
        except Exception as ex:
            parity = {"error": str(ex)}
    return dict(cfg=cfg, value=value, ms_per_step=ms_max / K, achieved=achieved, peak=peak, peak_src=peak_src,
                bytes_per_step=total_bytes / K, wbytes=wbytes, clocks=clocks, e2e=e2e, parity=parity,
                launches=launches_per_step * K, launches_per_step=launches_per_step, host_w=host_w, attn=attn)


def parity_sample(args, cfg, host_w, e, B, n_slots=4, n_steps=8):
    """Untimed: the engine that was just benchmarked decodes n_steps teacher-forced positions from 0 (all B slots, random
    tokens); n_slots of them are replayed through oracle/_ref (run.cc / runq.c compiled unmodified) and compared."""
    from oracle_lib import Ref32, RefQ8, ref_available
    from pkgload import load_pkg
    ck = load_pkg("checkpoint")
    q8 = args.quant == "q8"
    kind = "q8" if q8 else "fp32"
    if not ref_available(kind):
        return {"error": "oracle/_ref not built"}
    rng = np.random.default_rng(4321)
    toks = rng.integers(3, cfg.vocab_size, size=(n_steps, B)).astype(np.int32)
    sample = sorted(set(int(x) for x in np.linspace(0, B - 1, n_slots)))
    with tempfile.TemporaryDirectory() as td:
        path = os.path.join(td, "model.bin")
        (ck.write_v2 if q8 else ck.write_v0)(path, cfg, host_w)
        ref = (RefQ8 if q8 else Ref32)()
        h0, _ = ref.open(path)
        hs = [h0] + [(ref.lib.refq8_clone if q8 else ref.lib.ref32_clone)(h0) for _ in sample[1:]]
        worst_abs = worst_rel = 0.0
        same_argmax = True
        for stp in range(n_steps):
            pos = np.full(B, stp, np.int32)
            got = e.forward_batch(toks[stp], pos).numpy()
            for h, b in zip(hs, sample):
                want = ref.forward(h, int(toks[stp, b]), stp, cfg.vocab_size)
                ad = np.abs(got[b] - want)
                worst_abs = max(worst_abs, float(ad.max()))
                worst_rel = max(worst_rel, float(ad.max() / max(np.abs(want).max(), 1e-30)))
                same_argmax = same_argmax and int(got[b].argmax()) == int(want.argmax())
    return {"slots": sample, "steps": n_steps, "max_abs_err": worst_abs, "max_err_over_max_logit": worst_rel,
            "argmax_identical": bool(same_argmax), "tolerance": "fp32: 1e-4 abs-or-rel (tests); Q8_0: see tests/test_gpu_baseline_shapes.py",
            "oracle": "oracle/_ref (%s compiled unmodified), untimed" % ("runq.c" if q8 else "run.cc")}


def resident_tok_s(e, cfg, B, W, K, device, pos0=0, seed=1):
    """tokens/s of the resident greedy loop (device token / pos / argmax / advance), CUDA events on the launching stream."""
    import torch
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        rng = np.random.default_rng(seed)
        tok = torch.from_numpy(rng.integers(3, cfg.vocab_size, size=B).astype(np.int32)).to(device)
        pos = torch.full((B,), pos0, dtype=torch.int32, device=device)
        nxt = torch.zeros(B, dtype=torch.int32, device=device)
        logits = torch.zeros(B, cfg.vocab_size, dtype=torch.float32, device=device)
        for _ in range(W):
            e.decode_greedy(tok, pos, nxt, logits, stream=stream)
        ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        ev0.record(stream)
        for _ in range(K):
            e.decode_greedy(tok, pos, nxt, logits, stream=stream)
        ev1.record(stream)
        stream.synchronize()
    ms = ev0.elapsed_time(ev1)
    return B * K / (ms * 1e-3), ms / K


def extra_records(args, device, peak):
    """Bounded sub-records of the configurations the headline line does not cover; a few
    seconds each, rank 0 of a data-parallel run, random-init weights generated on the device."""
    import dataclasses
    import gc
    import torch
    from pkgload import load_pkg
    eng, ck = load_pkg("engine"), load_pkg("checkpoint")
    out = {}

    def free():
        gc.collect()
        torch.cuda.empty_cache()

    def decode_record(cfg, dw, B, W, K, label):
        e = eng.Engine(dw, B, device=device, with_att=False)
        v, ms = resident_tok_s(e, cfg, B, W, K, device)
        nbytes = sum(step_bytes(cfg, dw.nbytes(), p, B) for p in range(W, W + K)) / K
        rec = {"workload": label, "value": v, "unit": UNIT, "ms_per_step": ms, "launches_per_step": e.last_step_launches() + (1 if e.q8 else 0),
               "bytes_per_step": nbytes, "achieved_gbs": nbytes / ms / 1e6, "hbm_frac": nbytes / ms / 1e6 / peak}
        del e
        free()
        return rec

    try:   # stories110M Q8_0
        cfg = ck.STORIES110M
        dw = eng.device_random_weights(cfg, q8=True, seed=1337, device=device)
        out["s110m_q8_B256"] = decode_record(cfg, dw, 256, 5, 20, "stories110M Q8_0 batched greedy decode, 256 slots, positions 5..24")
        out["s110m_q8_B1"] = decode_record(cfg, dw, 1, 5, 20, "stories110M Q8_0 greedy decode, 1 slot, positions 5..24")
        del dw
        free()
    except Exception as ex:
        out["s110m_q8"] = {"error": str(ex)}
    try:   # Llama-2-7B Q8_0 at 1 / 8 / 64 slots
        cfg = ck.LLAMA2_7B
        dw = eng.device_random_weights(cfg, q8=True, seed=1337, device=device)
        for B in (1, 8, 64):
            c = dataclasses.replace(cfg, seq_len=512) if B == 64 else cfg   # 64 slots x 2048 positions of fp32 KV is 137 GB
            dw.cfg = c
            out[f"7b_q8_B{B}"] = decode_record(c, dw, B, 4, 12, f"Llama-2-7B Q8_0 batched greedy decode, {B} slots, positions 4..15, "
                                               f"KV slab of {c.seq_len} positions")
        # the same 64 slots with the full 2048-position context: only possible with the PAGED cache (dense fp32 KV would be
        # 137 GB); pool = 8 blocks of 16 positions per slot
        c = cfg
        dw.cfg = c
        paged = eng.PagedKV(c, 64, n_blocks=64 * 8)
        tab = np.zeros((64, paged.nrow), np.int32)
        tab[:, :8] = ((np.arange(64)[:, None] * 8 + np.arange(8)[None, :]) * 37) % (64 * 8)   # scattered over the pool, one owner per block
        paged.set_table(tab)
        e = eng.Engine(dw, 64, device=device, with_att=False, paged=paged)
        v, ms = resident_tok_s(e, c, 64, 4, 12, device)
        out["7b_q8_B64_paged_seq2048"] = {"workload": "Llama-2-7B Q8_0, 64 slots, context 2048, PAGED KV cache (512 blocks of 16 positions = 8.6 GB "
                                                      "instead of a 137 GB slab), positions 4..15", "value": v, "unit": UNIT, "ms_per_step": ms}
        del e
        paged.close()
        del paged, dw
        free()
    except Exception as ex:
        out["7b_q8"] = {"error": str(ex)}
    try:   # Llama-2-7B fp32, prompt of 2048 positions in one pass + first decode steps
        cfg = dataclasses.replace(ck.LLAMA2_7B, seq_len=2304)   # room for decode positions behind the 2048-position prompt
        dw = eng.device_random_weights(cfg, q8=False, seed=1337, device=device)
        e = eng.Engine(dw, 1, device=device, with_att=False)
        rng = np.random.default_rng(0)
        T = 2048
        seqs = [(0, 0, rng.integers(3, cfg.vocab_size, size=T).astype(np.int32))]
        st = torch.cuda.Stream()
        logits = torch.zeros(1, cfg.vocab_size, device=device)
        nxt = torch.zeros(1, dtype=torch.int32, device=device)
        with torch.cuda.stream(st):
            e.prefill(seqs, logits, nxt, stream=st)
            st.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(st)
            reps = 3
            for _ in range(reps):
                e.prefill(seqs, logits, nxt, stream=st)
            e1.record(st)
            st.synchronize()
        ms = e0.elapsed_time(e1) / reps
        d, h, L, kvd = cfg.dim, cfg.hidden_dim, cfg.n_layers, cfg.kv_dim
        pmm = L * (2 * d * d + 2 * d * kvd + 3 * d * h)
        flops = 2.0 * T * pmm + 2.0 * L * T * T * d + 2.0 * cfg.vocab_size * d
        try:
            tf_peak = float(json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))["bf16_tflops_sustained"])
        except Exception:
            tf_peak = 1381.0
        out["prefill_7b_f32_2048"] = {"workload": "Llama-2-7B fp32, one prompt of 2048 positions through tha_prefill_f32 (tensor-core matmuls: three fp16 products of split operands)",
                                      "ms": ms, "prompt_tok_per_s": T / ms * 1e3, "useful_tflops": flops / ms / 1e9,
                                      "tensor_frac_of_sustained_bf16": flops / ms / 1e9 / tf_peak,
                                      "note": "useful flops = 2 * T * weights + causal attention; three fp16 MMAs of split operands per useful one"}
        v, msd = resident_tok_s(e, cfg, 1, 2, 8, device, pos0=T)
        nb = step_bytes(cfg, dw.nbytes(), T + 5, 1)
        out["decode_7b_f32_B1_after_prefill"] = {"workload": "Llama-2-7B fp32 greedy decode, 1 slot, positions 2050..2057", "value": v, "unit": UNIT,
                                                 "ms_per_step": msd, "achieved_gbs": nb / msd / 1e6, "hbm_frac": nb / msd / 1e6 / peak}
        del e
        free()
        e = eng.Engine(dw, 8, device=device, with_att=False)   # 8 slots x 2304 positions of fp32 KV: 19 GB
        v, msd = resident_tok_s(e, cfg, 8, 2, 8, device, pos0=5)
        nb = step_bytes(cfg, dw.nbytes(), 10, 8)
        out["7b_f32_B8"] = {"workload": "Llama-2-7B fp32 greedy decode, 8 slots, positions 7..14 (tensor-core row pipeline from five slots on)",
                            "value": v, "unit": UNIT, "ms_per_step": msd, "achieved_gbs": nb / msd / 1e6, "hbm_frac": nb / msd / 1e6 / peak}
        del e, dw
        free()
    except Exception as ex:
        out["prefill_7b_f32_2048"] = {"error": str(ex)}
    try:   # Llama-2-7B bf16: prompt of 2048 positions (tensor-core matmuls AND attention), decode at 1 and 64 slots
        cfg = dataclasses.replace(ck.LLAMA2_7B, seq_len=2304)
        dw = eng.DeviceWeightsBF16.random(cfg, seed=1337, device=device)
        e = eng.Engine(dw, 1, device=device, with_att=False)
        rng = np.random.default_rng(0)
        T = 2048
        seqs = [(0, 0, rng.integers(3, cfg.vocab_size, size=T).astype(np.int32))]
        st = torch.cuda.Stream()
        logits = torch.zeros(1, cfg.vocab_size, device=device)
        nxt = torch.zeros(1, dtype=torch.int32, device=device)
        with torch.cuda.stream(st):
            e.prefill(seqs, logits, nxt, stream=st)
            st.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(st)
            reps = 3
            for _ in range(reps):
                e.prefill(seqs, logits, nxt, stream=st)
            e1.record(st)
            st.synchronize()
        ms = e0.elapsed_time(e1) / reps
        d, h, L, kvd = cfg.dim, cfg.hidden_dim, cfg.n_layers, cfg.kv_dim
        flops = 2.0 * T * L * (2 * d * d + 2 * d * kvd + 3 * d * h) + 2.0 * L * T * T * d + 2.0 * cfg.vocab_size * d
        try:
            tf_peak = float(json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))["bf16_tflops_sustained"])
        except Exception:
            tf_peak = 1381.0
        out["prefill_7b_bf16_2048"] = {"workload": "Llama-2-7B bf16, one prompt of 2048 positions through tha_prefill_bf16 (tcgen05 kind::f16 matmuls "
                                                   "and prompt attention)", "ms": ms, "prompt_tok_per_s": T / ms * 1e3,
                                       "useful_tflops": flops / ms / 1e9, "tensor_frac_of_sustained_bf16": flops / ms / 1e9 / tf_peak}
        v, msd = resident_tok_s(e, cfg, 1, 2, 8, device, pos0=T)
        nb = step_bytes(cfg, dw.nbytes(), T + 5, 1, elem_bytes_emb=2)
        out["decode_7b_bf16_B1_after_prefill"] = {"workload": "Llama-2-7B bf16 greedy decode, 1 slot, positions 2050..2057", "value": v, "unit": UNIT,
                                                  "ms_per_step": msd, "achieved_gbs": nb / msd / 1e6, "hbm_frac": nb / msd / 1e6 / peak}
        del e
        c64 = dataclasses.replace(ck.LLAMA2_7B, seq_len=512)
        dw.cfg = c64
        e = eng.Engine(dw, 64, device=device, with_att=False)
        v, msd = resident_tok_s(e, c64, 64, 4, 12, device)
        nb = sum(step_bytes(c64, dw.nbytes(), p_, 64, elem_bytes_emb=2) for p_ in range(4, 16)) / 12
        out["7b_bf16_B64"] = {"workload": "Llama-2-7B bf16 batched greedy decode, 64 slots, positions 4..15, KV slab of 512 positions", "value": v,
                              "unit": UNIT, "ms_per_step": msd, "achieved_gbs": nb / msd / 1e6, "hbm_frac": nb / msd / 1e6 / peak}
        del e, dw
        free()
    except Exception as ex:
        out["prefill_7b_bf16_2048"] = {"error": str(ex)}
    return out


def tp_extra(args, rank, world, local_rank, B=64, W=3, K=10):
    """Llama-2-7B Q8_0, ONE replica split over the `world` GPUs of this run (all-reduce after wo / w2 fused into its
    consumer over NVLink peer memory), 64 slots, KV slab of 512 positions: tok/s (strong scaling against extra.7b_q8_B64
    of the 1-GPU line).  Every rank takes part; rank 0 reports."""
    import argparse as _ap
    import gc
    import torch
    from pkgload import load_pkg
    device = f"cuda:{local_rank}"
    a2 = _ap.Namespace(model="7b", quant="q8", seq_len=512, batch=B)
    cfg, dw, _, e = build_tp_rank(a2, device, rank, world)
    e.connect_distributed()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        tok = torch.full((B,), 17, dtype=torch.int32, device=device)
        pos = torch.zeros(B, dtype=torch.int32, device=device)
        nxt = torch.zeros(B, dtype=torch.int32, device=device)
        logits = torch.zeros(B, cfg.vocab_size, dtype=torch.float32, device=device)
        for _ in range(W):
            e.decode_step(tok, pos, logits, nxt, advance=True, stream=stream)
        stream.synchronize()
        torch.distributed.barrier()
        torch.cuda.synchronize()
        ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        ev0.record(stream)
        for _ in range(K):
            e.decode_step(tok, pos, logits, nxt, advance=True, stream=stream)
        ev1.record(stream)
        stream.synchronize()
    ms = load_pkg("dp").max_over_ranks(ev0.elapsed_time(ev1), device)
    err = e.check_error()
    rec = {"workload": f"Llama-2-7B Q8_0, ONE replica tensor-parallel over {world} GPUs, {B} slots, positions {W}..{W + K - 1}",
           "value": B * K / (ms * 1e-3), "unit": UNIT, "ms_per_step": ms / K, "scaling": "strong", "peer_wait_timed_out": bool(err)}
    del e, dw
    gc.collect()
    torch.cuda.empty_cache()
    return rec


# ------------------------------------------------------------------ the reference's CPU path ----
class ReferenceMissing(RuntimeError):
    """The reference's own sources were not there to be compiled."""


def cpu_reference(args, cfg, host_w, n_seqs, n_threads, max_steps, warmup, budget_s):
    """Time oracle/_ref (run.cc / runq.c compiled unmodified; -O3 -mavx2 -mfma build) on the host.
    fp32: run.cc has no OpenMP pragma, so threads run independent sequences (one forward() each per
    step, the reference driver's one-thread-per-replica scheme); q8: runq.c's own OpenMP matmul.
    Returns (tok/s, steps timed, kind, threads used)."""
    from oracle_lib import Ref32, RefQ8, ref_available, cpu_has_avx2_fma
    from pkgload import load_pkg
    ck = load_pkg("checkpoint")
    q8 = args.quant == "q8"
    kindname = "q8" if q8 else "fp32"
    fast = cpu_has_avx2_fma() and ref_available(kindname, fast=True)
    if not ref_available(kindname, fast=fast):
        raise ReferenceMissing("oracle/_ref is not built (run __graft_entry__.build() where the reference's sources are)")
    if host_w is None:
        host_w = ck.random_weights(cfg, seed=1337, std=0.02)
    with tempfile.TemporaryDirectory() as td:
        path = os.path.join(td, "model.bin")
        (ck.write_v2 if q8 else ck.write_v0)(path, cfg, host_w)
        ref = (RefQ8 if q8 else Ref32)(fast=fast)
        h0, _ = ref.open(path)
        hs = [h0] + [ref.lib.refq8_clone(h0) if q8 else ref.lib.ref32_clone(h0) for _ in range(n_seqs - 1)]
        rng = np.random.default_rng(1234)
        tok = rng.integers(3, cfg.vocab_size, size=n_seqs).astype(np.int32)
        pos = np.zeros(n_seqs, np.int32)
        vocab = cfg.vocab_size
        import ctypes as C

        def one_step():
            ref.forward_many(hs, tok, pos, n_threads)
            for i, h in enumerate(hs):   # greedy sampler (sample_argmax, run.cc:619-630)
                lg = ref.lib.refq8_state_ptr(h, 7) if q8 else ref.lib.ref32_state_ptr(h, 7)
                tok[i] = (ref.lib.refq8_argmax if q8 else ref.lib.ref32_argmax)(lg, vocab)
            pos[:] += 1

        if q8:
            ref.lib.refq8_argmax.restype = C.c_int
            ref.lib.refq8_argmax.argtypes = [C.POINTER(C.c_float), C.c_int]
        for _ in range(warmup):
            one_step()
        t0 = time.perf_counter()
        done = 0
        while done < max_steps:
            one_step()
            done += 1
            if budget_s and time.perf_counter() - t0 > budget_s:
                break
        dt = time.perf_counter() - t0
    return n_seqs * done / dt, done, ("reference" if True else "port"), n_threads, fast


def host_cores():
    try:
        return len(os.sched_getaffinity(0))
    except AttributeError:
        return os.cpu_count() or 1


def base_line(args, cfg, world):
    B = args.batch
    return {
        "metric": METRIC, "unit": UNIT, "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "f32" if args.quant == "f32" else "int8+f32", "data": "synthetic",
        "config": {
            "workload": f"{model_label(args.model)} {'fp32' if args.quant == 'f32' else 'Q8_0'} batched greedy decode, "
                        f"{B} slots per {'replica' if args.tp > 1 else 'GPU'}, positions {args.pos0 + args.warmup}..{args.pos0 + args.warmup + args.steps - 1}, "
                        + (f"ONE replica tensor-parallel over {args.tp} GPUs (all-reduce after wo / w2 fused into its consumer over "
                           "NVLink peer memory)" if args.tp > 1 else "sequences sharded over GPUs (replicated weights, no collective)"),
            "batch_per_gpu": B, "global_batch": B * (1 if args.tp > 1 else world), "parallelism": (f"tp{args.tp}" if args.tp > 1 else f"dp{world}"), "vocab": cfg.vocab_size, "seq_len": cfg.seq_len,
            "weights": "seeded random-init N(0,0.02) of the named architecture",
            "l2": "inputs larger than L2 (weights read once per step: %d MB > 126 MB L2); no flush" %
                  (0,),
        },
    }


def main():
    args = parse_args()
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if args.design:
        if rank != 0:
            return 0
        if args.kernels:
            os.environ["THA_TRACE"] = "1"
        from pkgload import load_pkg
        bd = load_pkg("bench_designs")
        res = bd.run(load_pkg, args.design_sizes.split(","), prompt_len=args.design_prompt, batch=args.design_batch, steps=max(4, min(args.steps, 32)),
                     warmup=max(3, min(args.warmup, 8)), kernels=args.kernels, llama=not (args.kernels or args.design_only), design=args.design)
        print(json.dumps({"design": args.design, "dtype": "bf16", "data": "synthetic (random weights)", "n_gpus": 1,
                          "timing": "wall clock around the engine's step call (rows up, wanted logits back, stream synchronised), median",
                          "sizes": res}))
        return 0
    cfg, _ = model_config(args.model)

    if args.impl == "reference":
        if rank != 0:
            return 0
        cores = host_cores()
        n_seqs = min(args.batch * max(world, 1), 2 * cores)
        threads = cores if args.quant == "q8" else min(cores, n_seqs)
        try:
            v, done, kind, used, fast = cpu_reference(args, cfg, None, n_seqs, threads, args.steps, min(args.warmup, 2), 150.0)
        except ReferenceMissing as ex:
            print(json.dumps({"impl": "reference", "unavailable": str(ex)}), flush=True)
            return 0
        line = base_line(args, cfg, world)
        sample = (f"{n_seqs} sequences x {done} greedy decode positions from pos 0 through oracle/_ref "
                  f"({'runq.c' if args.quant == 'q8' else 'run.cc'} compiled unmodified, "
                  f"{'-O3 -mavx2 -mfma' if fast else '-O2'}), {used} host threads")
        line.update({"impl": "reference", "value": v, "ms_per_step": 1e3 * n_seqs / v, "steps": done,
                     "cpu_baseline": {"value": v, "unit": UNIT, "cores": used, "kind": kind, "sample": sample},
                     "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
                     "gpu_launches": 0})
        line["config"]["l2"] = "n/a (CPU)"
        print(json.dumps(line), flush=True)
        return 0

    import torch
    import torch.distributed as dist
    if world > 1:
        os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
        torch.cuda.set_device(local_rank)
        dist.init_process_group("nccl", device_id=torch.device(f"cuda:{local_rank}"))
    r = run_ours(args, rank, world, local_rank)
    tp_rec = None
    if world > 1 and args.tp == 1 and not args.no_extra and args.model == "s110m" and args.quant == "f32":
        # the optional tensor-parallel split (Llama-2-7B 2/4/8-way), one replica over all ranks of this run
        try:
            tp_rec = tp_extra(args, rank, world, local_rank)
        except Exception as ex:
            tp_rec = {"error": str(ex)}
    if rank == 0:
        cfg = r["cfg"]
        line = base_line(args, cfg, world)
        if args.tp > 1:
            line["scaling"] = "strong"
        line["config"]["l2"] = ("inputs larger than L2: %.0f MB of weights streamed once per step vs 126 MB L2; no flush"
                                % (r["wbytes"] / 1e6)) if r["wbytes"] > 126e6 else \
            "weights (%.0f MB) fit the 126 MB L2: number is L2-assisted, not an HBM figure" % (r["wbytes"] / 1e6)
        line.update({"value": r["value"], "ms_per_step": r["ms_per_step"], "e2e": r["e2e"],
                     "gpu_launches": r["launches"], "clocks": r["clocks"]})
        line["roofline"] = {"bound": "hbm", "achieved": r["achieved"], "peak": r["peak"], "unit": "GB/s",
                            "frac": r["achieved"] / r["peak"], "traffic": measured_traffic(args),
                            "kernel": ("mega_step_kernel (whole decode step, 1 persistent launch)" if r["launches_per_step"] == 1 else
                                       "decode step (%d kernels per step, CUDA-graph replay)" % r["launches_per_step"]),
                            "bytes_per_step": r["bytes_per_step"], "peak_source": r["peak_src"],
                            "frac_of_nominal_8TBs": r["achieved"] / 8000.0,
                            "live_shares_us": r["attn"]["live_shares_us"], "dominant_kernel": r["attn"]["dominant_kernel"]}
        if r.get("parity") is not None:
            line["parity_sample"] = r["parity"]
        if not args.no_cpu_baseline:
            try:
                if args.model == "7b":
                    raise RuntimeError("7B CPU sample skipped (26 GB checkpoint on tmpfs)")
                nth = 1 if args.quant == "f32" else host_cores()
                v, done, kind, used, fast = cpu_reference(args, cfg, r["host_w"], 1, nth, 256, 1, args.cpu_seconds)
                line["cpu_baseline"] = {"value": v, "unit": UNIT, "cores": used, "kind": kind,
                                        "sample": f"1 sequence x {done} greedy decode positions from pos 0, oracle/_ref "
                                                  f"({'runq.c' if args.quant == 'q8' else 'run.cc'} unmodified, "
                                                  f"{'-O3 -mavx2 -mfma' if fast else '-O2'}); run.cc has no OpenMP pragma"}
            except Exception as ex:  # the oracle being absent must not hide the GPU number
                line["cpu_baseline"] = {"value": None, "unit": UNIT, "cores": 0, "kind": "reference", "sample": f"unavailable: {ex}"}
        if tp_rec is not None:
            line.setdefault("extra", {})["tp_7b_q8_B64"] = tp_rec
        if not args.no_extra and args.tp == 1 and world == 1 and args.model == "s110m" and args.quant == "f32":
            try:
                import torch
                line.setdefault("extra", {}).update(extra_records(args, f"cuda:{local_rank}", r["peak"]))
            except Exception as ex:
                line.setdefault("extra", {})["error"] = str(ex)
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
