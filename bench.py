#!/usr/bin/env python3
"""Benchmark of the cudaCompress hot path on B200.

Workload (default): the 3-component 256^3 float32 vector field - each
component a seeded k^(-5/3) random-phase field (1024 modes, |k| <= 64, unit
std) - compressed with the lossy volume codec (3-level CDF 9/7 DWT, deadzone
quantization with step 0.01*std, zero-run RLE + Huffman, coding block 128)
and decompressed again.  One step = encode + decode of all 3 components
through the batched codec (one batch of 3 volumes, each stream byte-identical
to the plain single-volume codec's, replayed as CUDA graphs).

  value   raw field bytes / step time, inputs and outputs resident in HBM
          (GB/s raw, encode+decode), with consecutive steps in flight on 1-3
          batches (each on its own stream; the count chosen by a short
          untimed trial, `in_flight_batches`); latency_ms_per_step is one step
          at a time, and encode_gbs / decode_gbs split that sequential step;
          plain_path_ms_per_step times the per-component plain codec
  e2e     the same through the public API with host buffers: H2D of the
          fields, D2H of the streams (to page-locked host memory), H2D of the
          streams, D2H of the reconstructions, every step, inside the timed
          region; steps are software-pipelined (copy engines overlap the
          codec; consecutive steps alternate between two batches); the
          median of three runs of max(40, K) steps, all three in the line
  q0_sweep  the vector field at q0 in {0.002, 0.01, 0.05} std: per q0 the
          compression ratio, PSNR per component, encode / decode GB/s raw of
          one step at a time, and the FP32-vs-FP64 error of component 0
          (coefficients against the FP64 transform with the same taps,
          reconstruction against the FP64 inverse of the same symbols)
  batched_vs_per_brick  the 4096 uneven bricks (edges {16..64} per axis, q0
          log-uniform [0.002, 0.05]) in one batch vs one plain call per brick,
          coding block chosen by the autotuner
  serving the continuous-batching brick service at 10k req/s (Poisson, 90%
          decode, edges {32, 64, 128}): p50 / p99 latency, bricks/s
  roofline  the whole codec step against the measured HBM copy bandwidth:
          algorithmic bytes = raw + compressed bytes each way (intermediate
          passes do not count) over the in-flight step time; `traffic` is the
          step's DRAM bytes from ncu (profiles/traffic.json); beside it the
          step's dominant kernel section and every bandwidth section (CUDA
          events inside the library) with its own algorithmic bytes
  pipeline_roofline  the same fraction, plus encode and decode of one step
          at a time
  cpu_baseline  the reference's own CPU coder (src/CPU RunLengthCPU /
          HuffmanTableCPU / HuffmanCPU, built from the reference sources into
          oracle/_ref) plus the oracle's CPU DWT/quantize port (the reference
          has no CPU DWT), on one component, all host threads

Other workloads: --workload bricks-4096 (the full batched-bricks config; under
torchrun the brick set is partitioned across ranks by byte size, "scaling":
"strong"), --workload serving (1k / 10k / 50k req/s), --workload volume-128,
--workload heightfield-2048 (the lossless 2D codec, 2048^2 int16, 4 levels).
`--impl reference` times the CPU path as the reference arm.  Multi-GPU runs
(torchrun) are weak-scaling replicas: every rank codes its own field, no
collective on the data path; the time is the max over ranks.
"""
from __future__ import annotations

import argparse
import ctypes
import gc
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

WORKLOADS = {
    "vector-field-256": dict(n=256, comps=3, levels=3, q0=0.01, seeds=(1002, 1003, 1004), modes=1024, kmax=64,
                             desc="3 x 256^3 float32 k^-5/3 velocity, 3-level CDF 9/7, q0=0.01*std, RLE+Huffman cb=128"),
    "volume-128": dict(n=128, comps=1, levels=3, q0=0.01, seeds=(1000,), modes=512, kmax=32,
                       desc="128^3 float32 k^-5/3 field, 3-level CDF 9/7, q0=0.01*std, RLE+Huffman cb=128"),
}
WORKLOADS["bricks-4096"] = dict(count=4096, levels=2, seed=1005, plain_sample=256,
                                desc="4096 float32 bricks, edges {16,24,32,48,64} per axis, q0 log-uniform "
                                     "[0.002,0.05]*std, 2-level CDF 9/7, RLE+Huffman cb=128, per-brick tables")
WORKLOADS["serving"] = dict(rates=(1000.0, 10000.0, 50000.0), requests=100000, max_seconds=20.0,
                           edges=(32, 64, 128), decode_frac=0.9,
                           q0=0.01, levels=3, slots={32: 64, 64: 16, 128: 4}, bricks_per_edge=16, seed=1006,
                           desc="open-loop Poisson brick requests, 90% decode / 10% encode, cubic edge {32,64,128}, "
                                "q0=0.01*std, 3-level CDF 9/7, 4 GB HBM admission budget")
WORKLOADS["heightfield-2048"] = dict(n=2048, levels=4, seed=1001,
                                     desc="2048^2 int16 fBm terrain (10 octaves, H=0.8, [-2000, 8000]), 4-level "
                                          "CDF 5/3 integer DWT, lossless, RLE+Huffman cb=128")
FALLBACK_HBM_GBS = 6650.0
Q0_SWEEP = (0.002, 0.01, 0.05)
# sections that time a group of other sections (not one kernel)
COMPOSITE_SECTIONS = ("batch.lowpass_encode",)
SECTION_NOTES = {
    "lp.enc.table_build": "k_tableBuild: latency-bound, one CTA per Huffman table replaying libstdc++'s heap and "
                          "introsort exactly (sequential merge of ~1670 leaves per lowpass table)",
    "enc.table_build": "k_tableBuild: latency-bound (sequential libstdc++-order heap merge per table)",
}
L2_BYTES = 126 * 1024 * 1024


def load_peak():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(p) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    except Exception:
        return FALLBACK_HBM_GBS, "fallback"


class ClockSampler:
    """SM clock and throttle-reason samples taken during the timed region.
    The timed regions last tens of milliseconds, so NVML is polled from a
    thread every millisecond (read-only queries; the GPU is found by its PCI
    bus id, which CUDA_VISIBLE_DEVICES does not renumber); nvidia-smi at 200
    ms is the fallback."""
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
    NAMES = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")
    BITS = (0x8, 0x40, 0x20, 0x4)   # NVML clocks event reason bits, in NAMES order

    def __init__(self, gpu_index: int, period_s: float = 0.001):
        self.lines, self.samples = [], []
        self.proc, self.nvml = None, None
        self.period = period_s
        self._halt = threading.Event()
        try:
            import pynvml
            import torch
            pynvml.nvmlInit()
            try:
                pr = torch.cuda.get_device_properties(gpu_index)
                h = pynvml.nvmlDeviceGetHandleByPciBusId(
                    f"{pr.pci_domain_id:08x}:{pr.pci_bus_id:02x}:{pr.pci_device_id:02x}.0")
            except Exception:
                h = pynvml.nvmlDeviceGetHandleByIndex(gpu_index)
            self.nvml, self.h = pynvml, h
            self.max_mhz = float(pynvml.nvmlDeviceGetMaxClockInfo(h, pynvml.NVML_CLOCK_SM))
            self.thread = threading.Thread(target=self._poll, daemon=True)
            self.thread.start()
            return
        except Exception:
            self.nvml = None
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                                          "-lms", "200", "-i", str(gpu_index)], stdout=subprocess.PIPE,
                                         stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except Exception:
            self.proc = None

    def _poll(self):
        nv, h = self.nvml, self.h
        while not self._halt.is_set():
            try:
                sm = float(nv.nvmlDeviceGetClockInfo(h, nv.NVML_CLOCK_SM))
                rs = int(nv.nvmlDeviceGetCurrentClocksEventReasons(h))
                self.samples.append((sm, rs))
            except Exception:
                return
            time.sleep(self.period)

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self):
        if self.nvml is not None:
            self._halt.set()
            self.thread.join(timeout=2)
            sm = [a for a, _ in self.samples]
            reasons = {nm for _, rs in self.samples for nm, b in zip(self.NAMES, self.BITS) if rs & b}
            return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": self.max_mhz,
                    "reasons": sorted(reasons), "samples": len(sm), "source": "nvml, 1 ms"}
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        self.thread.join(timeout=2)
        sm, smax, reasons = [], [], set()
        for ln in self.lines:
            parts = [p.strip() for p in ln.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                smax.append(float(parts[2]))
            except ValueError:
                continue
            for nm, v in zip(self.NAMES, parts[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(smax) if smax else None,
                "reasons": sorted(reasons), "samples": len(sm), "source": "nvidia-smi, 200 ms"}


# ------------------------------------------------------------------ fields
def make_fields(wl, rank=0):
    from cudacompress_b200 import fields
    from cudacompress_b200.replicas import rank_seeds
    return [fields.turbulence_field(wl["n"], wl["modes"], wl["kmax"], s) for s in rank_seeds(wl["seeds"], rank)]


# -------------------------------------------------------------- CPU paths
def cpu_reference_step(vol, wl, threads):
    """Reference CPU coder on one component of the workload."""
    return cpu_reference_volume(vol, wl["levels"], wl["q0"], threads)


_ORACLE = []


def cpu_reference_volume(vol, L, q0, threads):
    """Reference CPU coder on one float32 volume (any z, y, x sizes): oracle
    DWT + quantize (the reference has no CPU DWT), the reference's own src/CPU
    RLE+Huffman for every band stream, then the inverse.  Returns
    (encode_s, decode_s, kind)."""
    sys.path.insert(0, os.path.join(ROOT, "tests"))
    from helpers import Oracle
    if not _ORACLE:
        _ORACLE.append(Oracle())
    orc = _ORACLE[0]
    orc.lib.orc_set_threads(threads)
    vol = np.ascontiguousarray(vol, np.float32)
    nz, ny, nx = vol.shape
    total = vol.size
    refcpu_path = os.path.join(ROOT, "oracle", "_ref", "libref_cpu.so")
    t0 = time.perf_counter()
    syms = np.zeros(total, np.uint16)
    orc.lib.orc_volume_symbols(vol, nx, ny, nz, L, q0, syms)
    if os.path.exists(refcpu_path):
        kind = "reference"
        ref = ctypes.CDLL(refcpu_path)
        vp = ctypes.c_void_p
        ref.refcpu_encode_rlhuff.restype = ctypes.c_long
        ref.refcpu_encode_rlhuff.argtypes = [vp, ctypes.c_uint32, ctypes.c_uint32, ctypes.c_uint32, ctypes.c_int, vp,
                                             ctypes.c_long, vp]
        ref.refcpu_decode_rlhuff.restype = ctypes.c_int
        ref.refcpu_decode_rlhuff.argtypes = [vp, vp, ctypes.c_uint32, ctypes.c_uint32, ctypes.c_uint32, ctypes.c_int, vp]
        # stream groups as the codec calls them: LP (1 stream), then per level
        # coarse->fine the 7 bands (equal sizes, contiguous)
        def band(shift):
            return (nx >> shift) * (ny >> shift) * (nz >> shift)
        groups = [(0, 1, band(L))]
        off = band(L)
        for l in range(L - 1, -1, -1):
            bn = band(l + 1)
            groups.append((off, 7, bn))
            off += 7 * bn
        outs = []
        for (o, S, cnt) in groups:
            cap = S * cnt * 2 + 4096 * S
            words = np.zeros(cap, np.uint32)
            sw = np.zeros(S, np.uint32)
            r = ref.refcpu_encode_rlhuff(syms[o:].ctypes.data, S, cnt, 128, threads, words.ctypes.data,
                                         ctypes.c_long(cap), sw.ctypes.data)
            assert r >= 0
            outs.append((words, sw, o, S, cnt))
        t1 = time.perf_counter()
        dec = np.zeros(total, np.uint16)
        for (words, sw, o, S, cnt) in outs:
            ref.refcpu_decode_rlhuff(words.ctypes.data, sw.ctypes.data, S, cnt, 128, threads, dec[o:].ctypes.data)
        rec = np.zeros(vol.shape, np.float32)
        orc.lib.orc_volume_from_symbols(dec, rec, nx, ny, nz, L, q0)
        t2 = time.perf_counter()
        assert np.array_equal(dec, syms), "reference CPU coder round trip mismatch"
        return t1 - t0, t2 - t1, kind
    kind = "port"
    words, bits = orc.compress_volume(vol, L, q0)
    t1 = time.perf_counter()
    orc.decompress_volume(words, bits, vol.shape, L, q0)
    t2 = time.perf_counter()
    return t1 - t0, t2 - t1, kind


def reference_line(args, wl, value, unit, step_s, kind, threads, sample):
    return {
        "impl": "reference", "metric": METRIC, "value": value, "unit": unit, "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": step_s * 1e3, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {"workload": args.workload, "desc": wl["desc"], "sample": sample},
        "cpu_baseline": {"value": value, "unit": unit, "cores": threads, "kind": kind, "sample": sample},
        "e2e": {"value": value, "unit": unit, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }


def run_reference_bricks(args, wl, threads):
    """The reference CPU coder over a bounded sample of the brick set: each
    step codes the next 64 bricks one after another (encode + decode)."""
    from cudacompress_b200 import fields
    bricks, q = fields.brick_set(wl["count"], wl["seed"])
    per = 64
    kind = "port"
    k = 0

    def one_step():
        nonlocal k, kind
        t = 0.0
        raw = 0
        for _ in range(per):
            b = bricks[k % len(bricks)]
            e, d, kind = cpu_reference_volume(b, wl["levels"], float(q[k % len(bricks)]), threads)
            t += e + d
            raw += b.size * 4
            k += 1
        return t, raw

    for _ in range(args.warmup):
        one_step()
    tt, rr = 0.0, 0
    for _ in range(args.steps):
        t, r = one_step()
        tt += t
        rr += r
    value = rr / tt / 1e9
    print(json.dumps(reference_line(args, wl, value, "GB/s", tt / args.steps, kind, threads,
                                    f"{per} bricks per step, encode+decode one brick at a time")), flush=True)


def run_reference_serving(args, wl, threads):
    """The reference CPU coder serving the same request mix one request at a
    time (encode: code the source brick; decode: decode its stream), bricks/s
    over a bounded sample of 200 requests per step."""
    from cudacompress_b200 import fields, serving
    rng = np.random.default_rng(wl["seed"])
    src = fields.turbulence_field(128, 1024, 64, wl["seed"])
    sources = {}
    for e in wl["edges"]:
        bl = []
        for _ in range(wl["bricks_per_edge"]):
            o = [int(rng.integers(0, 128 - e + 1)) for _ in range(3)]
            bl.append(np.ascontiguousarray(src[o[0]:o[0] + e, o[1]:o[1] + e, o[2]:o[2] + e]))
        sources[e] = bl
    per = 200
    reqs = serving.poisson_requests(per * (args.steps + args.warmup), 1e12, wl["edges"], wl["decode_frac"],
                                    wl["bricks_per_edge"], wl["seed"] + 2)
    kind = "port"

    def one_step(chunk):
        nonlocal kind
        t = 0.0
        for r in chunk:
            e, d, kind = cpu_reference_volume(sources[r.edge][r.brick], wl["levels"], wl["q0"], threads)
            t += e if r.op == serving.ENCODE else d
        return t

    for w in range(args.warmup):
        one_step(reqs[w * per:(w + 1) * per])
    tt = 0.0
    for st in range(args.steps):
        a = (args.warmup + st) * per
        tt += one_step(reqs[a:a + per])
    value = per * args.steps / tt
    print(json.dumps(reference_line(args, wl, value, "bricks/s", tt / args.steps, kind, threads,
                                    f"{per} requests per step, one at a time")), flush=True)


def run_reference(args, wl):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    threads = os.cpu_count() or 1
    if args.workload.startswith("bricks"):
        return run_reference_bricks(args, wl, threads)
    if args.workload == "serving":
        return run_reference_serving(args, wl, threads)
    if args.workload.startswith("heightfield"):
        from cudacompress_b200 import fields
        img = fields.fbm_heightfield(wl["n"], wl["seed"])
        for _ in range(args.warmup):
            cpu_reference_heightfield(img, wl["levels"])
        times = [sum(cpu_reference_heightfield(img, wl["levels"])) for _ in range(args.steps)]
        step = sum(times) / len(times)
        value = wl["n"] ** 2 * 2 / step / 1e9
        line = reference_line(args, wl, value, "GB/s", step, "port", 1,
                              f"the whole {wl['n']}^2 field per step, oracle port (one thread)")
        line["dtype"] = "int16"
        print(json.dumps(line), flush=True)
        return
    vols = make_fields(wl)
    # every step codes every component of the workload (encode + decode); the
    # warm-up steps code component 0 only
    for _ in range(args.warmup):
        cpu_reference_step(vols[0], wl, threads)
    times = []
    kind = "port"
    for _ in range(args.steps):
        t = 0.0
        for v in vols:
            e, d, kind = cpu_reference_step(v, wl, threads)
            t += e + d
        times.append(t)
    raw = wl["n"] ** 3 * 4 * len(vols)
    step = sum(times) / len(times)
    value = raw / step / 1e9
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": "GB/s", "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": step * 1e3, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {"workload": args.workload, "desc": wl["desc"], "sample": "all components per step"},
        "cpu_baseline": {"value": value, "unit": "GB/s", "cores": threads, "kind": kind,
                         "sample": f"all {wl['comps']} components ({wl['n']}^3 f32) encode+decode per step"},
        "e2e": {"value": value, "unit": "GB/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


METRIC = "enc/dec GB/s raw (%HBM peak); batched vs per-brick GB/s at fixed PSNR; p99"


# ---------------------------------------------------------- section bytes
# per-unit algorithmic bytes of the sections the roofline may pick
SECTION_UNITS = {
    "batch.dwt_forward": "per level (one fused k_bLevelFwd launch): the level's input read once (4 B/voxel) and "
                         "its outputs written once: 7 highpass octants as 2-byte symbols, the lowpass octant as "
                         "float (4 B) or, at the coarsest level, as 2-byte symbols",
    "batch.dwt_inverse": "per level (two launches: k_bSymbolCols, k_bPlanes): the level's inputs "
                         "read once (2 B/highpass symbol, 4 B/lowpass voxel) and its output written once "
                         "(4 B/voxel); the intermediate passes' traffic is not credited",
}


def section_bytes(name, wl, coded_bytes, counts):
    """Compulsory HBM bytes of one timed section over one step (algorithmic:
    each launch's inputs read once, its outputs written once)."""
    n, L, C = wl["n"], wl["levels"], wl["comps"]
    vols = [(n >> l) ** 3 for l in range(L)]
    hp = sum(7 * v // 8 for v in vols)
    lp = vols[-1] // 8
    m = {
        "pipe.dwt_forward": sum(8 * v for v in vols) * C,
        "batch.dwt_forward": sum(4 * v + 2 * (7 * v // 8) + (2 if i == len(vols) - 1 else 4) * (v // 8)
                                 for i, v in enumerate(vols)) * C,
        "batch.dwt_inverse": sum(4 * (v // 8) + 2 * (7 * v // 8) + 4 * v for v in vols) * C,
        "batch.quantize": (hp + lp) * 6 * C,
        "pipe.dwt_inverse": sum(4 * v // 8 + 2 * (7 * v // 8) + 4 * v for v in vols) * C,
        "pipe.quantize": (hp + lp) * 6 * C,
        "enc.rle_summary": hp * 2 * C,
        "enc.summary": hp * 2 * C,
        "enc.rle_write_hist": hp * 2 * C + counts.get("compact", 0) * 4,
        "enc.histogram": lp * 2 * C,
        "enc.block_bits": 2 * counts.get("compact", 0) * 2,
        "enc.pack": 2 * counts.get("compact", 0) * 2 + coded_bytes,
        "lp.enc.summary": lp * 2 * C,
        "lp.enc.rle_write_hist": lp * 2 * C,
        "lp.enc.block_bits": lp * 2 * C,
        "lp.enc.pack": lp * 2 * C + lp * C,
        "dec.huffman": lp * 2 * C,
        "dec.zero_counts": counts.get("compact", 0) * 2,
        "dec.symbols_scatter": counts.get("compact", 0) * 4 + hp * 2 * C,
    }
    return m.get(name)


# ---------------------------------------------------------------- bricks
def measure_bricks(count, levels, seed, steps, warmup, plain_sample, local, autotune=False):
    """Batched uneven bricks (one batch, CUDA graphs) against per-brick calls
    of the plain codec (cc_compress_volume_float / cc_decompress_volume_float
    one brick at a time) on the same bricks; both give the same streams and
    reconstructions, hence the same PSNR (checked on the sampled bricks)."""
    import torch
    import cudacompress_b200 as cc
    from cudacompress_b200 import fields
    dev = torch.device("cuda", local)
    bricks, q = fields.brick_set(count, seed)
    vols = [torch.from_numpy(b).to(dev) for b in bricks]
    raw = sum(b.size for b in bricks) * 4
    tuned = None
    cb, zc = 128, 0
    if autotune:
        from cudacompress_b200 import autotune as at
        cb, zc, tt = at.tune(local, vols, levels, [float(v) for v in q])
        tuned = {"coding_block": cb, "z_chunk": zc, "ms_per_pass": tt}
    inst = cc.Instance(local, 7, 32 ** 3, cb, 14)
    batch = cc.VolumeBatch(inst, [b.shape for b in bricks], levels, [float(v) for v in q], graph=True, z_chunk=zc)
    outs = [torch.empty_like(v) for v in vols]
    for _ in range(max(warmup, 1)):
        batch.compress(vols)
        batch.decompress(outs)
    batch.status()
    s0, e0 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    s0.record()
    for _ in range(steps):
        batch.compress(vols)
        batch.decompress(outs)
    e0.record()
    torch.cuda.synchronize()
    batch.status()
    batch_ms = s0.elapsed_time(e0) / steps
    # per-brick plain path on a sample (every brick a call of its own)
    P = min(plain_sample, count)
    pinst = inst if cb == 128 else cc.Instance(local, 7, 32 ** 3, 128, 14)
    cap = cc.volume_stream_capacity_words(64, 64, 64)
    words = torch.empty(cap, dtype=torch.int32, device=dev)
    pout = [torch.empty_like(vols[i]) for i in range(P)]

    def plain(i):
        _, b = cc.compress_volume_float(pinst, vols[i], levels, float(q[i]), words)
        cc.decompress_volume_float(pinst, pout[i], levels, float(q[i]), words, b)

    for i in range(min(P, 8)):
        plain(i)
    torch.cuda.synchronize()
    s1, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s1.record()
    for i in range(P):
        plain(i)
    e1.record()
    torch.cuda.synchronize()
    plain_ms_per_brick = s1.elapsed_time(e1) / P
    same = all(torch.equal(pout[i].view(torch.int32), outs[i].view(torch.int32)) for i in range(P))
    ps = [fields.psnr(bricks[i], outs[i].cpu().numpy()) for i in range(P)]
    bits = sum(batch.read_stream(i)[1] for i in range(min(count, 64)))
    batch.close()
    if pinst is not inst:
        pinst.close()
    inst.close()
    batched_bps = count / (batch_ms / 1e3)
    plain_bps = 1e3 / plain_ms_per_brick
    return {
        "bricks": count, "levels": levels, "raw_bytes": raw,
        "batched_ms_per_pass": batch_ms, "batched_bricks_per_s": batched_bps,
        "batched_gbs_raw": raw / (batch_ms / 1e3) / 1e9,
        "per_brick_ms": plain_ms_per_brick, "per_brick_bricks_per_s": plain_bps,
        "per_brick_sample": P, "speedup": batched_bps / plain_bps,
        "same_reconstruction_on_sample": bool(same), "psnr_db_mean_sample": float(np.mean(ps)),
        "sample_bits_per_voxel": bits / sum(bricks[i].size for i in range(min(count, 64))),
        "autotune": tuned, "coding_block": cb, "z_chunk": zc or 32,
    }


def measure_serving(wl, local, requests=None, rates=None):
    """Open-loop Poisson runs of the continuous-batching brick service at
    each rate (p50/p99 arrival -> result latency, bricks/s) and an offline
    run of the same requests all arriving at once (batched throughput)."""
    import torch
    from cudacompress_b200 import fields, serving
    rng = np.random.default_rng(wl["seed"])
    src = fields.turbulence_field(128, 1024, 64, wl["seed"])
    sources = {}
    for e in wl["edges"]:
        bl = []
        for _ in range(wl["bricks_per_edge"]):
            o = [int(rng.integers(0, 128 - e + 1)) for _ in range(3)]
            bl.append(torch.from_numpy(np.ascontiguousarray(src[o[0]:o[0] + e, o[1]:o[1] + e, o[2]:o[2] + e]))
                      .cuda(local))
        sources[e] = bl
    srv = serving.BrickServer(local, sources, wl["slots"], wl["levels"], wl["q0"], budget_bytes=4 << 30)
    n = requests or wl["requests"]
    out = {"requests_per_rate": {}, "store_bytes": srv.store_bytes, "budget_bytes": srv.budget}
    warm = serving.poisson_requests(200, 1e9, wl["edges"], wl["decode_frac"], wl["bricks_per_edge"], wl["seed"] + 1)
    srv.run(warm)                     # captures the graphs of the common fill levels
    offline = serving.poisson_requests(min(n, 20000), 1e12, wl["edges"], wl["decode_frac"], wl["bricks_per_edge"],
                                       wl["seed"] + 2)
    out["offline"] = serving.latency_stats(srv.run(offline))
    for rate in (rates or wl["rates"]):
        # at most max_seconds of arrivals per rate (10^5 requests at 10k req/s)
        nr = min(n, int(rate * wl.get("max_seconds", 20.0)))
        out["requests_per_rate"][str(int(rate))] = nr
        # a short run at the same rate first: fill levels met only at this
        # rate get their graphs captured outside the measured run
        srv.run(serving.poisson_requests(max(200, nr // 10), rate, wl["edges"], wl["decode_frac"],
                                         wl["bricks_per_edge"], wl["seed"] + int(rate) + 7))
        reqs = serving.poisson_requests(nr, rate, wl["edges"], wl["decode_frac"], wl["bricks_per_edge"],
                                        wl["seed"] + int(rate))
        gc.collect()
        gc.disable()   # no collector pause inside the measured run
        try:
            done = srv.run(reqs)
        finally:
            gc.enable()
        st = serving.latency_stats(done)
        dec = [r for r in reqs if r.op == serving.DECODE and r.edge == min(wl["edges"])]
        if dec:
            lat = np.array([r.done - r.arrival for r in dec]) * 1e3
            st["p99_ms_single_brick_decode_edge%d" % min(wl["edges"])] = float(np.percentile(lat, 99))
        out["rate_%d" % int(rate)] = st
    srv.close()
    return out


def run_serving(args, wl):
    import torch
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    sampler = ClockSampler(local)
    r = measure_serving(wl, local)
    clocks = sampler.stop()
    best = max(v["bricks_per_s"] for k, v in r.items() if k.startswith("rate_"))
    line = {
        "metric": METRIC, "value": best, "unit": "bricks/s", "n_gpus": 1, "steps": 1, "warmup": 1,
        "ms_per_step": None, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic (seeded k^-5/3 random-phase fields)",
        "config": {"workload": args.workload, "desc": wl["desc"], "parallelism": "replicas1"},
        "serving": r, "clocks": clocks,
    }
    print(json.dumps(line), flush=True)


def run_bricks_partitioned(args, wl, world, rank, local):
    """The brick set split across ranks by byte size (no collective on the
    data path): each rank codes its share as one batch; the job's pass time
    is the max over ranks; compressed sizes are gathered on the host."""
    import datetime

    import torch
    import torch.distributed as dist
    import cudacompress_b200 as cc
    from cudacompress_b200 import fields, replicas
    dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    dev = torch.device("cuda", local)
    bricks, q = fields.brick_set(wl["count"], wl["seed"])
    sizes = [b.size * 4 for b in bricks]
    mine = replicas.partition_by_bytes(sizes, world)[rank]
    inst = cc.Instance(local, 7, 32 ** 3, 128, 14)
    batch = cc.VolumeBatch(inst, [bricks[i].shape for i in mine], wl["levels"], [float(q[i]) for i in mine],
                           graph=True) if mine else None
    vols = [torch.from_numpy(bricks[i]).to(dev) for i in mine]
    outs = [torch.empty_like(v) for v in vols]

    def one_pass():
        if batch is not None:
            batch.compress(vols)
            batch.decompress(outs)

    for _ in range(max(args.warmup, 1)):
        one_pass()
    torch.cuda.synchronize()
    dist.barrier()
    sampler = ClockSampler(local)
    s0, e0 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s0.record()
    for _ in range(args.steps):
        one_pass()
    e0.record()
    torch.cuda.synchronize()
    clocks = sampler.stop()
    ms = replicas.max_over_ranks([s0.elapsed_time(e0) / args.steps], dist, dev)[0]
    if batch is not None:
        batch.status()
    coded = replicas.gather_on_host({i: batch.read_stream(j)[1] for j, i in enumerate(mine)} if mine else {}, dist)
    raw = sum(sizes)
    if rank == 0:
        line = {
            "metric": METRIC, "value": raw / (ms / 1e3) / 1e9, "unit": "GB/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "strong",
            "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded k^-5/3 random-phase fields)",
            "config": {"workload": args.workload, "desc": wl["desc"],
                       "parallelism": f"bricks partitioned by bytes over {world} ranks",
                       "l2": f"inputs {raw >> 20} MiB per pass"},
            "compressed_bytes": sum(coded.values()) // 8, "bricks_coded": len(coded), "clocks": clocks,
        }
        print(json.dumps(line), flush=True)
    if batch is not None:
        batch.close()
    inst.close()
    dist.barrier()
    dist.destroy_process_group()


def run_bricks(args, wl):
    import torch
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    if world > 1:
        return run_bricks_partitioned(args, wl, world, rank, local)
    sampler = ClockSampler(local)
    r = measure_bricks(wl["count"], wl["levels"], wl["seed"], args.steps, args.warmup, wl["plain_sample"], local,
                       autotune=True)
    clocks = sampler.stop()
    ms = r["batched_ms_per_pass"]
    line = {
        "metric": METRIC, "value": r["batched_gbs_raw"], "unit": "GB/s", "n_gpus": 1, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded k^-5/3 random-phase fields)",
        "config": {"workload": args.workload, "desc": wl["desc"], "parallelism": "replicas1",
                   "l2": f"inputs {r['raw_bytes'] >> 20} MiB per pass"},
        "batched_vs_per_brick": r, "clocks": clocks,
    }
    print(json.dumps(line), flush=True)


# ---------------------------------------------------------------- ours
def pipelined_e2e(torch, batches, vols_h, vols, dev, C, cc, steps=None):
    """Times the codec end to end with host buffers (see run_ours): steps
    alternate between two batches (each with its own stream and buffers), so
    one step's stream round trip and decode overlap the next step's encode.
    Returns the device-timed ms per step, the stream bytes moved each way per
    step and whether the last reconstruction equals the device-resident
    path's."""
    steps = steps or 10
    nb = len(batches)
    s_in, s_out = torch.cuda.Stream(dev), torch.cuda.Stream(dev)
    s_comp = [torch.cuda.Stream(dev) for _ in range(nb)]
    inst_stream = [cc.lib().cc_get_instance_stream(b.inst.handle) for b in batches]
    for b, st in zip(batches, s_comp):
        b.set_stream(st)
    pinned_in = [torch.from_numpy(v).pin_memory() for v in vols_h]
    dev_in = [[torch.empty_like(v) for v in vols] for _ in range(nb)]
    rec = [[torch.empty_like(v) for v in vols] for _ in range(nb)]
    pinned_out = [[torch.empty(v.shape, dtype=torch.float32).pin_memory() for v in vols_h] for _ in range(nb)]
    cap = sum(cc.volume_stream_capacity_words(*v.shape[::-1]) for v in vols_h)
    h_words = [torch.empty(cap, dtype=torch.int32).pin_memory() for _ in range(nb)]
    h_ext = [torch.zeros(2 * C, dtype=torch.int64).pin_memory() for _ in range(nb)]
    ev_in, ev_in_free, ev_rec, ev_out = ([torch.cuda.Event() for _ in range(nb)] for _ in range(4))

    def one(k):
        b = k % nb
        sc, bt = s_comp[b], batches[b]
        with torch.cuda.stream(s_in):
            s_in.wait_event(ev_in_free[b])           # this slot's previous encode has read dev_in[b]
            for c in range(C):
                dev_in[b][c].copy_(pinned_in[c], non_blocking=True)
            ev_in[b].record(s_in)
        sc.wait_event(ev_in[b])
        bt.compress(dev_in[b])
        ev_in_free[b].record(sc)
        bt.download_streams(h_words[b], h_ext[b])
        bt.upload_streams(h_words[b], h_ext[b])
        sc.wait_event(ev_out[b])                     # this slot's previous reconstruction has left rec[b]
        bt.decompress(rec[b])
        ev_rec[b].record(sc)
        with torch.cuda.stream(s_out):
            s_out.wait_event(ev_rec[b])
            for c in range(C):
                pinned_out[b][c].copy_(rec[b][c], non_blocking=True)
            ev_out[b].record(s_out)

    for k in range(2 * nb):                          # warm-up
        one(k)
    torch.cuda.synchronize()
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    start.record(s_in)
    for st in s_comp + [s_out]:
        st.wait_stream(s_in)
    for k in range(steps):
        one(k)
    for st in s_comp + [s_out]:
        s_in.wait_stream(st)
    end.record(s_in)
    torch.cuda.synchronize()
    for b in batches:
        b.status()
    ms = start.elapsed_time(end) / steps
    last = (steps - 1) % nb
    ext = h_ext[last].numpy()
    stream_bytes = int(sum((int(ext[C + c]) + 31) // 32 for c in range(C)) * 4)
    # the last reconstruction against the device-resident path's
    for b, st in zip(batches, inst_stream):
        b.set_stream(st)
    ref = [torch.empty_like(v) for v in vols]
    batches[0].compress(vols)
    batches[0].decompress(ref)
    torch.cuda.synchronize()
    identical = all(torch.equal(pinned_out[last][c], ref[c].cpu()) for c in range(C))
    return {"ms": ms, "stream_bytes": stream_bytes, "identical": identical}


def cpu_reference_heightfield(img, L):
    """The oracle's port of the heightfield codec (the reference's CPU coder
    has no 2D integer DWT); one thread.  Returns (encode_s, decode_s)."""
    sys.path.insert(0, os.path.join(ROOT, "tests"))
    from helpers import Oracle
    if not _ORACLE:
        _ORACLE.append(Oracle())
    orc = _ORACLE[0]
    t0 = time.perf_counter()
    words, bits = orc.compress_heightfield(img, L)
    t1 = time.perf_counter()
    rec = orc.decompress_heightfield(words, bits, img.shape, L)
    t2 = time.perf_counter()
    assert np.array_equal(rec, img), "oracle heightfield round trip mismatch"
    return t1 - t0, t2 - t1


def run_heightfield(args, wl):
    """The lossless 2D heightfield codec (C1): one step = compress + decompress
    of one 2048^2 int16 terrain per rank (weak-scaling replicas), through
    cc_compress_heightfield / cc_decompress_heightfield; the decode is checked
    bit-exact every run."""
    import torch
    import cudacompress_b200 as cc
    from cudacompress_b200 import fields, replicas

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    dev = torch.device("cuda", local)
    n, L = wl["n"], wl["levels"]
    img_h = fields.fbm_heightfield(n, wl["seed"] + 100 * rank)
    img = torch.from_numpy(img_h).to(dev)
    # 5 streams of a level-0 band: room for every level's streams in one
    # decode call (the codec falls back to one call per level otherwise)
    inst = cc.Instance(local, 5, (n // 2) ** 2, 128, 14)
    words = torch.empty(n * n + 64 * 1024, dtype=torch.int32, device=dev)
    out = torch.empty_like(img)
    bits = [0]

    def step():
        _, b = cc.compress_heightfield(inst, img, L, words)
        cc.decompress_heightfield(inst, out, L, words, b)
        bits[0] = b

    for _ in range(max(args.warmup, 1)):
        step()
    torch.cuda.synchronize()
    if not torch.equal(out, img):
        raise RuntimeError("heightfield round trip is not lossless")
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    if dist:
        dist.barrier()
    torch.cuda.synchronize()
    launches0 = cc.lib().cc_kernel_launches()
    sampler = ClockSampler(local)
    start.record()
    for _ in range(args.steps):
        step()
    end.record()
    torch.cuda.synchronize()
    clocks = sampler.stop()
    launches = cc.lib().cc_kernel_launches() - launches0
    ms = replicas.max_over_ranks([start.elapsed_time(end) / args.steps], dist, dev)[0]
    raw = n * n * 2
    coded = (bits[0] + 7) // 8
    value = replicas.job_gbs(world, raw, ms)
    # end to end: image in from pinned host memory, stream out and back, image out
    pin_in = torch.from_numpy(img_h).pin_memory()
    pin_out = torch.empty_like(pin_in).pin_memory()
    pin_words = torch.empty(words.numel(), dtype=torch.int32).pin_memory()
    dimg, dwords = torch.empty_like(img), torch.empty_like(words)

    def e2e_step():
        dimg.copy_(pin_in, non_blocking=True)
        _, b = cc.compress_heightfield(inst, dimg, L, words)
        nw = (b + 31) // 32
        pin_words[:nw].copy_(words[:nw], non_blocking=True)
        dwords[:nw].copy_(pin_words[:nw], non_blocking=True)
        cc.decompress_heightfield(inst, out, L, dwords, b)
        pin_out.copy_(out, non_blocking=True)
        return nw * 4

    e2e_step()
    torch.cuda.synchronize()
    s2, e2 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s2.record()
    for _ in range(args.steps):
        nbytes = e2e_step()
    e2.record()
    torch.cuda.synchronize()
    if not torch.equal(pin_out, pin_in):
        raise RuntimeError("heightfield end-to-end round trip is not lossless")
    e2e_ms = replicas.max_over_ranks([s2.elapsed_time(e2) / args.steps], dist, dev)[0]
    # per-kernel sections of one extra step (event timing on)
    lib = cc.lib()
    lib.cc_reset_timings(inst.handle)
    lib.cc_set_timing(inst.handle, 1)
    step()
    torch.cuda.synchronize()
    sections = {}
    for i in range(lib.cc_timing_count(inst.handle)):
        name, t_ms, cnt = ctypes.c_char_p(), ctypes.c_double(), ctypes.c_uint32()
        lib.cc_timing_entry(inst.handle, i, ctypes.byref(name), ctypes.byref(t_ms), ctypes.byref(cnt))
        sections[name.value.decode()] = round(t_ms.value, 4)
    lib.cc_set_timing(inst.handle, 0)
    peak, peak_kind = load_peak()
    alg = 2 * (raw + coded)
    achieved = alg / (ms / 1e3) / 1e9
    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        e, d = cpu_reference_heightfield(img_h, L)
        cpu = {"value": raw / (e + d) / 1e9, "unit": "GB/s", "cores": 1, "kind": "port",
               "sample": f"the whole {n}^2 field, compress + decompress, oracle port (one thread)"}
    if rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": "GB/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "int16", "data": "synthetic (seeded fBm terrain)",
            "config": {"workload": args.workload, "desc": wl["desc"], "parallelism": f"replicas{world}",
                       "l2": f"input {raw >> 20} MiB per step fits L2 (latency-bound config)"},
            "compression_ratio": raw / max(coded, 1), "lossless": True,
            "e2e": {"value": replicas.job_gbs(world, raw, e2e_ms), "unit": "GB/s", "h2d_bytes_per_step": raw + nbytes,
                    "d2h_bytes_per_step": raw + nbytes},
            "gpu_launches": launches,
            "roofline": {"bound": "hbm", "kernel": "whole codec (raw + compressed bytes, both directions)",
                         "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
                         "peak_source": peak_kind, "traffic": None},
            "sections_ms": dict(sorted(sections.items(), key=lambda kv: -kv[1])),
            "clocks": clocks, "cpu_baseline": cpu,
        }
        print(json.dumps(line), flush=True)
    inst.close()
    if dist:
        dist.destroy_process_group()


def run_profile(args):
    """A small self-contained case for profilers (ncu): one batch of
    `--comps` seeded n^3 float32 fields (the vector field's generator and
    seeds), or with `--workload bricks-4096` the 4096 uneven bricks, `--warmup`
    encode + decode passes, then `--steps` more; no timing, no other legs.  Launch order per step: the forward transform (one fused
    launch per level, the quantizer included), the encoders, then the
    decoder and the inverse transform (three passes per level)."""
    import torch
    import cudacompress_b200 as cc
    from cudacompress_b200 import fields
    if args.workload == "bricks-4096":
        # the batched-vs-per-brick leg's brick set in one batch, at the
        # autotuner's usual choice (coding block 64, tile depth 64)
        wl = WORKLOADS["bricks-4096"]
        bricks, q = fields.brick_set(wl["count"], wl["seed"])
        vols = [torch.from_numpy(b).cuda() for b in bricks]
        outs = [torch.empty_like(v) for v in vols]
        with cc.Instance(0, 7, 32 ** 3, 64, 14) as inst:
            with cc.VolumeBatch(inst, [v.shape for v in vols], wl["levels"], [float(x) for x in q], graph=True,
                                z_chunk=64) as batch:
                for _ in range(args.warmup + args.steps):
                    batch.compress(vols)
                    batch.decompress(outs)
                torch.cuda.synchronize()
                batch.status()
        print(json.dumps({"profile_case": {"workload": args.workload, "passes": args.warmup + args.steps}}))
        return
    n, C = args.n, args.comps
    vols = [torch.from_numpy(fields.turbulence_field(n, 1024, min(64, n // 4), seed)).cuda()
            for seed in fields.SEED_C2[:C]]
    outs = [torch.empty_like(v) for v in vols]
    with cc.Instance(0, 7, (n // 2) ** 3, 128, 14) as inst:
        with cc.VolumeBatch(inst, [v.shape for v in vols], 3, [args.q0] * C, graph=True) as batch:
            for _ in range(args.warmup + args.steps):
                batch.compress(vols)
                batch.decompress(outs)
            torch.cuda.synchronize()
            batch.status()
    print(json.dumps({"profile_case": {"n": n, "comps": C, "q0": args.q0, "passes": args.warmup + args.steps}}))


def compact_count(cc, torch, vol, levels, q0):
    """Run-length output entries (nonzero symbols plus one (0, 255) entry per
    whole 256 zeros before them; RunLengthKernels.cui:5-45) of every highpass
    band of one volume: the compact-symbol count of its encoder.  Symbols
    from the library's own transform and quantizer."""
    from cudacompress_b200 import accuracy
    coef = accuracy.multilevel_fp32(vol, levels)
    nz, ny, nx = vol.shape
    total = 0
    for lvl in range(levels):
        step = float(np.float32(q0) / np.float32(1 << lvl))
        hz, hy, hx = nz >> (lvl + 1), ny >> (lvl + 1), nx >> (lvl + 1)
        sym = torch.empty((hz, hy, hx), dtype=torch.int16, device=vol.device)
        for b in range(1, 8):
            x0, y0, z0 = (b & 1) * hx, ((b >> 1) & 1) * hy, (b >> 2) * hz
            cc.quantize_to_symbols(sym, coef[z0:z0 + hz, y0:y0 + hy, x0:x0 + hx], hx, hy, hz, step, nx, nx * ny)
            idx = torch.nonzero(sym.reshape(-1)).reshape(-1)
            if idx.numel():
                prev = torch.cat([torch.tensor([-1], device=idx.device), idx[:-1]])
                total += int(idx.numel() + ((idx - prev - 1) // 256).sum())
    return total


def measure_q0_sweep(inst, vols, vols_h, levels, q0s, steps, warmup):
    """The vector field's quantization sweep: per q0 one batch of all
    components (CUDA graphs), sequential steps with encode and decode split by
    events; compression ratio, PSNR per component, GB/s raw, and the FP32 vs
    FP64 error of component 0 (cudacompress_b200.accuracy: coefficients
    against the FP64 transform, reconstruction against the FP64 inverse of the
    same symbols)."""
    import torch
    import cudacompress_b200 as cc
    from cudacompress_b200 import accuracy, fields
    C = len(vols)
    raw = sum(v.numel() for v in vols) * 4
    recon = [torch.empty_like(v) for v in vols]
    err = accuracy.error_report(inst, vols[0], levels, q0s)
    out = {"fp64_coefficients_component0": err["coefficients"]}
    for q0 in q0s:
        b = cc.VolumeBatch(inst, [v.shape for v in vols], levels, [q0] * C, graph=True)
        for _ in range(max(warmup, 1)):
            b.compress(vols)
            b.decompress(recon)
        evs = [[torch.cuda.Event(enable_timing=True) for _ in range(3)] for _ in range(steps)]
        torch.cuda.synchronize()
        for k in range(steps):
            evs[k][0].record()
            b.compress(vols)
            evs[k][1].record()
            b.decompress(recon)
            evs[k][2].record()
        torch.cuda.synchronize()
        b.status()
        enc_ms = sum(e[0].elapsed_time(e[1]) for e in evs) / steps
        dec_ms = sum(e[1].elapsed_time(e[2]) for e in evs) / steps
        coded = sum(b.read_stream(c)[1] for c in range(C)) / 8
        b.close()
        out[str(q0)] = {
            "compression_ratio": raw / coded, "bits_per_voxel": 8 * coded / (raw / 4),
            "psnr_db": [fields.psnr(vols_h[c], recon[c].cpu().numpy()) for c in range(C)],
            "encode_ms": enc_ms, "decode_ms": dec_ms, "gbs_raw": 2 * raw / ((enc_ms + dec_ms) / 1e3) / 1e9,
            "encode_gbs": raw / (enc_ms / 1e3) / 1e9, "decode_gbs": raw / (dec_ms / 1e3) / 1e9,
            "fp64_reconstruction_component0": err["reconstruction"][str(q0)],
        }
    return out


def run_ours(args, wl):
    import torch
    import cudacompress_b200 as cc
    from cudacompress_b200 import fields, replicas

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    dev = torch.device("cuda", local)
    n, L, q0, C = wl["n"], wl["levels"], wl["q0"], wl["comps"]
    vols_h = make_fields(wl, rank)
    vols = [torch.from_numpy(v).to(dev) for v in vols_h]
    inst = cc.Instance(local, 7, (n // 2) ** 3, 128, 14)
    # the batched codec: all components in one batch, the whole step replayed as CUDA graphs
    batch = cc.VolumeBatch(inst, [v.shape for v in vols], L, [q0] * C, graph=True)
    recon = [torch.empty_like(v) for v in vols]

    def step(ev=None):
        if ev is not None:
            ev[0].record()
        batch.compress(vols)
        if ev is not None:
            ev[1].record()
        batch.decompress(recon)
        if ev is not None:
            ev[2].record()

    for _ in range(max(args.warmup, 1)):
        step()
    batch.status()
    # quality and parity (not timed): each batch stream equals the plain codec's
    psnr = [fields.psnr(vols_h[c], recon[c].cpu().numpy()) for c in range(C)]
    streams = [batch.read_stream(c) for c in range(C)]
    coded_bytes = sum(b // 8 for _, b in streams)
    cap = cc.volume_stream_capacity_words(n, n, n)
    plain_words = torch.empty(cap, dtype=torch.int32, device=dev)
    _, pbits = cc.compress_volume_float(inst, vols[0], L, q0, plain_words)
    torch.cuda.synchronize()
    same_as_plain = pbits == streams[0][1] and np.array_equal(
        plain_words[: (pbits + 31) // 32].cpu().numpy().view(np.uint32), streams[0][0])
    # latency: one step at a time (encode / decode split by events)
    evs = [[torch.cuda.Event(enable_timing=True) for _ in range(3)] for _ in range(args.steps)]
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    start.record()
    for k in range(args.steps):
        step(evs[k])
    end.record()
    torch.cuda.synchronize()
    batch.status()
    lat_ms = start.elapsed_time(end) / args.steps
    enc_ms = sum(evs[k][0].elapsed_time(evs[k][1]) for k in range(args.steps)) / args.steps
    dec_ms = sum(evs[k][1].elapsed_time(evs[k][2]) for k in range(args.steps)) / args.steps
    lat_ms, enc_ms, dec_ms = replicas.max_over_ranks([lat_ms, enc_ms, dec_ms], dist, dev)

    # throughput (value): consecutive steps in flight on `nb` batches, each on
    # its own stream, so one step's latency-bound phases (table builds, the
    # decoder's walk) overlap another's bandwidth-bound passes; every step
    # still encodes and decodes all components.  nb in {1, 2, 3, 4} is chosen
    # by a short untimed trial (more batches in flight contend for HBM and L2).
    pool = [batch] + [cc.VolumeBatch(inst, [v.shape for v in vols], L, [q0] * C, graph=True) for _ in range(3)]
    pstreams = [torch.cuda.Stream(dev) for _ in pool]
    inst_stream = cc.lib().cc_get_instance_stream(inst.handle)
    prec = [[torch.empty_like(v) for v in vols] for _ in pool]

    def inflight(nb, steps):
        for b, st in zip(pool[:nb], pstreams):
            b.set_stream(st)
        for st in pstreams[:nb]:
            st.wait_stream(torch.cuda.current_stream())
        for k in range(steps):
            i = k % nb
            pool[i].compress(vols)
            pool[i].decompress(prec[i])
        for st in pstreams[:nb]:
            torch.cuda.current_stream().wait_stream(st)

    trial = {}
    for nb in (1, 2, 3, 4):
        inflight(nb, 2 * nb)
        torch.cuda.synchronize()
        a, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        inflight(nb, 6)
        e.record()
        torch.cuda.synchronize()
        trial[nb] = a.elapsed_time(e) / 6
    nb = min(trial, key=trial.get)
    nb = int(replicas.max_over_ranks([nb], dist, dev)[0])      # every rank runs the same count
    inflight(nb, max(args.warmup, 2 * nb))
    if dist:
        dist.barrier()
    torch.cuda.synchronize()
    launches0 = cc.lib().cc_kernel_launches()
    sampler = ClockSampler(local)
    start.record()
    inflight(nb, args.steps)
    end.record()
    torch.cuda.synchronize()
    clocks = sampler.stop()
    launches = cc.lib().cc_kernel_launches() - launches0
    for b in pool:
        b.status()
    for b in pool:
        b.set_stream(inst_stream)
    if dist:
        dist.barrier()
    ms = replicas.max_over_ranks([start.elapsed_time(end) / args.steps], dist, dev)[0]
    raw_step = C * n ** 3 * 4
    value = replicas.job_gbs(world, raw_step, ms)
    same_inflight = all(torch.equal(prec[(args.steps - 1) % nb][c], recon[c]) for c in range(C))

    # the plain per-component path (cc_compress_volume_float / decompress), for comparison
    plain_out = torch.empty_like(vols[0])

    def plain_step():
        for c in range(C):
            _, b = cc.compress_volume_float(inst, vols[c], L, q0, plain_words)
            cc.decompress_volume_float(inst, plain_out, L, q0, plain_words, b)

    plain_step()
    torch.cuda.synchronize()
    s0, e0 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s0.record()
    for _ in range(max(1, args.steps // 2)):
        plain_step()
    e0.record()
    torch.cuda.synchronize()
    plain_ms = s0.elapsed_time(e0) / max(1, args.steps // 2)

    # end to end through the public API with host buffers, software-pipelined
    # over steps: the H2D of the next step's fields and the D2H of the previous
    # step's reconstruction (copy engines) overlap the steps' compress ->
    # stream download to pinned host memory -> stream upload from it ->
    # decompress, which alternate between two batches on their own streams.
    # Every step moves its own fields in, its streams out and back in, and its
    # reconstruction out.  At least 40 steps are timed (about 0.2 s): the
    # pipeline's fill (the first step's copy in and codec) and drain (the
    # last step's copy out) are a tenth of a 10-step region.  The PCIe link
    # is shared with the host's other GPUs, so three such runs are timed and
    # the median reported (all three are in the line).
    e2e_steps = max(args.steps, 40)
    e2e_runs = [pipelined_e2e(torch, pool[:2], vols_h, vols, dev, C, cc, steps=e2e_steps) for _ in range(3)]
    e2e_runs_ms = [r["ms"] for r in e2e_runs]
    e2e = sorted(e2e_runs, key=lambda r: r["ms"])[1]
    e2e["identical"] = all(r["identical"] for r in e2e_runs)
    e2e_ms = replicas.max_over_ranks([e2e["ms"]], dist, dev)[0]
    e2e_value = replicas.job_gbs(world, raw_step, e2e_ms)
    h2d = raw_step + e2e["stream_bytes"]
    d2h = raw_step + e2e["stream_bytes"]
    if not e2e["identical"]:
        raise RuntimeError("pipelined end-to-end reconstruction differs from the device-resident one")

    # per-kernel sections (one extra step with event timing on)
    lib = cc.lib()
    lib.cc_reset_timings(inst.handle)
    lib.cc_set_timing(inst.handle, 1)
    lib.cc_volume_batch_use_graph(batch.handle, 0)
    step()
    torch.cuda.synchronize()
    batch.collect_timings()
    lib.cc_volume_batch_use_graph(batch.handle, 1)
    nsec = lib.cc_timing_count(inst.handle)
    sections = {}
    for i in range(nsec):
        name = ctypes.c_char_p()
        t_ms = ctypes.c_double()
        cnt = ctypes.c_uint32()
        lib.cc_timing_entry(inst.handle, i, ctypes.byref(name), ctypes.byref(t_ms), ctypes.byref(cnt))
        sections[name.value.decode()] = (t_ms.value, cnt.value)
    lib.cc_set_timing(inst.handle, 0)
    peak, peak_kind = load_peak()
    # compact symbols of all highpass streams (algorithmic bytes of the
    # entropy sections)
    counts = {"compact": sum(compact_count(cc, torch, vols[c], L, q0) for c in range(C))}
    kernel_secs = {k: v for k, v in sections.items() if k not in COMPOSITE_SECTIONS}
    total_sec = sum(v[0] for v in kernel_secs.values()) or 1.0
    bw = {}
    for k, (t, cnt) in kernel_secs.items():
        b = section_bytes(k, wl, coded_bytes, counts)
        if b and t > 0:
            bw[k] = {"ms": t, "algorithmic_bytes": b, "gbs": b / (t / 1e3) / 1e9, "frac": b / (t / 1e3) / 1e9 / peak,
                     "launches": cnt, "share": t / total_sec}
            if k in SECTION_UNITS:
                bw[k]["per_unit"] = SECTION_UNITS[k]
    top = max(kernel_secs.items(), key=lambda kv: kv[1][0]) if kernel_secs else ("none", (0.0, 0))
    top_bytes = section_bytes(top[0], wl, coded_bytes, counts) or 0
    # whole codec (algorithmic: raw + compressed bytes; intermediate passes do not count)
    step_alg = 2 * (raw_step + coded_bytes)
    enc_gbs_alg = (raw_step + coded_bytes) / (enc_ms / 1e3) / 1e9
    dec_gbs_alg = (raw_step + coded_bytes) / (dec_ms / 1e3) / 1e9
    traffic = None
    tpath = os.path.join(ROOT, "profiles", "traffic.json")
    if os.path.exists(tpath):
        with open(tpath) as f:
            traffic = json.load(f).get("step_total")
    pipeline = {"achieved": step_alg / (ms / 1e3) / 1e9, "peak": peak, "unit": "GB/s",
                "frac": step_alg / (ms / 1e3) / 1e9 / peak,
                "algorithmic_bytes_per_step": step_alg,
                "encode_frac": enc_gbs_alg / peak, "decode_frac": dec_gbs_alg / peak}
    # the headline roofline is the whole codec step (every kernel of encode +
    # decode; algorithmic bytes = raw + compressed each way), with the step's
    # dominant kernel section and every bandwidth section beside it
    roofline = {"bound": "hbm", "kernel": "whole codec step (encode + decode, all kernels)",
                "achieved": pipeline["achieved"], "peak": peak, "unit": "GB/s", "frac": pipeline["frac"],
                "peak_source": peak_kind, "traffic": traffic, "algorithmic_bytes_per_step": step_alg,
                "per_unit": "raw field bytes in + compressed bytes out (encode), compressed in + raw out (decode)",
                "dominant_section": {"name": top[0], "ms": top[1][0], "share": top[1][0] / total_sec,
                                     "algorithmic_bytes": top_bytes,
                                     "frac": (top_bytes / (top[1][0] / 1e3) / 1e9 / peak) if top[1][0] else None,
                                     "note": SECTION_NOTES.get(top[0])},
                "sections": bw}

    bricks = None
    if rank == 0 and world == 1 and not args.no_bricks:
        bw3 = WORKLOADS["bricks-4096"]
        bricks = measure_bricks(bw3["count"], bw3["levels"], bw3["seed"], max(2, args.steps // 2), 2, 128, local,
                                autotune=True)
    sweep = None
    if rank == 0 and world == 1 and not args.no_sweep:
        sweep = measure_q0_sweep(inst, vols, vols_h, L, Q0_SWEEP, max(3, args.steps // 2), 2)
    serve = None
    if rank == 0 and world == 1 and not args.no_bricks:
        serve = measure_serving(WORKLOADS["serving"], local, requests=20000, rates=(10000.0,))

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        threads = os.cpu_count() or 1
        e, d, kind = cpu_reference_step(vols_h[0], wl, threads)
        e1, d1, _ = cpu_reference_step(vols_h[0], wl, 1)
        cpu = {"value": n ** 3 * 4 / (e + d) / 1e9, "unit": "GB/s", "cores": threads, "kind": kind,
               "sample": f"1 of {C} components ({n}^3 f32) encode+decode; DWT/quantize stages are the oracle port",
               "single_core": {"value": n ** 3 * 4 / (e1 + d1) / 1e9, "unit": "GB/s", "cores": 1,
                               "encode_s": e1, "decode_s": d1},
               "all_cores": {"encode_s": e, "decode_s": d, "cores": threads}}
    if rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": "GB/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded k^-5/3 random-phase fields)",
            "in_flight_batches": nb, "in_flight_trial_ms": {str(k): round(v, 4) for k, v in trial.items()},
            "latency_ms_per_step": lat_ms, "reconstruction_identical_in_flight": bool(same_inflight),
            "config": {"workload": args.workload, "desc": wl["desc"], "parallelism": f"replicas{world}",
                       "l2": f"inputs {C * n ** 3 * 4 >> 20} MiB per step > L2 126 MiB"},
            "encode_gbs": replicas.job_gbs(world, raw_step, enc_ms),
            "decode_gbs": replicas.job_gbs(world, raw_step, dec_ms),
            "compression_ratio": raw_step / max(coded_bytes, 1), "psnr_db": psnr,
            "plain_path_ms_per_step": plain_ms, "streams_identical_to_plain_codec": bool(same_as_plain),
            "q0_sweep": sweep, "compact_symbols_per_step": counts["compact"],
            "batched_vs_per_brick": bricks, "serving": serve,
            "e2e": {"value": e2e_value, "unit": "GB/s", "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
                    "steps": e2e_steps, "runs_ms_per_step": [round(x, 4) for x in e2e_runs_ms], "reported": "median of 3"},
            "gpu_launches": launches,
            "roofline": roofline, "pipeline_roofline": pipeline,
            "sections_ms": {k: round(v[0], 4) for k, v in sorted(sections.items(), key=lambda kv: -kv[1][0])},
            "clocks": clocks, "cpu_baseline": cpu,
        }
        print(json.dumps(line), flush=True)
    for b in pool:
        b.close()
    inst.close()
    if dist:
        dist.destroy_process_group()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--workload", choices=sorted(WORKLOADS), default="vector-field-256")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-bricks", action="store_true", help="skip the batched-vs-per-brick measurement")
    ap.add_argument("--no-sweep", action="store_true", help="skip the q0 sweep of the vector field")
    ap.add_argument("--profile", action="store_true",
                    help="a small case for profilers only: one batch of --comps n^3 fields, --warmup + --steps passes")
    ap.add_argument("--n", type=int, default=256, help="--profile: field edge")
    ap.add_argument("--comps", type=int, default=3, help="--profile: components")
    ap.add_argument("--q0", type=float, default=0.01, help="--profile: quantization step (times std)")
    args = ap.parse_args()
    wl = WORKLOADS[args.workload]
    if args.profile:
        run_profile(args)
    elif args.impl == "reference":
        run_reference(args, wl)
    elif args.workload.startswith("bricks"):
        run_bricks(args, wl)
    elif args.workload == "serving":
        run_serving(args, wl)
    elif args.workload.startswith("heightfield"):
        run_heightfield(args, wl)
    else:
        run_ours(args, wl)


if __name__ == "__main__":
    main()
