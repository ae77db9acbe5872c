"""Performance cases of the simulator: what a user of it has it do, from one
testbench cycle of a small design to the batched evaluation of the largest
benchmark design, through the public Python API.

A case names a design (a generator configuration of workloads.DESIGNS, with
overrides), the way it is run (`kind`) and the run's size:

  testbench  set_register / eval per cycle, then read_registers: a testbench
             driving one stream cycle by cycle (latency, launches, copies)
  free       reset, inputs written, eval_free_running: one stream running on
             its own, and the registers it ends with
  batch      every stream resident, equal lengths, the way the benchmark
             configures a workload (workloads.bench_simulator); inputs from
             the seed on the device, or uploaded as a host table (`table`)
  queue      streams of log-uniform length queued onto resident slots,
             optionally ending at their stop op
  inspect    state read back after a batch: register pools and digests of
             single streams
  gradient   the learned cost model's gradient over a set of profiled samples
"""
from __future__ import annotations

import math
import tempfile
from pathlib import Path

import numpy as np

from toucangpurt_gb300 import sim, workloads

# Designs: a benchmark workload's generator configuration with overrides.
# "ragged" is a mid-size design with every kind of op and odd sizes, whose
# streams stop on their own.
_RAGGED = dict(n_lut=100_003, levels=29, operands=3, palette_pct=40, fanout_alpha=2.2, max_fanout=512, ff_bits=8_200,
               pi_bits=68, n_mems=5, mem_depth=2048, mem_width=20, mem_read_ports=2, mem_write_ports=1, n_vec_ops=51,
               vec_nibbles=8, luts_per_part=3_000, mpart_width=32, cone_depth=3, with_stop=2)


def listed():
    return [
        # a testbench around the small design: 32 clock cycles, inputs set before each
        {"name": "testbench small", "kind": "testbench", "design": "small", "cycles": 32},
        # free running on one stream, the reference's own benchmark call
        {"name": "free small", "kind": "free", "design": "small", "cycles": 1000},
        {"name": "free 1M", "kind": "free", "design": "scale", "cycles": 300},
        # a regression run: hundreds of short tests of a small design, queued
        {"name": "queue small 1024", "kind": "queue", "design": "small", "streams": 1024, "short": 50, "long": 2000,
         "stop": False},
        # the same on a ragged mid-size design whose tests end at a stop op
        {"name": "queue ragged 203", "kind": "queue", "design": "ragged", "streams": 203, "short": 20, "long": 150,
         "stop": True},
        # few streams, not a multiple of the word's eight
        {"name": "batch ragged 13", "kind": "batch", "design": "ragged", "streams": 13, "cycles": 100, "table": True},
        # batched runs of the 1M-LUT design with final and per-cycle digests
        {"name": "batch 1M 64", "kind": "batch", "design": "scale", "streams": 64, "cycles": 100, "table": False},
        # mixed regions (deep control cones, memories), the learned-partitioner workload
        {"name": "batch mixed 4M 256", "kind": "batch", "design": "learned", "streams": 256, "cycles": 20, "table": False},
        # the headline workload: 16M LUTs, 64 streams, inputs uploaded per call
        {"name": "batch 16M 64", "kind": "batch", "design": "largest", "streams": 64, "cycles": 100, "table": True},
        # its plain form: one stream
        {"name": "batch 16M 1", "kind": "batch", "design": "largest", "streams": 1, "cycles": 100, "table": False},
        # state of single streams read back after a batch
        {"name": "inspect 1M 64", "kind": "inspect", "design": "scale", "streams": 64, "cycles": 4},
        # the cost model's gradient over the samples that the benchmark profiles
        {"name": "gradient 200K", "kind": "gradient", "samples": 200_000},
    ]


def _between(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["testbench", "free", "queue", "batch", "batch", "batch", "inspect", "gradient"])
    if kind == "gradient":
        return {"kind": kind, "samples": _between(rng, 10_000, 600_000)}
    if kind == "testbench":
        return {"kind": kind, "design": rng.choice(["small", "ragged"]), "seed": rng.randrange(1, 1000),
                "cycles": rng.randint(1, 60)}
    if kind == "free":
        design = rng.choice(["small", "ragged", "scale"])
        return {"kind": kind, "design": design, "seed": rng.randrange(1, 1000),
                "n_lut": 4096 if design == "small" else _between(rng, 20_000, 1 << 20),
                "cycles": _between(rng, 30, 2000 if design == "small" else 300)}
    if kind == "queue":
        design = rng.choice(["small", "ragged"])
        short = rng.randint(5, 100)
        return {"kind": kind, "design": design, "seed": rng.randrange(1, 1000), "streams": _between(rng, 20, 1500),
                "short": short, "long": short + _between(rng, 5, 1500 if design == "small" else 150),
                "stop": design == "ragged" and rng.random() < 0.5}
    design = rng.choice(["ragged", "scale", "learned", "largest"])
    n_lut = _between(rng, 50_000, 4 << 20)
    streams = _between(rng, 2, 256) if kind == "inspect" else rng.choice([1, _between(rng, 2, 256), _between(rng, 2, 256)])
    case = {"kind": kind, "design": design, "seed": rng.randrange(1, 1000), "n_lut": n_lut, "streams": streams,
            # lookups of a pass up to a sixteenth of the largest listed case's
            "cycles": max(2, min(200, int(6.4e9 / n_lut / max(8, streams))))}
    if kind == "batch":
        case["table"] = rng.random() < 0.5
    return case


# ---- designs and handles -----------------------------------------------------

def _design_config(case):
    name = case["design"]
    cfg = dict(_RAGGED, seed=77) if name == "ragged" else workloads.design_config(name)
    n = case.get("n_lut")
    if n and n != cfg["n_lut"]:
        # a smaller design of the same make: state and ports shrink with it
        f = n / cfg["n_lut"]
        cfg["n_lut"] = n
        for k, least in (("ff_bits", 256), ("n_vec_ops", 8), ("n_mems", 2)):
            if cfg.get(k):
                cfg[k] = max(least, int(cfg[k] * f))
        if name == "largest":
            cfg["mem_depth"] = 16 * 1024
    if case.get("seed"):
        cfg["seed"] = case["seed"]
    return cfg


_dir = None     # the process's design files
_files = {}     # configuration -> (design file, symbol file, generator info)
_handle = None  # (key, simulator): the program's current simulator


def _design(case):
    global _dir
    cfg = _design_config(case)
    key = tuple(sorted(cfg.items()))
    if key not in _files:
        if _dir is None:
            _dir = tempfile.TemporaryDirectory(prefix="perf_designs_")
        dp, sp = Path(_dir.name) / f"{len(_files)}.bin", Path(_dir.name) / f"{len(_files)}.sym"
        _files[key] = (dp, sp, sim.generate(dp, sp, **cfg))
    return key, _files[key]


def _simulator(case):
    """The simulator a program keeps while it runs one stimulus after another
    on a design: loaded once, every run starts from the initial state."""
    global _handle
    key, (dp, sp, _) = _design(case)
    key = (key, case["kind"], case.get("streams"))
    if _handle is None or _handle[0] != key:
        if _handle is not None:
            _handle[1].cleanup()
            _handle = None
        if case["kind"] == "batch":
            s, _ = workloads.bench_simulator(case["design"], dp, sp, streams=case["streams"], schedule="greedy")
        else:
            s = sim.Simulator()
            s.init(0, dp, sp, False, False)
        _handle = (key, s)
    return _handle[1]


def _lengths(case, rng):
    lo, hi = math.log(case["short"]), math.log(case["long"])
    return np.exp(rng.uniform(lo, hi, case["streams"])).astype(np.uint32)


def _mlp_arrays(case, seed):
    """Parameters of a partly trained model and standardised samples."""
    rng = np.random.default_rng(seed)
    p = rng.normal(0, 0.2, 5313).astype(np.float32)
    X = np.log1p(rng.integers(0, 64, (case["samples"], 16))).astype(np.float32)
    y = rng.normal(0, 1, case["samples"]).astype(np.float32)
    return p, X, y


def prepare(case, seed):
    kind = case["kind"]
    if kind == "gradient":
        return {"case": case, "arrays": _mlp_arrays(case, seed)}
    rng = np.random.default_rng(seed)
    _, (dp, sp, info) = _design(case)
    ids, bits = info["pi_ids"], info["pi_bits"]
    if kind == "testbench":
        # a testbench owns its simulator and drives it on from call to call
        s = sim.Simulator()
        s.init(0, dp, sp, False, False)
        regs = sim.symbol_registers(sp)
        ins = sorted(n for n in regs if n.startswith("pi_"))[:1]
        outs = sorted(n for n in regs if n.startswith("ff_"))[:8]
        limit = 1 << sum(w for _, w in regs[ins[0]])
        vals = [int(v) for v in rng.integers(0, min(limit, 1 << 62), case["cycles"])]
        return {"case": case, "sim": s, "ins": ins, "outs": outs, "vals": vals}
    if kind == "inspect":
        # the state read back belongs to this state's own simulator
        s, _ = workloads.bench_simulator(case["design"], dp, sp, streams=case["streams"], schedule="greedy")
    else:
        s = _simulator(case)
    if kind == "free":
        s.reset_state()
        init = s.reg_pool(0)
        init[ids] = rng.integers(0, 16, ids.size).astype(np.uint8) & ((1 << bits.astype(np.int64)) - 1).astype(np.uint8)
        return {"case": case, "sim": s, "init": init}
    name = "batch" if case["design"] in ("small", "ragged") else case["design"]
    stim = sim.StimulusSpec(int(seed), ids, bits, workloads.toggles(name, bits))
    if kind == "queue":
        return {"case": case, "sim": s, "stim": stim, "lengths": _lengths(case, rng)}
    cyc = np.full(case["streams"], case["cycles"], np.uint32)
    if case.get("table"):
        shape = (case["cycles"], ids.size, case["streams"])
        buf = sim.PinnedBuffer(shape)
        s.reset_state()
        prev = np.repeat(s.reg_pool(0)[ids][:, None], case["streams"], axis=1)
        sim.stimulus_table(stim, case["streams"], 0, case["cycles"], out=buf.array, prev=prev)
        stim = sim.StimulusSpec(int(seed), ids, bits, table=buf.array)
        return {"case": case, "sim": s, "stim": stim, "lengths": cyc, "buf": buf}
    if kind == "inspect":
        s.batch_run(cyc, stim, final_digests=False)
        picked = [int(x) for x in rng.integers(0, case["streams"], 4)]
        return {"case": case, "sim": s, "streams": picked}
    return {"case": case, "sim": s, "stim": stim, "lengths": cyc}


def _out(o):
    r = [o.final_reg_digest, o.final_mem_digest, o.rolling_digest]
    if o.cycle_digest is not None:
        r.append(o.cycle_digest)
    return [a.view(np.int64) for a in r] + [o.stop_cycle.astype(np.int64)]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "gradient":
        return sim.mlp_grad(*state["arrays"])
    s = state["sim"]
    if kind == "testbench":
        for v in state["vals"]:
            for n in state["ins"]:
                s.set_register(n, v)
            s.eval()
        return np.array(s.read_registers(state["outs"]), np.uint64).view(np.int64)
    if kind == "free":
        s.reset_state()
        s.write_reg_pool(state["init"])
        s.eval_free_running(case["cycles"])
        return s.reg_pool(0)
    if kind == "queue":
        return _out(s.batch_run(state["lengths"], state["stim"], stop_exit=case["stop"]))
    if kind == "inspect":
        return [np.array([s.digest(q) for q in state["streams"]], np.uint64).view(np.int64),
                [s.reg_pool(q) for q in state["streams"]]]
    # the 16M-LUT design carries 0.5 GiB of memories per stream: like the
    # benchmark's end-to-end steps, its runs read the rolling digests back
    big = case["design"] == "largest"
    o = s.batch_run(state["lengths"], state["stim"], cycle_digests=not big, final_digests=not big)
    return _out(o) + [s.reg_pool(case["streams"] - 1)]


def work(case):
    """Bytes: 4 per LUT op and cycle (an instruction word is read once for all
    streams) and half a byte per state nibble and stream, read and written
    every cycle; flops: one per table lookup."""
    if case["kind"] == "gradient":
        n = case["samples"]
        return {"bytes": 4.0 * (17 * n + 2 * 5313), "flops": 6.0 * 5248 * n}
    cfg = _design_config(case)
    state = cfg["ff_bits"] / 4
    if case["kind"] == "inspect":
        mem = cfg["n_mems"] * cfg["mem_depth"] * cfg["mem_width"] / 4
        return {"bytes": 4 * (mem + 1.5 * state), "flops": 0.0}
    if case["kind"] == "queue":
        # mean of a log-uniform length
        cycles = (case["long"] - case["short"]) / math.log(case["long"] / case["short"])
        total, longest = cycles * case["streams"], case["long"]
    else:
        total, longest = case["cycles"] * case.get("streams", 1), case["cycles"]
    return {"bytes": 4.0 * cfg["n_lut"] * longest + 0.5 * 2 * state * total, "flops": float(cfg["n_lut"]) * total}


def exact(case, seed):
    """The gradient in 64 bits; every other output is a whole number."""
    if case["kind"] != "gradient":
        return None
    p, X, y = (a.astype(np.float64) for a in _mlp_arrays(case, seed))
    n = len(y)
    W1, b1, W2, b2, W3, b3 = (p[:1024].reshape(64, 16), p[1024:1088], p[1088:5184].reshape(64, 64), p[5184:5248],
                              p[5248:5312], p[5312])
    h1 = np.maximum(X @ W1.T + b1, 0)
    h2 = np.maximum(h1 @ W2.T + b2, 0)
    d = h2 @ W3 + b3 - y
    dy = 2 * d / n
    d2 = np.where(h2 > 0, dy[:, None] * W3, 0)
    d1 = np.where(h1 > 0, d2 @ W2, 0)
    g = [d1.T @ X, d1.sum(0), d2.T @ h1, d2.sum(0), h2.T @ dy, dy.sum()]
    return np.concatenate([np.ravel(v) for v in g]), float(np.mean(d * d))
