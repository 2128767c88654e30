"""Performance cases of the scan library: the calls a program makes, with the
sizes, data types and options it makes them with.

Operations:
  scan     one device-wide prefix scan (Plan.scan), chained or reduce-then-scan
  batched  thousands of independent scans in one launch (Plan.scan_segmented)
  select   stream compaction by flag bytes (Plan.select)
  graph    a captured sequence of small scans, replayed

Sizes span a few kilobytes to 1 GiB of input. `in_off` / `out_off` are element
offsets of the input and output views from a 16-byte boundary (a slice of a
larger array); only integer plans take them.
"""
import math

import numpy as np
import torch

from gpuprefixsums_gb300 import Plan

# Bytes of one scanned element, and the torch type its words are held in.
ELEM = {"u32": 4, "u64": 8, "f32": 4, "f32c": 4, "u32x4": 16}
WORD = {"u32": torch.int32, "u64": torch.int64, "f32": torch.float32, "f32c": torch.float32, "u32x4": torch.int32}


def listed():
    return [
        # A call of a few kilobytes: bucket offsets, block counts. Latency only.
        {"name": "scan_u32_1000", "op": "scan", "algo": "csdl", "dtype": "u32", "n": 1000, "inclusive": False,
         "in_off": 0, "out_off": 0},
        # The library's verification size, 2^20 elements.
        {"name": "scan_u32_1m", "op": "scan", "algo": "csdl", "dtype": "u32", "n": 1 << 20, "inclusive": True,
         "in_off": 0, "out_off": 0},
        # A slice x[1:] of an array, of no round length, into an output of its own.
        {"name": "scan_u32_slice_10m", "op": "scan", "algo": "csdl", "dtype": "u32", "n": 10_000_019,
         "inclusive": False, "in_off": 1, "out_off": 0},
        # The headline benchmark: 2^28 u32, exclusive.
        {"name": "scan_u32_256m", "op": "scan", "algo": "csdl", "dtype": "u32", "n": 1 << 28, "inclusive": False,
         "in_off": 0, "out_off": 0},
        # 64-bit offsets at the same number of bytes.
        {"name": "scan_u64_128m", "op": "scan", "algo": "csdl", "dtype": "u64", "n": 1 << 27, "inclusive": False,
         "in_off": 0, "out_off": 0},
        # The other algorithm a program can ask for.
        {"name": "rts_u32_64m", "op": "scan", "algo": "rts", "dtype": "u32", "n": 1 << 26, "inclusive": True,
         "in_off": 0, "out_off": 0},
        # An ordinary floating-point scan (a cumulative distribution), no round length.
        {"name": "scan_f32_1m", "op": "scan", "algo": "csdl", "dtype": "f32", "n": 1_000_003, "inclusive": True,
         "in_off": 0, "out_off": 0},
        # The large compensated scan of the precision benchmark.
        {"name": "scan_f32c_64m", "op": "scan", "algo": "csdl", "dtype": "f32c", "n": 1 << 26, "inclusive": True,
         "in_off": 0, "out_off": 0},
        # The batched benchmark: 4096 scans of log-uniform lengths up to 2^20.
        {"name": "batched_u32_4096", "op": "batched", "dtype": "u32", "lengths": "loguniform", "low": 1,
         "high": 1 << 20, "count": 4096, "lengths_seed": 3, "inclusive": False},
        # A small ragged batch: 500 sequences with Zipf lengths, compensated.
        {"name": "batched_f32c_500", "op": "batched", "dtype": "f32c", "lengths": "zipf", "low": 32,
         "high": 1 << 16, "count": 500, "lengths_seed": 5, "inclusive": True},
        # Compaction of 2^28 values by Bernoulli(0.3) flags.
        {"name": "select_u32_256m", "op": "select", "dtype": "u32", "n": 1 << 28, "p": 0.3},
        # A step that scans many small arrays, captured once: 32 scans of 2^16.
        {"name": "graph_u32_64k_x32", "op": "graph", "dtype": "u32", "n": 1 << 16, "count": 32, "inclusive": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges."""
    pick = rng.random()
    if pick < 0.5:
        dtype = rng.choice(["u32", "u32", "u64", "f32", "f32c", "u32x4"])
        algo = "rts" if dtype in ("u32", "u64") and rng.random() < 0.25 else "csdl"
        # Up to 1 GiB of input for the chained integer scans, 256 MiB for the others.
        top = 1 << 30 if dtype in ("u32", "u64") and algo == "csdl" else 1 << 28
        n = _log_int(rng, 1000, top // ELEM[dtype])
        off = dtype in ("u32", "u64") and rng.random() < 0.3
        last = 16 // ELEM[dtype] - 1
        if off:  # an element-aligned slice costs more than an aligned buffer
            n = min(n, (1 << 27) // ELEM[dtype])
        return {"op": "scan", "algo": algo, "dtype": dtype, "n": n, "inclusive": rng.random() < 0.5,
                "in_off": rng.randint(1, last) if off else 0, "out_off": rng.randint(0, last) if off else 0}
    if pick < 0.75:
        dtype = rng.choice(["u32", "u64", "f32", "f32c", "u32x4"])
        low = rng.choice([1, 32])
        return {"op": "batched", "dtype": dtype, "lengths": rng.choice(["loguniform", "zipf"]), "low": low,
                "high": _log_int(rng, 1 << 10, 1 << 20), "count": _log_int(rng, 16, 10_000),
                "lengths_seed": rng.randrange(1 << 20), "inclusive": rng.random() < 0.5}
    if pick < 0.9:
        dtype = rng.choice(["u32", "u64", "f32"])
        p = round(rng.uniform(0.02, 0.95), 3)
        top = 1 << 30 if p < 0.4 else 1 << 29
        return {"op": "select", "dtype": dtype, "n": _log_int(rng, 1000, top // ELEM[dtype]), "p": p}
    return {"op": "graph", "dtype": rng.choice(["u32", "u64", "f32", "f32c"]), "n": _log_int(rng, 256, 1 << 18),
            "count": rng.randint(8, 48), "inclusive": rng.random() < 0.5}


def _offsets(case):
    """CSR offsets of a batch: lengths from the case alone, cut where the input passes its limit."""
    r = np.random.default_rng(case["lengths_seed"])
    u = r.uniform(0.0, 1.0, size=case["count"])
    low, high = case["low"], case["high"]
    if case["lengths"] == "loguniform":
        lengths = np.floor(np.exp(math.log(low) + u * (math.log(high) - math.log(low))))
    else:  # Zipf, exponent 1.2, truncated to [low, high]
        a, b = low ** -0.2, high ** -0.2
        lengths = np.clip(np.floor((a - u * (a - b)) ** -5.0), low, high)
    ends = np.cumsum(lengths.astype(np.int64))
    top = {"u32": 1_230_000_000, "u64": 1 << 30, "u32x4": 1 << 30}.get(case["dtype"], 1 << 28)
    cap = top // ELEM[case["dtype"]]
    keep = max(1, int(np.searchsorted(ends, cap, side="right")))
    return np.concatenate([[0], ends[:keep]])


def _values(dtype, words, gen):
    if dtype in ("f32", "f32c"):
        return torch.randn(words, device="cuda", generator=gen)
    if dtype == "u64":
        return torch.randint(-(1 << 63), (1 << 63) - 1, (words,), dtype=torch.int64, device="cuda", generator=gen)
    if dtype == "u32x4":
        return torch.randint(-(1 << 31), (1 << 31) - 1, (words,), dtype=torch.int32, device="cuda", generator=gen)
    return torch.randint(0, 256, (words,), dtype=torch.int32, device="cuda", generator=gen)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    op, dtype = case["op"], case["dtype"]
    members = 4 if dtype == "u32x4" else 1
    if op == "scan":
        words = case["n"] * members
        x = _values(dtype, words + case["in_off"], gen)[case["in_off"]:]
        out = torch.zeros(words + case["out_off"], dtype=WORD[dtype], device="cuda")[case["out_off"]:]
        return {"op": op, "plan": Plan(case["algo"], dtype, max_n=case["n"]), "x": x, "out": out,
                "inclusive": case["inclusive"]}
    if op == "batched":
        offs = _offsets(case)
        n = int(offs[-1])
        x = _values(dtype, n * members, gen)
        d_off = torch.from_numpy(offs.astype(np.uint32).view(np.int32)).cuda()
        return {"op": op, "plan": Plan("csdl", dtype, max_n=n), "x": x, "offsets": d_off,
                "out": torch.zeros_like(x), "inclusive": case["inclusive"]}
    if op == "select":
        n = case["n"]
        x = _values(dtype, n, gen)
        flags = (torch.rand(n, device="cuda", generator=gen) < case["p"]).to(torch.uint8)
        return {"op": op, "plan": Plan("csdl", dtype, max_n=n), "x": x, "flags": flags,
                "out": torch.zeros_like(x), "count": torch.zeros(1, dtype=torch.int64, device="cuda")}
    # graph: rows of one array, each scanned on its own, in one captured sequence
    n, count = case["n"], case["count"]
    pitch = -(-n // 4) * 4  # rows start on 16-byte boundaries
    x = _values(dtype, pitch * count, gen).view(count, pitch)
    out = torch.zeros_like(x)
    plan = Plan("csdl", dtype, max_n=n)

    def scans():
        for i in range(count):
            plan.scan(x[i, :n], out=out[i, :n], inclusive=case["inclusive"])

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        scans()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        scans()
    return {"op": op, "plan": plan, "graph": graph, "x": x, "out": out}


def run(state):
    op = state["op"]
    if op == "scan":
        return state["plan"].scan(state["x"], out=state["out"], inclusive=state["inclusive"])
    if op == "batched":
        return state["plan"].scan_segmented(state["x"], state["offsets"], out=state["out"],
                                            inclusive=state["inclusive"])
    if op == "select":
        return list(state["plan"].select(state["x"], state["flags"], out=state["out"],
                                         num_selected=state["count"]))
    state["graph"].replay()
    return state["out"]


def work(case):
    es, op = ELEM[case["dtype"]], case["op"]
    adds = 4 if case["dtype"] == "u32x4" else 1
    if op == "scan":
        return {"bytes": 2 * case["n"] * es, "flops": case["n"] * adds}
    if op == "batched":
        offs = _offsets(case)
        return {"bytes": 2 * int(offs[-1]) * es + 4 * len(offs), "flops": int(offs[-1]) * adds}
    if op == "select":
        n = case["n"]
        return {"bytes": n * es + n + int(case["p"] * n) * es + 8, "flops": n}
    return {"bytes": 2 * case["n"] * case["count"] * es, "flops": case["n"] * case["count"]}


def _prefix64(x, inclusive):
    c = torch.cumsum(x.double(), dim=-1)
    return c if inclusive else c - x.double()


def exact(case, seed):
    """Floating-point outputs in 64 bits; integer results are exact as they are."""
    if case["dtype"] not in ("f32", "f32c"):
        return None
    s = prepare(case, seed)
    x = s["x"]
    if case["op"] == "scan":
        return _prefix64(x, case["inclusive"])
    if case["op"] == "batched":
        offs = torch.from_numpy(_offsets(case)).cuda()
        before = torch.cat([torch.zeros(1, dtype=torch.float64, device="cuda"), torch.cumsum(x.double(), 0)])
        base = torch.repeat_interleave(before[offs[:-1]], offs[1:] - offs[:-1])
        return (before[1:] if case["inclusive"] else before[:-1]) - base
    if case["op"] == "select":
        got = torch.masked_select(x, s["flags"].bool()).double()
        out = torch.zeros(case["n"], dtype=torch.float64, device="cuda")
        out[:got.numel()] = got
        return [out, torch.tensor([got.numel()], dtype=torch.int64, device="cuda")]
    out = torch.zeros_like(x, dtype=torch.float64)
    out[:, :case["n"]] = _prefix64(x[:, :case["n"]], case["inclusive"])
    return out
