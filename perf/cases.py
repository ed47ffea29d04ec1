"""Performance cases: the work a user of this package has it do, through its public entry points.

`listed()` gives the fixed cases, `draw(rng)` one more case of the same ranges,
`prepare(case, seed)` what a program holds before the call (tables on the GPU, a
plan, a server), `run(state)` one call and its whole outputs, `work(case)` the
bytes and operations one call cannot do without, and `exact(case, seed)` the
outputs evaluated in 64 bits by torch alone.
"""
from __future__ import annotations

import ctypes
import math

import torch

from nt2_gb300 import api, video
from nt2_gb300._lib import check, lib
from nt2_gb300.server import Server

RATE, SIGMA = 0.02, 0.30
DTYPES = {"f32": torch.float32, "f64": torch.float64}

# One-argument functors: the interval of arguments a program passes, and the
# function in 64 bits.
_SQRT_HALF = math.sqrt(0.5)
MAPS = {
    "exp": (-20.0, 20.0, torch.exp),
    "log": (1e-3, 1e3, torch.log),
    "sqrt": (0.0, 1e3, torch.sqrt),
    "erfc": (-4.0, 4.0, torch.special.erfc),
    "normcdf": (-5.0, 5.0, lambda x: 0.5 * torch.special.erfc(-_SQRT_HALF * x)),
    "exp2": (-30.0, 30.0, torch.exp2),
    "log2": (1e-3, 1e3, torch.log2),
    "log10": (1e-3, 1e3, torch.log10),
    "expm1": (-2.0, 2.0, torch.expm1),
    "log1p": (-0.9, 10.0, torch.log1p),
    "sin": (-60.0, 60.0, torch.sin),
    "cos": (-60.0, 60.0, torch.cos),
    "tan": (-60.0, 60.0, torch.tan),
    "asin": (-1.0, 1.0, torch.asin),
    "atan": (-10.0, 10.0, torch.atan),
    "sinh": (-10.0, 10.0, torch.sinh),
    "tanh": (-4.0, 4.0, torch.tanh),
    "asinh": (-60.0, 60.0, torch.asinh),
}
# Two-argument functors: the intervals of both arguments, and the function.
MAPS2 = {
    "pow": (0.0, 100.0, -10.0, 10.0, torch.pow),
    "atan2": (-10.0, 10.0, -10.0, 10.0, torch.atan2),
    "hypot": (-10.0, 10.0, -10.0, 10.0, torch.hypot),
}
# Operations of one element in NT2's algorithm (multiplies, adds, divisions and
# roots), rounded.
MAP_FLOPS = {"exp": 20, "log": 30, "sqrt": 1, "erfc": 45, "normcdf": 47, "exp2": 18, "log2": 32, "log10": 34,
             "expm1": 30, "log1p": 35, "sin": 20, "cos": 20, "tan": 25, "asin": 20, "atan": 25, "sinh": 25,
             "tanh": 28, "asinh": 40, "pow": 60, "atan2": 30, "hypot": 8}


def listed():
    return [
        # a pricing request of the smallest usual size: latency and launch
        {"name": "bs_f32_request", "kind": "bs", "n": 1000, "dtype": "f32", "cdf": "normcdf", "precision": "exact"},
        # the benchmark's pricing batch, float and double tables
        {"name": "bs_f32_batch", "kind": "bs", "n": 1 << 24, "dtype": "f32", "cdf": "normcdf", "precision": "exact"},
        {"name": "bs_f64_batch", "kind": "bs", "n": 1 << 24, "dtype": "f64", "cdf": "normcdf", "precision": "exact"},
        # the benchmark's saxpy
        {"name": "saxpy_f32", "kind": "saxpy", "n": 1 << 24, "dtype": "f32"},
        # single functors over a table: double of a ragged length, and the costliest float one
        {"name": "sin_f64_ragged", "kind": "map", "op": "sin", "n": 3000001, "dtype": "f64"},
        {"name": "pow_f32", "kind": "map2", "op": "pow", "n": 1 << 24, "dtype": "f32"},
        # the benchmark's dot product and its row sums
        {"name": "dot_f32", "kind": "dot", "n": 1 << 26, "dtype": "f32", "compensated": True},
        {"name": "sum_rows_f32", "kind": "reduce", "op": "sum", "rows": 8192, "cols": 4096, "dim": 2, "dtype": "f32"},
        # statistics of the columns of a double table of odd sizes
        {"name": "stdev_cols_f64", "kind": "reduce", "op": "stdev", "rows": 10001, "cols": 777, "dim": 1,
         "dtype": "f64"},
        # a running sum over one long vector
        {"name": "cumsum_f32_long", "kind": "scan", "op": "cumsum", "rows": 1 << 26, "cols": 1, "dim": 1,
         "dtype": "f32"},
        # the benchmark's background subtraction: 256 uneven streams of 8 frames, one captured launch
        {"name": "sigmadelta_256x8", "kind": "sigmadelta", "streams": 256, "frames": 8, "mix": 3},
        # a burst of pricing requests of mixed sizes through the server
        {"name": "server_burst", "kind": "server", "requests": 64, "max_n": 1 << 18, "mix": 5},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _table(rng, cells_hi):
    cells = _log_int(rng, 4096, cells_hi)
    rows = _log_int(rng, 16, cells // 16)
    return rows, max(1, cells // rows)


def draw(rng):
    kind = rng.choice(["bs", "bs", "bs", "saxpy", "map", "map", "map", "map2", "dot", "reduce", "reduce", "scan",
                       "scan", "sigmadelta"])
    dtype = rng.choice(["f32", "f64"])
    if kind == "bs":
        f32 = dtype == "f32"
        return {"kind": kind, "n": _log_int(rng, 256, 1 << 24), "dtype": dtype,
                "cdf": rng.choice(["normcdf", "normcdf", "fastnormcdf"]) if f32 else "normcdf",
                "precision": rng.choice(["exact", "fused", "fast"]) if f32 else rng.choice(["exact", "fused"])}
    if kind == "saxpy":
        return {"kind": kind, "n": _log_int(rng, 256, 1 << 25), "dtype": dtype}
    if kind == "map":
        return {"kind": kind, "op": rng.choice(sorted(MAPS)), "n": _log_int(rng, 256, 1 << 24), "dtype": dtype}
    if kind == "map2":
        return {"kind": kind, "op": rng.choice(sorted(MAPS2)), "n": _log_int(rng, 256, 1 << 24), "dtype": dtype}
    if kind == "dot":
        return {"kind": kind, "n": _log_int(rng, 256, 1 << 26), "dtype": dtype,
                "compensated": rng.choice([True, True, False])}
    if kind == "reduce":
        rows, cols = _table(rng, 1 << 25)
        return {"kind": kind, "op": rng.choice(["sum", "sum", "mean", "stdev", "norm2", "max"]), "rows": rows,
                "cols": cols, "dim": rng.choice([1, 2, 0]), "dtype": dtype}
    if kind == "scan":
        rows, cols = _table(rng, 1 << 25) if rng.random() < 0.5 else (_log_int(rng, 4096, 1 << 26), 1)
        return {"kind": kind, "op": rng.choice(["cumsum", "cumsum", "cummax"]), "rows": rows, "cols": cols,
                "dim": rng.choice([1, 2]) if cols > 1 else 1, "dtype": dtype}
    return {"kind": kind, "streams": _log_int(rng, 1, 128), "frames": rng.randint(2, 8),
            "mix": rng.randint(1, 1 << 20)}


# ------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(g, n, lo, hi, dtype):
    return torch.rand(n, generator=g, device="cuda", dtype=dtype).mul_(hi - lo).add_(lo)


def _normal(g, n, dtype):
    return torch.randn(n, generator=g, device="cuda", dtype=dtype)


def _options(g, n, dtype):
    return (_uniform(g, n, 5.0, 30.0, dtype), _uniform(g, n, 1.0, 100.0, dtype), _uniform(g, n, 0.25, 10.0, dtype))


def _request_sizes(case):
    """The sizes of the burst's requests, log-uniform; "mix" names one draw of them."""
    g = torch.Generator()
    g.manual_seed(case["mix"])
    u = torch.rand(case["requests"], generator=g, dtype=torch.float64)
    lo, hi = math.log(256), math.log(case["max_n"])
    return [int(round(math.exp(lo + (hi - lo) * v))) for v in u.tolist()]


def _inputs(case, seed):
    g, kind = _gen(seed), case["kind"]
    dtype = DTYPES[case.get("dtype", "f32")]
    if kind == "bs":
        return _options(g, case["n"], dtype)
    if kind == "saxpy":
        return _uniform(g, case["n"], -1.0, 1.0, dtype), _uniform(g, case["n"], -1.0, 1.0, dtype)
    if kind == "map":
        lo, hi, _ = MAPS[case["op"]]
        return (_uniform(g, case["n"], lo, hi, dtype),)
    if kind == "map2":
        lo0, hi0, lo1, hi1, _ = MAPS2[case["op"]]
        return _uniform(g, case["n"], lo0, hi0, dtype), _uniform(g, case["n"], lo1, hi1, dtype)
    if kind == "dot":
        return _normal(g, case["n"], dtype), _normal(g, case["n"], dtype)
    if kind in ("reduce", "scan"):
        return (_normal(g, case["rows"] * case["cols"], dtype),)
    if kind == "server":
        return [_options(g, n, dtype) for n in _request_sizes(case)]
    raise ValueError(kind)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sigmadelta":
        return _prepare_streams(case, seed)
    x = _inputs(case, seed)
    st = dict(case, x=x)
    if kind == "bs":
        st["call"], st["put"] = torch.empty_like(x[0]), torch.empty_like(x[0])
    elif kind == "saxpy":
        st["y"] = torch.empty_like(x[1])
    elif kind in ("map", "map2"):
        st["out"] = torch.empty_like(x[0])
    elif kind == "scan":
        st["out"] = torch.empty_like(x[0])
    elif kind == "server":
        st["server"] = Server(budget_bytes=1 << 30)
        total = sum(S.numel() for S, _, _ in x)
        st["call"], st["put"] = torch.empty(total, device="cuda"), torch.empty(total, device="cuda")
        torch.cuda.synchronize()        # a request's tables are ready when it is submitted
    return st


def _prepare_streams(case, seed):
    """The streams' planes in one buffer each of labels, backgrounds and variances, and the captured launch."""
    sizes = video.stream_sizes(case["streams"], case["mix"])
    entries = video.make_batch(case["streams"], case["frames"], seed, sizes=sizes)
    bufs = {}
    for key in ("labels", "bkg", "var"):
        padded = [(e[key].numel() + 255) // 256 * 256 for e in entries]
        bufs[key] = torch.zeros(sum(padded), dtype=torch.uint8, device="cuda")
        at = 0
        for e, step in zip(entries, padded):
            e[key] = bufs[key][at:at + e[key].numel()]
            at += step
    plan = api.SigmaDeltaPlan(entries, case["frames"], init=True)
    return {"kind": "sigmadelta", "entries": entries, "bufs": bufs, "plan": plan}


def run(st):
    kind, x = st["kind"], st.get("x")
    if kind == "bs":
        return api.blackscholes(*x, RATE, SIGMA, call=st["call"], put=st["put"], cdf=st["cdf"],
                                precision=st["precision"])
    if kind == "saxpy":
        # y = 2.5*x + y works in place on the program's y; each pass accumulates into a fresh copy
        st["y"].copy_(x[1])
        return api.saxpy(2.5, x[0], st["y"])
    if kind == "map":
        return api.map_(st["op"], x[0], out=st["out"])
    if kind == "map2":
        return api.map2(st["op"], x[0], x[1], out=st["out"])
    if kind == "dot":
        return api.dot(x[0], x[1], compensated=st["compensated"])
    if kind == "reduce":
        return api.reduce(st["op"], x[0], st["rows"], st["cols"], dim=st["dim"])
    if kind == "scan":
        return api.cumulative(st["op"], x[0], st["rows"], st["cols"], dim=st["dim"], out=st["out"])
    if kind == "sigmadelta":
        st["plan"].launch()
        return st["bufs"]
    return _run_server(st)


def _run_server(st):
    """Submit the burst, copy each finished request's prices out, then give the slots back."""
    server, stream = st["server"], torch.cuda.current_stream()
    tickets = [server.submit(S, K, T, RATE, SIGMA) for S, K, T in st["x"]]
    at = 0
    for ticket, (S, _, _) in zip(tickets, st["x"]):
        n = S.numel()
        for dst, src in zip((st["call"][at:at + n], st["put"][at:at + n]), server.wait(ticket)):
            check(lib().nt2cuda_memcpy_d2d(ctypes.c_void_p(dst.data_ptr()), ctypes.c_void_p(src), 4 * n,
                                           ctypes.c_void_p(stream.cuda_stream)), "copy out")
        at += n
    stream.synchronize()
    for ticket in tickets:
        server.release(ticket)
    return st["call"], st["put"]


# --------------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    size = 8 if case.get("dtype") == "f64" else 4
    if kind == "bs":
        # S, K, T in, call and put out; a log, an exp, a root, four divisions and two erfc
        return {"bytes": 5 * size * case["n"], "flops": 160 * case["n"]}
    if kind == "saxpy":
        return {"bytes": 3 * size * case["n"], "flops": 2 * case["n"]}
    if kind == "map":
        return {"bytes": 2 * size * case["n"], "flops": MAP_FLOPS[case["op"]] * case["n"]}
    if kind == "map2":
        return {"bytes": 3 * size * case["n"], "flops": MAP_FLOPS[case["op"]] * case["n"]}
    if kind == "dot":
        return {"bytes": 2 * size * case["n"] + size, "flops": 2 * case["n"]}
    if kind == "reduce":
        outs = {0: 1, 1: case["cols"], 2: case["rows"]}[case["dim"]]
        per = {"sum": 1, "mean": 1, "stdev": 3, "norm2": 2, "max": 1}[case["op"]]
        return {"bytes": size * (case["rows"] * case["cols"] + outs), "flops": per * case["rows"] * case["cols"]}
    if kind == "scan":
        return {"bytes": 2 * size * case["rows"] * case["cols"], "flops": case["rows"] * case["cols"]}
    if kind == "sigmadelta":
        # every frame in; a label plane of all but the first, the background and the variance out
        pixels = sum(w * h for w, h in video.stream_sizes(case["streams"], case["mix"]))
        return {"bytes": pixels * (2 * case["frames"] + 1), "flops": pixels * 10 * (case["frames"] - 1)}
    total = sum(_request_sizes(case))
    return {"bytes": 20 * total, "flops": 160 * total}


# -------------------------------------------------------------------- exact
def _bs_exact(S, K, T, r, v):
    S, K, T = S.double(), K.double(), T.double()
    cdf = MAPS["normcdf"][2]
    vda = v * T.sqrt()
    d1 = ((S / K).log() + (0.5 * v * v + r) * T) / vda
    d2 = d1 - vda
    e = K * torch.exp(-r * T)
    return S * cdf(d1) - e * cdf(d2), e * cdf(-d2) - S * cdf(-d1)


def _scalar(v, dtype):
    """The value a call in this type receives for the Python number v."""
    return torch.tensor(v, dtype=dtype).double().item()


def exact(case, seed):
    kind = case["kind"]
    if kind == "sigmadelta":        # bytes: no rounding in them
        return None
    dtype = DTYPES[case.get("dtype", "f32")]
    r, v = _scalar(RATE, dtype), _scalar(SIGMA, dtype)
    x = _inputs(case, seed)
    if kind == "bs":
        return _bs_exact(*x, r, v)
    if kind == "server":
        prices = [_bs_exact(*t, r, v) for t in x]
        return torch.cat([c for c, _ in prices]), torch.cat([p for _, p in prices])
    x = [t.double() for t in x]
    if kind == "saxpy":
        return 2.5 * x[0] + x[1]
    if kind == "map":
        return MAPS[case["op"]][2](x[0])
    if kind == "map2":
        return MAPS2[case["op"]][4](x[0], x[1])
    if kind == "dot":
        return (x[0] * x[1]).sum().reshape(1)
    A = x[0].view(case["cols"], case["rows"])       # column-major: one column per row of the view
    if kind == "reduce":
        axis = {0: (0, 1), 1: 1, 2: 0}[case["dim"]]
        op = case["op"]
        if op == "sum":
            res = A.sum(axis)
        elif op == "mean":
            res = A.mean(axis)
        elif op == "stdev":
            res = A.std(axis, correction=1)
        elif op == "norm2":
            res = A.square().sum(axis).sqrt()
        else:
            res = A.amax(axis)
        return res.reshape(-1)
    axis = 1 if case["dim"] == 1 else 0
    res = A.cumsum(axis) if case["op"] == "cumsum" else A.cummax(axis).values
    return res.reshape(-1)
