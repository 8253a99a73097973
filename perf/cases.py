"""Performance cases: what a user of this package has it compute, through its
public entry points, from the smallest calls to the largest.

``listed()`` names the cases that are always timed, ``draw(rng)`` makes one
more of the same ranges, ``prepare`` builds what a program has in hand before
the call, ``run`` is one call, ``work`` the bytes and floating-point
operations it cannot do without, and ``exact`` the result in 64-bit
arithmetic from plain torch.

Kinds of case:

* ``host``    numpy CSR in, numpy matrix out: ``sb.pdist`` / ``sb.cdist`` /
              ``sb.l2_kernel``, as most programs call the package.
* ``device``  CUDA CSR in, condensed CUDA matrix out (``autograd.pdist`` /
              ``autograd.l2_kernel`` without gradients).
* ``grad``    forward and backward of the same.
* ``batch``   many independent problems in one planned launch.
* ``dense``   condensed storage to the dense matrix and back, on the device.

PCFs are those of the repository's own workloads (``synthetic.py``), drawn on
the GPU: Exp(1) gaps, with N(0, 1) values ("gaussian"), non-increasing
integer values over lengths from 16 to 4096 ("stable_rank"), or the integer
walk of a Betti curve ("betti"); the last value is always 0.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import stablebear_gb300 as sb
from stablebear_gb300 import autograd
from stablebear_gb300.batch import PairwiseBatch
from stablebear_gb300.device import condensed_to_dense, dense_to_condensed

#: Operations per merged rectangle: compare, width, difference or product, scale, accumulate.
OPS_PER_RECTANGLE = 5
#: exact() is skipped above this many (breakpoint, other PCF) evaluations.
MOST_EVALUATIONS = 1.7e10


def listed():
    return [
        # a notebook call: a hundred PCFs, latency is all that counts
        dict(name="host_l1_n100", kind="host", call="pdist", p=1.0, n=100, lengths="uniform", lo=10, hi=200,
             values="gaussian", dtype="float32"),
        # the small pdist workload on data already on the GPU
        dict(name="device_l1_n1000", kind="device", op="l1", n=1000, lengths="uniform", lo=10, hi=200,
             values="gaussian", dtype="float32"),
        # the headline workload: the largest distance matrix
        dict(name="device_l1_n100000", kind="device", op="l1", n=100000, lengths="poisson", lo=256, hi=2,
             values="gaussian", dtype="float32"),
        # an ordinary call end to end from host memory
        dict(name="host_l1_n6007", kind="host", call="pdist", p=1.0, n=6007, lengths="poisson", lo=256, hi=2,
             values="gaussian", dtype="float32"),
        # a distance of general order
        dict(name="host_l3_n2000", kind="host", call="pdist", p=3.0, n=2000, lengths="uniform", lo=10, hi=200,
             values="gaussian", dtype="float32"),
        # cross distances of two sets of different sizes in double precision, arbitrary values
        dict(name="host_cdist_l1_f64", kind="host", call="cdist", p=1.0, n=1003, m=701, lengths="uniform", lo=10,
             hi=300, values="gaussian", dtype="float64"),
        # kernel matrix of persistence stable ranks, double precision, very uneven lengths
        dict(name="device_kernel_f64_rank", kind="device", op="kernel", n=3500, lengths="log", lo=16, hi=4096,
             values="stable_rank", dtype="float64"),
        # and their L2 distances
        dict(name="device_l2_f64_rank", kind="device", op="l2", n=2501, lengths="log", lo=16, hi=4096,
             values="stable_rank", dtype="float64"),
        # training on the kernel matrix: forward and backward
        dict(name="grad_kernel_n4096", kind="grad", op="kernel", n=4096, lengths="uniform", lo=16, hi=512,
             values="gaussian", dtype="float32"),
        # training on L2 distances, a smaller batch
        dict(name="grad_l2_n1021", kind="grad", op="l2", n=1021, lengths="uniform", lo=16, hi=512,
             values="gaussian", dtype="float32"),
        # many small and middling problems of uneven size at once
        dict(name="batch_l1_24", kind="batch", op="l1", problems=24, lo_n=50, hi_n=2000, lengths="uniform", lo=8,
             hi=1024, values="betti", dtype="float32"),
        # a result handed on to code that wants the full matrix
        dict(name="dense_from_condensed_n30011", kind="dense", direction="expand", storage="distance", n=30011,
             dtype="float32"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "host", "device", "device", "device", "grad", "grad", "batch", "dense"])
    if kind == "dense":
        return dict(kind=kind, direction=rng.choice(["expand", "condense"]),
                    storage=rng.choice(["distance", "symmetric"]), n=_log_int(rng, 400, 40000),
                    dtype=rng.choice(["float32", "float32", "float64"]))
    if kind == "batch":
        return dict(kind=kind, op=rng.choice(["l1", "l2_kernel", "lp"]), problems=rng.randint(3, 40), lo_n=50,
                    hi_n=rng.choice([300, 2000]), lengths="uniform", lo=8, hi=rng.randint(40, 1024), values="betti",
                    dtype="float32")
    c = dict(kind=kind, dtype="float32", values="gaussian")
    shape = rng.choice(["uniform", "poisson"])
    c.update(lengths=shape, lo=256 if shape == "poisson" else rng.randint(4, 32),
             hi=2 if shape == "poisson" else rng.randint(60, 512))
    if kind == "grad":
        c.update(op=rng.choice(["kernel", "l2", "l1"]), n=_log_int(rng, 100, 4000))
        return c
    if kind == "device":
        if rng.random() < 0.4:
            c.update(dtype="float64", n=_log_int(rng, 100, 3000))
            if rng.random() < 0.6:
                c.update(lengths="log", lo=16, hi=rng.choice([512, 4096]), values="stable_rank")
        else:
            c.update(n=_log_int(rng, 200, 90000))
        c.update(op=rng.choice(["l1", "l2", "kernel"]))
        return c
    c.update(call=rng.choice(["pdist", "pdist", "cdist", "l2_kernel"]), p=rng.choice([1.0, 1.0, 2.0, 3.0, 1.5]))
    f64 = rng.random() < 0.3
    if f64:
        c["dtype"] = "float64"
    c["n"] = _log_int(rng, 20, 1500 if f64 else 9000)
    if c["call"] == "cdist":
        c["n"] = _log_int(rng, 20, 1500 if f64 else 4000)
        c["m"] = _log_int(rng, 20, 1500 if f64 else 4000)
    return c


# --- inputs -----------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _lengths(case, n):
    """The lengths are the case's own, the same for every seed."""
    lo, hi, g = case["lo"], case["hi"], _generator(n)
    if case["lengths"] == "uniform":
        return torch.randint(lo, hi + 1, (n,), generator=g, device="cuda")
    if case["lengths"] == "poisson":
        return torch.poisson(torch.full((n,), float(lo), device="cuda"), generator=g).long() + hi
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    return torch.exp(math.log(lo) + u * (math.log(hi) - math.log(lo))).round().long()


def _pcfs(case, n, g):
    """CSR of n PCFs on the GPU: points (M, 2) and int64 offsets.  A gap is
    Exp(1) plus a thousandth, so times stay apart in float32 too.  Gaps are
    summed as whole numbers, whose sums are the same in any order."""
    lens = _lengths(case, n)
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(lens, 0)
    total = int(off[-1])
    first = off[:-1]
    gaps = torch.empty(total, dtype=torch.float64, device="cuda").exponential_(1.0, generator=g) + 1e-3
    ticks = (gaps * 2.0 ** 24).long()
    ticks[first] = 0
    ticks = torch.cumsum(ticks, 0)
    ticks = ticks - torch.repeat_interleave(ticks[first], lens)
    t = ticks.double() * (math.sqrt(0.999) / 2.0 ** 24)  # times with all their digits
    if case["values"] == "gaussian":
        v = torch.randn(total, generator=g, device="cuda", dtype=torch.float64)
    else:
        if case["values"] == "stable_rank":
            step = -torch.empty(total, dtype=torch.float64, device="cuda").geometric_(0.3, generator=g)
            v0 = torch.randint(1, 501, (n,), generator=g, device="cuda").double()
        else:
            step = torch.randint(0, 2, (total,), generator=g, device="cuda").double() * 2 - 1
            v0 = torch.randint(0, 11, (n,), generator=g, device="cuda").double()
        step[first] = 0
        walk = torch.cumsum(step, 0)
        walk = walk - torch.repeat_interleave(walk[first], lens) + torch.repeat_interleave(v0, lens)
        v = walk.clamp(min=0) if case["values"] == "stable_rank" else walk.abs()
    v[off[1:] - 1] = 0
    dt = torch.float32 if case["dtype"] == "float32" else torch.float64
    return torch.stack([t.to(dt), v.to(dt)], dim=1).contiguous(), off, int(lens.max())


def _host_array(points, offsets):
    return sb.PcfArray.from_csr(points.cpu().numpy(), offsets.cpu().numpy().astype(np.uint64))


def _problem_sizes(case):
    """The sizes are the case's own, the same for every seed."""
    r = np.random.default_rng(case["problems"])
    return [int(x) for x in r.integers(case["lo_n"], case["hi_n"] + 1, size=case["problems"])]


def _condensed_count(storage, n):
    return n * (n + 1) // 2 if storage == "symmetric" else n * (n - 1) // 2


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind == "dense":
        dt = torch.float32 if case["dtype"] == "float32" else torch.float64
        n = case["n"]
        c = torch.rand(_condensed_count(case["storage"], n), generator=g, device="cuda", dtype=dt)
        if case["direction"] == "expand":
            return {"case": case, "storage": c}
        return {"case": case, "dense": condensed_to_dense(c, n, case["storage"])}
    if kind == "batch":
        problems = []
        for n in _problem_sizes(case):
            pts, off, _ = _pcfs(case, n, g)
            problems.append((pts.cpu().numpy(), off.cpu().numpy().astype(np.uint64)))
        return {"case": case, "batch": PairwiseBatch(problems, op=case["op"], p=2.0 if case["op"] == "lp" else 1.0)}
    pts, off, longest = _pcfs(case, case["n"], g)
    if kind == "host":
        state = {"case": case, "x": _host_array(pts, off)}
        if case["call"] == "cdist":
            state["y"] = _host_array(*_pcfs(case, case["m"], g)[:2])
        return state
    state = {"case": case, "points": pts, "offsets": off, "longest": longest}
    if kind == "grad":
        pts.requires_grad_(True)
        count = _condensed_count("symmetric" if case["op"] == "kernel" else "distance", case["n"])
        state["weight"] = torch.randn(count, generator=g, device="cuda", dtype=pts.dtype) / case["n"]
    return state


# --- one pass ---------------------------------------------------------------

def _device_matrix(case, points, offsets, longest):
    if case["op"] == "kernel":
        return autograd.l2_kernel(points, offsets, max_points=longest)
    return autograd.pdist(points, offsets, p=1 if case["op"] == "l1" else 2, max_points=longest)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "device":
        return _device_matrix(case, state["points"], state["offsets"], state["longest"])
    if kind == "grad":
        out = _device_matrix(case, state["points"], state["offsets"], state["longest"])
        grad, = torch.autograd.grad(out, state["points"], state["weight"])
        return out, grad
    if kind == "batch":
        return state["batch"].run()
    if kind == "dense":
        if case["direction"] == "expand":
            return condensed_to_dense(state["storage"], case["n"], case["storage"])
        return dense_to_condensed(state["dense"], case["storage"])
    if case["call"] == "cdist":
        return sb.cdist(state["x"], state["y"], p=case["p"])
    if case["call"] == "l2_kernel":
        return sb.l2_kernel(state["x"]).data
    return sb.pdist(state["x"], p=case["p"]).data


# --- what a pass cannot do without --------------------------------------------

def _mean_length(case):
    lo, hi = case["lo"], case["hi"]
    if case["lengths"] == "uniform":
        return (lo + hi) / 2
    if case["lengths"] == "poisson":
        return lo + hi
    return (hi - lo) / math.log(hi / lo)


def work(case):
    es = 4 if case["dtype"] == "float32" else 8
    kind = case["kind"]
    if kind == "dense":
        return {"bytes": es * (_condensed_count(case["storage"], case["n"]) + case["n"] ** 2), "flops": 0}
    mean = _mean_length(case)
    if kind == "batch":
        diag = "symmetric" if case["op"] == "l2_kernel" else "distance"
        sizes = _problem_sizes(case)
        pairs, pcfs = sum(_condensed_count(diag, n) for n in sizes), sum(sizes)
    elif case.get("call") == "cdist":
        pairs, pcfs = case["n"] * case["m"], case["n"] + case["m"]
    else:
        diag = "symmetric" if "kernel" in (case.get("op"), case.get("call", "")[3:]) else "distance"
        pairs, pcfs = _condensed_count(diag, case["n"]), case["n"]
    points = pcfs * mean
    size = es * (2 * points + pairs) + 8 * pcfs
    flops = OPS_PER_RECTANGLE * pairs * (2 * mean - 1)
    if kind == "grad":  # the weights in and the gradients out; both sides' terms of every rectangle again
        size += es * (2 * points + pairs)
        flops *= 3
    return {"bytes": size, "flops": flops}


# --- the same in 64 bits ------------------------------------------------------

def _padded(points, offsets):
    """Times (padded with inf) and values (with the last one) of shape
    (n, longest + 1), in float64."""
    p = points.detach().double()
    lens = offsets[1:] - offsets[:-1]
    width = int(lens.max()) + 1
    k = torch.arange(width, device=p.device)
    at = offsets[:-1, None] + torch.minimum(k[None, :], lens[:, None] - 1)
    t = p[:, 0][at]
    t[k[None, :] >= lens[:, None]] = math.inf
    return t, p[:, 1][at], lens


class _Side:
    def __init__(self, points, offsets):
        self.t, self.v, self.lens = _padded(points, offsets)
        p = points.detach().double()
        self.off, self.n, self.m = offsets, offsets.numel() - 1, p.shape[0]
        self.start, self.value = p[:, 0].contiguous(), p[:, 1].contiguous()
        self.pcf = torch.repeat_interleave(torch.arange(self.n, device=p.device), self.lens)
        last = torch.zeros(self.m, dtype=torch.bool, device=p.device)
        last[offsets[1:] - 1] = True
        self.end = torch.roll(self.start, -1).masked_fill(last, math.inf)
        self.first = offsets[:-1]

    def at(self, lo, hi, times):
        """For PCFs lo..hi at every one of the times: (value, where it ends,
        whether a breakpoint lies there, index of the segment)."""
        q = times[None, :].expand(hi - lo, -1).contiguous()
        k = torch.searchsorted(self.t[lo:hi], q, right=True) - 1
        return (torch.gather(self.v[lo:hi], 1, k), torch.gather(self.t[lo:hi], 1, k + 1),
                torch.gather(self.t[lo:hi], 1, k) == q, k)


def _phi(op, p, f, g):
    if op == "kernel":
        return f * g
    d = (f - g).abs()
    return d if p == 1 else d * d if p == 2 else d ** p


def _widths(begin, end):
    w = end - begin
    return torch.where(torch.isinf(w), torch.zeros_like(w), w)  # both PCFs are 0 there


def _matrix(rows, cols, op, p):
    """All pairs: every merged rectangle begins at a breakpoint of the row
    (counted for a block of columns) or at one of the column alone."""
    out = torch.zeros(rows.n, cols.n, dtype=torch.float64, device=rows.t.device)

    def half(a, b, skip_ties):
        step = max(1, int(4e7) // max(1, a.m))
        for lo in range(0, b.n, step):
            hi = min(b.n, lo + step)
            g, end, tie, _ = b.at(lo, hi, a.start)
            w = _widths(a.start[None, :], torch.minimum(end, a.end[None, :]))
            x = _phi(op, p, a.value[None, :], g) * w
            if skip_ties:
                x = x.masked_fill(tie, 0.0)
            x = torch.segment_reduce(x.t().contiguous(), "sum", lengths=a.lens, axis=0, unsafe=True)
            if a is rows and not skip_ties:
                out[:, lo:hi] += x
            else:
                out[lo:hi, :] += x.t()

    half(rows, cols, False)
    half(cols, rows, True)
    if op != "kernel" and p != 1:
        out = out ** (1 / p)
    return out


def _condense(full, with_diagonal):
    n = full.shape[0]
    i, j = torch.tril_indices(n, n, 0 if with_diagonal else -1, device=full.device)
    return full[i, j]


def _gradient(side, op, p, weight):
    n = side.n
    full = _matrix(side, side, op, p)
    w = torch.zeros(n, n, dtype=torch.float64, device=side.t.device)
    i, j = torch.tril_indices(n, n, 0 if op == "kernel" else -1, device=w.device)
    w[i, j] = weight.double()
    w = w + w.t()  # the kernel's diagonal counts for both of its sides
    if op != "kernel" and p == 2:
        w = torch.where(full > 0, w / full.clamp(min=1e-300), torch.zeros_like(w))
    scale = 0.5 if op != "kernel" and p == 2 else 1.0

    def slope(f, g):
        return g if op == "kernel" else torch.sign(f - g) if p == 1 else f - g

    gv = torch.zeros(side.m, dtype=torch.float64, device=w.device)
    gt = torch.zeros_like(gv)
    before = torch.roll(side.value, 1)
    inner = torch.ones(side.m, dtype=torch.bool, device=w.device)
    inner[side.first] = False
    step = max(1, int(2e7) // max(1, side.m))
    for lo in range(0, n, step):
        hi = min(n, lo + step)
        # rectangles that begin at the breakpoints of the PCF that takes the gradient
        g, end, tie, _ = side.at(lo, hi, side.start)
        wt = w[lo:hi][:, side.pcf]
        f = side.value[None, :]
        gv += (wt * slope(f, g) * _widths(side.start[None, :], torch.minimum(end, side.end[None, :]))).sum(0)
        delta = scale * (_phi(op, p, before[None, :], g) - _phi(op, p, f, g))
        own = side.pcf[None, :] == torch.arange(lo, hi, device=w.device)[:, None]
        if op == "kernel":  # of <f, f> with respect to f's own breakpoint, both sides at once
            delta = torch.where(own, 0.5 * (before * before - side.value * side.value)[None, :], delta)
        gt += torch.where(inner[None, :] & (~tie | own), wt * delta, torch.zeros_like(wt)).sum(0)
        # rectangles that begin at the other PCF's breakpoints alone
        f, end, tie, k = side.at(lo, hi, side.start)
        x = w[lo:hi][:, side.pcf] * slope(f, side.value[None, :])
        x = x * _widths(side.start[None, :], torch.minimum(end, side.end[None, :]))
        gv.index_add_(0, (k + side.first[lo:hi, None]).reshape(-1), x.masked_fill(tie, 0.0).reshape(-1))
    return _condense(full, op == "kernel"), torch.stack([gt, gv], dim=1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "dense":
        return None  # nothing is computed
    g = _generator(seed)
    if kind == "batch":
        sizes = _problem_sizes(case)
        if sum(n * n for n in sizes) * _mean_length(case) > MOST_EVALUATIONS:
            return None
        op = "kernel" if case["op"] == "l2_kernel" else "distance"
        out = []
        for n in sizes:
            s = _Side(*_pcfs(case, n, g)[:2])
            out.append(_condense(_matrix(s, s, op, 2 if case["op"] == "lp" else 1), op == "kernel"))
        return out
    n, m = case["n"], case.get("m", case["n"])
    if n * m * _mean_length(case) > MOST_EVALUATIONS / (2 if kind == "grad" else 1):
        return None
    rows = _Side(*_pcfs(case, n, g)[:2])
    if kind == "host":
        if case["call"] == "cdist":
            return _matrix(rows, _Side(*_pcfs(case, m, g)[:2]), "distance", case["p"]).cpu().numpy()
        op = "kernel" if case["call"] == "l2_kernel" else "distance"
        return _condense(_matrix(rows, rows, op, case["p"]), op == "kernel").cpu().numpy()
    op, p = ("kernel", 1) if case["op"] == "kernel" else ("distance", 1 if case["op"] == "l1" else 2)
    if kind == "device":
        return _condense(_matrix(rows, rows, op, p), op == "kernel")
    count = _condensed_count("symmetric" if op == "kernel" else "distance", n)
    dt = torch.float32 if case["dtype"] == "float32" else torch.float64
    weight = torch.randn(count, generator=g, device="cuda", dtype=dt) / n
    return _gradient(rows, op, p, weight)
