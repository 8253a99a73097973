"""Data that the float32 L2 gradients by contraction (csrc/backward_l2.cu) must
not be thrown off by, against the float64 gradients of the same numbers.

Tolerance, as in test_gpu_l2_gradient.py: 2e-6 in the norm of the whole
gradient, from about 600 rounded terms of random sign an entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 2e-6
KINDS = ["kernel", "l2"]


def _run(points, offsets, kind, w):
    import torch
    from stablebear_gb300 import autograd
    P = points.clone().requires_grad_(True)
    longest = int((offsets[1:] - offsets[:-1]).max())
    f = autograd.l2_kernel if kind == "kernel" else autograd.pdist
    out = f(P, offsets, max_points=longest)
    grad, = torch.autograd.grad(out, P, w)
    return out.detach(), grad


def _data(n, lo, hi, seed):
    import torch
    rng = np.random.default_rng(seed)
    ln = rng.integers(lo, hi + 1, n)
    off = np.zeros(n + 1, np.int64)
    np.cumsum(ln, out=off[1:])
    t = np.concatenate([np.r_[0.0, np.cumsum(rng.exponential(1.0, k - 1) + 1e-3)] for k in ln])
    v = rng.standard_normal(int(off[-1]))
    v[off[1:] - 1] = 0.0
    return torch.from_numpy(np.stack([t, v], 1).astype(np.float32)).cuda(), torch.from_numpy(off).cuda()


def _weights(n, kind, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(n * (n + 1) // 2 if kind == "kernel" else n * (n - 1) // 2, generator=g, device="cuda") / n


def _near(got, want):
    for c in range(2):
        err = float((got[:, c].double() - want[:, c]).norm() / want[:, c].norm())
        assert err <= TOL, (c, err)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("rows", ["nan", "stale"])
def test_rows_behind_the_last_pcf(kind, rows):
    """A points tensor may be longer than the offsets say; what stands in the
    rest is not read and gets no gradient."""
    import torch
    pts, off = _data(1000, 80, 150, seed=2)
    spare = torch.full((len(pts) // 50, 2), float("nan") if rows == "nan" else -3e8, device="cuda")
    both = torch.cat([pts, spare])
    w = _weights(1000, kind, 2)
    got = _run(both, off, kind, w)[1]
    assert bool((got[len(pts):] == 0).all())
    _near(got[:len(pts)], _run(pts.double(), off, kind, w.double())[1])


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n,points", [(7500, 2), (1000, 120)])
@pytest.mark.parametrize("where", ["zero", "negative zero", "twice"])
def test_elements_without_width(kind, n, points, where):
    """A breakpoint at time 0 (or -0.0) behind the first one, or two at one
    time: an element without width, whose time gradient is the walk's.  7500
    breakpoints fit one bin, 119,000 do not."""
    pts, off = _data(n, points, points, seed=n)
    k = off[:-1:7] + 1
    if where == "twice":
        if points < 3:
            pytest.skip("needs a third breakpoint")
        pts[k + 60, 0] = pts[k + 59, 0]
    else:
        pts[k, 0] = 0.0 if where == "zero" else -0.0
    w = _weights(n, kind, 3)
    _near(_run(pts, off, kind, w)[1], _run(pts.double(), off, kind, w.double())[1])


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("size", [1e38, 3e38])
def test_a_pcf_that_overflows(kind, size):
    """One PCF whose integrals are beyond float32 and whose pairs all have
    weight 0: it gets no gradient, and nobody gets one from it.  3e38: its
    steps from value to value overflow too."""
    import torch
    n, one = 1000, 123
    pts, off = _data(n, 80, 150, seed=7)
    a, b = int(off[one]), int(off[one + 1])
    pts[a:b - 1, 1] = size * torch.sign(pts[a:b - 1, 1])
    w = torch.zeros(n, n, device="cuda")
    i, j = torch.tril_indices(n, n, 0 if kind == "kernel" else -1, device="cuda")
    w[i, j] = _weights(n, kind, 7)
    w[one, :] = 0
    w[:, one] = 0
    w = w[i, j]
    got = _run(pts, off, kind, w)[1]
    assert bool((got[a:b] == 0).all())
    _near(got, _run(pts.double(), off, kind, w.double())[1])


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n,lo,hi", [(1000, 100, 200), (700, 300, 500), (2047, 60, 90)])
def test_each_value_gradient_against_its_own_terms(kind, n, lo, hi):
    """Segments from a millionth to a few units of time, far shorter and far
    longer than a bin.  An entry sums w_ij times the integral of |g_j|, and of
    |v| for distances, over its own segment: at most 256 + n / 256 rounded terms
    of the product, a bin's list over 32 lanes (under 64 each), 14 more; where a
    quarter of a bin is left of the whole, four times that."""
    import torch
    pts, off = _data(n, lo, hi, seed=n + 1)
    rng = np.random.default_rng(n)
    t = pts[:, 0].double().cpu().numpy()
    gaps = np.diff(t, append=0.0)
    short = rng.random(len(gaps)) < 0.3
    gaps[short] *= 10.0 ** rng.uniform(-6, 0, short.sum())
    o = off.cpu().numpy()
    for a, b in zip(o[:-1], o[1:]):
        t[a:b] = np.r_[0.0, np.cumsum(gaps[a:b - 1])]
        x = t[a:b].astype(np.float32)
        while np.any(np.diff(x) <= 0):  # times ascend in float32 too
            at = np.nonzero(np.diff(x) <= 0)[0] + 1
            x[at] = np.nextafter(x[at - 1], np.float32(np.inf))
        t[a:b] = x
    pts[:, 0] = torch.from_numpy(t).cuda()
    w = _weights(n, kind, 9)
    out, got = _run(pts, off, kind, w)
    dout, want = _run(pts.double(), off, kind, w.double())
    ap = pts.double().abs()
    i, j = torch.tril_indices(n, n, 0 if kind == "kernel" else -1, device="cuda")
    a = torch.zeros(n, n, device="cuda", dtype=torch.float64)
    a[i, j] = w.double().abs() if kind == "kernel" else (w.double() / dout).abs()
    k, m = torch.tril_indices(n, n, 0, device="cuda")
    scale = _run(ap, off, "kernel", a[k, m])[1][:, 1]
    if kind == "l2":
        total = (a + a.T).sum(1)
        owner = torch.repeat_interleave(torch.arange(n, device="cuda"), off[1:] - off[:-1])
        width = torch.zeros(len(pts), device="cuda", dtype=torch.float64)
        width[:-1] = (ap[1:, 0] - ap[:-1, 0]).clamp(min=0)
        scale = scale + total[owner] * ap[:, 1] * width
    last = torch.zeros(len(pts), dtype=torch.bool, device="cuda")
    last[off[1:] - 1] = True
    err = ((got[:, 1].double() - want[:, 1]).abs() / scale)[~last]
    assert float(err.max()) <= 4 * (256 + n / 256 + 64 + 14) * 2.0 ** -24, float(err.max())


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("each", [1, 3])
def test_elements_without_width_at_shared_times(kind, each):
    """Times on a grid, where other PCFs have breakpoints at the same time as
    an element without width; one such element in a PCF, or three, of which
    there are more than PCFs."""
    import torch
    n, points = 1000, 120
    pts, off = _data(n, points, points, seed=11)
    rng = np.random.default_rng(12)
    t = np.concatenate([np.r_[0.0, np.sort(rng.choice(2000, points - 1, replace=False) + 1) / 16] for _ in range(n)])
    pts[:, 0] = torch.from_numpy(t.astype(np.float32)).cuda()
    for e in range(each):
        k = off[:-1] + 20 + 30 * e
        pts[k, 0] = pts[k - 1, 0]
    if each == 3:
        pts[off[:-1:4] + 50 + 1, 0] = pts[off[:-1:4] + 50, 0]  # three breakpoints at one time
    w = _weights(n, kind, 13)
    _near(_run(pts, off, kind, w)[1], _run(pts.double(), off, kind, w.double())[1])


@pytest.mark.parametrize("n,points", [(4096, 128), (2048, 256), (1024, 1024)])
def test_pcfs_of_one_length(n, points):
    """Lengths that divide the stretches the edges are sampled from: the bins
    stay even and the contraction runs, whose kernel gradients add nothing
    atomically, so that a second run gives the same bits."""
    pts, off = _data(n, points, points, seed=points)
    w = _weights(n, "kernel", 5)
    got = _run(pts, off, "kernel", w)[1]
    assert bool((got == _run(pts, off, "kernel", w)[1]).all())
    _near(got, _run(pts.double(), off, "kernel", w.double())[1])
