"""The float32 L2 gradients by contraction (csrc/backward_l2.cu) against the
float64 gradients of the same float32 data (the walk of backward.cu, pinned to
the FP64 reference gradient in test_gpu_autograd.py).

Tolerance: in the norm of the whole gradient, 2e-6.  A gradient entry sums
about 600 rounded terms (chunks of 256 products, 16 chunk sums, a list of a
bin over 32 lanes, a few bins) of random sign, each to 2^-24: at most
600 * 2^-24 = 3.6e-5 of the sum of |terms|, and of its root-mean-square size,
which is what the norm sees, sqrt(600) * 2^-24 = 1.5e-6."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 2e-6


def _run(points, offsets, kind, w):
    import torch
    from stablebear_gb300 import autograd
    P = points.clone().requires_grad_(True)
    longest = int((offsets[1:] - offsets[:-1]).max())
    if kind == "kernel":
        out = autograd.l2_kernel(P, offsets, max_points=longest)
    else:
        out = autograd.pdist(P, offsets, p=2, max_points=longest)
    grad, = torch.autograd.grad(out, P, w)
    return out.detach(), grad


def _data(n, lens, seed, ticks=None, shift=0.0):
    import torch
    rng = np.random.default_rng(seed)
    ln = rng.choice(lens, size=n) if not callable(lens) else lens(rng, n)
    off = np.zeros(n + 1, np.int64)
    np.cumsum(ln, out=off[1:])
    t = np.concatenate([np.r_[0.0, np.cumsum(rng.exponential(1.0, k - 1) + 1e-3)] for k in ln])
    if ticks:
        # distinct within a PCF, shared between PCFs
        t = np.concatenate([np.r_[0.0, np.sort(rng.choice(ticks * int(ln.max()) * 2, k - 1, replace=False) + 1) / ticks]
                            for k in ln])
    v = rng.standard_normal(int(off[-1])) + shift
    v[off[1:] - 1] = 0.0
    pts = np.stack([t, v], 1).astype(np.float32)
    return torch.from_numpy(pts).cuda(), torch.from_numpy(off).cuda()


def _weights(n, kind, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(n * (n + 1) // 2 if kind == "kernel" else n * (n - 1) // 2, generator=g, device="cuda") / n


def _compare(pts, off, kind, w):
    out, got = _run(pts, off, kind, w)
    # the float64 weights of the distances use the float32 result, as the gradient does
    _, want = _run(pts.double(), off, kind, w.double())
    for c in range(2):
        err = float((got[:, c].double() - want[:, c]).norm() / want[:, c].norm())
        assert err <= TOL, (c, err)
    return got


@pytest.mark.parametrize("kind", ["kernel", "l2"])
@pytest.mark.parametrize("n,lo,hi", [(700, 200, 400), (1025, 1, 300), (1280, 90, 91), (2047, 2, 100), (310, 1100, 1300),
                                     (4100, 1, 30)])
def test_against_float64(kind, n, lo, hi):
    """Sizes around the tiles of the product, rows per CTA and panels of the
    length order; one-element PCFs; about one breakpoint to a bin and many."""
    pts, off = _data(n, lambda rng, m: rng.integers(lo, hi + 1, m), seed=n)
    a = _compare(pts, off, kind, _weights(n, kind, n))
    assert bool((a[off[:-1], 0] == 0).all())
    if kind == "kernel":  # nothing is added atomically (pairs of distances close together are)
        assert bool((a == _run(pts, off, kind, _weights(n, kind, n))[1]).all())


@pytest.mark.parametrize("kind", ["kernel", "l2"])
def test_shared_breakpoints(kind):
    """Times on a grid: many PCFs share a breakpoint, which then gets no time
    gradient from them."""
    pts, off = _data(1000, (40, 150, 160), seed=4, ticks=64)
    _compare(pts, off, kind, _weights(1000, kind, 4))


@pytest.mark.parametrize("kind", ["kernel", "l2"])
def test_a_common_offset(kind):
    """Values far from 0 but near one another."""
    pts, off = _data(1100, (80, 100, 120), seed=5, shift=30.0)
    got = _run(pts, off, kind, _weights(1100, kind, 5))[1]
    want = _run(pts.double(), off, kind, _weights(1100, kind, 5).double())[1]
    for c in range(2):
        assert float((got[:, c].double() - want[:, c]).norm() / want[:, c].norm()) <= 10 * TOL


@pytest.mark.parametrize("what", ["tail", "value", "weight", "nan weight", "one time", "start"])
def test_data_that_takes_the_walk(what):
    """A last value other than 0, values or weights that are not finite, more
    breakpoints at one time than a bin holds: the walk runs behind the gate, and non-finite entries appear
    where it puts them (in float64 the walk is the only path)."""
    import torch
    n = 9000 if what == "one time" else 800
    pts, off = _data(n, (3, 4) if what == "one time" else (150, 200), seed=6)
    if what == "one time":
        n = len(off) - 1
        first = off[:-1][(off[1:] - off[:-1]) > 1] + 1
        pts[first, 0] = 1e-4
        pts = torch.cat([pts, torch.zeros(0, 2, device="cuda")])
    w = _weights(n, "kernel", 6)
    k = int(off[5]) + 1
    if what == "tail":
        pts[off[6] - 1, 1] = 1e-30
    elif what == "value":
        pts[k, 1] = float("inf")
    elif what == "weight":
        w[1234] = float("inf")
    elif what == "nan weight":
        w[1234] = float("nan")
    elif what == "start":
        pts[off[7], 0] = 0.25
    got = _run(pts, off, "kernel", w)[1]
    want = _run(pts.double(), off, "kernel", w.double())[1]
    fin = torch.isfinite(want) & torch.isfinite(got)
    if what == "tail":
        # last values see a rectangle up to the type's largest number: no common value
        fin[off[1:] - 1, 1] = False
    assert bool((torch.isnan(got) == torch.isnan(want)).all())
    assert float((got.double() - want)[fin].norm() / want[fin].norm()) <= 5 * TOL


def test_pairs_close_together():
    """Near-duplicates, whose distances are far smaller than the PCFs: the
    contraction leaves them to the walk and adds its gradient."""
    import torch
    pts, off = _data(500, (150, 200, 250), seed=9)
    rng = torch.Generator(device="cuda")
    rng.manual_seed(1)
    twin = pts.clone()
    twin[:, 1] += 1e-3 * torch.randn(len(pts), generator=rng, device="cuda") * (pts[:, 1] != 0)
    both = torch.cat([pts, twin, pts])
    offs = torch.cat([off, off[1:] + len(pts), off[1:] + 2 * len(pts)])
    w = _weights(1500, "l2", 9)
    got = _run(both, offs, "l2", w)[1]
    want = _run(both.double(), offs, "l2", w.double())[1]
    # the float32 distance of a twin is itself off by some 1e-5 of it, here and in the walk alone
    for c in range(2):
        assert float((got[:, c].double() - want[:, c]).norm() / want[:, c].norm()) <= 2e-5


def test_panels_of_rows():
    """More rows than one product holds (1 GB of weights)."""
    n = 17500
    pts, off = _data(n, (1, 2, 6), seed=8)
    _compare(pts, off, "l2", _weights(n, "l2", 8))
