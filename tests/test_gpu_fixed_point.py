"""The fixed-point float64 path (csrc/fixed_point.cu) against the double-double
oracle and the direct kernels.

Tolerance: a pair is accepted with an error bound of 2^-47 of its sum of
|terms| and walked in double precision otherwise (64 naive steps: 63 * 2^-53);
both stay below 2^-46 = 1.4e-14 of the sum of |terms|.  For distances that sum
is the integral itself; for the L2 kernel it is bounded by the integral of
|f| |g|, computed by the oracle on absolute values."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 2.0 ** -46


def _pack(lists):
    off = np.zeros(len(lists) + 1, np.uint64)
    np.cumsum([len(p) for p in lists], out=off[1:])
    return np.concatenate([np.asarray(p, np.float64).reshape(-1, 2) for p in lists]), off


def _random(n, lens, values, seed, ticks=0):
    """`ticks`: times on a grid of that many per unit (ties), 0: anywhere."""
    rng = np.random.default_rng(seed)
    out = []
    for i in range(n):
        k = int(rng.choice(lens))
        t = np.concatenate([[0.0], np.cumsum(rng.exponential(1.0, k - 1))])
        if ticks:
            t = np.round(t * ticks) / ticks
        if values == "counts":
            v = rng.integers(0, 60, k).astype(float)
        elif values == "signed counts":
            v = rng.integers(-60, 60, k) * 0.25
        elif values == "wide counts":
            v = rng.integers(0, 1 << 20, k).astype(float)
        elif values == "steps":  # long runs of equal values
            v = np.repeat(rng.integers(0, 5, k), 7)[:k].astype(float)
        elif values == "positive":
            v = rng.random(k)
        else:
            v = rng.standard_normal(k) * (1e-30 if values == "tiny" else 1.0)
        v[-1] = 0.0
        out.append(np.stack([t, v], 1))
    return _pack(out)


def _check(pts, off, got_l1, got_l2, got_k):
    from oracle import oracle as orc
    ap = pts.copy()
    ap[:, 1] = np.abs(ap[:, 1])
    for got, kw in ((got_l1, dict(op=orc.OP_L1, mode=orc.MODE_PDIST)),
                    (got_l2, dict(op=orc.OP_LP, mode=orc.MODE_PDIST, p=2.0))):
        want = orc.evaluate(pts, off, truth=True, **kw)
        assert np.all(np.abs(got - want) <= TOL * np.abs(want)), kw
    want = orc.evaluate(pts, off, op=orc.OP_L2, mode=orc.MODE_KERNEL, truth=True)
    scale = orc.evaluate(ap, off, op=orc.OP_L2, mode=orc.MODE_KERNEL, truth=True)
    assert np.all(np.abs(got_k - want) <= TOL * scale)


VALUES = ["counts", "signed counts", "wide counts", "steps", "normal", "positive", "tiny"]


@pytest.mark.parametrize("values", VALUES)
@pytest.mark.parametrize("lens", [(1, 2, 3), (31, 32, 33), (2, 280, 300), (5, 390, 400, 1300), (3000, 7)])
def test_against_the_oracle(values, lens):
    """Both forms, signs, one and several windows and row pieces."""
    import stablebear_gb300 as sb
    n = 9 if max(lens) > 2000 else 77
    pts, off = _random(n, lens, values, seed=max(lens) + len(values), ticks=4 if max(lens) == 300 else 0)
    X = sb.PcfArray.from_csr(pts, off)
    _check(pts, off, sb.pdist(X).data, sb.pdist(X, p=2).data, sb.l2_kernel(X).data)


def _all(sb, X, Y):
    return [sb.pdist(X).data.copy(), sb.pdist(X, p=2).data.copy(), sb.l2_kernel(X).data.copy(),
            sb.cdist(X, Y).copy(), sb.cdist(X, Y, p=2).copy()]


@pytest.mark.parametrize("values", ["counts", "signed counts", "normal"])
def test_exact_sums_do_not_depend_on_order_bands_or_sides(values):
    """Integer sums: processing order, bands, which PCF of a pair is the row
    and how the call is cut change no bit."""
    import stablebear_gb300 as sb
    pts, off = _random(1100, (1, 3, 40, 90), values, seed=3, ticks=8)
    X = sb.PcfArray.from_csr(pts, off)
    Y = X[:333]
    try:
        base = _all(sb, X, Y)
        sb.set_tuning(order=1)
        for a, b in zip(_all(sb, X, Y), base):
            np.testing.assert_array_equal(a, b)
        sb.set_tuning(order=1, band_bytes=200 << 10)
        for a, b in zip(_all(sb, X, Y), base):
            np.testing.assert_array_equal(a, b)
        sb.set_tuning(band_bytes=200 << 10)
        for a, b in zip(_all(sb, X, Y), base):
            np.testing.assert_array_equal(a, b)
    finally:
        sb.set_tuning()
    C, D = sb.cdist(X, X), sb.pdist(X).to_dense()
    np.testing.assert_array_equal(C, C.T)
    np.testing.assert_array_equal(C, D)


@pytest.mark.parametrize("scale", [1e-6, 1e-10, 1e-16])
@pytest.mark.parametrize("values", ["counts", "positive", "normal"])
def test_products_that_end_early(values, scale):
    """PCFs of 1 to 400 elements that end, or change last, at a very early
    time (walked in double precision up to there) and some whose last value
    is not 0, among long ones."""
    import stablebear_gb300 as sb
    pts, off = _random(90, (1, 2, 33, 64, 400), values, seed=11)
    for i in range(0, 90, 4):
        a, b = int(off[i]), int(off[i + 1])
        if i % 8 == 0:
            pts[a:b, 0] *= scale
        elif b - a > 2:
            pts[a:a + 3, 0] *= scale
            pts[a + 2:b, 1] = 0.0
    X = sb.PcfArray.from_csr(pts, off)
    _check(pts, off, sb.pdist(X).data, sb.pdist(X, p=2).data, sb.l2_kernel(X).data)
    tails = pts.copy()
    tails[np.asarray(off[1::9], dtype=np.int64) - 1, 1] = 2.0
    X = sb.PcfArray.from_csr(tails, off)
    from oracle import oracle as orc
    want = orc.evaluate(tails, off, op=orc.OP_L2, mode=orc.MODE_KERNEL, truth=True)
    ap = np.abs(tails)
    bound = orc.evaluate(ap, off, op=orc.OP_L2, mode=orc.MODE_KERNEL, truth=True)
    fine = np.isfinite(bound) & (bound < 1e300)
    got = sb.l2_kernel(X).data
    assert np.all(np.abs(got - want)[fine] <= TOL * bound[fine])


def test_pairs_the_bound_refuses():
    """Near-identical PCFs, duplicates and functions that end at once: walked
    in double precision, or exactly 0."""
    import stablebear_gb300 as sb
    rng = np.random.default_rng(5)
    k = 500
    t = np.concatenate([[0.0], np.cumsum(rng.exponential(1.0, k - 1))])
    v = rng.standard_normal(k)
    v[-1] = 0
    lists = [np.stack([t, v], 1), np.stack([t, v], 1)]
    for eps in (1e-3, 1e-9, 1e-14):
        lists.append(np.stack([t, v + eps * np.r_[rng.standard_normal(k - 1), 0]], 1))
        lists.append(np.stack([t * (1 + eps), v], 1))
    lists += [[[0, 3], [1e-9, 0]], [[0, 2], [1e-13, 0]], [[0, 0]], [[0, 0], [5, 0]]]
    pts, off = _pack(lists)
    X = sb.PcfArray.from_csr(pts, off)
    _check(pts, off, sb.pdist(X).data, sb.pdist(X, p=2).data, sb.l2_kernel(X).data)
    assert sb.pdist(X).data[0] == 0 and sb.pdist(X, p=2).data[0] == 0
    cv = np.round(np.abs(v) * 9)
    lists = [np.stack([t, cv], 1), np.stack([t, cv], 1), np.stack([t, cv + (np.arange(k) == 7)], 1),
             [[0, 3], [1e-9, 0]], [[0, 2], [1e-13, 0]], [[0, 0]]]
    pts, off = _pack(lists)
    X = sb.PcfArray.from_csr(pts, off)
    _check(pts, off, sb.pdist(X).data, sb.pdist(X, p=2).data, sb.l2_kernel(X).data)
    assert sb.pdist(X).data[0] == 0


@pytest.mark.parametrize("what", ["outlier", "huge", "inf", "nan", "tails", "late", "subnormal", "tail"])
def test_data_without_a_form_takes_the_direct_kernels(what):
    """The default equals the forced direct kernel bit for bit where the
    record refuses the data; a non-zero last value gives what it gives there."""
    import stablebear_gb300 as sb
    pts, off = _random(70, (1, 5, 60, 300), "normal", seed=8)
    k = int(off[3]) + int(off[4] - off[3]) // 2
    if what == "outlier":
        pts[k, 1] = 1e9
    elif what == "huge":
        pts[:, 1] *= 1e200
    elif what == "inf":
        pts[k, 1] = np.inf
    elif what == "nan":
        pts[k, 1] = np.nan
    elif what == "late":
        pts[:, 0] *= 1e150
    elif what == "subnormal":
        pts[k, 1] = 5e-324
    elif what.startswith("tail"):
        pts[off[1:10].astype(int) - 1, 1] = [1.0, 1.0, -2.0, 3.0, 1e-300, 0.5, 1.0, 7.0, 1e-320]
    elif what == "tail":
        pts[off[3:4].astype(int) - 1, 1] = 5.0
    X = sb.PcfArray.from_csr(pts, off)
    Y = X[:40]
    got = _all(sb, X, Y)
    try:
        sb.set_tuning(variant=5)
        want = _all(sb, X, Y)
    finally:
        sb.set_tuning()
    for a, b in zip(got, want):
        if what.startswith("tail"):
            fin = np.isfinite(b)
            np.testing.assert_array_equal(np.isfinite(a), fin)
            np.testing.assert_array_equal(a[~fin], b[~fin])
            big = fin & (np.abs(b) > 1e100)
            np.testing.assert_allclose(a[big], b[big], rtol=TOL)
        else:
            np.testing.assert_array_equal(a, b)


def test_device_entry_bands_misaligned_points_and_capture():
    """The device entry: whole windows as bands give the whole call's bits, a
    points pointer that is only 8-byte aligned, and a call with max_points
    under graph capture."""
    import torch
    import stablebear_gb300 as sb
    from stablebear_gb300 import _native as nat
    pts, off = _random(1300, (2, 20, 50), "normal", seed=21)
    n = len(off) - 1
    want = sb.pdist(sb.PcfArray.from_csr(pts, off)).data
    flat = torch.zeros(pts.size + 1, dtype=torch.float64, device="cuda")
    flat[1:] = torch.from_numpy(pts.reshape(-1)).cuda()
    do = torch.from_numpy(off.astype(np.int64)).cuda()
    lmax = int(np.diff(off.astype(np.int64)).max())

    def call(out, rb, re, base):
        nat.check(nat.lib().sbg_pairwise_device(nat.F64, nat.OP_L1, 1.0, nat.SKIP_LOWER_NODIAG, flat.data_ptr() + 8,
                                                do.data_ptr(), n, None, None, 0, None, None, lmax, out.data_ptr(),
                                                base, rb, re,
                                                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))

    cut = 1024 * 1023 // 2
    lo = torch.empty(cut, dtype=torch.float64, device="cuda")
    hi = torch.empty(n * (n - 1) // 2 - cut, dtype=torch.float64, device="cuda")
    call(lo, 0, 1024, 0)
    call(hi, 1024, n, cut)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(torch.cat([lo, hi]).cpu().numpy(), want)
    out = torch.zeros(n * (n - 1) // 2, dtype=torch.float64, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(out, 0, 0, 0)
    for _ in range(2):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy(), want)


def test_a_low_allocation_limit_leaves_the_direct_path():
    import torch
    import stablebear_gb300 as sb
    from stablebear_gb300 import _native as nat
    pts, off = _random(300, (2, 20, 50), "normal", seed=22)
    X = sb.PcfArray.from_csr(pts, off)
    try:
        sb.set_tuning(variant=5)
        want = sb.pdist(X).data.copy()
    finally:
        sb.set_tuning()
    torch.cuda.synchronize()
    held = nat.lib().sbg_device_bytes_held()
    need = pts.nbytes + off.nbytes + 4 * 300 + want.nbytes
    try:
        assert nat.lib().sbg_set_alloc_limit(held + need + 1024) == 0
        np.testing.assert_array_equal(sb.pdist(X).data, want)
    finally:
        nat.lib().sbg_set_alloc_limit(nat.ALLOC_UNLIMITED)
