"""Where the fixed-point float64 path (csrc/fixed_point.cu) ends: lengths that
a caller states too small, and pairs that the error test has to judge."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pcfs(lens, values, seed):
    rng = np.random.default_rng(seed)
    lens = np.asarray(lens)
    off = np.zeros(len(lens) + 1, np.uint64)
    np.cumsum(lens, out=off[1:])
    t = np.concatenate([np.r_[0.0, np.cumsum(rng.exponential(1.0, k - 1))] for k in lens])
    m = int(off[-1])
    if values == "counts":
        v = rng.integers(0, 60, m).astype(float)
    elif values == "signed counts":
        v = rng.integers(-60, 60, m) * 0.25
    elif values == "positive":
        v = rng.random(m)
    else:
        v = rng.standard_normal(m)
    v[off[1:].astype(np.int64) - 1] = 0.0
    return np.stack([t, v], 1), off


def _device_pdist(pts, off, op, p, skip, max_points, fill):
    import torch
    from stablebear_gb300 import _native as nat
    n = len(off) - 1
    dp = torch.from_numpy(np.ascontiguousarray(pts)).cuda()
    do = torch.from_numpy(off.astype(np.int64)).cuda()
    out = torch.full((int(nat.lib().sbg_output_count(skip, n, n)),), fill, dtype=torch.float64, device="cuda")
    nat.check(nat.lib().sbg_pairwise_device(nat.F64, op, p, skip, dp.data_ptr(), do.data_ptr(), n, None, None, 0, None,
                                            None, max_points, out.data_ptr(), 0, 0, 0,
                                            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("stated,longest", [(100, 1200), (250, 1500)])
@pytest.mark.parametrize("values", ["counts", "normal"])
def test_a_stated_length_below_the_longest(stated, longest, values):
    """max_points sizes the buffers of sums that pass from one time window to
    the next; a longer PCF has to leave the call to the direct kernels (plain,
    then hybrid), which check lengths themselves."""
    import stablebear_gb300 as sb
    from stablebear_gb300 import _native as nat
    lens = np.random.default_rng(stated).integers(2, 60, 64)
    lens[17] = longest
    pts, off = _pcfs(lens, values, seed=stated)
    for op, p, skip in ((nat.OP_L1, 1.0, nat.SKIP_LOWER_NODIAG), (nat.OP_LP, 2.0, nat.SKIP_LOWER_NODIAG),
                        (nat.OP_L2_INNER, 1.0, nat.SKIP_LOWER)):
        got = _device_pdist(pts, off, op, p, skip, stated, -7.0)
        try:
            sb.set_tuning(variant=5 if stated == 100 else 4)
            want = _device_pdist(pts, off, op, p, skip, stated, -7.0)
        finally:
            sb.set_tuning()
        np.testing.assert_array_equal(got, want)


# A pair whose error bound is above 2^-47 of its sum of |terms| is walked in
# double precision (63 naive steps of 2^-53): both stay below 2^-46.
TOL = 2.0 ** -46


def _truth(rows, cols, p):
    from oracle import oracle as orc
    kw = dict(op=orc.OP_L1) if p == 1 else dict(op=orc.OP_LP, p=2.0)
    out = orc.evaluate(rows[0], rows[1], col_points=cols[0], col_offsets=cols[1], mode=orc.MODE_CROSS, truth=True, **kw)
    return out.reshape(len(rows[1]) - 1, len(cols[1]) - 1)


def _join(lists):
    off = np.zeros(len(lists) + 1, np.uint64)
    np.cumsum([len(x) for x in lists], out=off[1:])
    return np.concatenate(lists), off


@pytest.mark.parametrize("values", ["counts", "normal"])
def test_one_breakpoint_apart_by_less_than_a_unit(values):
    """Pairs of steps that end apart by the last bit of a time, far below its
    unit, at each of the 998 breakpoints of a long PCF that shares their
    column group: where a time window ends there, the walk sees no difference."""
    import stablebear_gb300 as sb
    k = 1000
    long, _ = _pcfs([k], values, seed=31)
    long[-1, 0] = 2.0 ** 20 * long[-2, 0]
    height = 3.0 if values == "counts" else float(np.pi)
    rows, cols = [], []
    for j in range(1, k - 1):
        if len(cols) % 32 == 0:
            cols.append(long)
        t = long[j, 0]
        rows.append(np.array([[0.0, height], [np.nextafter(t, np.inf), 0.0]]))
        cols.append(np.array([[0.0, height], [t, 0.0]]))
    steps = [i for i, c in enumerate(cols) if len(c) == 2]
    rows, cols = _join(rows), _join(cols)
    X, Y = sb.PcfArray.from_csr(*rows), sb.PcfArray.from_csr(*cols)
    try:
        sb.set_tuning(order=1)  # the groups as they are
        got = [sb.cdist(X, Y, p=p) for p in (1, 2)]
    finally:
        sb.set_tuning()
    for p in (1, 2):
        want = _truth(rows, cols, p)[np.arange(k - 2), steps]
        assert np.all(want > 0)
        assert np.all(np.abs(got[p - 1][np.arange(k - 2), steps] - want) <= TOL * want), p


def test_times_that_round_the_same_way():
    """A falling staircase whose times all lie 0.4375 units behind a whole
    one: their errors add up instead of evening out."""
    import stablebear_gb300 as sb
    steps = 4000
    t = np.r_[0.0, np.arange(1, steps + 1) * 2.0 ** 33 + 0.4375]
    stairs = np.stack([t, np.arange(steps, -1, -1.0)], 1)
    rows = _join([stairs, np.array([[0.0, 1.0], [2.0 ** 61, 0.0]])])
    cols = _join([np.zeros((1, 2)), np.array([[0.0, 1.0], [2.0 ** 43, 0.0]])])
    X, Y = sb.PcfArray.from_csr(*rows), sb.PcfArray.from_csr(*cols)
    for p in (1, 2):
        want = _truth(rows, cols, p)
        assert np.all(np.abs(sb.cdist(X, Y, p=p) - want) <= TOL * want), p


@pytest.mark.parametrize("values", ["counts", "signed counts", "normal"])
def test_long_and_close_pairs_do_not_depend_on_order_bands_or_sides(values):
    """Which pairs are walked again is a matter of the pair alone: several
    windows and row pieces, PCFs close together, early times below the unit."""
    import stablebear_gb300 as sb
    pts, off = _pcfs(np.random.default_rng(6).integers(400, 1500, 60), values, seed=6)
    rng = np.random.default_rng(7)
    lists = []
    for i in range(60):
        x = pts[int(off[i]):int(off[i + 1])].copy()
        if i % 10 == 3:
            x[:, 0] *= 0.01
        lists.append(x)
        for eps in (1e-3, 1e-7):
            y = x.copy()
            at = rng.integers(1, len(y) - 1, 5)
            y[at, 0] = np.nextafter(y[at, 0], np.inf)
            if values == "normal":
                y[:-1, 1] += eps * rng.standard_normal(len(y) - 1)
            lists.append(y)
    lists[-1][-1, 0] *= 40.0  # the others' times below 2^56 units
    lists += [np.array([[0.0, 1.0], [3.0, 0.0]])] * 900  # two processing-order windows
    X = sb.PcfArray.from_csr(*_join(lists))
    Y = X[:180]

    def every():
        return [sb.pdist(X).data.copy(), sb.pdist(X, p=2).data.copy(), sb.l2_kernel(X).data.copy(),
                sb.cdist(Y, X).copy(), sb.cdist(Y, X, p=2).copy()]

    try:
        base = every()
        for kw in (dict(order=1), dict(order=1, band_bytes=400 << 10), dict(band_bytes=400 << 10)):
            sb.set_tuning(**kw)
            for a, b in zip(every(), base):
                np.testing.assert_array_equal(a, b)
    finally:
        sb.set_tuning()
    for p, C in ((1, base[3]), (2, base[4])):
        np.testing.assert_array_equal(sb.cdist(X, Y, p=p), C.T)
        np.testing.assert_array_equal(sb.pdist(Y, p=p).to_dense(), sb.cdist(Y, Y, p=p))


@pytest.mark.parametrize("values", ["counts", "normal"])
@pytest.mark.parametrize("k", [2, 3, 31, 33, 64, 65, 1000])
def test_refused_pairs_alone_and_together(values, k):
    """Pairs too close together, or ending too early, for the error bound: few
    of a row are walked one after the other, a part to a lane, many at once, a
    pair to a lane; with the same bits and within the tolerance."""
    import stablebear_gb300 as sb
    from oracle import oracle as orc
    base, _ = _pcfs([k], values, seed=k)
    rng = np.random.default_rng(k)
    lists = []
    for i in range(40):
        x = base.copy()
        x[:, 0] *= 2.0 ** -40  # all of it far below the unit of the last PCF's time
        if i % 2 and k > 2:
            x = np.delete(x, rng.integers(1, k - 1), axis=0)
        x[1:, 0] *= 1 + 1e-9 * rng.random()
        lists.append(x)
    lists.append(np.array([[0.0, 1.0], [1e6, 0.0]]))
    pts, off = _join(lists)
    ap = np.abs(pts)
    X = sb.PcfArray.from_csr(pts, off)
    for name, got, kw in (("l1", sb.pdist(X).to_dense(), dict(op=orc.OP_L1, mode=orc.MODE_PDIST)),
                          ("l2", sb.pdist(X, p=2).to_dense(), dict(op=orc.OP_LP, p=2.0, mode=orc.MODE_PDIST)),
                          ("kernel", sb.l2_kernel(X).to_dense(), dict(op=orc.OP_L2, mode=orc.MODE_KERNEL))):
        want = orc.evaluate(pts, off, truth=True, **kw)
        scale = orc.evaluate(ap, off, truth=True, **kw) if name == "kernel" else want
        i, j = np.tril_indices(41, 0 if name == "kernel" else -1)
        assert np.all(np.abs(got[i, j] - want) <= TOL * scale), name
        if name == "kernel":
            continue
        # the last PCF keeps the unit of time; a column group of three
        for a in range(0, 40, 7):
            few = sb.PcfArray.from_csr(*_join([lists[a], lists[(a + 11) % 40], lists[40]]))
            C = sb.cdist(X, few, p=1 if name == "l1" else 2)
            np.testing.assert_array_equal(C[:40, 0], got[:40, a])
            np.testing.assert_array_equal(C[:40, 1], got[:40, (a + 11) % 40])


@pytest.mark.parametrize("values", ["counts", "signed counts", "normal"])
@pytest.mark.parametrize("longest", [60, 300])
def test_calls_whose_pairs_would_be_refused_take_the_direct_kernels(values, longest):
    """One PCF that ends far behind the others takes the unit of time with it:
    the direct kernels' bits (plain, then hybrid), also for two sets."""
    import stablebear_gb300 as sb
    lens = np.random.default_rng(longest).integers(20, longest, 70)
    lens[0] = longest
    pts, off = _pcfs(lens, values, seed=longest)
    pts[int(off[6]) - 1, 0] *= 1e6
    X = sb.PcfArray.from_csr(pts, off)
    Y = X[:30]

    def every():
        return [sb.pdist(X).data.copy(), sb.pdist(X, p=2).data.copy(), sb.l2_kernel(X).data.copy(),
                sb.cdist(X, Y).copy(), sb.cdist(Y, X, p=2).copy()]

    got = every()
    try:
        sb.set_tuning(variant=5 if longest == 60 else 4)
        want = every()
    finally:
        sb.set_tuning()
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)


def _pairs(X, which):
    """The distances, or products, of chosen pairs (i, j), i > j."""
    import stablebear_gb300 as sb
    D = {"l1": lambda: sb.pdist(X), "l2": lambda: sb.pdist(X, p=2), "kernel": lambda: sb.l2_kernel(X)}[which]().to_dense()
    return lambda i, j: D[i, j]


def test_early_times_are_as_exact_as_in_double_precision():
    """Steps that end 0.4375 units behind a whole one, against zero: exact in
    double precision.  A pair is taken with a usual error, 0.289 units here, of
    2^-51 of the integral: 0.5 / 0.289 of that at most."""
    import stablebear_gb300 as sb
    ends = [2.0 ** m + 0.4375 for m in range(30, 51)]
    lists = [np.zeros((1, 2)), np.array([[0.0, 1.0], [2.0 ** 61, 0.0]])] + [np.array([[0.0, 1.0], [t, 0.0]]) for t in ends]
    at = _pairs(sb.PcfArray.from_csr(*_join(lists)), "l1")
    for k, t in enumerate(ends):
        assert abs(at(2 + k, 0) - t) <= 1.74 * 2.0 ** -51 * t, k


def test_small_values_are_as_exact_as_in_double_precision():
    """A value near 2^-14 of the largest, a quarter of a unit off: one
    rectangle, exact in double precision, 2^-50.3 off where the value rounds."""
    import stablebear_gb300 as sb
    v = (337769972052787.0 + 0.25) * 2.0 ** -62  # 1.2 2^48 units
    pts, off = _pcfs([50] * 40, "positive", seed=41)
    lists = [pts[int(off[i]):int(off[i + 1])] for i in range(40)]
    lists += [np.zeros((1, 2)), np.array([[0.0, 0.75], [32.0, 0.0]]), np.array([[0.0, v], [32.0, 0.0]])]
    X = sb.PcfArray.from_csr(*_join(lists))
    for which, j, want in (("l1", 40, 32 * v), ("l2", 40, np.sqrt(32.0) * v), ("kernel", 41, 24 * v)):
        assert abs(_pairs(X, which)(42, j) - want) <= 2.0 ** -51 * want, which


def test_launch_shapes_are_the_callers():
    """Warps and rows per item, set or cached, reach the float64 kernel: one
    warp a CTA is far slower, and no shape changes a bit."""
    import torch
    import stablebear_gb300 as sb
    from stablebear_gb300 import _native as nat
    pts, off = _pcfs(np.random.default_rng(5).integers(20, 600, 900), "normal", seed=5)
    n, longest = len(off) - 1, int(np.diff(off.astype(np.int64)).max())
    dp, do = torch.from_numpy(pts).cuda(), torch.from_numpy(off.astype(np.int64)).cuda()
    out = torch.empty(n * (n - 1) // 2, dtype=torch.float64, device="cuda")

    def run():
        best = float("inf")
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            nat.check(nat.lib().sbg_pairwise_device(nat.F64, nat.OP_L1, 1.0, nat.SKIP_LOWER_NODIAG, dp.data_ptr(),
                                                    do.data_ptr(), n, None, None, 0, None, None, longest,
                                                    out.data_ptr(), 0, 0, 0,
                                                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best, out.cpu().numpy().copy()

    default, want = run()
    try:
        for warps, chunk in ((1, 0), (5, 1), (16, 8), (32, 32), (0, 3), (0, 1024)):
            sb.set_tuning(warps=warps, row_chunk=chunk)
            ms, got = run()
            np.testing.assert_array_equal(got, want)
            if warps == 1:
                assert ms > 3 * default
        sb.set_tuning()
        nat.check(nat.lib().sbg_tuning_cache_store(nat.F64, nat.OP_L1, 1.0, nat.SKIP_LOWER_NODIAG, n, longest, 1, 64))
        ms, got = run()
        np.testing.assert_array_equal(got, want)
        assert ms > 3 * default
    finally:
        sb.set_tuning()
        nat.check(nat.lib().sbg_tuning_cache_clear())


@pytest.mark.parametrize("values", ["counts", "normal"])
def test_one_last_value_that_is_not_zero(values):
    """A single PCF that never returns to zero: its last rectangle reaches to
    the largest double, as in the direct kernels."""
    import stablebear_gb300 as sb
    pts, off = _pcfs(np.random.default_rng(3).integers(1, 300, 70), values, seed=3)
    pts[int(off[4]) - 1, 1] = 5.0
    X = sb.PcfArray.from_csr(pts, off)

    def every():
        return [sb.pdist(X).data.copy(), sb.pdist(X, p=2).data.copy(), sb.l2_kernel(X).data.copy()]

    got = every()
    try:
        sb.set_tuning(variant=5)
        want = every()
    finally:
        sb.set_tuning()
    for a, b in zip(got, want):
        finite = np.isfinite(b)
        np.testing.assert_array_equal(np.isfinite(a), finite)
        np.testing.assert_array_equal(a[~finite], b[~finite])
        big = finite & (np.abs(b) > 1e100)
        np.testing.assert_allclose(a[big], b[big], rtol=TOL)


@pytest.mark.parametrize("values", ["counts", "normal"])
def test_equal_last_values_that_are_not_zero(values):
    """Distances of PCFs that end on one value other than 0 end where the later
    one does, also for pairs that are walked again."""
    import stablebear_gb300 as sb
    from oracle import oracle as orc
    pts, off = _pcfs(np.random.default_rng(4).integers(1, 200, 60), values, seed=4)
    pts[off[1:].astype(np.int64) - 1, 1] = 7.0
    for i in range(0, 60, 3):  # early ones, with points behind their last change
        a, b = int(off[i]), int(off[i + 1])
        pts[a:b, 0] *= 1e-9
        pts[a + (b - a) // 2:b, 1] = 7.0
    X = sb.PcfArray.from_csr(pts, off)
    for got, kw in ((sb.pdist(X).data, dict(op=orc.OP_L1)), (sb.pdist(X, p=2).data, dict(op=orc.OP_LP, p=2.0))):
        want = orc.evaluate(pts, off, mode=orc.MODE_PDIST, truth=True, **kw)
        assert np.all(np.abs(got - want) <= TOL * want)
