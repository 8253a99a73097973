"""Lp distances with the exponents that have their own kernels (1.5, 2.5, 3, 4):
against the double-double oracle and against pow() (a forced variant), at
short, long and windowed PCFs, with zero, equal and infinite values.

Tolerance: |d|^p is at most three correctly rounded operations, the root at
most two more and four ulp of pow(); with the compensated sum (eight, in
float64 64, naive steps) a result is within 63 + 9 units in the last place in
float64, 7 + 9 in float32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {np.float32: 16 * 2.0 ** -23, np.float64: 72 * 2.0 ** -52}


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("p", [1.5, 2.5, 3, 4, 3.5])
@pytest.mark.parametrize("hi", [3, 90, 700])
def test_against_the_oracle(dt, p, hi):
    import stablebear_gb300 as sb
    from stablebear_gb300 import synthetic
    from oracle import oracle as orc
    pts, off = synthetic.gaussian(45, synthetic.uniform_lengths(1, hi), dt, seed=hi)
    X = sb.PcfArray.from_csr(pts, off)
    Y = X[:20]
    want = orc.evaluate(pts, off, op=orc.OP_LP, p=p, truth=True)
    assert np.all(np.abs(sb.pdist(X, p=p).data - want) <= TOL[dt] * want)
    yp, yo = Y.csr()
    want = orc.evaluate(pts, off, op=orc.OP_LP, p=p, truth=True, mode=orc.MODE_CROSS, col_points=yp, col_offsets=yo)
    assert np.all(np.abs(sb.cdist(X, Y, p=p).reshape(-1) - want.reshape(-1)) <= TOL[dt] * want.reshape(-1))


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("p", [1.5, 2.5, 3, 4])
def test_special_values_as_pow_gives_them(dt, p):
    import stablebear_gb300 as sb
    big = 1e30 if dt == np.float32 else 1e200
    edge = 1e10 if dt == np.float32 else 1e80  # the fourth power overflows, the square does not
    lists = [[[0, edge], [1, 0]], [[0, 3 * edge], [2, edge], [3, 0]], [[0, 0], [1, np.inf], [2, 0]], [[0, 0], [1, 5], [3, 0]], [[0, -np.inf], [1, 0]], [[0, 0]],
             [[0, 0], [1, 5], [3, 0]], [[0, big], [1, 0]], [[0, np.nan], [2, 0]], [[0, 1], [1, 2]]]
    off = np.zeros(len(lists) + 1, np.uint64)
    np.cumsum([len(x) for x in lists], out=off[1:])
    X = sb.PcfArray.from_csr(np.concatenate([np.array(x, dt) for x in lists]), off)
    got = sb.pdist(X, p=p).data.copy()
    try:
        sb.set_tuning(variant=5)
        want = sb.pdist(X, p=p).data.copy()
    finally:
        sb.set_tuning()
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    np.testing.assert_array_equal(np.isinf(got), np.isinf(want))
    np.testing.assert_array_equal(got == 0, want == 0)
