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
