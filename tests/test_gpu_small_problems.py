"""Problems of few work items (csrc/engine.cu: launch_problem): halves of the
32-row chunks and items from the last one down give the bits of whole chunks in
order, at item counts around both limits; and the length order's permutation
at whole and part windows."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 16, 17, 33, 48, 300, 860, 900, 1340, 1380])
def test_parts_and_reversed_items_change_no_bit(n):
    import stablebear_gb300 as sb
    from stablebear_gb300 import synthetic
    pts, off = synthetic.gaussian(n, synthetic.uniform_lengths(1, 40), np.float32, seed=n)
    X = sb.PcfArray.from_csr(pts, off)
    Y = X[: max(1, n // 3)]

    def run():
        return [sb.pdist(X).data.copy(), sb.l2_kernel(X).data.copy(), sb.cdist(X, Y).copy(), sb.cdist(Y, X, p=2).copy()]

    got = run()
    try:
        sb.set_tuning(row_chunk=2)
        want = run()
        sb.set_tuning(order=1)
        caller = run()
    finally:
        sb.set_tuning()
    for a, b, c in zip(got, want, caller):
        np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(a, c)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 1023, 1024, 1025, 1057, 3000])
def test_length_order(n):
    import torch
    from stablebear_gb300 import _native as nat
    rng = np.random.default_rng(n)
    lens = rng.integers(1, 9, n)
    off = torch.from_numpy(np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)).cuda()
    perm = torch.full((n + 1,), -1, dtype=torch.int32, device="cuda")
    nat.check(nat.lib().sbg_length_order_device(off.data_ptr(), n, perm.data_ptr(),
                                                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    want = np.concatenate([w + np.argsort(lens[w:w + 1024], kind="stable") for w in range(0, n, 1024)])
    np.testing.assert_array_equal(perm.cpu().numpy(), np.append(want, -1))
