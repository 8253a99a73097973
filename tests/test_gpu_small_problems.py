"""Problems of few work items (csrc/engine.cu: launch_problem): halves of the
32-row chunks and items from the last one down give the bits of whole chunks in
order, at item counts around both limits; the length order's permutation at
whole and part windows; the batch's starting shapes (csrc/batch.cu) give the
bits of 8 warps and 32-row items."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 16, 17, 33, 48, 300, 860, 900, 1340, 1380, 2000, 2900])
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
        sb.set_tuning(row_chunk=8)
        want = run()
        sb.set_tuning(order=1)
        caller = run()
    finally:
        sb.set_tuning()
    for a, b, c in zip(got, want, caller):
        np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(a, c)


# Longer PCFs take the windowed kernel, whose windows follow from the column
# group: the same groups, so the same order, on both sides.
@pytest.mark.parametrize("n", [2, 16, 17, 33, 48, 300, 430, 480, 1340, 1380, 2100])
def test_windowed_parts_and_reversed_items_change_no_bit(n):
    import stablebear_gb300 as sb
    from stablebear_gb300 import synthetic
    pts, off = synthetic.gaussian(n, synthetic.uniform_lengths(1, 700), np.float32, seed=n)
    X = sb.PcfArray.from_csr(pts, off)
    Y = X[: max(1, n // 3)]

    def run():
        return [sb.pdist(X).data.copy(), sb.l2_kernel(X).data.copy(), sb.cdist(X, Y).copy(), sb.cdist(Y, X, p=2).copy()]

    got = run()
    try:
        sb.set_tuning(row_chunk=8)
        want = run()
    finally:
        sb.set_tuning()
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)


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


# (PCFs of each problem, longest): 128-row items and 32-row items, on both
# sides of 128 elements
@pytest.mark.parametrize("sizes,hi", [((2600, 700), 150), ((1100,), 128), ((300, 40, 2), 700), ((300, 40, 2), 66), ((90, 1, 33), 60)])
def test_batch_starting_shapes_change_no_bit(sizes, hi):
    import stablebear_gb300 as sb
    from stablebear_gb300 import synthetic
    from stablebear_gb300.batch import PairwiseBatch
    probs = [synthetic.gaussian(n, synthetic.uniform_lengths(1, hi), np.float32, seed=n) for n in sizes]
    outs = []
    try:
        for warps in (0, 8):
            sb.set_tuning(warps=warps)
            b = PairwiseBatch(probs, op="l1", graph=False)
            outs.append([o.cpu().numpy() for o in b.run()])
            b.close()
    finally:
        sb.set_tuning()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("cap,fits", [(440, True), (712, True), (736, False), (800, False), (1 << 20, False)])
def test_window_caps_taken_and_refused(cap, fits):
    import stablebear_gb300 as sb
    from stablebear_gb300 import synthetic
    from stablebear_gb300.batch import PairwiseBatch
    pts, off = synthetic.gaussian(70, synthetic.uniform_lengths(1, 1500), np.float32, seed=3)
    X = sb.PcfArray.from_csr(pts, off)
    want = sb.pdist(X).data.copy()
    sb.set_window_cap(cap)
    try:
        for make in (lambda: sb.pdist(X).data, lambda: PairwiseBatch([(pts, off)], op="l1", graph=False).run()[0].cpu().numpy()):
            if fits:
                # both sums are within 1e-6 of the integral (see test_gpu_window.py)
                np.testing.assert_allclose(make(), want, rtol=2e-6)
            else:
                with pytest.raises(Exception, match="does not fit"):
                    make()
    finally:
        sb.set_window_cap(0)
