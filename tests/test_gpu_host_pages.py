"""Host results of one band, copied straight into the caller's pages: outputs
that start inside a page, fresh or already written, small and large (pages made
by one and by several threads), with the bytes around them left alone."""
import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 40, 700, 3100])
@pytest.mark.parametrize("lead", [0, 1, 4097])
@pytest.mark.parametrize("fresh", [True, False])
def test_output_inside_a_mapping(n, lead, fresh):
    from stablebear_gb300 import _native as nat, synthetic
    import stablebear_gb300 as sb
    pts, off = synthetic.gaussian(n, synthetic.uniform_lengths(1, 6), np.float32, seed=n)
    count = n * (n - 1) // 2
    tail = 513
    m = mmap.mmap(-1, 4 * (lead + count + tail) + 3 * mmap.PAGESIZE)  # anonymous, no page made yet
    buf = np.frombuffer(m, np.float32)
    if not fresh:
        buf[:] = -7.0
    out = buf[lead:lead + count]
    nat.check(nat.lib().sbg_pairwise_host(nat.F32, nat.OP_L1, 1.0, nat.SKIP_LOWER_NODIAG, nat.ptr(pts), nat.ptr(off), n,
                                          None, None, 0, nat.ptr(out), 1))
    np.testing.assert_array_equal(out, sb.pdist(sb.PcfArray.from_csr(pts, off)).data)
    rest = 0.0 if fresh else -7.0
    assert (buf[:lead] == rest).all() and (buf[lead + count:] == rest).all()


def test_calls_from_several_threads_share_the_pool():
    import threading
    import stablebear_gb300 as sb
    from stablebear_gb300 import _native as nat, synthetic
    sets = [synthetic.gaussian(150 + 40 * k, synthetic.uniform_lengths(1, 90), np.float32 if k % 2 else np.float64, seed=k)
            for k in range(6)]
    want = [sb.pdist(sb.PcfArray.from_csr(*s)).data.copy() for s in sets]
    held = nat.lib().sbg_device_bytes_held()
    bad = []

    def work(k):
        X = sb.PcfArray.from_csr(*sets[k])
        for _ in range(15):
            if not np.array_equal(sb.pdist(X).data, want[k]):
                bad.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sets))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    assert nat.lib().sbg_device_bytes_held() == held
