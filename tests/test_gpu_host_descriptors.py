"""Descriptors in pageable host arrays (matching._ratio_match_bf): the same matches as from device memory on
both sides of the sizes at which copies are cut into pieces, from arrays at odd addresses and from
page-locked ones, and no slower way to the device than the driver's own copy."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("na,nb", [(40, 40), (2000, 2000), (4090, 12290), (20001, 3), (3, 70001)])
def test_matches_equal_device_arrays(na, nb):
    import torch
    import fieldstitch_b200 as F
    rng = np.random.default_rng(na + nb)
    raw_a, raw_b = (np.empty(n * 128 + 1, np.uint8) for n in (na, nb))
    a, b = raw_a[1:].reshape(na, 128), raw_b[1:].reshape(nb, 128)   # one byte past the allocation's alignment
    a[...] = rng.integers(0, 180, a.shape)
    b[...] = rng.integers(0, 180, b.shape)
    k = min(na, nb) // 2
    a[:k] = b[-k:]
    (q, t), = F.matching.ratio_match_bf_batch_d([torch.from_numpy(a.copy()).cuda()], [torch.from_numpy(b.copy()).cuda()],
                                                0.9, precision="fp32")
    pin = [torch.from_numpy(x.copy()).pin_memory().numpy() for x in (a, b)]
    for x, y in ((a, b), pin):
        hq, ht = F.matching._ratio_match_bf(x, y, 0.9)
        np.testing.assert_array_equal(hq, q.cpu().numpy())
        np.testing.assert_array_equal(ht, t.cpu().numpy())
    assert len(hq) >= k


def test_large_arrays_take_the_drivers_copy():
    """Two queries against 200 000 host descriptors against a plain copy of the same array, in turn: 1.10 times
    its time; staged through the context's ring it was 1.3 to 1.4."""
    import torch
    import fieldstitch_b200 as F
    a = np.random.default_rng(1).integers(0, 180, (2, 128)).astype(np.uint8)
    b = np.random.default_rng(2).integers(0, 180, (200000, 128)).astype(np.uint8)
    d, tb = torch.empty(b.shape, dtype=torch.uint8, device="cuda"), torch.from_numpy(b)

    def copy():
        d.copy_(tb)
        torch.cuda.synchronize()

    best = {}
    for _ in range(25):
        for name, fn in (("call", lambda: F.matching._ratio_match_bf(a, b, 0.9)), ("copy", copy)):
            t = time.perf_counter()
            fn()
            best[name] = min(best.get(name, 1.0), time.perf_counter() - t)
    assert best["call"] < 1.2 * best["copy"], best
