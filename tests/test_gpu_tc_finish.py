"""The finishing pass of the tensor-core matcher where its forms change: 4 and 16 rows per warp (the number
of query rows), chunks cut by the last target, fewer targets than two chunks, several column splits, equal
distances in one chunk and across chunks, rows of zeros and of 255. Every engine returns the pairs of the
plain-distance engine, which is compared with the reference elsewhere."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# query rows of 75 776 and more in all take 16 rows per warp
SIZES = {
    "few targets": [(37, 2), (64, 15), (5, 16), (130, 17), (33, 31), (700, 33)],
    "splits": [(300, 5003), (17, 9001)],
    "rows below the line": [(75775, 257)],
    "rows at the line": [(75000, 300), (771, 16), (5, 2)],
    "long, ragged": [(50001, 777), (31234, 1025), (1, 50), (2, 19)],
}


def _pair(rng, na, nb):
    b = rng.integers(0, 256, (nb, 128), dtype=np.uint8)
    b[rng.integers(0, nb, max(1, nb // 8))] = b[rng.integers(0, nb)]           # equal targets
    if nb > 4:
        b[nb // 2] = 0
        b[nb - 1] = 255
    a = rng.integers(0, 256, (na, 128), dtype=np.uint8)
    hit = rng.random(na) < 0.6
    src = b[rng.integers(0, nb, na)]
    noisy = np.clip(src.astype(np.int16) + rng.integers(-9, 10, src.shape), 0, 255).astype(np.uint8)
    a[hit] = noisy[hit]
    a[rng.random(na) < 0.05] = 0
    same = rng.random(na) < 0.05
    a[same] = src[same]
    return a, b


@pytest.mark.parametrize("prec", ["bf16", "fp8"])
@pytest.mark.parametrize("name", list(SIZES))
def test_finish_equals_plain_distances(name, prec):
    import torch

    import fieldstitch_b200 as F
    rng = np.random.default_rng(len(name))
    pairs = [_pair(rng, na, nb) for na, nb in SIZES[name]]
    da = [torch.from_numpy(a).cuda() for a, _ in pairs]
    db = [torch.from_numpy(b).cuda() for _, b in pairs]
    for ratio in (0.8, 1.0):
        want = F.matching.ratio_match_bf_batch_d(da, db, ratio, precision="fp32")
        got = F.matching.ratio_match_bf_batch_d(da, db, ratio, precision=prec)
        for (gq, gt), (wq, wt) in zip(got, want):
            np.testing.assert_array_equal(gq.cpu().numpy(), wq.cpu().numpy())
            np.testing.assert_array_equal(gt.cpu().numpy(), wt.cpu().numpy())
        assert sum(len(q) for q, _ in want) > 0
