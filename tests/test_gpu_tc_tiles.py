"""The tensor-core matcher at the edges of its 256-row target tiles, 16-column chunks, splits and its
schedule (uneven pairs in several rounds), with rows that exercise the packing (zeros, saturated rows,
single bytes at every power-of-two scale, bytes half way between two E4M3 values) and pairs with more
targets than one block compacts: the match lists equal the exact integer matcher's in every precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(na, nb, seed):
    from fieldstitch_b200 import synth
    a, b, _ = synth.synth_descriptors(na, nb, seed)
    rng = np.random.default_rng(seed)
    for x in (a, b):
        n = len(x)
        if n < 12:
            continue
        rows = rng.choice(n, 10, replace=False)
        x[rows[0]] = 0
        x[rows[1]] = 255
        for k in range(8):   # one non-zero byte: every scale exponent of the 8-bit operands
            x[rows[2 + k]] = 0
            x[rows[2 + k], 11 * k] = (1 << k) + (k > 3) * ((1 << max(k - 4, 0)) * 3)
        x[rows[0] - 1] = np.arange(128, 256, dtype=np.uint8)   # every rounding of the top binade
    return a, b


@pytest.mark.parametrize("precision", ["bf16", "fp8"])
@pytest.mark.parametrize("na,nb", [(2, 2), (1, 300), (255, 15), (256, 16), (257, 17), (300, 255), (128, 256), (129, 257),
                                   (1000, 511), (40, 513), (2, 4097)])
def test_tile_edges(na, nb, precision):
    import fieldstitch_b200 as F
    a, b = _problem(na, nb, na + 3 * nb)
    want = F.matching._ratio_match_bf(a, b, 0.85)
    got = F.matching._ratio_match_bf(a, b, 0.85, precision=precision)
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])


@pytest.mark.parametrize("precision", ["bf16", "fp8"])
@pytest.mark.parametrize("sizes", [[(300, 2000), (9000, 700), (5, 12000), (12000, 5), (4000, 4100), (7777, 9001)],
                                   [(6000, 500)] * 14, [(600, 33000), (500, 400)]])
def test_uneven_batches(sizes, precision):
    import torch

    import fieldstitch_b200 as F
    probs = [_problem(na, nb, 5 * na + nb + k) for k, (na, nb) in enumerate(sizes)]
    dev = [[torch.from_numpy(x).cuda() for x in p] for p in probs]
    for _ in range(2):
        got = F.matching.ratio_match_bf_batch_d([d[0] for d in dev], [d[1] for d in dev], 0.8, precision=precision)
        for (a, b), (q, t) in zip(probs, got):
            q1, t1 = F.matching._ratio_match_bf(a, b, 0.8)
            np.testing.assert_array_equal(q.cpu().numpy(), q1)
            np.testing.assert_array_equal(t.cpu().numpy(), t1)
