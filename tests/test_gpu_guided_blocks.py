"""The guided matcher's blocks hold one query per warp up to 64 000 queries of a call and four beyond: both
give the per-pair results (whose calls hold one) across that line, with ragged last blocks, and a call of
few queries spreads them over the GPU instead of queueing them behind one another."""
import time

import pytest

pytestmark = pytest.mark.gpu

W, H = 2640.0, 1978.0


def _problem(na, nb, seed):
    import torch
    from fieldstitch_b200 import synth
    a, b, _ = synth.synth_descriptors_device(na, nb, seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    wh = torch.tensor([W, H], dtype=torch.float64, device="cuda")
    bxy = torch.rand((nb, 2), generator=g, dtype=torch.float64, device="cuda") * wh
    pred = torch.rand((na, 2), generator=g, dtype=torch.float64, device="cuda") * wh
    return pred, a, bxy, b, (W, H)


@pytest.mark.parametrize("nas", [(30000, 30000, 3999, 1), (30000, 30000, 3999, 2), (64001, 3, 10003)])
@pytest.mark.parametrize("kc", [0, 16])
def test_batches_across_the_line_equal_single_pairs(nas, kc):
    import torch
    import fieldstitch_b200 as F
    probs = [_problem(na, 3001 + 7 * i, 900 + i) for i, na in enumerate(nas)]
    batch = F.matching.guided_from_pred_batch_d(probs, 60.0, kc, 0.9)
    found = 0
    for p, (q, t) in zip(probs, batch):
        (sq, st), = F.matching.guided_from_pred_batch_d([p], 60.0, kc, 0.9)
        assert torch.equal(q, sq) and torch.equal(t, st)
        found += len(q)
    assert found > 100


def test_few_queries_run_side_by_side():
    """2000 queries with a window of 8000 targets each, against four of them: within the GPU's warps, so about one
    query's time (four queries a warp took four times that)."""
    import torch
    import fieldstitch_b200 as F
    pred, a, bxy, b, wh = _problem(2000, 8000, 5)

    def best(n):
        prob = [(pred[:n].contiguous(), a[:n].contiguous(), bxy, b, wh)]
        times = []
        for _ in range(12):
            torch.cuda.synchronize()
            t = time.perf_counter()
            F.matching.guided_from_pred_batch_d(prob, 4000.0, 0, 0.9)
            torch.cuda.synchronize()
            times.append(time.perf_counter() - t)
        return min(times)

    few, many = best(4), best(2000)
    assert many < 2.2 * few, (few, many)
