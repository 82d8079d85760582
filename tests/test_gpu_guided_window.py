"""The guided matcher's window where its list can go wrong: windows cut by every side of the frame,
targets outside the frame (kept in the border cells), grids of one row or one column, radii from below
the keypoint spacing to beyond the frame, clusters of more than 32 candidates with the kc nearest taken
among them, repeated positions, query rows that are only 4-byte aligned, more targets than one block
compacts, and the refusal beyond 512 candidates. Distances are exact, so the lists are identical."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(na, nb, w, h, seed, cluster=0):
    from fieldstitch_b200 import synth
    rng = np.random.default_rng(seed)
    a, b, truth = synth.synth_descriptors(na, nb, seed)
    bxy = np.c_[rng.uniform(-20, w + 20, nb), rng.uniform(-20, h + 20, nb)]
    bxy[nb // 2:nb // 2 + 6] = bxy[nb // 2]   # one position, several keypoints
    if cluster:
        bxy[:cluster] = np.array([w / 3, h / 3]) + rng.uniform(-4, 4, (cluster, 2))
    pred = np.c_[rng.uniform(-60, w + 60, na), rng.uniform(-60, h + 60, na)]
    j = np.flatnonzero(truth >= 0)
    pred[truth[j]] = bxy[j] + rng.normal(0, 6, (len(j), 2))
    edge = np.array([[0, 0], [w, 0], [0, h], [w, h], [-1e-9, h / 2], [w / 2, -39.9], [w + 39.9, h / 2]])
    pred[:min(na, 7)] = edge[:min(na, 7)]
    return pred, a, bxy, b


@pytest.mark.parametrize("kc", [1, 16, 40, None])
@pytest.mark.parametrize("w,h,radius,cluster", [(400, 300, 40.0, 0), (400, 300, 3.0, 0), (60, 900, 70.0, 0),
                                                (900, 50, 60.0, 90), (400, 300, 25.0, 300)])
def test_window_matches_oracle(w, h, radius, cluster, kc):
    import fieldstitch_b200 as F
    from oracle import matching_ref
    pred, a, bxy, b = _problem(700, 800, w, h, int(w + radius) + cluster, cluster)
    got = F.matching.guided_from_pred(pred, a, bxy, b, (w, h), radius, kc, 0.85)
    want = matching_ref.guided_from_pred(pred, a, bxy, b, (w, h), radius, kc, 0.85, ties="index")
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])


@pytest.mark.parametrize("shift", [0, 4])
def test_unaligned_queries_and_batch(shift):
    import torch

    from fieldstitch_b200 import _lib
    import fieldstitch_b200 as F
    ctx = _lib.context(0)
    probs = [_problem(na, nb, 500, 400, na + nb, 60) for na, nb in [(1, 900), (17, 300), (500, 33000), (333, 1001)]]
    n = len(probs)
    keep, ptrs = [], [[], [], [], []]
    for p in probs:
        for k, x in enumerate(p):
            raw = np.ascontiguousarray(x).view(np.uint8).reshape(-1)
            off = shift if k == 1 else 0
            t = torch.zeros(raw.size + 16, dtype=torch.uint8, device="cuda")
            t[off:off + raw.size].copy_(torch.from_numpy(raw))
            keep.append(t)
            ptrs[k].append(t.data_ptr() + off)
    out = [[torch.empty(len(p[1]), dtype=torch.int64, device="cuda") for p in probs] for _ in range(2)]
    P, I, D = ctypes.c_void_p * n, ctypes.c_int32 * n, ctypes.c_double * n
    cnt = I()
    torch.cuda.synchronize()
    _lib.check(ctx.lib.fsb_match_guided_batch_d(
        ctx.handle, n, P(*ptrs[0]), P(*ptrs[1]), I(*[len(p[1]) for p in probs]), P(*ptrs[2]), P(*ptrs[3]),
        I(*[len(p[3]) for p in probs]), D(*[500.0] * n), D(*[400.0] * n), 30.0, 16, 0.85,
        P(*[t.data_ptr() for t in out[0]]), P(*[t.data_ptr() for t in out[1]]), cnt))
    for i, (pred, a, bxy, b) in enumerate(probs):
        q, t = F.matching.guided_from_pred(pred, a, bxy, b, (500, 400), 30.0, 16, 0.85)
        np.testing.assert_array_equal(out[0][i][:cnt[i]].cpu().numpy(), q)
        np.testing.assert_array_equal(out[1][i][:cnt[i]].cpu().numpy(), t)


def test_too_many_candidates_are_refused():
    import fieldstitch_b200 as F
    pred, a, bxy, b = _problem(50, 800, 400, 300, 5, 600)
    pred[10] = (400 / 3, 300 / 3)
    with pytest.raises(RuntimeError, match="capacity overflow"):
        F.matching.guided_from_pred(pred, a, bxy, b, (400, 300), 25.0, 16, 0.85)
    F.matching.guided_from_pred(pred, a, bxy, b, (400, 300), 25.0, None, 0.85)
