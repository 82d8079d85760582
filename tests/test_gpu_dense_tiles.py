"""The CUDA-core dense matcher's tiles: sizes on both sides of the 32 / 64 / 128-row blocks and of the
switch between the two block heights, splits with a ragged last tile, operands that are only 4-byte
aligned, saturated and zero rows, and batches (one set of launches) against single calls, including a
pair with more targets than one block compacts. Distances are integers, so the lists are identical."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(na, nb, seed):
    from fieldstitch_b200 import synth
    a, b, _ = synth.synth_descriptors(na, nb, seed)
    a[na // 2] = 0
    b[nb // 3] = 255
    if nb > 4:
        b[nb - 1] = b[nb // 2]   # a tie for the best distance fails the ratio test
    return a, b


def _oracle(a, b, ratio):
    from oracle import matching_ref
    return matching_ref.ratio_match_bf(a.astype(np.float32), b.astype(np.float32), ratio)


@pytest.mark.parametrize("na,nb", [(2, 2), (3, 129), (31, 127), (32, 128), (33, 130), (64, 257), (65, 1), (127, 255),
                                   (129, 641), (300, 2), (1501, 1499), (2200, 2177), (4100, 1025)])
@pytest.mark.parametrize("shift", [0, 4])
def test_tiles_match_oracle(na, nb, shift):
    import torch

    from fieldstitch_b200 import _lib
    a, b = _problem(na, nb, na + 7 * nb)
    ctx = _lib.context(0)
    buf = [torch.zeros(len(x) * 128 + 16, dtype=torch.uint8, device="cuda") for x in (a, b)]
    ptr = []
    for t, x in zip(buf, (a, b)):
        t[shift:shift + x.size].copy_(torch.from_numpy(x.reshape(-1)))
        ptr.append(ctypes.c_void_p(t.data_ptr() + shift))
    q = torch.empty(na, dtype=torch.int64, device="cuda")
    t = torch.empty(na, dtype=torch.int64, device="cuda")
    n = ctypes.c_int32()
    torch.cuda.synchronize()
    _lib.check(ctx.lib.fsb_match_bf_d(ctx.handle, ptr[0], na, ptr[1], nb, 0.85, 0, ctypes.c_void_p(q.data_ptr()),
                                      ctypes.c_void_p(t.data_ptr()), ctypes.byref(n)))
    want = _oracle(a, b, 0.85) if min(na, nb) > 1 else (np.zeros(0, np.int64),) * 2
    np.testing.assert_array_equal(q[:n.value].cpu().numpy(), want[0])
    np.testing.assert_array_equal(t[:n.value].cpu().numpy(), want[1])


@pytest.mark.parametrize("sizes", [[(500, 700)], [(130, 2), (2, 4000), (1, 50), (777, 778), (3000, 2900)],
                                   [(40, 33000), (900, 1000)]])
def test_batch_equals_single(sizes):
    import torch

    import fieldstitch_b200 as F
    probs = [_problem(na, nb, 3 * na + nb) for na, nb in sizes]
    dev = [[torch.from_numpy(x).cuda() for x in p] for p in probs]
    for _ in range(2):
        got = F.matching.ratio_match_bf_batch_d([d[0] for d in dev], [d[1] for d in dev], 0.8, precision="fp32")
        for (a, b), (q, t) in zip(probs, got):
            q1, t1 = F.matching._ratio_match_bf(a, b, 0.8)
            np.testing.assert_array_equal(q.cpu().numpy(), q1)
            np.testing.assert_array_equal(t.cpu().numpy(), t1)
