"""Staged host copies and the launch form of the batched extraction: image, descriptor and match copies
around the staging piece (512 KB) and the ring of four pieces, and batches that are launched directly,
captured and replayed in every order, against the per-image and device-resident results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pinned(a):
    import torch
    t = torch.empty(a.shape, dtype=torch.uint8, pin_memory=True)
    t.numpy()[:] = a
    return t


def test_batch_direct_capture_replay_in_any_order():
    import torch

    import fieldstitch_b200 as F
    from fieldstitch_b200 import synth
    dev = torch.device("cuda", 0)
    h, w, nf = 400, 501, 900
    imgs = [synth.synth_image(h, w, 70 + k) for k in range(5)]
    want = [F.features.sift_gpu_u8(im, nf) for im in imgs]

    class Set:
        def __init__(self, idx):
            self.idx = idx
            self.d = [torch.from_numpy(imgs[i]).to(dev) for i in idx]
            self.xy = [torch.zeros((nf, 2), dtype=torch.float32, device=dev) for _ in idx]
            self.u8 = [torch.zeros((nf, 128), dtype=torch.uint8, device=dev) for _ in idx]
            self.rs = [torch.zeros(nf, dtype=torch.float32, device=dev) for _ in idx]

    sets = {"a": Set([0, 1, 2]), "b": Set([3, 4]), "c": Set([2, 0, 4, 1, 3])}
    # new arguments (direct), the same again (capture), again (replay), others between, back to the
    # captured ones (replay) after direct calls of smaller and larger batches
    for step, name in enumerate("aaabaccabbac"):
        s = sets[name]
        for t in s.xy + s.u8 + s.rs:
            t.zero_()
        counts = F.features.sift_gpu_batch_d(s.d, [nf] * len(s.idx), s.xy, s.u8, s.rs, chains=2)
        for k, i in enumerate(s.idx):
            wxy, wu8, wrs = want[i]
            assert counts[k] == len(wxy) > 0, (step, name, k)
            np.testing.assert_array_equal(s.xy[k][:counts[k]].cpu().numpy(), wxy)
            np.testing.assert_array_equal(s.u8[k][:counts[k]].cpu().numpy(), wu8)
            np.testing.assert_array_equal(s.rs[k][:counts[k]].cpu().numpy(), wrs)


def test_batch_uploads_direct_between_replays():
    """Page-locked uploads: the nodes of the captured graph survive a direct call of another batch."""
    import fieldstitch_b200 as F
    from fieldstitch_b200 import synth
    h, w, nf = 300, 420, 600
    imgs = [synth.synth_image(h, w, 170 + k) for k in range(6)]
    want = [F.features.sift_gpu_u8(im, nf) for im in imgs]
    for idx in ([0, 1, 2], [0, 1, 2], [3, 4], [1, 2, 5], [5, 4, 3, 2], [2, 1, 0], [3, 3], [0, 5, 4]):
        hold = [_pinned(imgs[i]) for i in idx]
        got = F.features.sift_gpu_u8_batch([t.numpy() for t in hold], [nf] * len(idx), chains=2)
        for i, g in zip(idx, got):
            for x, y in zip(g, want[i]):
                np.testing.assert_array_equal(x, y)


# 1024 columns: a piece is exactly 512 rows
@pytest.mark.parametrize("h,w,pad", [(511, 1024, 0), (513, 1024, 3), (1025, 1023, 0), (2048, 1024, 0), (2051, 1500, 7)])
def test_image_upload_pieces(h, w, pad):
    import torch

    import fieldstitch_b200 as F
    from fieldstitch_b200 import synth
    wide = np.zeros((h, w + pad), np.uint8)
    wide[:, :w] = synth.synth_image(h, w, 9)
    img = wide[:, :w]
    a = F.features.sift_gpu_u8(img, 1500)
    hold = torch.empty((h, w), dtype=torch.uint8, pin_memory=True)   # page-locked: one transfer, no pieces
    hold.numpy()[:] = img
    b = F.features.sift_gpu_u8(hold.numpy(), 1500)
    assert len(a[0]) > 100
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


# 4096 descriptors of 128 bytes are one piece, 16384 the ring
@pytest.mark.parametrize("na,nb", [(2, 2), (4095, 4097), (4096, 8193), (9000, 7384), (9001, 7384), (70000, 500)])
def test_dense_match_from_host_arrays(na, nb):
    import torch

    import fieldstitch_b200 as F
    rng = np.random.default_rng(na + nb)
    b = rng.integers(0, 120, (nb, 128), dtype=np.uint8)
    a = rng.integers(0, 120, (na, 128), dtype=np.uint8)
    m = min(na, nb) // 2
    a[rng.permutation(na)[:m]] = b[rng.permutation(nb)[:m]]
    q, t = F.matching._ratio_match_bf(a, b, 0.8)
    [(dq, dt)] = F.matching.ratio_match_bf_batch_d([torch.from_numpy(a).cuda()], [torch.from_numpy(b).cuda()], 0.8,
                                                   precision="fp32")
    np.testing.assert_array_equal(q, dq.cpu().numpy())
    np.testing.assert_array_equal(t, dt.cpu().numpy())
    assert len(q) >= m
