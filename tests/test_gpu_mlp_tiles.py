"""The match filter's blocked kernels at the edges of their slices (128 samples), of their cluster sizes
(4 blocks per slice up to 32 slices, 2 up to 70, then 1) and of the inference tiles, against the float64
oracle with the tolerances of the whole-network tests (a slice of 128 samples sums in the same order for
every cluster size, so the bounds do not depend on it), and a training step that mixes both."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(0, 1, (n, 8)) * np.array([0.3, 0.5, 1.0, 0.4, 0.6, 0.02, 0.02, 2.0]) + 0.5
    y = ((x[:, 0] < 0.5) & (x[:, 4] < 0.7)).astype(np.float32)
    return x.astype(np.float32), y


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 32 * 128, 32 * 128 + 1, 70 * 128, 70 * 128 + 3])
def test_gradient_at_slice_edges(n):
    import torch

    from fieldstitch_b200 import match_filter as MF
    from oracle import mlp_ref as M
    x, y = _data(n, n)
    p = M.init_params(np.full(8, 0.5), np.array([0.3, 0.5, 1.0, 0.4, 0.6, 0.02, 0.02, 2.0]), seed=2)
    loss, g = MF.MatchFilter(p).grad(torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda())
    l_ref, g_ref = M.grad(p.astype(np.float64), x.astype(np.float64), y)
    assert abs(loss - l_ref) < 1e-5 * max(1.0, abs(l_ref))
    np.testing.assert_allclose(g.cpu().numpy(), g_ref, rtol=1e-3, atol=1e-5 * np.abs(g_ref).max())


@pytest.mark.parametrize("n", [1, 127, 128, 129, 2 * 148 * 128 + 1])
def test_inference_at_tile_edges(n):
    import torch

    from fieldstitch_b200 import match_filter as MF
    from oracle import mlp_ref as M
    x, _ = _data(n, 3 * n)
    p = M.init_params(np.full(8, 0.5), np.array([0.3, 0.5, 1.0, 0.4, 0.6, 0.02, 0.02, 2.0]), seed=4)
    mf, xt = MF.MatchFilter(p), torch.from_numpy(x).cuda()
    z, _ = M.forward(p.astype(np.float64), x.astype(np.float64))
    np.testing.assert_allclose(mf.predict(xt, bf16=False).cpu().numpy(), M.sigmoid(z), atol=2e-6)
    np.testing.assert_allclose(mf.predict(xt, bf16=True).cpu().numpy(), M.forward_bf16(p, x), atol=5e-3)


@pytest.mark.parametrize("batch", [128, 1024, 4096, 8192, 16384])
def test_steps_do_not_depend_on_earlier_calls(batch):
    """Two epochs of several steps: equal to the same call after unrelated work on the same buffers."""
    import torch

    from fieldstitch_b200 import match_filter as MF
    x, y = _data(40000, 9)
    xt, yt = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    out = []
    for k in range(2):
        mf = MF.MatchFilter()
        mf.init(xt, 1)
        losses = mf.fit(xt, yt, epochs=2, batch=batch, seed=5)
        out.append((losses, mf.params.cpu().numpy()))
        other = MF.MatchFilter()
        other.init(xt, 2)
        other.fit(xt[:777], yt[:777], epochs=3, batch=256, seed=8)
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
