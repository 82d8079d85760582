"""The fused layer groups on small tiles (32 x 16 for octaves that fit on the GPU at once, 64 x 16 beyond)
give the per-layer kernels' DoG, magnitude and angle atlases bit for bit: octaves smaller than a tile,
ragged last tiles, halos that reflect more than once, widths that are not a multiple of four, and both
tile sizes (an octave of 1990 x 2222 has more than three 32 x 16 tiles per SM)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hw", [(12, 13), (20, 31), (37, 53), (131, 151), (240, 320), (495, 661), (995, 1111)])
def test_small_tiles_bit_identical(monkeypatch, hw):
    import fieldstitch_b200 as f
    from fieldstitch_b200 import synth
    img = synth.synth_image(hw[0], hw[1], 3 + hw[0])
    monkeypatch.setenv("FSB_PYRAMID", "layer")
    k0, st0 = f.gsift.detect(img)
    ref = st0.atlas()
    monkeypatch.setenv("FSB_PYRAMID", "group_small")
    k1, st1 = f.gsift.detect(img)
    got = st1.atlas()
    assert got[0] == ref[0]
    for o in range(len(ref[0])):
        for k, name in ((1, "dog"), (2, "mag"), (3, "ang")):
            np.testing.assert_array_equal(got[k][o], ref[k][o], err_msg="%s octave %d" % (name, o))
    for key in ("x", "y", "size", "angle", "response"):
        np.testing.assert_array_equal(k1[key], k0[key])
