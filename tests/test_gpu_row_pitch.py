"""Octave widths that are not a multiple of four: planes are stored with a padded row pitch, the atlases
are read out packed. Sizes whose octaves leave 1, 2 and 3 columns past a multiple of four, narrower than
a tile and a tensor-copy box and just past them; DoG and magnitude are the oracle's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hw", [(21, 23), (37, 85), (64, 81), (85, 84), (131, 151), (90, 333)])
def test_packed_atlas_of_pitched_planes(hw):
    import fieldstitch_b200 as f
    from fieldstitch_b200 import synth
    from oracle import gsift_ref
    img = synth.synth_image(hw[0], hw[1], 5 + hw[1])
    octs = gsift_ref.build_pyramid(img)
    _, st = f.gsift.detect(img, exact=True)
    shapes, dog, mag, _ = st.atlas()
    _, fast = f.gsift.detect(img)
    _, fdog, fmag, _ = fast.atlas()
    assert shapes == [o["dog"].shape[1:] for o in octs]
    for o, oc in enumerate(octs):
        np.testing.assert_array_equal(dog[o], oc["dog"])
        np.testing.assert_array_equal(mag[o], gsift_ref.gradients(oc)[0])
        assert np.abs(fdog[o] - oc["dog"]).max() < 2e-6   # the float32 path's bound (test_atlas_fast_within_ulps)
        assert np.abs(fmag[o] - gsift_ref.gradients(oc)[0]).max() < 4e-6
