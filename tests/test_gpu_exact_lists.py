"""Exact mode against the oracle without slack. Positions, responses, octaves and layers are free of
transcendental functions, so the keypoint lists are equal row by row: sizes around the strips of 62 columns, the
blocks of four strips and the chunk heights of the extremum test, plateaus, a repeated tile, and thresholds on
both sides of the 24-bit ranking. A descriptor's entries are within 0.02 for every keypoint: the gradient angles
agree to 1e-3 degrees, which moves 2.2e-5 of a sample between two orientation bins, 0.011 of a descriptor of
length 512, and everything else is float64; a pixel missed or taken twice is far above that."""
import numpy as np
import pytest

from test_gpu_describe_edges import H, W, _keypoints

pytestmark = pytest.mark.gpu


def _image(h, w, kind):
    from fieldstitch_b200 import synth
    if kind == "tile":
        return np.ascontiguousarray(np.tile(synth.synth_image(48, 64, 8), (h // 48 + 1, w // 64 + 1))[:h, :w])
    img = synth.synth_image(h, w, 2 * h + w)
    return np.kron(img[::4, ::4], np.ones((4, 4), np.uint8))[:h, :w] if kind == "plateau" else img


@pytest.mark.parametrize("hw", [(20, 22), (24, 36), (36, 66), (37, 67), (43, 129), (61, 128), (66, 131), (131, 253), (205, 260), (333, 91)])
@pytest.mark.parametrize("kind", ["photo", "plateau", "tile"])
@pytest.mark.parametrize("contrast", [0.0, 1e-6, 0.004, 0.015])
def test_keypoint_lists_are_equal(hw, kind, contrast):
    import fieldstitch_b200 as f
    from oracle import gsift_ref
    img = _image(*hw, kind)
    ref, _ = gsift_ref.detect(img, max_kp=100000, contrast=contrast, edge=12.0)
    got, _ = f.gsift.detect(img, max_kp=100000, contrast=contrast, edge=12.0, exact=True)
    for key in ("x", "y", "response", "octave", "layer"):
        np.testing.assert_array_equal(got[key], ref[key], err_msg=key)


@pytest.mark.parametrize("angle", [0.0, 90.0, 180.0, 270.0, 45.0, 225.0, 89.9999, 180.0001, 26.565, 333.3])
def test_every_descriptor_is_close(angle):
    import fieldstitch_b200 as f
    from fieldstitch_b200 import synth
    from oracle import gsift_ref
    img = synth.synth_image(H, W, 77)
    state = gsift_ref.State(gsift_ref.build_pyramid(img))
    kps = _keypoints(angle)
    sel = np.arange(len(kps["x"]))
    _, st = f.gsift.detect(img, exact=True)
    want = gsift_ref.describe(state, kps, sel)
    err = np.abs(f.gsift.describe(st, kps, sel) - want).max(1)
    assert err.max() <= 0.02, (angle, err.argmax(), err.max())
    st.close()
