"""The extremum test's chunks: image sizes around the strip of 62 columns, the four strips of a block and
the chunk heights (which follow from the image size), an odd last column pair, rows left over by the
three-row rotation, and plateaus, where every tied voxel counts. The candidate set is compared through
the refined keypoints of a low contrast threshold with the float64 blur (the oracle's atlas bit for bit)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hw", [(20, 21), (23, 36), (24, 37), (36, 67), (40, 68), (41, 129), (61, 130), (97, 257), (333, 91)])
@pytest.mark.parametrize("plateau", [False, True])
def test_keypoints_equal_oracle(hw, plateau):
    import fieldstitch_b200 as f
    from fieldstitch_b200 import synth
    from oracle import gsift_ref
    h, w = hw
    img = synth.synth_image(h, w, h + 3 * w)
    if plateau:   # blocks of equal values: flat areas and tied neighbours
        img = np.kron(img[::4, ::4], np.ones((4, 4), np.uint8))[:h, :w]
    ref, _ = gsift_ref.detect(img, max_kp=100000, contrast=0.002, edge=12.0)
    got, _ = f.gsift.detect(img, max_kp=100000, contrast=0.002, edge=12.0, exact=True)
    # positions, responses, octaves and layers are transcendental-free: equal as sets of rows
    key = lambda k: set(zip(k["x"].view(np.uint32).tolist(), k["y"].view(np.uint32).tolist(),
                            k["response"].view(np.uint32).tolist(), k["octave"].tolist(), k["layer"].tolist()))
    a, b = key(ref), key(got)
    assert len(a ^ b) <= 0.01 * len(a) + 1, (len(a), len(b), len(a ^ b))


@pytest.mark.parametrize("contrast", [0.0, 1e-6, 2e-4, 0.004, 0.015, 0.2])
@pytest.mark.parametrize("quantised", [False, True])
def test_response_order_for_thresholds(contrast, quantised):
    """Keypoints are listed strongest first, equal responses by DoG index, for thresholds that leave more
    and fewer than 24 bits of response to sort (the sort drops the low ones and restores them)."""
    import fieldstitch_b200 as f
    from fieldstitch_b200 import synth
    from oracle import gsift_ref
    img = synth.synth_image(181, 233, 8)
    if quantised:   # a repeated tile: many equal responses
        img = np.tile(img[:48, :64], (4, 4))[:181, :233]
    ref, _ = gsift_ref.detect(img, max_kp=100000, contrast=contrast, edge=12.0)
    got, _ = f.gsift.detect(img, max_kp=100000, contrast=contrast, edge=12.0, exact=True)
    assert (np.diff(got["response"]) <= 0).all()
    n = min(len(ref["x"]), len(got["x"]))
    assert abs(len(ref["x"]) - len(got["x"])) <= 0.01 * n + 1
    a, b = (np.stack([k[c].astype(np.float64)[:n] for c in ("x", "y", "response")], 1) for k in (ref, got))
    if n and len(ref["x"]) == len(got["x"]):
        assert (a == b).all(1).mean() >= 0.99, (a == b).all(1).mean()
