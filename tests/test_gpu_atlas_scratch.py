"""Reading a state's atlases back takes a bounded amount of device memory beside the state's own, whatever the
image's size, and gives every row of every layer across the pieces that it is copied in."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hw", [(61, 90), (700, 1301), (1300, 2001)])
def test_scratch_is_bounded(hw):
    import fieldstitch_b200 as f
    from fieldstitch_b200 import _lib, synth
    from oracle import gsift_ref
    img = synth.synth_image(hw[0], hw[1], 4)

    def read():   # on a thread, and so a context, of its own
        _, st = f.gsift.detect(img, exact=True)
        before = _lib.context(0).device_bytes()
        atlas = st.atlas()
        more = _lib.context(0).device_bytes() - before
        st.close()
        return atlas, more

    with ThreadPoolExecutor(1) as ex:
        (shapes, dog, mag, ang), more = ex.submit(read).result()
    assert more <= 16 << 20, more
    for o in range(len(shapes)):
        assert np.isfinite(dog[o]).all() and (mag[o] >= 0).all() and (ang[o] >= 0).all() and (ang[o] <= 360).all()
    if hw[0] < 1000:
        for o, oc in enumerate(gsift_ref.build_pyramid(img)):
            np.testing.assert_array_equal(dog[o], oc["dog"], err_msg="octave %d" % o)
            np.testing.assert_array_equal(mag[o], gsift_ref.gradients(oc)[0], err_msg="octave %d" % o)
