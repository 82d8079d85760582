"""A detect state that outlives its context (objects collected in any order at interpreter exit): what it can
still be asked is answered with an error, and freeing it touches nothing of the freed context."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HEAD = """
import ctypes
import numpy as np
import fieldstitch_b200 as F
from fieldstitch_b200 import _lib, synth
img = synth.synth_image(131, 150, 77)
"""

AFTER = HEAD + """
ctx = _lib.context(0)
states = [F.gsift.detect(img)[1] for _ in range(5)]
states[1].close()
n = ctypes.c_int32()
x = np.zeros(100000, np.float32)
ctx.close()
lib = _lib.load()
for st in (states[0], states[2], states[4]):
    assert lib.fsb_state_geometry(st.handle, ctypes.byref(n), None, None) == 5      # FSB_ERR_STATE
    assert lib.fsb_state_keypoints(st.handle, _lib.ptr(x), None, None, None, None, None, None) == 5
    assert lib.fsb_state_atlas(st.handle, 0, _lib.ptr(x), 1) == 5
    assert b"context was destroyed" in lib.fsb_last_error()
for st in states:
    assert st.handle is None or lib.fsb_state_free(st.handle) == 0
    st.handle = None
_lib._tls.ctxs.clear()
kps, st = F.gsift.detect(img)      # a context made afterwards
assert len(kps["x"]) > 50
print("ok")
"""

AT_EXIT = HEAD + """
class Holder:      # a cycle that holds context and states, left to the collector at exit
    pass
a, b = Holder(), Holder()
a.other, b.other = b, a
a.state = F.gsift.detect(img)[1]
b.ctx = _lib.context(0)
more = [F.gsift.detect(synth.synth_image(20 + 3 * k, 21 + 5 * k, k))[1] for k in range(12)]
a.more = more
for k in range(40):
    got, _ = F.gsift.detect(synth.synth_image(20 + k, 30 + k, k), max_kp=100000, contrast=0.002)
print("ok")
"""


@pytest.mark.parametrize("body", [AFTER, AT_EXIT], ids=["after", "at_exit"])
def test_state_outlives_its_context(body):
    env = dict(os.environ, PYTHONPATH=ROOT + os.pathsep + os.environ.get("PYTHONPATH", ""))
    r = subprocess.run([sys.executable, "-c", body], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stdout, r.stderr)
