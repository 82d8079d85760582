"""The allocation-free matcher in a second context of a device (after cudaDeviceReset): its scratch and the
kernel's shared memory belong to a context, and the second one has the first one's handle. In a process of
its own, without torch."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

BODY = """
import ctypes
import numpy as np
from fieldstitch_b200 import _lib
from oracle import matching_ref
lib = _lib.load()
rt = ctypes.CDLL("libcudart.so.12")
rng = np.random.default_rng(5)


def ok(status):
    assert status == 0, (status, lib.fsb_last_error())


def device(nbytes, src=None):
    p = ctypes.c_void_p()
    ok(rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(max(nbytes, 256))))
    if src is not None:
        ok(rt.cudaMemcpy(p, ctypes.c_void_p(src.ctypes.data), ctypes.c_size_t(src.nbytes), 1))
    return p


def match(a, b, ratio):
    da, db = device(a.nbytes, a), device(b.nbytes, b)
    dq, dt, dn = device(8 * len(a)), device(8 * len(a)), device(4)
    ok(lib.fsb_match_bf_noalloc(da, len(a), db, len(b), ratio, dq, dt, dn, None))
    ok(rt.cudaDeviceSynchronize())
    n = np.zeros(1, np.int32)
    ok(rt.cudaMemcpy(ctypes.c_void_p(n.ctypes.data), dn, ctypes.c_size_t(4), 2))
    out = [np.zeros(int(n[0]), np.int64) for _ in range(2)]
    for h, d in zip(out, (dq, dt)):
        ok(rt.cudaMemcpy(ctypes.c_void_p(h.ctypes.data), d, ctypes.c_size_t(h.nbytes), 2))
    return out


sets = []
for na, nb in ((300, 200), (3000, 2500)):   # two queries' blocks: 47 and 57 KB of shared memory
    b = rng.integers(0, 180, (nb, 128)).astype(np.uint8)
    a = rng.integers(0, 180, (na, 128)).astype(np.uint8)
    a[:nb // 2] = np.clip(b[:nb // 2].astype(int) + rng.integers(-3, 4, (nb // 2, 128)), 0, 255)
    sets.append((a, b))
first = [match(a, b, 0.8) for a, b in sets]
assert all(len(q) >= len(b) // 2 for (q, t), (a, b) in zip(first, sets))
for _ in range(2):
    ok(rt.cudaDeviceReset())
    for (a, b), (q, t) in reversed(list(zip(sets, first))):
        q2, t2 = match(a, b, 0.8)
        np.testing.assert_array_equal(q2, q)
        np.testing.assert_array_equal(t2, t)
want = matching_ref.ratio_match_bf(sets[0][0], sets[0][1], 0.8) if hasattr(matching_ref, "ratio_match_bf") else None
if want is not None:
    np.testing.assert_array_equal(first[0][0], want[0])
    np.testing.assert_array_equal(first[0][1], want[1])
print("ok")
"""


def test_second_context_of_a_device():
    env = dict(os.environ, PYTHONPATH=ROOT + os.pathsep + os.environ.get("PYTHONPATH", ""))
    r = subprocess.run([sys.executable, "-c", BODY], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.endswith("ok\n"), (r.returncode, r.stdout, r.stderr)
