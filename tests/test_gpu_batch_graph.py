"""The graph of a batched extraction is a cache: a call whose work is done returns its results whether or
not a graph could be made from it. The capture is made to fail on the host: a preloaded
cudaGraphInstantiate that returns an error stands before the CUDA runtime's."""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
static int calls, fail;
int shim_calls(void) { return calls; }
void shim_fail(int on) { fail = on; }
int cudaGraphInstantiate(void** exec, void* graph, unsigned long long flags) {
    int (*real)(void**, void*, unsigned long long) = dlsym(RTLD_NEXT, "cudaGraphInstantiate");
    if (!real) {
        void* rt = dlopen("libcudart.so.12", RTLD_NOW | RTLD_NOLOAD);
        if (rt) real = dlsym(rt, "cudaGraphInstantiate");
    }
    ++calls;
    if (fail || !real) return 2; /* out of memory */
    return real(exec, graph, flags);
}
"""

BODY = """
import ctypes, sys
import numpy as np, torch
import fieldstitch_b200 as F
from fieldstitch_b200 import synth
shim = ctypes.CDLL(sys.argv[1])
dev = torch.device("cuda", 0)


class Batch:
    def __init__(self, imgs, nfeats):
        self.nf = nfeats
        self.want = [F.features.sift_gpu_u8(im, nf) for im, nf in zip(imgs, nfeats)]
        self.img = [torch.from_numpy(im).to(dev) for im in imgs]
        m = max(nfeats)
        self.xy = [torch.zeros((m, 2), device=dev) for _ in imgs]
        self.u8 = [torch.zeros((m, 128), dtype=torch.uint8, device=dev) for _ in imgs]
        self.rs = [torch.zeros(m, device=dev) for _ in imgs]

    def call(self, host=None):
        for t in self.xy + self.u8 + self.rs:
            t.zero_()
        n = F.features.sift_gpu_batch_d(self.img, self.nf, self.xy, self.u8, self.rs, chains=2, host_images=host)
        for k, (wxy, wu8, wrs) in enumerate(self.want):
            assert n[k] == len(wxy) > 0
            np.testing.assert_array_equal(self.xy[k][:n[k]].cpu().numpy(), wxy)
            np.testing.assert_array_equal(self.u8[k][:n[k]].cpu().numpy(), wu8)
            np.testing.assert_array_equal(self.rs[k][:n[k]].cpu().numpy(), wrs)

"""


def _run(tmp_path, body):
    src, so, prog = tmp_path / "shim.c", tmp_path / "shim.so", tmp_path / "prog.py"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(so), str(src), "-ldl"], check=True)
    prog.write_text(BODY + textwrap.dedent(body))
    env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=ROOT + os.pathsep + os.environ.get("PYTHONPATH", ""))
    r = subprocess.run([sys.executable, str(prog), str(so)], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr


def test_failed_capture_is_no_failed_call(tmp_path):
    _run(tmp_path, """
    b = Batch([synth.synth_image(240, 320, 40 + k) for k in range(3)], [600, 200, 900])
    shim.shim_fail(1)
    for _ in range(5):
        b.call()
    tried = shim.shim_calls()
    assert tried > 0           # the preloaded function was reached
    for _ in range(3):
        b.call()
    assert shim.shim_calls() == tried   # what failed is not tried at every call
    shim.shim_fail(0)
    c = Batch([synth.synth_image(200, 300, 50 + k) for k in range(3)], [600, 200, 900])
    for _ in range(4):
        c.call()
    assert shim.shim_calls() > tried    # another size gets its graph
    """)


@pytest.mark.parametrize("hw", [(240, 320), (101, 333)])
def test_graphs_are_made_once_per_size(tmp_path, hw):
    """What a batch keeps for later calls is made by the first call of a size: a second call with the same
    buffers, calls with other buffers, smaller caps, fewer images and page-locked uploads make no more of it,
    and every one of them returns the per-image results. A few thresholds that take turns have a graph each;
    one beyond the number kept takes the place of one that was replayed, else none until it repeats."""
    _run(tmp_path, """
    H, W = %d, %d
    imgs = [synth.synth_image(H, W, 60 + k) for k in range(6)]
    nf = [600, 200, 900, 50, 900, 20]
    a, b = Batch(imgs[:5], nf[:5]), Batch(imgs[1:], nf[1:])
    a.call()
    made = shim.shim_calls()
    assert made > 0
    for _ in range(3):
        a.call()
    for _ in range(2):
        b.call()
    few = Batch(imgs[:3], [100, 700, 30])
    few.call()
    a.call([torch.from_numpy(im).pin_memory() for im in imgs[:5]])
    a.call()
    assert shim.shim_calls() == made, (made, shim.shim_calls())
    def at(contrast, k=0):
        want = F.features.sift_gpu_u8(imgs[k], nf[k], contrast=contrast)
        n = F.features.sift_gpu_batch_d(a.img, nf[:5], a.xy, a.u8, a.rs, chains=2, contrast=contrast)
        assert n[k] == len(want[0])
        np.testing.assert_array_equal(a.u8[k][:n[k]].cpu().numpy(), want[1])
        return shim.shim_calls()
    for contrast in (0.03, 0.02, 0.01):
        two = at(contrast)
    assert two == made + 3 * 2              # one per chain and threshold
    for contrast in (0.03, 0.02, 0.01, 0.015, 0.03):
        assert at(contrast) == two          # kept
    for k, contrast in enumerate((0.031, 0.032, 0.033, 0.034)):
        assert at(contrast) == two + 2 * (k + 1)   # in the place of the four above
    for contrast in (0.035, 0.036):
        assert at(contrast) == two + 8      # none of those was replayed
    assert at(0.036) == two + 10
    assert at(0.036) == two + 10
    assert at(0.034) == two + 10            # kept all the while
    """ % hw)


@pytest.mark.parametrize("exact", [False, True])
def test_slots_carry_every_call_s_own_arguments(exact):
    """More images than chains, other caps and outputs at each call (none for the responses, a cap of zero among
    them), padded rows, both pyramids: the launches kept from the first call take all of it from the slots."""
    import numpy as np
    import torch
    import fieldstitch_b200 as F
    from fieldstitch_b200 import synth
    dev = torch.device("cuda", 0)
    h, w = 150, 203
    imgs = [synth.synth_image(h, w, 80 + k) for k in range(7)]
    for call in range(4):
        rng = np.random.default_rng(call)
        pick = [int(k) for k in rng.permutation(7)[:5 + call % 3]]
        caps = [int(rng.integers(1, 900)) for _ in pick]
        caps[call % len(caps)] = 0
        pitch = w if call < 2 else w + 5   # another row pitch: graphs of its own
        d = [torch.zeros((h, pitch), dtype=torch.uint8, device=dev)[:, :w] for _ in pick]
        for t, k in zip(d, pick):
            t.copy_(torch.from_numpy(imgs[k]))
        xy = [torch.full((1000, 2), -7.0, device=dev) for _ in pick]
        u8 = [torch.full((1000, 128), 9, dtype=torch.uint8, device=dev) for _ in pick]
        rs = [torch.full((1000,), -7.0, device=dev) for _ in pick] if call % 2 else None
        n = F.features.sift_gpu_batch_d(d, caps, xy, u8, rs, chains=3, exact=exact)
        for i, (k, cap) in enumerate(zip(pick, caps)):
            if cap == 0:
                assert n[i] == 0
            else:
                wxy, wu8, wrs = F.features.sift_gpu_u8(imgs[k], cap, exact=exact)
                assert n[i] == len(wxy)
                np.testing.assert_array_equal(xy[i][:n[i]].cpu().numpy(), wxy)
                np.testing.assert_array_equal(u8[i][:n[i]].cpu().numpy(), wu8)
                if rs is not None:
                    np.testing.assert_array_equal(rs[i][:n[i]].cpu().numpy(), wrs)
            # nothing behind the image's own rows
            assert (xy[i][n[i]:] == -7.0).all() and (u8[i][n[i]:] == 9).all()
            assert rs is None or (rs[i][n[i]:] == -7.0).all()
