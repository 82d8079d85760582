"""The bounds of a candidate chunk of the tensor-core matcher, for every value that a record can hold (a dense
kernel that gave up leaves some unwritten): compiled for the host and compared with 64-bit arithmetic."""
import ctypes
import os
import random
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fieldstitch_b200", "csrc")


def test_columns_stay_inside_the_targets(tmp_path):
    src, so = tmp_path / "c.cpp", tmp_path / "c.so"
    src.write_text('#include "tc_chunk.cuh"\nextern "C" int columns(int ch, int nb) { return fsb::chunk_columns(ch, nb); }\n')
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", CSRC, "-o", str(so), str(src)], check=True)
    f = ctypes.CDLL(str(so)).columns
    rng = random.Random(1)
    top = 2 ** 31 - 1
    chunks = [-1, 0, 1, 2, 0x07ffffff, 0x08000000, 0x0fffffff, 0x10000000, 0x10000001, 0x18000000, top, -top - 1]
    sizes = [1, 2, 15, 16, 17, 31, 32, 33, 16384, 2 ** 27, top]
    cases = [(c, n) for c in chunks for n in sizes] + [(rng.randint(-top - 1, top), rng.randint(1, top)) for _ in range(20000)]
    cases += [(n // 16 + d, n) for n in sizes for d in (-1, 0, 1)]
    for ch, nb in cases:
        want = max(0, min(16, nb - 16 * ch)) if ch >= 0 else 0
        assert f(ch, nb) == want, (ch, nb)
