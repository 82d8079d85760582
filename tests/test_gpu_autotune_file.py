"""Choices kept in a tuning file: those of this library are taken without timing, those of a library whose
variants were numbered otherwise (no version in the key) are not, and are tuned again."""
import os
import re
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

BODY = """
import hashlib
import fieldstitch_b200 as F
from fieldstitch_b200 import synth
xy, u8, resp = F.features.sift_gpu_u8(synth.synth_image(610, 830, 3), 2000)
print(len(xy), hashlib.sha256(u8.tobytes() + xy.tobytes()).hexdigest())
"""


def _run(path):
    env = dict(os.environ, FSB_AUTOTUNE_FILE=str(path), PYTHONPATH=ROOT + os.pathsep + os.environ.get("PYTHONPATH", ""))
    for k in ("FSB_AUTOTUNE", "FSB_PYRAMID", "FSB_LAYER_VARIANT"):
        env.pop(k, None)
    r = subprocess.run([sys.executable, "-c", BODY], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    return r.stdout, [line for line in path.read_text().splitlines() if "k_octave" in line]


def test_choices_of_other_variants_are_tuned_again(tmp_path):
    path = tmp_path / "tuning"
    out, made = _run(path)
    assert len(made) >= 3
    same, kept = _run(path)
    assert same == out and kept == made                      # this library's choices: nothing to tune
    old = tmp_path / "old"
    # lines as an earlier library wrote them, every octave with the last variant
    old.write_text("".join(re.sub(r"/v\d+/", "/", line).rsplit(" ", 1)[0] + " 2\n" for line in made))
    again, lines = _run(old)
    assert again == out
    assert [line.rsplit(" ", 1)[0] for line in lines[len(made):]] == [line.rsplit(" ", 1)[0] for line in made]
