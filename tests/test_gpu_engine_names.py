"""FSB_PYRAMID's names: each forces the engine that it says, the names of retired fused engines the layer groups
(told apart by the number of launches: five per octave and two), and an unknown name chooses as unset."""
import pytest

pytestmark = pytest.mark.gpu


def test_names_force_their_engines(monkeypatch):
    import fieldstitch_b200 as f
    from fieldstitch_b200 import _lib, synth
    img = synth.synth_image(200, 300, 6)
    monkeypatch.setenv("FSB_AUTOTUNE", "0")   # unset: the per-layer kernels
    count = {}
    for name in (None, "layer", "group", "group_small", "strip", "fused", "other"):
        if name is None:
            monkeypatch.delenv("FSB_PYRAMID", raising=False)
        else:
            monkeypatch.setenv("FSB_PYRAMID", name)
        f.gsift.detect(img)[1].close()
        n0 = _lib.launch_count()
        _, st = f.gsift.detect(img)
        count[name] = _lib.launch_count() - n0
        st.close()
    assert count["layer"] == count[None] == count["other"]
    assert count["group"] == count["group_small"] < count["layer"]
    assert count["strip"] == count["fused"] == count["group"], count
