"""Models that share kernels: loading a second potential must not take shared
memory away from the launches of one that is in use.  The limit of dynamic
shared memory belongs to a kernel, and nets of one block width, activation and
precision share theirs: the larger net is loaded first, then the smaller, then
the first computes again."""
import numpy as np
import pytest

from tmd_b200 import TensorMDModel, TensorMDSystem, synth

pytestmark = pytest.mark.gpu

WIDE = dict(nelt=4, num_filters=32, rc=6.0, max_moment=3)
SLIM = dict(nelt=1, num_filters=16, rc=6.0, max_moment=3)
# (keyword, larger net, smaller net)
PAIRS = {
    "fp32-128": ("", dict(SLIM, hidden=(128,) * 4, actfn=3), dict(SLIM, hidden=(128,) * 2, actfn=3)),
    "fp32-64": ("", dict(SLIM, hidden=(64,) * 5, actfn=2), dict(SLIM, hidden=(64,), actfn=2)),
    "tiled-bf16": ("precision bf16", dict(SLIM, hidden=(64,) * 4, actfn=1, resnet=1),
                   dict(SLIM, hidden=(64,) * 3, actfn=1, resnet=1)),
    "persistent-bf16": ("precision bf16", dict(SLIM, hidden=(64,) * 3, actfn=2),
                        dict(SLIM, hidden=(64,) * 2, actfn=2)),
    "streamed-bf16x3": ("precision bf16x3", dict(WIDE, hidden=(128,) * 3, actfn=1),
                        dict(WIDE, nelt=3, hidden=(64,) * 3, actfn=1)),
    "streamed-tf32x3": ("precision tf32x3", dict(WIDE, hidden=(128,) * 3, actfn=1),
                        dict(SLIM, hidden=(64,) * 2, actfn=1)),
    "fp8": ("precision fp8", dict(SLIM, hidden=(64,) * 4, actfn=2), dict(SLIM, hidden=(64,) * 2, actfn=2)),
}


def _system(path, keyword, net):
    syms = synth.gaussian_potential(path, seed=5, **net)
    x, t, box, _ = synth.build_system("fcc", 3.6, (5, 5, 5), sigma=0.05, nelt=net["nelt"], seed=3)
    s = TensorMDSystem(TensorMDModel(f"{path} {' '.join(syms)} {keyword}"), len(x), 1.0)
    s.set_box(box)
    s.set_atoms(x, t)
    return s


@pytest.mark.parametrize("form", sorted(PAIRS))
def test_second_model_leaves_the_first_usable(tmp_path, form):
    keyword, large, small = PAIRS[form]
    first = _system(tmp_path / "a.npz", keyword, large)
    ref = first.compute(1, 1)
    second = _system(tmp_path / "b.npz", keyword, small)
    second.compute(1, 1)
    again = first.compute(1, 1)
    assert np.array_equal(again["f"], ref["f"]) and again["energy"] == ref["energy"]
