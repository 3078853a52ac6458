"""set_atoms allocates nothing for the FP32 MLP: its act' scratch is part of the
system, so a larger or differently mixed set of atoms neither waits for the
device's allocator nor can fail half way.  Free device memory must not change
when the atom count grows, the rows of the neighbor list being long enough."""
import numpy as np
import pytest

from tmd_b200 import TensorMDModel, TensorMDSystem, synth

pytestmark = pytest.mark.gpu


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_growing_atom_sets_allocate_nothing(tmp_path):
    p = tmp_path / "m.npz"
    syms = synth.gaussian_potential(p, nelt=2, num_filters=4, rc=3.0, max_moment=1,
                                    hidden=(128, 128, 128, 128), actfn=3, resnet=1, seed=2)
    m = TensorMDModel(f"{p} {' '.join(syms)}")
    x, _, box, _ = synth.build_system("fcc", 3.6, (20, 20, 20), sigma=0.05, nelt=1, seed=3)
    s = TensorMDSystem(m, len(x), 1.0)
    s.set_box(box)
    rng = np.random.default_rng(4)

    def use(n):
        some = np.sort(rng.permutation(len(x))[:n])
        s.set_atoms(x[some], rng.integers(1, 3, n).astype(np.int32))
        return s.compute(1, 1)

    use(64)
    before = _free()
    for n in (500, 4000, 12000, len(x)):
        use(n)
    assert _free() == before
