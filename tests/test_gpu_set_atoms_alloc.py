"""set_atoms allocates nothing for the FP32 MLP: its act' scratch is part of the
system, so a larger or differently mixed set of atoms neither waits for the
device's allocator nor can fail half way.  Free device memory must not change
when the atom count grows, the rows of the neighbor list being long enough."""
import numpy as np
import pytest

from tmd_b200 import TensorMDModel, TensorMDSystem, TmdError, synth

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
    rng = np.random.default_rng(4)

    def use(s, n):
        some = np.sort(rng.permutation(len(x))[:n])
        s.set_atoms(x[some], rng.integers(1, 3, n).astype(np.int32))
        return s.compute(1, 1)

    sizes = (500, 4000, 12000, len(x))
    first = TensorMDSystem(m, len(x), 1.0)  # loads every kernel that the sizes take
    first.set_box(box)
    for n in (64, *sizes):
        use(first, n)
    s = TensorMDSystem(m, len(x), 1.0)
    s.set_box(box)
    use(s, 64)
    before = _free()
    for n in sizes:
        use(s, n)
    assert _free() == before


@pytest.mark.parametrize("ghost", [False, True])
def test_refused_atoms_leave_nothing_to_compute(tmp_path, ghost):
    """set_atoms beyond 4,096 neighbors per atom is refused; the atoms of the call
    before are gone by then, so a compute is refused too, until atoms are set."""
    p = tmp_path / "m.npz"
    syms = synth.gaussian_potential(p, nelt=1, num_filters=4, rc=6.0, max_moment=1, hidden=(16,),
                                    actfn=2, seed=2)
    s = TensorMDSystem(TensorMDModel(f"{p} {' '.join(syms)}"), 2500, 1.0)
    x, t, box, _ = synth.build_system("fcc", 3.6, (4, 4, 4), sigma=0.05, nelt=1, seed=3)

    def use(x, t):
        if ghost:
            s.set_atoms_ghost(len(x) // 2, x, t)
        else:
            s.set_atoms(x, t)

    s.set_box(box)
    use(x, t)
    ref = s.compute(1, 1)
    dense = np.random.default_rng(5).uniform(0.0, 8.0, (2500, 3))  # 5 atoms per A^3
    if not ghost:
        s.set_box(np.array([0, 0, 0, 8.0, 8.0, 8.0, 0, 0, 0]))
    with pytest.raises(TmdError) as err:
        use(dense, np.ones(2500, dtype=np.int32))
    assert err.value.code == -4
    with pytest.raises(TmdError) as err:
        s.compute(1, 1)
    assert "set_atoms" in str(err.value)
    if not ghost:
        s.set_box(box)
    use(x, t)
    again = s.compute(1, 1)
    assert np.array_equal(again["f"], ref["f"]) and again["energy"] == ref["energy"]
