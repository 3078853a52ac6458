"""Default descriptor form: wide, and split for table radials on 8,192 (local)
atoms and more.  The choice follows the atom count of the launch, so a cell must get
the same bits from both forms: descriptors, forces, energy and virial of the
wide and the split form are compared bitwise over filter counts, radial kinds,
ranks and elements."""
import numpy as np
import pytest

from tmd_b200 import TensorMDBatch, TensorMDModel, TensorMDSystem, synth

pytestmark = pytest.mark.gpu


def _system(tmp_path, cells, table, **kw):
    p = tmp_path / "m.npz"
    syms = synth.gaussian_potential(p, rc=5.0, hidden=(16, 16), actfn=2, seed=8, **kw)
    m = TensorMDModel(f"{p} {' '.join(syms)}" + (" interp 0.005" if table else ""))
    x, t, box, _ = synth.build_system("bcc", 2.9, cells, sigma=0.08, nelt=kw["nelt"], seed=6)
    s = TensorMDSystem(m, len(x), 1.0)
    s.set_box(box)
    s.set_atoms(x, t)
    return s


@pytest.mark.parametrize("table", [False, True], ids=["gauss", "table"])
@pytest.mark.parametrize("K,mm,nelt", [(4, 3, 2), (8, 2, 1), (16, 3, 1), (32, 3, 2), (64, 3, 1),
                                       (16, 1, 2)])
def test_wide_and_split_agree_bitwise(tmp_path, K, mm, nelt, table):
    s = _system(tmp_path, (5, 5, 6), table, nelt=nelt, num_filters=K, max_moment=mm)
    got = []
    for form in ("wide", "split"):
        s.set_descriptor_variant(form)
        out = s.compute(1, 1)
        got.append((s.descriptors(), out["f"], out["energy"], out["virial"]))
    assert np.array_equal(got[0][0], got[1][0])
    assert np.array_equal(got[0][1], got[1][1])
    assert got[0][2] == got[1][2]
    assert np.array_equal(got[0][3], got[1][3])


def test_default_follows_kind_and_size(tmp_path):
    kw = dict(nelt=1, num_filters=8, max_moment=1)
    assert _system(tmp_path, (6, 6, 6), True, **kw).descriptor_variant() == "wide"
    assert _system(tmp_path, (16, 16, 16), False, **kw).descriptor_variant() == "wide"
    s = _system(tmp_path, (16, 16, 16), True, **kw)  # 8,192 atoms
    assert s.descriptor_variant() == "split"
    s.set_descriptor_variant("wide")  # the caller's choice stands
    assert s.descriptor_variant() == "wide"


def test_default_counts_local_atoms(tmp_path):
    p = tmp_path / "m.npz"
    syms = synth.gaussian_potential(p, rc=3.0, hidden=(16,), actfn=2, seed=8, nelt=1,
                                    num_filters=8, max_moment=1)
    m = TensorMDModel(f"{p} {' '.join(syms)} interp 0.005")
    x, _, _, _ = synth.build_system("bcc", 2.9, (16, 16, 17), sigma=0.05, nelt=1, seed=6)
    t = np.ones(len(x), dtype=np.int32)
    s = TensorMDSystem(m, len(x), 0.5)
    s.set_atoms_ghost(8191, x, t)  # the kernels run over the local atoms
    assert s.descriptor_variant() == "wide"
    s.set_atoms_ghost(8192, x, t)
    assert s.descriptor_variant() == "split"


@pytest.mark.parametrize("nelt,K", [(1, 16), (3, 32)])
def test_wide_and_split_agree_bitwise_in_batches(tmp_path, nelt, K):
    """Cells of one batch, each with its own box, above the split form's line."""
    p = tmp_path / "m.npz"
    syms = synth.gaussian_potential(p, rc=5.0, hidden=(16, 16), actfn=2, seed=8, nelt=nelt,
                                    num_filters=K, max_moment=3)
    m = TensorMDModel(f"{p} {' '.join(syms)} interp 0.005")
    cells = [synth.build_system(lat, a, rep, sigma=0.08, nelt=nelt, seed=k)[:3]
             for k in range(24) for lat, a, rep in (("bcc", 2.9, (5, 5, 6)), ("fcc", 3.6, (3, 4, 3)))]
    b = TensorMDBatch(m, [len(c[0]) for c in cells], 1.0)
    b.set_cells(np.stack([c[2] for c in cells]))
    b.set_atoms(np.concatenate([c[0] for c in cells]), np.concatenate([c[1] for c in cells]))
    assert sum(len(c[0]) for c in cells) >= 8192
    assert b.system().descriptor_variant() == "split"
    got = {}
    for form in ("split", "wide"):
        b.system().set_descriptor_variant(form)
        got[form] = b.compute()
    for k in got["split"]:
        assert np.array_equal(got["split"][k], got["wide"][k]), k
    k = int(np.argmax([len(c[0]) for c in cells]))  # a cell alone gives the same forces
    s = TensorMDSystem(m, len(cells[k][0]), 1.0)
    s.set_box(cells[k][2])
    s.set_atoms(cells[k][0], cells[k][1])
    at = sum(len(c[0]) for c in cells[:k])
    assert np.array_equal(s.compute(1, 1)["f"], got["split"]["f"][at:at + len(cells[k][0])])
