"""FP32 MLP kernel at the edges of its tiles, column blocks and chunks.

The tile height follows the number of atoms (1, 2, 4 or 8 rows per thread) and
the block width the widest hidden layer (32, 64, 128 columns; wider layers take
several blocks).  Sums run over the reduction index in one order whatever the
tile, so a cell's results must not depend on the tile height or on how many
cells share the launch.  test_tiles_and_blocks: one cell (smallest tiles) against
the oracle, then the same cell among copies of it, bitwise, with the heights that
the library picks.  test_every_tile_height: every height of every block width,
bitwise against the smallest and that against the oracle, with one element's
atoms at one row less than a tile, a full tile and one row more."""
import numpy as np
import pytest

from pack import Oracle, load_npz
from tmd_b200 import TensorMDBatch, TensorMDModel, TensorMDSystem, synth
from tmd_testutil import rel_rms

pytestmark = pytest.mark.gpu

NETS = [dict(hidden=(8, 8), actfn=2),                       # 32-column blocks
        dict(hidden=(30, 7), actfn=3),                      # widths not multiples of 4
        dict(hidden=(48, 48, 48), actfn=1, resnet=1),       # 64, residual
        dict(hidden=(64,), actfn=0),                        # one hidden layer
        dict(hidden=(96, 80), actfn=2),                     # 128, unequal
        dict(hidden=(160, 160, 160), actfn=3, resnet=1)]    # two blocks, residual


@pytest.mark.parametrize("net", NETS, ids=lambda n: "-".join(map(str, n["hidden"])))
def test_tiles_and_blocks(tmp_path, net):
    p = tmp_path / "m.npz"
    syms = synth.gaussian_potential(p, nelt=2, num_filters=4, rc=4.5, max_moment=2, seed=3, **net)
    m = TensorMDModel(f"{p} {' '.join(syms)}")
    orc = Oracle(load_npz(p))
    rng = np.random.default_rng(4)
    x0, box = synth.lattice("fcc", 3.6, 3, 3, 3)
    x0 = synth.wrap(x0 + rng.normal(0.0, 0.08, x0.shape), box)
    for first in (1, 16, 33):  # atoms of element 0; the rest are element 1
        t = np.full(len(x0), 2, dtype=np.int32)
        t[:first] = 1
        s = TensorMDSystem(m, len(x0), 1.0)
        s.set_box(box)
        s.set_atoms(x0, t)
        out = s.compute(1, 1)
        ref = orc.compute(x0, t - 1, box, [1, 1, 1], skin=1.0)
        assert rel_rms(out["f"], ref["f"]) <= 1e-5
        # FP32 hidden layers: relative to the energy for residual nets, whose
        # atoms carry a sum of 100 inputs
        tol = max(5e-7 * len(x0), 2e-7 * abs(ref["energy"]))
        assert abs(out["energy"] - ref["energy"]) <= tol
        for copies in (40, 400):
            b = TensorMDBatch(m, [len(x0)] * copies, 1.0)
            b.set_cells(np.tile(box, (copies, 1)))
            b.set_atoms(np.tile(x0, (copies, 1)), np.tile(t, copies))
            many = b.compute()
            assert np.array_equal(many["f"].reshape(copies, -1, 3),
                                  np.broadcast_to(out["f"], (copies,) + out["f"].shape))
            b.close()


WIDTHS = [dict(hidden=(24, 32), actfn=1),
          dict(hidden=(64, 64, 64), actfn=2, resnet=1),
          dict(hidden=(128, 100), actfn=3)]


@pytest.mark.parametrize("net", WIDTHS, ids=["32", "64", "128"])
def test_every_tile_height(tmp_path, net):
    p = tmp_path / "m.npz"
    syms = synth.gaussian_potential(p, nelt=2, num_filters=4, rc=4.5, max_moment=2, seed=3, **net)
    m = TensorMDModel(f"{p} {' '.join(syms)}")
    orc = Oracle(load_npz(p))
    rng = np.random.default_rng(4)
    x, box = synth.lattice("fcc", 3.6, 5, 4, 4)
    x = synth.wrap(x + rng.normal(0.0, 0.08, x.shape), box)
    s = TensorMDSystem(m, len(x), 1.0)
    s.set_box(box)
    heights = s.mlp_rows()[1]
    block = 32 if max(net["hidden"]) <= 32 else (64 if max(net["hidden"]) <= 64 else 128)
    assert heights == [1024 // block * r for r in (1, 2, 4, 8)]
    for first in sorted({h + d for h in heights for d in (-1, 0, 1)}):
        t = np.full(len(x), 2, dtype=np.int32)
        t[:first] = 1
        got = []
        for h in heights:
            s.set_mlp_rows(h)
            s.set_atoms(x, t)
            assert s.mlp_rows()[0] == h
            got.append(s.compute(1, 1))
        ref = orc.compute(x, t - 1, box, [1, 1, 1], skin=1.0)
        assert rel_rms(got[0]["f"], ref["f"]) <= 1e-5
        for g in got[1:]:
            assert np.array_equal(g["f"], got[0]["f"]) and g["energy"] == got[0]["energy"]
    s.set_mlp_rows(0)
    s.set_atoms(x, t)
    assert s.mlp_rows()[0] in heights


# (hidden layers, atoms): the heights that the choice must be among, each at
# least 5% faster than the others in timings of all four (1,024 / block width x
# 1, 2, 4, 8 atoms; the 128,000 and 126,976 atoms differ in how full the last
# wave of 128-atom tiles is)
CHOICES = [((32, 32, 32), 432, (32,)), ((32, 32, 32), 97556, (64, 128)),
           ((64, 64), 432, (16,)), ((64, 64), 8192, (32,)), ((64, 64), 126976, (128,)),
           ((64, 64), 128000, (64,)),
           ((128, 128, 128), 432, (8,)), ((128, 128, 128), 2048, (16,)),
           ((128, 128, 128), 23040, (64,)), ((128, 128, 128), 202612, (32, 64))]


@pytest.mark.parametrize("hidden,n,best", CHOICES, ids=[f"{h[0]}-{n}" for h, n, _ in CHOICES])
def test_height_follows_the_timings(tmp_path, hidden, n, best):
    p = tmp_path / "m.npz"
    syms = synth.gaussian_potential(p, nelt=1, num_filters=4, rc=2.0, max_moment=1, seed=3,
                                    hidden=hidden, actfn=2)
    s = TensorMDSystem(TensorMDModel(f"{p} {' '.join(syms)}"), n, 0.5)
    k = int(np.ceil(n ** (1 / 3)))
    s.set_box(np.array([0, 0, 0, 3.0 * k, 3.0 * k, 3.0 * k, 0, 0, 0]))
    x = 3.0 * np.stack(np.unravel_index(np.arange(n), (k, k, k)), -1).astype(float)
    s.set_atoms(x, np.ones(n, dtype=np.int32))
    assert s.mlp_rows()[0] in best
