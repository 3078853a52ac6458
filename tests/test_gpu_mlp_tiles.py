"""FP32 MLP kernel at the edges of its tiles, column blocks and chunks.

The tile height follows the number of atoms (1, 2, 4 or 8 rows per thread) and
the block width the widest hidden layer (32, 64, 128 columns; wider layers take
several blocks).  Sums run over the reduction index in one order whatever the
tile, so a cell's results must not depend on how many cells share the launch:
one cell (smallest tiles) against the oracle, then the same cell among enough
copies to reach the larger tiles, bitwise.  Cell sizes put every element's last
tile at one row, a full tile and one row more."""
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
