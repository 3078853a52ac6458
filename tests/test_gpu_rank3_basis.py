"""The rank-3 descriptor is summed over 16 functions on the sphere and put
together again; what that does must not shift every atom alike.

In a perfect cubic crystal P_xx = P_yy = P_zz = P_0 / 3 and the off-diagonal
sums vanish, so G_2 = G_0^2 / 3 whatever the radial functions' own errors.  Each
side rounds to about 1e-7; over 32 filters and 36 crystals a common part of
more than 2e-8 shows (constants that do not add up gave 4e-8)."""
import numpy as np
import pytest

from tmd_b200 import TensorMDModel, TensorMDSystem, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["filter4", "wide", "wide2", "split"])
def test_no_common_shift_in_cubic_crystals(tmp_path, form):
    p = tmp_path / "m.npz"
    syms = synth.gaussian_potential(p, nelt=1, num_filters=32, rc=6.0, max_moment=3,
                                    hidden=(16,), actfn=2, seed=4)
    m = TensorMDModel(f"{p} {' '.join(syms)}")
    off = []
    for lattice, a0 in (("fcc", 3.4), ("bcc", 2.7)):
        for a in a0 * np.linspace(1.0, 1.3, 18):
            x, box = synth.lattice(lattice, a, 5, 5, 5)
            s = TensorMDSystem(m, len(x), 0.5)
            s.set_box(box)
            s.set_atoms(x, np.ones(len(x), dtype=np.int32))
            s.set_descriptor_variant(form)
            g = s.descriptors().reshape(len(x), 32, 4)
            use = g[..., 0] > 1e-3 * g[..., 0].max()
            off.append(np.mean(3 * g[use][:, 2] / g[use][:, 0] ** 2 - 1))
    assert abs(np.mean(off)) < 2e-8, np.mean(off)
