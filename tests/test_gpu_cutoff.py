"""Pair geometry near the cutoff: forces of isolated dimers against the FP64
oracle, relative to each dimer's own force.

There f_c goes as (1 - z)^2 and f_c' as 1 - z with z = r / rc, so what counts
is the relative accuracy of the cutoff's sine and cosine and of the distance.
FP32 leaves the rounding of z = fl(r fl(1/rc)): 2^-25 / sqrt(3) rms from the
product and up to 2^-25, the same for every pair, from 1/rc; an error dz is
2 dz / (1 - z) of f_c.  Over z uniform in [a, b] the rms of 1 / (1 - z) is
1 / sqrt((1 - a)(1 - b))."""
import numpy as np
import pytest

from pack import Oracle, load_npz
from tmd_b200 import TensorMDBatch, TensorMDModel, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rank", [1, 3])
def test_dimers_near_the_cutoff(tmp_path, rank):
    n, rc, lo, hi = 1500, 5.0, 4.9, 4.99
    p = tmp_path / "m.npz"
    # one linear hidden layer: the potential adds no rounding that varies
    syms = synth.gaussian_potential(p, nelt=1, num_filters=4, rc=rc, hidden=(8,), actfn=0, seed=3,
                                    max_moment=rank)
    rng = np.random.default_rng(1)
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    x = np.empty((n, 2, 3))
    x[:, 0] = 7.0 + rng.uniform(0.0, 1.0, (n, 3))
    x[:, 1] = x[:, 0] + u * rng.uniform(lo, hi, n)[:, None]
    box = np.array([0, 0, 0, 20.0, 20.0, 20.0, 0, 0, 0])
    b = TensorMDBatch(TensorMDModel(f"{p} {' '.join(syms)}"), [2] * n, 1.0)
    b.set_cells(np.tile(box, (n, 1)))
    b.set_atoms(x.reshape(-1, 3), np.ones(2 * n, dtype=np.int32))
    f = b.compute()["f"].reshape(n, 2, 3)[:, 0]
    b.close()
    orc = Oracle(load_npz(p))
    elem = np.zeros(2, dtype=np.int32)
    ref = np.stack([orc.compute(c, elem, box, [1, 1, 1], skin=1.0)["f"][0] for c in x])
    err = np.linalg.norm(f - ref, axis=1) / np.linalg.norm(ref, axis=1)
    dz = 2.0 ** -25 / np.sqrt(3.0) + 2.0 ** -25
    assert np.sqrt(np.mean(err ** 2)) <= 2 * dz / np.sqrt((1 - lo / rc) * (1 - hi / rc))
