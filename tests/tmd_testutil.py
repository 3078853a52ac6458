"""Shared helpers of the test suite (fixtures, data files, tolerances)."""
from __future__ import annotations

import json
from pathlib import Path

import numpy as np

from tmd_b200.synth import frac_wrap, read_data  # noqa: F401  (re-exported)

ROOT = Path(__file__).resolve().parent.parent
GOLDEN = ROOT / "tests" / "golden"
NKTV2P = 1.6021765e6  # metal units, update.cpp:187-206


# FIRE starts (seed of a 64-atom packing, iterations) whose trajectories are
# stable: the FP64 oracle, started 1e-7 A away, stays within 2e-4 A of its own
# (test_fire_starts.py).  Most packings come near a zero of the power F.v
# within 200 iterations, and a 1e-8 A change of the start then flips a branch;
# these do not, or (90 iterations) end before they do.
FIRE_STARTS = [(23, 200), (26, 200), (21, 90), (28, 90)]


def fire_start(seed):
    from tmd_b200 import synth
    rng = np.random.default_rng(seed)
    x, box = synth.random_packing(64, rng)
    return x, rng.integers(1, 5, size=64).astype(np.int32), box


def fire_potential(path):
    """The four-element random-weight potential of the serving tests."""
    from tmd_b200 import synth
    return synth.gaussian_potential(path, seed=31, nelt=4, num_filters=16, rc=6.0, max_moment=3,
                                    hidden=(64, 64), actfn=2)


def cell_distance(a, b, box):
    """Largest coordinate difference of two configurations of an orthogonal cell."""
    d = a - b
    return float(np.abs(d - np.round(d / box[3:6]) * box[3:6]).max())


def published():
    return json.loads((GOLDEN / "published.json").read_text())


def volume(box):
    return box[3] * box[4] * box[5]


def kinetic_pressure(natoms, temp, vol):
    """Kinetic part of LAMMPS's pressure in bar: dof k_B T / (3 V) with
    dof = 3 N - 3 (ComputeTemp::dof_compute, compute_temp.cpp:58-62, extra_dof
    = dimension, compute.cpp:84) and metal k_B (update.cpp:188)."""
    return (3 * natoms - 3) * 8.617343e-5 * temp / (3 * vol) * NKTV2P


def bcc_lattice(a, nx, ny, nz):
    """Perfect BCC cells (LAMMPS `lattice bcc a` + `create_atoms`): positions
    and the orthogonal box as (xlo, ylo, zlo, xhi, yhi, zhi, xy, xz, yz)."""
    g = np.stack(np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"),
                 -1).reshape(-1, 3).astype(float)
    x = np.concatenate([g, g + 0.5]) * a
    return x, np.array([0, 0, 0, nx * a, ny * a, nz * a, 0, 0, 0], dtype=float)


def canonical_pairs(off, ent):
    """Sorted (i, j, sx, sy, sz) tuples of a neighbor list."""
    n = len(off) - 1
    i = np.repeat(np.arange(n), np.diff(off))
    t = np.concatenate([i[:, None], ent[:, :4]], 1).astype(np.int64)
    order = np.lexsort(t.T[::-1])
    return t[order]


def rel_rms(a, b):
    a = np.asarray(a, dtype=np.float64).ravel()
    b = np.asarray(b, dtype=np.float64).ravel()
    return float(np.sqrt(np.mean((a - b) ** 2)) / max(np.sqrt(np.mean(b ** 2)), 1e-300))
