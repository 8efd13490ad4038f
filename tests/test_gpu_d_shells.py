"""Molecules with d shells, whose orbital pairs the integral and gradient kernels deal out by cost.

GFN2 energies, forces and charges against the numpy oracle, GFN1 forces against central differences
of its energies, at sizes on both sides of a run of 128 orbital rows and of a block of 128 pairs;
and the bits of molecules without d shells, which must not depend on others in the batch.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import TOL_E, TOL_F, TOL_Q
from oracle import gfn2
from xtbloom_b200 import abi
from xtbloom_b200 import workloads as W

pytestmark = pytest.mark.gpu

T = 3.83 / np.sqrt(3.0)
SICL4 = (np.array([14, 17, 17, 17, 17], np.int32),
         np.array([[0, 0, 0], [T, T, T], [T, -T, -T], [-T, T, -T], [-T, -T, T]]))
H2S = (np.array([16, 1, 1], np.int32), np.array([[0, 0, 0], [1.8, 1.76, 0], [1.8, -1.76, 0]]))
HCL = (np.array([17, 1], np.int32), np.array([[0, 0, 0], [2.41, 0, 0]]))


def lattice(molecule, spacing, count):
    """count molecules on a cubic lattice, every atom moved a little."""
    z, x = molecule
    edge = int(np.ceil(count ** (1 / 3)))
    cells = [(i, j, k) for i in range(edge) for j in range(edge) for k in range(edge)][:count]
    rng = np.random.default_rng(count)
    return (np.concatenate([z] * count).astype(np.int32),
            np.concatenate([x + spacing * np.array(c) + rng.normal(0, 0.05, x.shape) for c in cells]))


def ragged(mols):
    return abi.ragged_from_lists([m[0] for m in mols], [m[1] for m in mols])


# 45, 180 orbitals of d atoms alone; 22 and 132 with hydrogens; 10 and 110
MOLECULES = [lattice(SICL4, 9.5, 1), lattice(SICL4, 9.5, 4), lattice(H2S, 7.5, 2), lattice(H2S, 7.5, 12),
             lattice(HCL, 7.5, 1), lattice(HCL, 7.5, 11)]


def test_gfn2_matches_the_oracle(cuda_lib):
    b = ragged(MOLECULES)
    out = cuda_lib.compute(b, cuda_lib.make_options(ctol=1e-9, etol=1e-12))
    for i, (z, x) in enumerate(MOLECULES):
        r = gfn2.singlepoint(z, x)
        a0, a1 = b.atom_offsets[i], b.atom_offsets[i + 1]
        assert out["per_system_status"][i] == 0
        assert abs(out["energies"][i] - r.energy) < TOL_E
        assert np.abs(out["forces"][3 * a0:3 * a1] + r.gradient.ravel()).max() < TOL_F
        assert np.abs(out["atomic_charges"][a0:a1] - r.charges).max() < TOL_Q


def test_gfn1_forces_are_the_energy_slope(cuda_lib):
    """Central differences along one random direction a molecule: the step of 1e-3 leaves an error
    of h^2 E''' / 6, about 1e-7 for third derivatives of order one."""
    opt = cuda_lib.make_options(model=abi.MODEL_GFN1, ctol=1e-10, etol=1e-13)
    rng = np.random.default_rng(3)
    u = [rng.normal(size=x.shape) for _, x in MOLECULES]
    u = [v / np.linalg.norm(v) for v in u]
    h = 1e-3
    b, up, down = (ragged([(z, x + s * h * v) for (z, x), v in zip(MOLECULES, u)]) for s in (0, 1, -1))
    out, e_up, e_down = (cuda_lib.compute(q, opt) for q in (b, up, down))
    assert all((o["per_system_status"] == 0).all() for o in (out, e_up, e_down))
    for i, v in enumerate(u):
        a0, a1 = b.atom_offsets[i], b.atom_offsets[i + 1]
        slope = (e_up["energies"][i] - e_down["energies"][i]) / (2 * h)
        assert abs(slope + out["forces"][3 * a0:3 * a1] @ v.ravel()) < 2e-6


@pytest.mark.parametrize("model", [1, 2])
def test_molecules_without_d_shells_keep_their_bits_beside_them(cuda_lib, model):
    plain = [W.water_cluster(3, np.random.default_rng(1)), W.hetero_alkane(9, np.random.default_rng(2))]
    opt = cuda_lib.make_options(model=model)
    # the same number and sizes of systems, so that the launches are alike
    alone = cuda_lib.compute(ragged(plain + [W.hetero_alkane(7, np.random.default_rng(3))]), opt)
    beside = cuda_lib.compute(ragged(plain + [lattice(SICL4, 9.5, 1)]), opt)
    n = 3 * sum(len(z) for z, _ in plain)
    assert np.array_equal(alone["energies"][:2], beside["energies"][:2])
    assert np.array_equal(alone["forces"][:n], beside["forces"][:n])
    assert np.array_equal(alone["atomic_charges"][:n // 3], beside["atomic_charges"][:n // 3])
