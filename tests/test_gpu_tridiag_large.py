"""Eigenpairs of systems above the register-resident Householder kernel's size.

One SCC iteration of water clusters whose orbital counts sit at the edges of
the cluster kernel's tiles (rows of 8, columns of 64, odd counts), for the
launch shapes its rule picks (8 and 16 CTAs a system, small systems in the
same call; at 2190 orbitals 16 CTAs no longer have the shared memory, above 2208
eight warps a CTA do not either), and for batches on both sides of the line to
the single-CTA path: 33 x 262 are one wave of clusters, 60 x 360 two, more than
run at once; 40 x 302 and 70 x 360 take the single CTAs, and 160 x 402, more
than one wave of those, the clusters again.  The eigenvalues must be those of
X H X (LAPACK), and the density, formed from the back-transformed vectors,
LAPACK's: a backward-stable solver moves an occupied projector by about
n eps ||A|| / gap, under 1e-11 here; 1e-9 leaves two orders.
"""
from __future__ import annotations

import numpy as np
import pytest

from xtbloom_b200 import abi
from xtbloom_b200 import workloads as W

pytestmark = pytest.mark.gpu


def cluster(n):
    """A molecule of n orbitals: waters, then H2 (2 orbitals) or H3O+ (7) beside them."""
    extra, charge = n % 6, 0.0
    add = []
    if extra % 2:
        add.append("H3O+")
        charge, n = 1.0, n - 7
    add += ["H2"] * ((n % 6) // 2)
    z, x = W.water_cluster(n // 6, np.random.default_rng(n))
    far = np.abs(x).max() + 6.0
    for k, what in enumerate(add):
        if what == "H2":
            z, x = np.append(z, [1, 1]), np.vstack([x, [[far, 6.0 * k, 0], [far, 6.0 * k, 1.4]]])
        else:
            z = np.append(z, [8, 1, 1, 1])
            x = np.vstack([x, np.array([[0, 0, 0.3], [1.75, 0, 0], [-0.875, 1.516, 0], [-0.875, -1.516, 0]]) + [far, 6.0 * k, 0]])
    return z, x, charge


@pytest.mark.parametrize("sizes", [
    [258], [257, 259, 264], [320, 321, 319, 12], [384, 30, 200], [481], [600, 480], [1000], [2190], [2214],
    [262] * 33, [258] * 9 + [90] * 40, [360] * 60, [302] * 40, [360] * 70, [402] * 160,
    [600, 594, 588, 577, 569, 560, 552, 537, 520, 513, 504, 481]], ids=lambda s: "%dx%d" % (len(s), s[0]))
def test_eigenpairs_match_lapack(cuda_lib, sizes):
    mols = [cluster(n) for n in sizes]
    b = abi.ragged_from_lists([m[0] for m in mols], [m[1] for m in mols], [m[2] for m in mols])
    cuda_lib.compute(b, cuda_lib.make_options(max_iter=1))
    for i in sorted({0, len(sizes) // 2, len(sizes) - 1}):
        ev = cuda_lib.fetch("eigenvalues", i, capacity=4096)
        n = len(ev)
        assert n == sizes[i]
        h, x, p = (cuda_lib.fetch(k, i, capacity=n * n).reshape(n, n) for k in ("hamiltonian", "x", "density"))
        a = x @ h @ x
        ref, vec = np.linalg.eigh(0.5 * (a + a.T))
        k = int((ev < 1e300).sum())
        assert np.abs(ev[:k] - ref[:k]).max() < 1e-10 * max(1.0, np.abs(ref).max())
        occupied = int(round(cuda_lib.fetch("occupations", i, capacity=4096).sum())) // 2
        assert ref[occupied] - ref[occupied - 1] > 0.05
        c = x @ vec[:, :occupied]
        assert np.abs(p - 2.0 * c @ c.T).max() < 1e-9
