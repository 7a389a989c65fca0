"""The warp forms of the class kernels (eriWarpKernel) and of the gradient contraction (eriD1WarpKernel)
against the C restatement: bras with d and f functions under thin kets, in store, J/K and gradient
mode, in bases with one- and several-primitive pairs, and the kernels that were launched.

Tolerances: 1e-12 per integral, 1e-11 for J/K sums, 1e-10 for gradients (as the other tests of these
modes); 1e-6 Eh/bohr against central differences of step 1e-4 bohr, 1e-7 against the five-point formula of
step 4e-3 bohr (truncation h^4 / 30 = 8.5e-12 of the fifth derivative, some 1e2 to 1e3 Eh/bohr^5 at the most)."""
import numpy as np
import pytest
from launches import launched

from lible_b200 import ints as L
from lible_b200.workloads import random_density, water_cluster
from oracle import port

pytestmark = pytest.mark.gpu


FORWARD = {f"eriWarpKernel<{c}>" for c in ("2,2,1,0", "2,2,2,0", "3,1,2,0", "3,2,1,1", "3,3,0,0", "3,3,3,0")}
GRADIENT = {f"eriD1WarpKernel<{c}>" for c in ("2,1,0,0", "2,1,2,0", "2,2,1,0", "3,0,2,1", "3,2,3,0", "3,3,2,0")}


@pytest.mark.parametrize("basis", ["def2-tzvp", "cc-pvtz"])
def test_warp_form_integrals_match_the_restatement(basis):
    Z, xyz, _ = water_cluster(1, seed=41)
    s = L.Structure(basis, Z, xyz, units="bohr")
    assert np.abs(L.eri4(s) - port.PortMolecule(basis, Z, xyz).eri4()).max() <= 1e-12
    assert FORWARD <= launched(lambda: L.eri4(s)).keys()


@pytest.mark.parametrize("basis,waters", [("def2-tzvp", 1), ("cc-pvtz", 1), ("cc-pvtz", 2)])
def test_warp_form_jk_and_gradient_match_the_restatement(basis, waters):
    Z, xyz, rng = water_cluster(waters, seed=42)
    s = L.Structure(basis, Z, xyz, units="bohr")
    D = random_density(s.nao, 5 * waters, rng)
    J, K, _ = L.jk(s, D, schwarz=0.0)
    Jr, Kr = port.jk(basis, Z, xyz, D)
    assert np.abs(J - Jr).max() <= 1e-11 and np.abs(K - Kr).max() <= 1e-11
    assert FORWARD <= launched(lambda: L.jk(s, D, schwarz=0.0)).keys()
    if waters == 1:
        g = L.jk_energy_backward(s, D, schwarz=0.0)
        assert np.abs(g - port.PortMolecule(basis, Z, xyz).jk_grad(D)).max() <= 1e-10
        assert GRADIENT <= launched(lambda: L.jk_energy_backward(s, D, schwarz=0.0)).keys()


@pytest.mark.parametrize("basis,aux,forms", [("cc-pvtz", "def2-universal-jkfit", GRADIENT),
                                             ("def2-tzvp", "def2-qzvp-rifit", {"eriD1WarpKernel<4,0,4,0>",
                                                                               "eriD1WarpKernel<5,0,1,1>"})])
def test_warp_form_of_the_ri_gradient_against_the_energy(basis, aux, forms):
    Z, xyz, rng = water_cluster(1, seed=45)

    def build(x):
        return L.Structure(basis, Z, x, aux, units="bohr")

    s = build(xyz)
    D = random_density(s.nao, 5, rng)
    g, _ = L.rij_grad(s, D, schwarz=0.0)
    assert forms <= launched(lambda: L.rij_grad(s, D, schwarz=0.0)).keys()
    for atom, x in ((0, 1), (1, 0), (2, 2)):
        e = {}
        for k in (-2, -1, 1, 2):
            moved = xyz.copy()
            moved[atom, x] += 4e-3 * k
            e[k] = L.rij_grad(build(moved), D, schwarz=0.0)[1]
        assert abs((e[-2] - 8 * e[-1] + 8 * e[1] - e[2]) / (12 * 4e-3) - g[atom, x]) <= 1e-7


def test_warp_form_gradient_beyond_the_shared_memory_atoms():
    """More than 512 atoms: the warps add to the output directly instead of to the block's copy."""
    n = 520
    xyz = np.array([[12.0 * (i % 9), 12.0 * (i // 9 % 9), 12.0 * (i // 81)] for i in range(n)])
    xyz[1] = [1.5, 0.9, 0.4]
    basis = [[(0, [0.8], [1.0])] for _ in range(n)]
    for a in (0, 1):
        basis[a] = [(0, [0.9], [1.0]), (1, [1.1], [1.0]), (2, [0.7], [1.0])]

    def build(x):
        return L.Structure(basis, [1] * n, x, units="bohr")

    s = build(xyz)
    D = random_density(s.nao, 8, np.random.default_rng(43))
    D[:18, :18] += 0.5 * np.eye(18)
    g = L.jk_energy_backward(s, D, schwarz=0.0)
    assert "eriD1WarpKernel<2,2,1,0>" in launched(lambda: L.jk_energy_backward(s, D, schwarz=0.0))
    assert np.abs(g.sum(axis=0)).max() <= 1e-10
    # the two atoms with d functions, and a neighbour on the grid
    for atom, x in ((0, 0), (0, 1), (0, 2), (1, 0), (1, 1), (1, 2), (9, 1)):
        e = []
        for d in (1e-4, -1e-4):
            moved = xyz.copy()
            moved[atom, x] += d
            e.append(L.jk_energy_forward(build(moved), D, schwarz=0.0))
        assert abs((e[0] - e[1]) / 2e-4 - g[atom, x]) <= 1e-6


@pytest.mark.parametrize("waters,aux", [(1, "def2-universal-jkfit"), (2, "cc-pvdz-rifit")])
def test_rij_solves_the_metric_equations(waters, aux):
    """d of RI-J against the metric itself: the refinement's residual kernel at row lengths that are and
    are not multiples of its 128-element step.  Bound: a backward-stable solve's 1e-12 of |M| |d|."""
    Z, xyz, rng = water_cluster(waters, seed=44)
    s = L.Structure("cc-pvdz", Z, xyz, aux, units="bohr")
    D = random_density(s.nao, 5 * waters, rng)
    J, gamma, d = L.rij(s, D, schwarz=0.0)
    M = L.eri2(s)
    assert L.rij_last_solve(s)["method"] == "cholesky"
    assert np.abs(M @ d - gamma).max() <= 1e-12 * (np.abs(M) @ np.abs(d)).max()
    T = L.eri3(s)
    assert np.abs(np.einsum("mnP,P->mn", T, d) - J).max() <= 1e-10
    assert np.abs(np.einsum("mnP,mn->P", T, D) - gamma).max() <= 1e-10
