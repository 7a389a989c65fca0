"""The split form of the register path (one warp per heavily contracted quartet) against the C
restatement of the integrals.  Molecules this small send every quartet of at least 8 primitive pairs of a
class with a split form to it, in both orientations ((dd|ss) runs as (ss|dd)), next to the ordinary
launch of the rest.

Tolerances: 1e-11 for J/K sums (as the other J/K tests), 1e-12 per integral, and for mixed precision
1e-6 in the Frobenius norm."""
import numpy as np
import pytest

from lible_b200 import ints as L
from lible_b200.workloads import random_density, water_cluster
from oracle import port

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("basis,waters,precision", [("cc-pvdz", 1, "fp64"), ("cc-pvtz", 1, "fp64"), ("6-31+g", 2, "fp64"),
                                                    ("def2-svp", 2, "fp64"), ("cc-pvdz", 2, "mixed")])
def test_split_jk_matches_the_restatement(basis, waters, precision):
    Z, xyz, rng = water_cluster(waters, seed=31)
    s = L.Structure(basis, Z, xyz, units="bohr")
    D = random_density(s.nao, 5 * waters, rng)
    J, K, st = L.jk(s, D, schwarz=0.0, precision=precision, fp32_threshold=1e-2)
    Jr, Kr = port.jk(basis, Z, xyz, D)
    if precision == "fp64":
        assert np.abs(J - Jr).max() <= 1e-11 and np.abs(K - Kr).max() <= 1e-11
    else:
        assert st["n_fp32"] > 0
        assert np.linalg.norm(J - Jr) <= 1e-6 and np.linalg.norm(K - Kr) <= 1e-6


@pytest.mark.parametrize("basis", ["cc-pvdz", "def2-svp"])
def test_split_store_matches_the_restatement(basis):
    Z, xyz, _ = water_cluster(1, seed=32)
    s = L.Structure(basis, Z, xyz, units="bohr")
    assert np.abs(L.eri4(s) - port.PortMolecule(basis, Z, xyz).eri4()).max() <= 1e-12
