"""The split form of the register path (one warp per heavily contracted quartet) against the C
restatement of the integrals, next to the ordinary launch of the rest, and the kernels that were launched.
Split are the quartets of at least 28 primitive pairs and the launch's even share, in launches that give
every quartet a warp of its own those of at least 4; f shells have it in both orientations (FP64 (ff|ss) runs
as (ss|ff), (fd|ps) as (ps|fd)).

Tolerances: 1e-11 for J/K sums (as the other J/K tests), 1e-12 per integral, and for mixed precision
1e-6 in the Frobenius norm."""
import numpy as np
import pytest
from launches import launched

from lible_b200 import ints as L
from lible_b200.workloads import random_density, water_cluster
from oracle import port

pytestmark = pytest.mark.gpu


def _split(*classes, arithmetic="double"):
    return {f"eriSplitKernel<{c},{arithmetic}>" for c in classes}


SPD = ("0,0,0,0", "1,0,1,0", "1,1,1,1", "2,0,0,0", "2,1,1,0", "2,2,0,0")
F64 = ("3,0,0,0", "3,1,1,0", "0,0,3,3", "1,0,3,2")
F32 = ("3,0,1,0", "3,1,2,0", "3,2,0,0", "3,3,0,0")


@pytest.mark.parametrize("basis,waters,precision,split", [
    ("cc-pvdz", 1, "fp64", _split(*SPD)), ("cc-pvtz", 1, "fp64", _split(*SPD, *F64)),
    ("6-31+g", 2, "fp64", _split(*SPD[:3])), ("def2-svp", 2, "fp64", _split(*SPD)),
    ("cc-pvdz", 2, "mixed", _split(*SPD) | _split(*SPD, arithmetic="float")),
    ("cc-pvtz", 1, "mixed", _split(*SPD, *F64) | _split(*F32, arithmetic="float"))])
def test_split_jk_matches_the_restatement(basis, waters, precision, split):
    Z, xyz, rng = water_cluster(waters, seed=31)
    s = L.Structure(basis, Z, xyz, units="bohr")
    D = random_density(s.nao, 5 * waters, rng)

    def build():
        return L.jk(s, D, schwarz=0.0, precision=precision, fp32_threshold=1e-2)

    J, K, st = build()
    Jr, Kr = port.jk(basis, Z, xyz, D)
    if precision == "fp64":
        assert np.abs(J - Jr).max() <= 1e-11 and np.abs(K - Kr).max() <= 1e-11
    else:
        assert st["n_fp32"] > 0
        assert np.linalg.norm(J - Jr) <= 1e-6 and np.linalg.norm(K - Kr) <= 1e-6
    assert split <= launched(build).keys()


@pytest.mark.parametrize("basis", ["cc-pvdz", "def2-svp"])
def test_split_store_matches_the_restatement(basis):
    Z, xyz, _ = water_cluster(1, seed=32)
    s = L.Structure(basis, Z, xyz, units="bohr")
    assert np.abs(L.eri4(s) - port.PortMolecule(basis, Z, xyz).eri4()).max() <= 1e-12
    assert _split("0,0,0,0", "1,0,1,0", "2,0,0,0", "2,2,0,0") <= launched(lambda: L.eri4(s)).keys()
