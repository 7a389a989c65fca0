"""The J/K gradient with its launches on all stream branches (below 4.3e10 operations) and in order (above), against
central differences of the energy: step 1e-4 bohr, 1e-6 Eh/bohr as the other gradient tests."""
import numpy as np
import pytest

from lible_b200 import ints as L
from lible_b200.workloads import random_density, water_cluster

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("waters,small", [(4, True), (5, False)])
def test_gradient_on_both_sides_of_the_stream_rule(waters, small):
    Z, xyz, rng = water_cluster(waters, seed=77)

    def build(x):
        return L.Structure("cc-pvtz", Z, x, units="bohr")

    s = build(xyz)
    assert (L.jk_plan(s, 1e-12, "fp64")["flops_fp64"] < 4.3e10) == small
    D = random_density(s.nao, 5 * waters, rng)
    g = L.jk_energy_backward(s, D)
    for atom, x in ((0, 0), (4, 2)):
        e = []
        for d in (1e-4, -1e-4):
            moved = xyz.copy()
            moved[atom, x] += d
            e.append(L.jk_energy_forward(build(moved), D))
        assert abs((e[0] - e[1]) / 2e-4 - g[atom, x]) <= 1e-6
    assert np.abs(L.jk_energy_backward(s, D) - g).max() <= 1e-10
