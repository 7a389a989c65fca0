"""(gs|ps) and (gs|ds) of the RI calls: the warp form in short launches, the register form in long ones.

Both forms against each other over the same integrals, 1e-12 per integral (the bound of the other
integral tests), and which of them a kernel batch and an RI contraction take on the two sides of the rule:
four quartets per warp slot (16 an SM) for a work queue, eight for a list."""
import numpy as np
import pytest
import torch
from launches import launched

from lible_b200 import ints as L
from lible_b200.workloads import random_density, water_cluster

pytestmark = pytest.mark.gpu

FORMS = {True: "eriWarpKernel<4,0,%s,0>", False: "eriKernel<4,0,%s,0,double,0>"}


@pytest.mark.parametrize("lk", [1, 2])
def test_forms_agree_and_the_rule_chooses(lk):
    limit = 128 * torch.cuda.get_device_properties(0).multi_processor_count
    Z, xyz, _ = water_cluster(2, seed=61)
    s = L.Structure("cc-pvtz", Z, xyz, "def2-qzvp-rifit", units="bohr")
    sp = next(x for x in L.shellPairData(True, s) if x.getLPair() == (lk, 0))
    g = next(x for x in L.shellDataAux(s) if x.l_ == 4)
    pairs = np.stack(np.unravel_index(np.arange(sp.n_pairs_ * g.n_shells_), (sp.n_pairs_, g.n_shells_)), 1)
    idx = np.resize(pairs, (limit, 2)).astype(np.uint32)
    k = L.ERI3Kernel(sp, g)
    long, short = k.batch(idx), k.batch(idx[:-1])
    assert np.abs(long[:-1] - short).max() <= 1e-12
    assert FORMS[False] % lk in launched(lambda: k.batch(idx))
    assert FORMS[True] % lk in launched(lambda: k.batch(idx[:-1]))


@pytest.mark.parametrize("waters,short", [(2, True), (10, False)])
def test_form_of_an_ri_contraction(waters, short):
    Z, xyz, rng = water_cluster(waters, seed=62)
    s = L.Structure("cc-pvtz", Z, xyz, "def2-qzvp-rifit", units="bohr")
    D = random_density(s.nao, 5 * waters, rng)
    names = launched(lambda: L.ri_contract(s, D))
    for lk in (1, 2):
        assert FORMS[short] % lk in names and FORMS[not short] % lk not in names
