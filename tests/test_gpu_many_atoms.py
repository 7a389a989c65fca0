"""The J/K gradient of many atoms: up to 2,048 the register form sums a block's gradient in shared memory.

Distant s functions with a diagonal density are point charges D_aa: dE/dR_a = -D_aa sum_b D_bb R_ab / R_ab^3
(erf(sqrt(0.8) 12) = 1 in double precision).  Bound: 1e-12 relative, for sums of 2,000 terms of one size."""
import numpy as np
import pytest
from launches import launched

from lible_b200 import ints as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,form", [(1877, "eriD1RegKernel"), (1878, "eriD1RegKernel"), (2048, "eriD1RegKernel"),
                                    (2049, "eriD1Kernel")])
def test_gradient_of_distant_atoms(n, form):
    xyz = 12.0 * np.stack(np.unravel_index(np.arange(n), (13, 13, 13)), 1).astype(float)
    s = L.Structure([[(0, [0.8], [1.0])]] * n, [1] * n, xyz, units="bohr")
    q = np.random.default_rng(4).uniform(0.5, 1.5, n)
    D = np.diag(q)
    g = L.jk_energy_backward(s, D, schwarz=1e-10)
    r = xyz[:, None, :] - xyz[None, :, :]
    d = np.linalg.norm(r, axis=2)
    np.fill_diagonal(d, np.inf)
    want = -q[:, None] * np.einsum("abx,ab->ax", r, q[None, :] / d ** 3)
    assert np.abs(g - want).max() <= 1e-12 * np.abs(want).max()
    names = launched(lambda: L.jk_energy_backward(s, D, schwarz=1e-10))
    assert [k for k in names if k.startswith("eriD1")] == [f"{form}<0,0,0,0>"]
