"""The RI metric beside its Cholesky factor: what a context keeps of it, and the solve that uses it.

naux^2 doubles hold the factor and, in its unused half, the metric.  The memory bound leaves half a matrix
(0.18 GB) beside them and the fitted tensor for library workspaces and kernels loaded on the way.
The solve's bound is that of a backward-stable solve, 1e-12 of |M| |d|, at row lengths on both sides of the
residual kernel's 32-row blocks and 128-column steps."""
import numpy as np
import pytest
import torch

from lible_b200 import ints as L

pytestmark = pytest.mark.gpu


def _oxygens(n, aux):
    """n distant atoms with one s function each and the oxygen fitting set."""
    xyz = [[12.0 * (i % 4), 12.0 * (i // 4 % 4), 12.0 * (i // 16)] for i in range(n)]
    return L.Structure([[(0, [0.8], [1.0])]] * n, [8] * n, xyz, L.basis_atoms(aux, [8] * n, L.AUX_BASIS_ROOT),
                       units="bohr")


def test_context_keeps_no_second_copy_of_the_metric():
    C = np.eye(48)[:, :2].copy()
    L.rik(_oxygens(2, "def2-universal-jkfit"), C=C[:2].copy())  # libraries and kernels loaded
    s = _oxygens(48, "def2-qzvp-rifit")
    M, tensor = 8 * s.naux ** 2, 8 * s.naux * s.nao ** 2
    assert M > 0.3e9
    before = torch.cuda.mem_get_info()[0]
    L.rik(s, C=C)
    L.rik(s, C=C)
    assert before - torch.cuda.mem_get_info()[0] <= tensor + 1.5 * M
    L.rij(s, np.eye(s.nao))
    assert L.rij_last_solve(s)["method"] == "cholesky"


@pytest.mark.parametrize("n,extra", [(1, 0), (2, 0), (2, 1), (3, 2)])
def test_solve_at_ragged_sizes(n, extra):
    aux = L.basis_atoms("def2-universal-jkfit", [8] * n, L.AUX_BASIS_ROOT)
    for k in range(extra):
        aux[k] = aux[k][:-1 - k]
    s = L.Structure([[(0, [0.8], [1.0]), (1, [1.1], [1.0])]] * n, [8] * n, [[2.0 * i, 0.3 * i, 0.0] for i in range(n)], aux,
                    units="bohr")
    D = np.random.default_rng(3).standard_normal((s.nao, s.nao))
    J, gamma, d = L.rij(s, D + D.T, schwarz=0.0)
    M = L.eri2(s)
    assert L.rij_last_solve(s)["method"] == "cholesky"
    assert np.abs(M @ d - gamma).max() <= 1e-12 * (np.abs(M) @ np.abs(d)).max()
