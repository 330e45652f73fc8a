"""Convergence before the restart's end, in the first, the second and later chunks of Arnoldi steps: the fused
Gram-Schmidt up to 31 columns (whose tail kernel raises the flag that the host reads), the warp's back substitution up to 32,
and the modified Gram-Schmidt beyond."""
import numpy as np
import pytest

from test_gpu_gmres import _inputs
from test_gpu_induction import OP_TOL, _np, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rtol", [0.3, 3e-2, 1e-3, 1e-6, 1e-10])
@pytest.mark.parametrize("restart", [30, 31, 32, 60])
def test_early_exit_solves_the_oracles_system(restart, rtol):
    """A (E - Eo) is the difference of the two residuals on the free rows: at most the sum of their stated norms, plus the
    operators' own rounding (OP_TOL of the largest entry, per row)."""
    h, di, oi, rng = _setup("box", True, True, rtol=rtol, max_it=200, restart=restart)
    dirichlet, Phi, Ee = _inputs(h, rng)
    free, dt = dirichlet == 0, 0.05
    b = Ee + oi.apply_F(Phi)
    Eo, ito, rro = oi.solve(Phi, Ee, dirichlet, dt, False)
    AEo = oi.apply_A(Eo, dt)
    for _ in range(2):  # the second solve reuses the captured chunks
        E, it, rr = di.solve(Phi, Ee, dirichlet, dt, False)
        assert rr <= rtol and rro <= rtol and abs(it - ito) <= 2
        AE = oi.apply_A(_np(E), dt)
        rounding = 2 * OP_TOL * np.sqrt(b.size) * max(np.abs(x).max() for x in (AE, AEo, b))
        assert np.linalg.norm((AE - AEo)[free]) <= (rr + rro) * np.linalg.norm(b) + rounding
        assert np.array_equal(_np(E)[~free], Ee[~free])
