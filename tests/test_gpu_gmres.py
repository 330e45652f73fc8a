"""The restart cycle's chunks of Arnoldi steps: restart lengths around a chunk, the iteration cap inside and at the end of
one, and convergence before the restart's end, against the oracle's solve."""
import numpy as np
import pytest

from test_gpu_induction import _np, _setup, port, rel_err  # noqa: F401

pytestmark = pytest.mark.gpu


def _inputs(h, rng):
    return (np.asarray(h["edge_mode"]) == 2).astype(np.int8), rng.uniform(-1, 1, h.n_faces), rng.uniform(-1, 1, h.n_edges)


@pytest.mark.parametrize("max_it", [5, 13])
@pytest.mark.parametrize("restart", [1, 4, 5, 6, 10, 11, 16])
def test_capped_solve_takes_the_oracles_steps(restart, max_it):
    """Thirteen FP64 steps of dots over 1e3 edges, far above the rounding floor: the iterates agree to 1e-9, the
    residuals to 1e-6."""
    h, di, oi, rng = _setup("box", True, True, rtol=1e-15, max_it=max_it, restart=restart)
    args = _inputs(h, rng)
    for _ in range(2):  # the second solve reuses the captured chunks
        E, it, rr = di.solve(args[1], args[2], args[0], 0.05, False)
        Eo, ito, rro = oi.solve(args[1], args[2], args[0], 0.05, False)
        assert it == ito == max_it
        assert rr == pytest.approx(rro, rel=1e-6)
        assert rel_err(_np(E), Eo) <= 1e-9


@pytest.mark.parametrize("rtol", [1e-1, 1e-3, 1e-6, 1e-10])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_early_exit_meets_the_tolerance(precision, rtol):
    h, di, oi, rng = _setup("box", True, True, rtol=rtol, max_it=200, restart=60, precision=precision)
    args = _inputs(h, rng)
    E, it, rr = di.solve(args[1], args[2], args[0], 0.05, False)
    Eo, ito, rro = oi.solve(args[1], args[2], args[0], 0.05, False)
    assert rr <= rtol and rro <= rtol
    if precision == "fp64":
        assert abs(it - ito) <= 2
    assert np.array_equal(_np(E)[args[0] != 0], args[2][args[0] != 0])
