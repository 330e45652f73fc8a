"""The first-order scheme (second_order = 0: every face state is its cell's) on the device: the step against the oracle's
zero-gradient step, and the adjoint gradient against the tangent-linear run."""
import numpy as np
import pytest

from test_gpu_fp64_kernels import _workload

pytestmark = pytest.mark.gpu


def _state(wl):
    from mpcns_uns_b200 import gpu
    p = gpu.step_params(wl.n_species, wl.gamma, fs=wl.fs, mass=wl.mass, u_inf=wl.u_inf, B_imf=wl.B_imf, second_order=False)
    st = gpu.ResidentState(gpu.DeviceMesh(wl.mesh), p)
    st.set(wl.U, wl.Phi, wl.PhiAdd)
    return st


@pytest.mark.parametrize("kind,nsp", [("box_tet_111", 1), ("box_tet_421", 2), ("box_tet_433", 1), ("shell_tet", 2)])
def test_gradient_equals_tangent(kind, nsp):
    """Two steps of chains of a few hundred rounded operations, summed over at most 1e3 entries: 1e-11 of the sum of the
    absolute products, as in the second-order test."""
    from mpcns_uns_b200 import gpu
    wl = _workload(kind, nsp, "noise")
    h = wl.mesh
    st = _state(wl)
    rng = np.random.default_rng(1)
    fn = gpu.DeviceFunction(st, 10.0 ** rng.uniform(-3, -1, h.n_cells), np.ones(h.n_cells, np.int8), 2, 1, 1e-3)
    de, du = 1e-2 * rng.normal(size=h.n_cells), rng.normal(size=3)
    J = fn.forward()
    ge, gu = fn.backward()
    Jt, dJ = fn.tangent(de, du)
    assert Jt == J
    assert abs(ge @ de + gu @ du - dJ) < 1e-11 * (np.abs(ge * de).sum() + np.abs(gu * du).sum())
