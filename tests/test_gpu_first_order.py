"""The first-order scheme (second_order = 0: every face state is its cell's) on the device: the step against the oracle's
zero-gradient step, and the adjoint gradient against the tangent-linear run."""
import numpy as np
import pytest

from oracle import port
from test_gpu_fp64_kernels import _workload

pytestmark = pytest.mark.gpu


def _state(wl):
    from mpcns_uns_b200 import gpu
    p = gpu.step_params(wl.n_species, wl.gamma, fs=wl.fs, mass=wl.mass, u_inf=wl.u_inf, B_imf=wl.B_imf, second_order=False)
    st = gpu.ResidentState(gpu.DeviceMesh(wl.mesh), p)
    st.set(wl.U, wl.Phi, wl.PhiAdd)
    return st


class _Oracle(port.PortMesh):
    @staticmethod
    def step_params(*args, **kw):
        p = port.PortMesh.step_params(*args, **kw)
        p.second_order = 0
        return p


@pytest.mark.parametrize("nsp", [1, 2, 3])
@pytest.mark.parametrize("kind", ["box_tet_111", "box_tet_433", "box_hex_443", "shell_tet", "shell_hex"])
def test_step_equals_oracle(kind, nsp):
    """The face pass of the first-order stage in the reference's operation order: equal bits."""
    wl = _workload(kind, nsp, "noise")
    st, pm = _state(wl), _Oracle(wl.mesh)
    U, Phi = [np.array(u) for u in wl.U], np.array(wl.Phi)
    Badd = pm.cell_vector(wl.PhiAdd)
    for _ in range(2):
        st.step(2e-3)
        pm.rk2_step(wl, U, Phi, Badd, 2e-3)
    for s in range(nsp):
        assert np.array_equal(st.U(s), U[s])
    assert np.array_equal(st.Phi(), Phi)
    # per stage: prepare, face candidates, edge EMF, CT, and for every pair of species the face values, the flux and
    # the update; and the kernel that sets the step size
    assert st.launches() == 2 * (1 + 2 * (4 + 3 * ((nsp + 1) // 2)))


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
