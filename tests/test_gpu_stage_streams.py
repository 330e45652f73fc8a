"""A stage's fluid and EMF passes on two streams give the bits of the single stream that the profiler keeps them on."""
import numpy as np
import pytest

from helpers import SHELL_BC, SOURCE_EXTRA, source_fields
from mpcns_uns_b200.mesh import HostMesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsp,sources", [(1, False), (2, False), (2, True), (5, False)])
@pytest.mark.parametrize("cells,precision", [("tet", "fp64"), ("tet", "mixed"), ("hex", "fp64")])
@pytest.mark.parametrize("n", [3, 14])
def test_two_streams_equal_one(n, cells, precision, nsp, sources):
    from mpcns_uns_b200 import gpu, workloads
    h = HostMesh.shell(n, 2 * n, 1.0, 2.0, 1.1, tets=cells == "tet").compute_geometry().boundary(*SHELL_BC)
    rng = np.random.default_rng(n + nsp)
    W = np.empty((nsp, h.n_cells, 5))
    W[..., 0], W[..., 4] = rng.uniform(0.9, 1.1, (nsp, h.n_cells)), rng.uniform(0.09, 0.11, (nsp, h.n_cells))
    W[..., 1:4] = rng.uniform(-0.1, 0.1, (nsp, h.n_cells, 3))
    U = [workloads.to_cons(w, workloads.GAMMA).ravel() for w in W]
    Phi = workloads.d1(h, workloads.fourier_potential(h, 3, amp=0.05))
    PhiAdd = np.asarray(h["face_area"]) @ np.array([0.1, -0.2, 0.3])
    p = gpu.step_params(nsp, workloads.GAMMA, fs=[(1.0, 0.0, 0.0, 0.0, 0.1)] * nsp, mass=[1.0, 23.0, 16.0, 4.0, 32.0][:nsp],
                        u_inf=(0.0, 0.0, 0.0), B_imf=(0.0, 0.0, -0.5), precision=precision, lorentz=sources,
                        induce_coeff=0.7 if sources else 0.0, extra=SOURCE_EXTRA if sources else None)
    dm, runs = gpu.DeviceMesh(h), []
    for one in (True, False):
        st = gpu.ResidentState(dm, p)
        st.set(U, Phi, PhiAdd)
        if sources:
            st.set_source_fields(*source_fields(h.n_cells))
        st.profile(one)
        dts = [st.step() for _ in range(3)]
        st.step(dts[-1], sync=False)
        runs.append((dts, [st.U(s) for s in range(nsp)], st.Phi()))
    assert runs[0][0] == runs[1][0]
    assert np.array_equal(runs[0][2], runs[1][2])
    for a, b in zip(runs[0][1], runs[1][1]):
        assert np.array_equal(a, b)
