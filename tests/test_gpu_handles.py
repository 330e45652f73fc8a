"""Handles may be destroyed in any order: a mesh or a state that others were made on stays usable for them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_owners_destroyed_first():
    from mpcns_uns_b200 import gpu, workloads
    wl = workloads.shell(3, 4)
    dm = gpu.DeviceMesh(wl.mesh)
    st = gpu.ResidentState(dm, gpu.step_params(2, wl.gamma, fs=wl.fs, mass=wl.mass, u_inf=wl.u_inf, B_imf=wl.B_imf))
    st.set(wl.U, wl.Phi, wl.PhiAdd)
    nc = wl.mesh.n_cells
    fn = gpu.DeviceFunction(st, np.full(nc, 1e-3), np.ones(nc, np.int8), 2, 1, 1e-3)
    ind = gpu.DeviceInduction(dm, np.ones(wl.mesh.n_edges))
    J = fn.forward()
    fn.reset()
    L = gpu.lib()
    for h, destroy in ((dm, L.mhd_gpu_mesh_destroy), (st, L.mhd_gpu_state_destroy)):
        gpu.check(destroy(h._h))
        h._h = None
    assert fn.forward() == J
    gpu.check(L.mhd_gpu_induction_destroy(ind._h))
    gpu.check(L.mhd_gpu_fn_destroy(fn._h))
    ind._h = fn._h = None
