"""The FP64 step's table-driven kernels against the oracle's C restatement, at the sizes where they can go wrong.

Cell counts below, at and just past one warp's and one block's cells, the tetrahedral (4 faces), hexahedral (6 faces)
and mixed-polyhedra forms, every face kind, one to three species (a species pair and a lone one), and states whose
limiter meets its special cases: constant neighbourhoods (zero numerators), ties between the two bounds, and face
values that are not positive.  The kernels keep the reference's operation order, so the states are equal bit for bit;
with the sources the device's sin and cos of the gyration allow 1e-12.
"""
import numpy as np
import pytest

from helpers import MIXED_BOX_BC, SHELL_BC, SOURCE_EXTRA, rel_err, source_fields
from oracle import port

pytestmark = pytest.mark.gpu


def _mesh(kind):
    from mpcns_uns_b200.mesh import HostMesh
    if kind.startswith("box"):
        nx, ny, nz = (int(v) for v in kind.split("_")[2])
        h = HostMesh.box(nx, ny, nz, tets="tet" in kind, jitter=0.1, seed=3)
        return h.compute_geometry().boundary(*MIXED_BOX_BC), MIXED_BOX_BC[2]
    h = HostMesh.shell(3, 4, 1.0, 3.0, 1.1, n_solid=1, tets="tet" in kind)
    return h.compute_geometry().boundary(*SHELL_BC), SHELL_BC[2]


def _workload(kind, nsp, state, seed=5):
    from mpcns_uns_b200 import workloads
    h, u_inf = _mesh(kind)
    rng = np.random.default_rng(seed)
    U, fs = [], []
    for s in range(nsp):
        W = np.zeros((h.n_cells, 5))
        W[:, 0], W[:, 1:4], W[:, 4] = 1.0, u_inf, 0.1
        if state == "noise":
            W[:, 0] = rng.uniform(0.5, 1.5, h.n_cells)
            W[:, 1:4] = rng.uniform(-1.0, 1.0, (h.n_cells, 3))
            W[:, 4] = rng.uniform(0.05, 0.15, h.n_cells)
        elif state == "steps":      # two values only: ties of the bounds, constant neighbourhoods
            W[:, 0] = np.where(rng.uniform(size=h.n_cells) < 0.3, 2.0, 1.0)
            W[:, 4] = np.where(rng.uniform(size=h.n_cells) < 0.3, 0.2, 0.1)
        elif state == "vacuum":     # six decades: extrapolated densities and pressures fall below zero
            W[:, 0] = 10.0 ** rng.uniform(-6, 0, h.n_cells)
            W[:, 4] = 10.0 ** rng.uniform(-6, 0, h.n_cells)
        U.append(workloads.to_cons(W, workloads.GAMMA).ravel())
        fs.append((1.0, *u_inf, 0.1))
    Phi = workloads.d1(h, workloads.fourier_potential(h, seed, amp=0.1))
    return workloads.Workload(name=kind, mesh=h, n_species=nsp, gamma=workloads.GAMMA, U=U, Phi=Phi,
                              PhiAdd=np.asarray(h["face_area"]) @ np.array([0.1, -0.2, 0.3]), fs=fs, mass=[1.0, 23.0, 16.0][:nsp],
                              u_inf=tuple(u_inf), B_imf=(0.0, 0.0, -0.5))


def _both(wl, steps=2, dt=2e-3, sources=False):
    from mpcns_uns_b200 import gpu
    kw = dict(lorentz=True, induce_coeff=0.7) if sources else {}
    p = gpu.step_params(wl.n_species, wl.gamma, fs=wl.fs, mass=wl.mass, u_inf=wl.u_inf, B_imf=wl.B_imf,
                        extra=SOURCE_EXTRA if sources else None, **kw)
    st = gpu.ResidentState(gpu.DeviceMesh(wl.mesh), p)
    st.set(wl.U, wl.Phi, wl.PhiAdd)
    extra = None
    if sources:
        photo, vst = source_fields(wl.mesh.n_cells)
        st.set_source_fields(photo, vst)
        extra = dict(SOURCE_EXTRA, photo=photo, vst=vst)
    pm = port.PortMesh(wl.mesh)
    U, Phi = [np.array(u) for u in wl.U], np.array(wl.Phi)
    Badd = pm.cell_vector(wl.PhiAdd)
    assert np.array_equal(st.download(gpu.FIELD_BADD), Badd)
    for _ in range(steps):
        st.step(dt)
        pm.rk2_step(wl, U, Phi, Badd, dt, extra=extra, **kw)
    return [st.U(s) for s in range(wl.n_species)], st.Phi(), U, Phi


@pytest.mark.parametrize("state", ["noise", "steps", "vacuum"])
@pytest.mark.parametrize("nsp", [1, 2, 3])
@pytest.mark.parametrize("kind", ["box_tet_111", "box_tet_421", "box_tet_433", "box_hex_331", "box_hex_443", "shell_tet", "shell_hex"])
def test_step_equals_oracle(kind, nsp, state):
    U, Phi, Ur, Pr = _both(_workload(kind, nsp, state))
    for a, b in zip(U, Ur):
        assert np.array_equal(a, b)
    assert np.array_equal(Phi, Pr)


@pytest.mark.parametrize("kind", ["box_tet_433", "box_hex_443", "shell_tet", "shell_hex"])
def test_full_model_step_equals_oracle(kind):
    U, Phi, Ur, Pr = _both(_workload(kind, 2, "noise"), sources=True)
    for a, b in zip(U, Ur):
        assert rel_err(a, b) < 1e-12
    assert rel_err(Phi, Pr) < 1e-12


@pytest.mark.parametrize("rel_limit", [0.0, 0.3])
@pytest.mark.parametrize("kind,nsp", [("box_tet_111", 1), ("box_tet_421", 2), ("box_tet_433", 1), ("shell_tet", 2)])
def test_gradient_equals_tangent(kind, nsp, rel_limit):
    """The adjoint gradient along a direction equals the tangent-linear run's derivative, every face kind and limiter
    branch among the cells.  Two steps of chains of a few hundred rounded operations, summed over at most 1e3 entries:
    1e-11 of the sum of the absolute products."""
    from mpcns_uns_b200 import gpu
    wl = _workload(kind, nsp, "noise")
    h = wl.mesh
    p = gpu.step_params(nsp, wl.gamma, fs=wl.fs, mass=wl.mass, u_inf=wl.u_inf, B_imf=wl.B_imf, rel_limit=rel_limit)
    st = gpu.ResidentState(gpu.DeviceMesh(h), p)
    st.set(wl.U, wl.Phi, wl.PhiAdd)
    rng = np.random.default_rng(1)
    fn = gpu.DeviceFunction(st, 10.0 ** rng.uniform(-3, -1, h.n_cells), np.ones(h.n_cells, np.int8), 2, 1, 1e-3)
    de, du = 1e-2 * rng.normal(size=h.n_cells), rng.normal(size=3)
    J = fn.forward()
    ge, gu = fn.backward()
    Jt, dJ = fn.tangent(de, du)
    assert Jt == J
    assert abs(ge @ de + gu @ du - dJ) < 1e-11 * (np.abs(ge * de).sum() + np.abs(gu * du).sum())
