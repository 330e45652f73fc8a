"""Performance cases: what users of this library run on one GPU, through its public entry points.

A case is a dict of plain values; ``prepare`` makes the inputs (seeded, on the GPU) and the handles that a program
keeps (the device mesh, the resident state, the induction handle), ``run`` is one pass over them, ``work`` its
compulsory bytes and operations, and ``exact`` the same results from a plain torch restatement in 64 bits.

Kinds:
  step      explicit SSP-RK2 steps of a resident state with the CFL step on the device (ResidentState.step)
  semi      the semi-implicit step: forward Euler fluid, EMF from the induction solve (step_semi_implicit)
  solve     one cold GMRES solve of the Hall + resistive induction (DeviceInduction.solve)
  adjoint   forward run and adjoint sweep of the differentiated explicit run (DeviceFunction)
  calls     one explicit stage through the single functions that a host code calls in place of its CPU bodies
Meshes: ``box`` (jittered unit cube), ``shell`` (cubed sphere); ``cells`` "tet" (6 per hexahedron) or "hex".
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mpcns_uns_b200 import gpu, workloads
from mpcns_uns_b200.mesh import HostMesh

GAMMA = 5.0 / 3.0
# a sheath flow (subsonic past the dipole): the model stays stable in it over thousands of passes on one state
U_INF, B_IMF, P_REL, NOISE = (-1.0, 0.0, 0.0), (0.0, 0.0, -0.5), 3.0, 0.01
RHO_FLOOR, P_FLOOR, NE_FLOOR = 1e-10, 1e-12, 0.01
R_OUT = 6.0
# switches and constants of the full two-ion model (J x B and gyration with the ambipolar and chemistry terms)
FULL = dict(ambipolar=True, chemistry=True, pressure_coef=0.3, a1_Na=0.5, a4=0.2, a5=1e-6, a6=1e-7, state_coeff_H=1.0,
            state_coeff_Na=1.0 / 23.0, T_ref=1e4, Tn0=600.0)
TEN_RHO = [1.0, 0.3, 0.1, 3e-2, 1e-2, 5e-3, 2e-3, 1e-3, 4e-4, 2e-4]


def listed():
    step = dict(kind="step", mesh="shell", cells="tet", ions=2, sources="lorentz", steps=1)
    return [
        # the smallest run users make (24,576 tetrahedra, one ion): a time loop that reads each step's dt, so launches,
        # their gaps and the read-back count
        dict(step, name="fp64 step box 24k", mesh="box", n=16, ions=1, sources="none", precision="fp64"),
        # the same box in mixed precision as a burst of 20 steps queued without reading dt in between
        dict(step, name="mixed 20 steps box 24k", mesh="box", n=16, ions=1, sources="none", precision="mixed", steps=20),
        # a development-size two-ion shell with the J x B force and gyration
        dict(step, name="mixed step shell 221k", n=16, nr=24, precision="mixed"),
        # the production two-ion shell (the benchmark's mesh)
        dict(step, name="mixed step shell 14.2M", n=64, nr=96, precision="mixed"),
        # the reference-exact FP64 step that the mixed one is validated with
        dict(step, name="fp64 step shell 1.8M", n=32, nr=48, precision="fp64"),
        # the hexahedral shells that the reference's own generator makes, with every model term on; odd sizes
        dict(step, name="fp64 step hex 307k full model", cells="hex", n=33, nr=47, precision="fp64", sources="full"),
        # the ten-ion hot path: the fluid passes dominate
        dict(step, name="mixed step ten ions 1.3M", n=24, nr=64, ions=10, precision="mixed", sources="none"),
        # one explicit stage through the functions a host code calls one by one (the drop-in's use), odd size
        dict(kind="calls", name="calls box 73k", mesh="box", cells="tet", n=23),
        # a converged FP64 induction solve
        dict(kind="solve", name="fp64 solve 263k edges", mesh="shell", cells="tet", n=16, nr=24, precision="fp64", max_it=600),
        # a large mixed-precision solve under an iteration cap (the basis is far larger than L2)
        dict(kind="solve", name="mixed solve 2.8M edges", mesh="shell", cells="tet", n=32, nr=64, precision="mixed", max_it=60),
        # the reference's default run mode
        dict(kind="semi", name="semi-implicit step 746k", mesh="shell", cells="tet", n=24, nr=36, ions=2, sources="lorentz"),
        # gradient of a functional of the run: forward with checkpoints, then the adjoint sweep
        dict(kind="adjoint", name="adjoint 8 steps 295k", mesh="shell", cells="tet", n=16, nr=32, ions=2, sources="none", steps=8,
             every=4),
    ]


def draw(rng):
    """One more case of the same ranges: sizes log-uniform from a few thousand cells, odd ones among them."""
    def shell(lo, hi, tet=True):
        cells = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        n = max(5, round((cells / (6 * (6 if tet else 1)) / rng.uniform(1.2, 2.2)) ** (1 / 3)))
        return dict(mesh="shell", n=n, nr=max(6, round(cells / ((36 if tet else 6) * n * n))))

    kind = rng.choice(["mixed", "mixed", "mixed", "fp64", "fp64", "hex", "ten", "calls", "solve", "solve", "semi", "adjoint"])
    if kind in ("mixed", "fp64"):
        c = dict(kind="step", cells="tet", precision=kind, steps=rng.choice([1, 1, 1, 2, 5]))
        if rng.random() < 0.25:
            return dict(c, mesh="box", n=rng.randint(9, 41), ions=1, sources="none")
        return dict(c, ions=2, sources=rng.choice(["none", "lorentz", "lorentz", "full"]), **shell(2e4, 4e6))
    if kind == "hex":
        return dict(kind="step", cells="hex", precision="fp64", ions=2, steps=1, sources=rng.choice(["none", "lorentz", "full"]),
                    **shell(1e4, 6e5, tet=False))
    if kind == "ten":
        return dict(kind="step", cells="tet", precision=rng.choice(["mixed", "mixed", "fp64"]), ions=rng.choice([3, 5, 10]), steps=1,
                    sources="none", **shell(3e4, 1.2e6))
    if kind == "calls":
        return dict(kind="calls", mesh="box", cells=rng.choice(["tet", "hex"]), n=rng.randint(9, 35))
    if kind == "solve":
        p = rng.choice(["fp64", "mixed"])
        return dict(kind="solve", cells="tet", precision=p, max_it=60, **shell(3e4, 1.5e6))
    if kind == "semi":
        return dict(kind="semi", cells="tet", ions=2, sources="lorentz", **shell(3e4, 9e5))
    return dict(kind="adjoint", cells="tet", ions=2, sources="none", steps=rng.choice([3, 4, 6]), every=rng.choice([2, 3]),
                **shell(3e4, 3e5))


# ------------------------------------------------------------------ meshes (kept by a program for its whole run)
_MESH = {}


def _mesh(case):
    """(host mesh, device mesh, tensors) of a case: the last one is kept, as a program keeps its mesh across states."""
    r_in, r_out = (0.8, R_OUT) if case["kind"] == "solve" else (1.0, 8.0 if case.get("ions", 1) > 2 else R_OUT)
    key = (case["mesh"], case["cells"], case["n"], case.get("nr", 0), r_in, r_out)
    if key not in _MESH:
        _MESH.clear()
        if case["mesh"] == "box":
            h = HostMesh.box(case["n"], case["n"], case["n"], tets=case["cells"] == "tet", jitter=0.15, seed=0)
            h = h.compute_geometry().boundary("outflow")
        elif case["cells"] == "tet":
            h, _ = workloads.shell_mesh(case["n"], case["nr"], r_in, r_out, None, U_INF, device_geometry=True)
        else:
            h = HostMesh.shell(case["n"], case["nr"], r_in, r_out, workloads.shell_stretch(case["n"], case["nr"], r_in, r_out))
            h = h.compute_geometry().boundary("outflow", {"inner": "wall", "outer": "farfield"}, U_INF)
        t = {k: torch.as_tensor(np.array(h[k]), device="cuda") for k in (
            "cell_center", "edge_mid", "edge_vec", "face_area", "star1", "f2e_ptr", "f2e_idx", "f2e_sgn")}
        _MESH[key] = (h, gpu.DeviceMesh(h), t)
    return _MESH[key]


def _rows(ptr):
    n = ptr[1:] - ptr[:-1]
    return torch.repeat_interleave(torch.arange(n.numel(), device=ptr.device), n)


def _d1(t, A):
    """(d1 A)_f: circulation of an edge potential around every face."""
    rows = _rows(t["f2e_ptr"])
    out = torch.zeros(t["f2e_ptr"].numel() - 1, dtype=torch.float64, device="cuda")
    return out.index_add_(0, rows, t["f2e_sgn"].double() * A[t["f2e_idx"].long()])


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uni(g, *shape):
    return 2.0 * torch.rand(*shape, generator=g, dtype=torch.float64, device="cuda") - 1.0


def _fourier_flux(t, g, amp, modes=8):
    """Divergence-free induced flux: d1 of a few Fourier modes of an edge potential."""
    x, a = t["edge_mid"], 0.0
    for _ in range(modes):
        k = torch.randint(1, 3, (3,), generator=g, device="cuda").double() * torch.sign(_uni(g, 3))
        d = _uni(g, 3)
        a = a + torch.cos(2 * math.pi * (x @ k) + math.pi * _uni(g, 1))[:, None] * (amp * d / d.norm())
    return _d1(t, (a * t["edge_vec"]).sum(1))


def _cons(W):
    ke = 0.5 * W[..., 0] * (W[..., 1:4] ** 2).sum(-1)
    return torch.cat([W[..., :1], W[..., :1] * W[..., 1:4], (W[..., 4] / (GAMMA - 1.0) + ke)[..., None]], -1)


def _inputs(case, seed):
    """Seeded state of a case: U (ions, cells, 5), induced and background face flux, free stream, masses, m_edge, ..."""
    h, _, t = _mesh(case)
    g = _gen(seed)
    nc, ions = h.n_cells, case.get("ions", 1)
    s = {"mass": [1.0], "u_inf": U_INF, "B_imf": B_IMF}
    W = torch.empty(ions, nc, 5, dtype=torch.float64, device="cuda")
    noise = lambda: 1.0 + NOISE * _uni(g, nc)
    if case["mesh"] == "box":
        s.update(u_inf=(1.0, 0.0, 0.0), B_imf=(0.0, 0.0, 0.0), fs=[(1.0, 1.0, 0.0, 0.0, 0.1)])
        W[0] = torch.stack([noise(), noise(), 0.01 * _uni(g, nc), 0.01 * _uni(g, nc), 0.1 * noise()], 1)
        B0 = torch.tensor([0.1, 0.2, 0.0], dtype=torch.float64, device="cuda")
        A0 = 0.5 * (torch.linalg.cross(B0.expand_as(t["edge_mid"]), t["edge_mid"]) * t["edge_vec"]).sum(1)
        s["Phi"] = _fourier_flux(t, g, 0.05) + _d1(t, A0)
        s["PhiAdd"] = torch.zeros_like(s["Phi"])
    else:
        rho0 = TEN_RHO[:ions] if ions > 2 else [1.0, 1e-3]
        s["mass"] = workloads.TEN_ION_MASSES[:ions] if ions > 2 else [1.0, 23.0]
        prof = torch.exp(-(t["cell_center"].norm(dim=1) - 1.0) / 0.2)
        s["fs"] = []
        for k in range(ions):
            ex = torch.exp(0.5 * torch.randn(nc, generator=g, dtype=torch.float64, device="cuda")) * prof if k else 0.0
            far = 1.0 if k == 0 or ions > 2 else 1e-3          # two ions: the second is an exosphere above a thin stream
            W[k, :, 0] = rho0[k] * (far + ex) * noise()
            W[k, :, 1:4] = torch.tensor(U_INF, dtype=torch.float64, device="cuda") + NOISE * abs(U_INF[0]) * _uni(g, nc, 3)
            W[k, :, 4] = P_REL * W[k, :, 0] * noise()
            s["fs"].append((rho0[k] * far, *U_INF, P_REL * rho0[k] * far))
        s["Phi"] = _fourier_flux(t, g, 0.02)
        r = t["edge_mid"] - torch.tensor([0.0, 0.0, 0.2], dtype=torch.float64, device="cuda")
        d2 = (r * r).sum(1) + 1e-6
        m = torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64, device="cuda").expand_as(r)
        dip = torch.linalg.cross(m, r) / (d2 * d2.sqrt())[:, None]
        s["PhiAdd"] = t["face_area"] @ torch.tensor(B_IMF, dtype=torch.float64, device="cuda") + _d1(t, (dip * t["edge_vec"]).sum(1))
        if case.get("sources") == "full":
            sun = 0.5 * (1.0 + t["cell_center"][:, 0] / t["cell_center"].norm(dim=1))
            s["photo"], s["vst"] = 1e-3 * prof * sun * noise(), 2e-2 * prof * noise()
    s["U"] = _cons(W)
    r_e = t["edge_mid"].norm(dim=1)
    if case["kind"] == "solve":
        # the semi-implicit solve of a resistive core with a whistler-stiff exterior
        s["m_edge"] = torch.where(r_e < 1.0, 1.0, 1e-3) / t["star1"]
        s["B0"] = _dipole(t["cell_center"])
        s["ne"] = 1.0 + 0.25 * (1.0 + _uni(g, nc))
        s["Phi"] = _fourier_flux(t, g, 0.05)
        u = torch.tensor(U_INF, dtype=torch.float64, device="cuda").expand_as(t["edge_mid"])
        s["E"] = -(torch.linalg.cross(u, _dipole(t["edge_mid"])) * t["edge_vec"]).sum(1)
        s["dir"] = torch.as_tensor(np.array(h["edge_mode"]) == 2, device="cuda").to(torch.int8)
        s["dt"] = 20.0 * workloads.whistler_dt(h, s["B0"].cpu().numpy(), s["ne"].cpu().numpy(), 1.0, 1.0)
    if case["kind"] == "semi":
        s["m_edge"] = torch.where(r_e < 1.2, 1e-2, 1e-4) / t["star1"]
    if case["kind"] == "adjoint":
        s["eta"] = 10.0 ** (-3.0 + _uni(g, nc))
        x, r = t["cell_center"], t["cell_center"].norm(dim=1)
        s["mask"] = ((r >= 1.2) & (r <= 1.6) & (x[:, 0] > 0)).to(torch.int8)
    return s


def _dipole(x):
    r = x - torch.tensor([0.0, 0.0, 0.2], dtype=torch.float64, device="cuda")
    d = r.norm(dim=1, keepdim=True)
    rh, m = r / d, torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64, device="cuda")
    return (3.0 * (rh @ m)[:, None] * rh - m) / d ** 3 + torch.tensor(B_IMF, dtype=torch.float64, device="cuda")


class _View:
    """A resident field as a tensor: the state's own device buffer."""

    def __init__(self, state, field, shape):
        self.state = state
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f8", data=(state.device_ptr(field), False), version=3)


def _params(case, s):
    src = case.get("sources", "none")
    return gpu.step_params(len(s["mass"]), GAMMA, fs=s["fs"], mass=s["mass"], u_inf=s["u_inf"], B_imf=s["B_imf"], cfl=0.4,
                           precision=case.get("precision", "fp64"), lorentz=src != "none", induce_coeff=1.0 if src != "none" else 0.0,
                           extra=FULL if src == "full" else None)


def prepare(case, seed):
    h, dm, t = _mesh(case)
    s = _inputs(case, seed)
    if case["kind"] == "solve":
        ind = gpu.DeviceInduction(dm, s["m_edge"].cpu().numpy(), hall=True, hall_coef=1.0, hall_r_min=1.0, hall_r_max=1.012, rtol=1e-8,
                                  max_it=case["max_it"], restart=30, precision=case["precision"])
        ind.set_frozen_state(s["B0"].reshape(-1), s["ne"])
        return {"case": case, "ind": ind, **{k: s[k] for k in ("Phi", "E", "dir", "dt")}}
    if case["kind"] == "calls":
        W = dm.to_prim(s["U"][0].reshape(-1), GAMMA)
        return {"case": case, "dm": dm, "U": s["U"][0].reshape(-1).clone(), "Phi": s["Phi"], "fs": s["fs"][0], "u_inf": s["u_inf"],
                "B_imf": s["B_imf"], "dt": 1e-3 / case["n"], "W": W}
    st = gpu.ResidentState(dm, _params(case, s))
    st.set([u.reshape(-1).cpu().numpy() for u in s["U"]], s["Phi"].cpu().numpy(), s["PhiAdd"].cpu().numpy())
    if "photo" in s:
        st.set_source_fields(s["photo"].cpu().numpy(), s["vst"].cpu().numpy())
    out = {"case": case, "st": st, "U": torch.as_tensor(_View(st, gpu.FIELD_U, (len(s["mass"]), 5, h.n_cells)), device="cuda"),
           "Phi": torch.as_tensor(_View(st, gpu.FIELD_PHI, (h.n_faces,)), device="cuda")}
    if case["kind"] == "semi":
        # the Hall coefficient puts the initial CFL step at twice the explicit whistler limit
        out["ind"] = gpu.DeviceInduction(dm, s["m_edge"].cpu().numpy(), hall=True, hall_coef=_semi_hall(case, s, st.cfl_dt()),
                                         hall_r_min=1.0, hall_r_max=1.012, rtol=1e-8, max_it=200, restart=30)
    if case["kind"] == "adjoint":
        out["fn"] = gpu.DeviceFunction(st, s["eta"].cpu().numpy(), s["mask"].cpu().numpy(), case["steps"], case["every"], st.cfl_dt())
    return out


def _semi_hall(case, s, dt):
    h, dm, _ = _mesh(case)
    ne = (s["U"][0, :, 0] / s["mass"][0] + s["U"][1, :, 0] / s["mass"][1]).cpu().numpy()
    B = dm.reconstruct_cell_vector(s["Phi"] + s["PhiAdd"]).cpu().numpy()
    return 2.0 * workloads.whistler_dt(h, B, np.sqrt(ne * ne + NE_FLOOR ** 2), 1.0, 1.0) / dt


def run(state):
    case = state["case"]
    if case["kind"] == "step":
        st = state["st"]
        if case["steps"] == 1:
            return {"dt": st.step(), "U": state["U"], "Phi": state["Phi"]}
        for _ in range(case["steps"]):
            st.step(sync=False)
        return {"U": state["U"], "Phi": state["Phi"]}
    if case["kind"] == "semi":
        dt, it, _ = state["st"].step_semi_implicit(state["ind"])
        return {"dt": dt, "iterations": it, "U": state["U"], "Phi": state["Phi"]}
    if case["kind"] == "solve":
        # the residual estimate is a diagnostic of the field that comes back
        E, it, _ = state["ind"].solve(state["Phi"], state["E"], state["dir"], state["dt"], warm=False)
        return {"E": E, "iterations": it}
    if case["kind"] == "adjoint":
        J = state["fn"].forward()
        ge, gu = state["fn"].backward()
        return {"J": J, "eta": ge, "u_inf": gu}
    dm, Phi, fs, dt = state["dm"], state["Phi"], state["fs"], state["dt"]
    W = dm.to_prim(state["U"], GAMMA)
    grad = dm.limited_gradients(W, 0, fs)
    rhs = dm.fluid_flux_rhs(GAMMA, 0, fs, W, grad)
    B = dm.reconstruct_cell_vector(Phi)
    u = W.view(-1, 5)[:, 1:4].reshape(-1)
    E = dm.edge_modes(state["u_inf"], state["B_imf"], dm.add_ideal_emf(u, B, B, Phi, Phi))
    return {"W": W, "grad": grad, "rhs": rhs, "B": B, "E": E, "Phi": dm.faraday_update(E, Phi, dt), "J": dm.cell_current(B)}


def work(case):
    """Compulsory traffic of one pass: each input (state, fluxes, topology, metric) read once per application of the
    operator, each output written once; operations counted per cell, face and edge of the scheme."""
    tet = case["cells"] == "tet"
    n, hexes = case["n"], case["n"] ** 3 if case["mesh"] == "box" else 6 * case["n"] ** 2 * case["nr"]
    nc, nf, ne, fpc = (6 * hexes, 12 * hexes, 7 * hexes, 4) if tet else (hexes, 3 * hexes, 3 * hexes, 6)
    epf = 3 if tet else 4
    ions = case.get("ions", 1)
    val = 4.0 if case.get("precision") == "mixed" else 8.0      # metric and work values; the state stays 8
    topo = nc * fpc * 5.0 + nf * (8 + 5 * epf + 1) + ne * (5.0 * epf * nf / ne + 1)
    metric = val * (4 * nc + 7 * nf + 7 * ne)
    state = 8.0 * (5 * ions * nc + nf)
    fl = ions * (nc * (60 + 5 * (20 + 22 * fpc)) + nf * 130) + nf * 60 + ne * (60 + nf * epf / ne * 60) + 6.0 * nc * fpc * 4
    if case["kind"] == "step":
        k = case["steps"]
        return {"bytes": k * (2 * state + 8.0 * nf + topo + metric), "flops": k * 2.0 * fl}
    if case["kind"] == "calls":
        return {"bytes": state + topo + metric + 8.0 * nc * (5 + 15 + 5 + 3 + 3) + 8.0 * (ne + nf), "flops": fl}
    op = 8.0 * 2 * ne + topo + val * (3 * nc * fpc + 3 * nf + 4 * nc + 4 * ne)   # x in, y out, tables
    opfl = nf * 2 * epf + nc * fpc * 20 + ne * 40
    if case["kind"] == "solve":
        its = min(case["max_it"], 170)
        basis = 8.0 * ne * (2 * 16 + 4)                              # the mean column's basis, for the dots and the update
        return {"bytes": its * (op + basis), "flops": its * (opfl + 4.0 * ne * 16)}
    if case["kind"] == "semi":
        its = 6
        return {"bytes": 2 * state + topo + metric + its * (op + 8.0 * ne * 12), "flops": fl + its * opfl}
    k = case["steps"]
    return {"bytes": k * 3.0 * (2 * state + topo + metric) + 8.0 * 2 * nc, "flops": k * 2.0 * fl * 5}


# ------------------------------------------------------------------ the same results in plain torch, 64 bits
def _dot(a, b):
    return (a * b).sum(-1)


def _cross(a, b):
    return torch.linalg.cross(a, b)


class _Exact:
    """The scheme restated on one mesh with torch index operations (any polyhedra), differentiable."""

    def __init__(self, h):
        T = lambda k: torch.as_tensor(np.array(h[k]), device="cuda")
        self.nc, self.nf, self.ne, self.nn = h.n_cells, h.n_faces, h.n_edges, h.n_nodes
        for k in ("cell_center", "cell_volume", "face_area", "face_center", "face_area_mag", "edge_vec", "edge_mid", "edge_len",
                  "star1", "star2", "ec_weight", "ef_weight"):
            setattr(self, k, T(k))
        self.mat, self.kind, self.mode = T("cell_material"), T("face_kind").long(), T("edge_mode").long()
        self.fluid = self.mat == 0
        for a in ("c2f", "f2e", "e2f", "f2c"):
            ptr = T(a + "_ptr").long()
            setattr(self, a, (_rows(ptr), T(a + "_idx").long(), T(a + "_sgn").double()))
            setattr(self, a + "_ptr", ptr)
        self.ec = (_rows(T("ec_ptr").long()), T("ec_cell").long())
        self.ec_n = T("ec_ptr").long().diff()
        self.ec_pad = self._pad(T("ec_ptr").long(), self.ec[1])
        self.nodes = T("e2n_idx").long().reshape(-1, 2)
        self.n = self.face_area / self.face_area_mag[:, None]
        fr, fc, fs = self.f2c
        self.L = torch.full((self.nf,), -1, dtype=torch.long, device="cuda")
        self.R = self.L.clone()
        self.L[fr[fs > 0]], self.R[fr[fs < 0]] = fc[fs > 0], fc[fs < 0]
        self.cnt = self.f2c_ptr.diff()
        self.inner = (self.cnt == 2) & (self.kind == 0)
        # least-squares stencil: neighbour across interior faces, the mirrored point elsewhere
        c, f, sg = self.c2f
        self.nb = torch.where(self.L[f] == c, self.R[f], self.L[f])
        self.int_e, self.skip = self.inner[f], self.kind[f] == 4
        xc, no = self.cell_center[c], sg[:, None] * self.n[f]
        d = torch.where(self.int_e[:, None], self.cell_center[self.nb.clamp(min=0)] - xc,
                        2.0 * _dot(self.face_center[f] - xc, no)[:, None] * no)
        self.no, self.dx = no, self.face_center[f] - xc
        w = torch.where(self.skip, 0.0, 1.0 / _dot(d, d).clamp(min=1e-300))
        M = torch.zeros(self.nc, 3, 3, dtype=torch.float64, device="cuda").index_add_(0, c, w[:, None, None] * d[:, :, None] * d[:, None, :])
        det = torch.linalg.det(M)
        sc = torch.diagonal(M, dim1=1, dim2=2).amax(1).clamp(min=1e-300)
        self.valid = (det.abs() >= 1e-9 * sc ** 3) & self.fluid
        eye = torch.eye(3, dtype=torch.float64, device="cuda")
        inv = torch.linalg.inv(torch.where(self.valid[:, None, None], M, eye))
        self.fit = torch.einsum("eij,ej->ei", inv[c], w[:, None] * d)     # gradient = sum fit dq
        Mb = torch.zeros(self.nc, 3, 3, dtype=torch.float64, device="cuda").index_add_(
            0, c, self.face_area_mag[f][:, None, None] * self.n[f][:, :, None] * self.n[f][:, None, :])
        self.rec = torch.einsum("eij,ej->ei", torch.linalg.inv(Mb)[c], self.n[f])
        # edge geometry of the upwind EMF
        e, f, _ = self.e2f
        self.th = self.edge_vec / self.edge_len[:, None]
        v = self.face_center[f] - self.edge_mid[e]
        v = v - _dot(v, self.th[e])[:, None] * self.th[e]
        self.m = v / v.norm(dim=1, keepdim=True)
        self.sig = _dot(self.th[e], _cross(self.m, self.n[f]))
        ax = torch.where((self.th[:, 0].abs() < 0.9)[:, None], eye[0], eye[1])
        e1 = _cross(self.th, ax)
        self.e1 = e1 / e1.norm(dim=1, keepdim=True)
        self.e2 = _cross(self.th, self.e1)

    @staticmethod
    def _pad(ptr, idx):
        n = int(ptr.diff().max())
        k = ptr[:-1, None] + torch.arange(n, device="cuda")
        return torch.where(k < ptr[1:, None], idx[k.clamp(max=idx.numel() - 1)], -1)

    def _sum(self, n, rows, v):
        return torch.zeros((n, *v.shape[1:]), dtype=torch.float64, device="cuda").index_add(0, rows, v)

    def cell_vector(self, phi):
        c, f, _ = self.c2f
        return self._sum(self.nc, c, self.rec * phi[f][:, None])

    def d1(self, E):
        f, e, s = self.f2e
        return self._sum(self.nf, f, s * E[e])

    @staticmethod
    def prims(U):
        r = U[:, 0].clamp(min=RHO_FLOOR)
        u = U[:, 1:4] / r[:, None]
        p = ((GAMMA - 1.0) * (U[:, 4] - 0.5 * r * _dot(u, u))).clamp(min=P_FLOOR)
        return torch.cat([r[:, None], u, p[:, None]], 1)

    @staticmethod
    def ghost(kind, absorb, W, n, fs):
        un = _dot(W[:, 1:4], n)
        wall = torch.cat([W[:, :1], W[:, 1:4] - 2 * un[:, None] * n, W[:, 4:]], 1)
        if absorb:
            wall = torch.tensor([1e-12, 0, 0, 0, 1e-12], dtype=torch.float64, device="cuda").expand_as(W)
        k = kind[:, None]
        return torch.where(k == 1, wall, torch.where(k == 2, fs.expand_as(W), W))

    def gradients(self, W, absorb, fs):
        c, f, _ = self.c2f
        wn = torch.where(self.int_e[:, None], W[self.nb.clamp(min=0)], self.ghost(self.kind[f], absorb, W[c], self.no, fs))
        wn = torch.where(self.skip[:, None], W[c], wn)
        g = torch.stack([self._sum(self.nc, c, self.fit * (wn - W[c])[:, q:q + 1]) for q in range(5)], 1)
        i5 = c[:, None].expand(-1, 5)
        hi = W.scatter_reduce(0, i5, wn, "amax", include_self=True)
        lo = W.scatter_reduce(0, i5, wn, "amin", include_self=True)
        dl = torch.einsum("eqa,ea->eq", g[c], self.dx)
        one = torch.ones_like(dl)
        q = torch.where(dl > 1e-300, (hi - W)[c] / torch.where(dl > 1e-300, dl, one),
                        torch.where(dl < -1e-300, (lo - W)[c] / torch.where(dl < -1e-300, dl, one), one))
        psi = torch.ones_like(W).scatter_reduce(0, i5, q, "amin", include_self=True).clamp(0.0, 1.0)
        return torch.where(self.valid[:, None, None], psi[:, :, None] * g, 0.0)

    def flux_rhs(self, W, g, absorb, fs):
        on = torch.zeros(self.nf, dtype=torch.bool, device="cuda")
        fr, fc, fsg = self.f2c
        on[fr[self.fluid[fc]]] = True
        on &= self.kind != 4
        def state(c):
            w = W[c] + torch.einsum("fqa,fa->fq", g[c], self.face_center - self.cell_center[c])
            return torch.where(((w[:, 0] > 0) & (w[:, 4] > 0))[:, None], w, W[c])
        inL = (self.L >= 0) & self.fluid[self.L.clamp(min=0)]
        c1 = torch.where(inL, self.L, self.R).clamp(min=0)                # the inside cell of a boundary face
        s1 = torch.where(inL, 1.0, -1.0)[:, None].double()
        a, b = state(self.L.clamp(min=0)), state(self.R.clamp(min=0))
        ins = torch.where(inL[:, None], a, b)
        gh = self.ghost(self.kind, absorb, ins, s1 * self.n, fs)
        Ls = torch.where(self.inner[:, None], a, torch.where(s1 > 0, ins, gh))
        Rs = torch.where(self.inner[:, None], b, torch.where(s1 > 0, gh, ins))
        def parts(w):
            u = _cons(w)
            un = _dot(w[:, 1:4], self.n)
            F = torch.cat([(w[:, 0] * un)[:, None], (w[:, 0] * un)[:, None] * w[:, 1:4] + w[:, 4:] * self.n,
                           (un * (u[:, 4] + w[:, 4]))[:, None]], 1)
            return u, F, un.abs() + (GAMMA * w[:, 4] / w[:, 0]).sqrt()
        one = torch.ones(5, dtype=torch.float64, device="cuda")
        uL, FL, sL = parts(torch.where(on[:, None], Ls, one))
        uR, FR, sR = parts(torch.where(on[:, None], Rs, one))
        F = 0.5 * (FL + FR) - 0.5 * torch.maximum(sL, sR)[:, None] * (uR - uL)
        F = torch.where(on[:, None], F * self.face_area_mag[:, None], 0.0)
        c, f, s = self.c2f
        return torch.where(self.fluid[:, None], self._sum(self.nc, c, -s[:, None] * F[f]) / self.cell_volume[:, None], 0.0)

    def ideal_emf(self, u, Bt, Bi, phi_tot, phi, cuct=0.5):
        n, one = self.n, self.cnt == 1
        L = torch.where(self.L >= 0, self.L, self.R)
        R = torch.where(self.R >= 0, self.R, self.L)
        Bn = (phi_tot / self.face_area_mag)[:, None]
        flux = lambda c: _dot(u[c], n)[:, None] * Bt[c] - Bn * u[c]
        a = torch.maximum(_dot(u[L], n).abs(), _dot(u[R], n).abs())[:, None]
        F = torch.where(one[:, None], flux(L), 0.5 * (flux(L) + flux(R)) - 0.5 * a * (Bi[R] - Bi[L]))
        Ef = -_cross(n, F)
        e, f, _ = self.e2f
        w = self.ef_weight
        Ec = self._sum(self.ne, e, w * _dot(Ef[f], self.edge_vec[e]))
        aef = None
        for k in range(self.ec_pad.shape[1]):
            c = self.ec_pad[:, k]
            d = torch.where((c >= 0)[e], _dot(u[c.clamp(min=0)][e], self.m).abs(), 0.0)
            aef = d if aef is None else torch.maximum(aef, d)
        as_ = aef * self.sig
        qa, qb = as_ * _dot(n[f], self.e1[e]), as_ * _dot(n[f], self.e2[e])
        S = lambda v: self._sum(self.ne, e, v)
        M11, M12, M22, g1, g2 = S(w * qa * qa), S(w * qa * qb), S(w * qb * qb), S(w * qa), S(w * qb)
        tr = M11 + M22
        eps = 1e-14 * tr
        det = (M11 + eps) * (M22 + eps) - M12 * M12
        ok = (tr > 0) & (det > 0)
        dd = torch.where(ok, det, 1.0)
        l1 = torch.where(ok, ((M22 + eps) * g1 - M12 * g2) / dd, 0.0)
        l2 = torch.where(ok, ((M11 + eps) * g2 - M12 * g1) / dd, 0.0)
        Eu = S(w * (1.0 - (qa * l1[e] + qb * l2[e])) * as_ * (phi / self.face_area_mag)[f])
        fl = torch.zeros(self.ne, dtype=torch.bool, device="cuda")
        fl[self.ec[0][self.fluid[self.ec[1]]]] = True
        return torch.where(fl, Ec + 2.0 * cuct * self.edge_len * Eu, 0.0)

    def edge_modes(self, E, u_inf, B_imf):
        Einf = -_cross(u_inf, B_imf)
        return torch.where(self.mode == 1, 0.0, torch.where(self.mode == 2, self.edge_vec @ Einf, E))

    def current(self, B):
        c, f, s = self.c2f
        o = torch.where(self.L[f] == c, self.R[f], self.L[f])
        bf = torch.where((o >= 0)[:, None], 0.5 * (B[c] + B[o.clamp(min=0)]), B[c])
        return self._sum(self.nc, c, _cross(s[:, None] * self.face_area[f], bf)) / self.cell_volume[:, None]

    def induction(self, p, m_edge, B0, ne, hall_coef, r_min=1.0, r_max=1.012):
        """F of the semi-implicit induction: phi per face -> EMF per edge."""
        r = self.cell_center.norm(dim=1)
        taper = 0.5 * (1.0 + torch.tanh(2.0 * (r - 0.5 * (r_min + r_max)) / (r_max - r_min)))
        alpha = torch.where((ne > 0) & self.fluid, taper * hall_coef / ne.clamp(min=1e-300), 0.0)[:, None]
        e, f, s = self.e2f
        ee, cc = self.ec

        def F(phi):
            g = alpha * _cross(self.current(self.cell_vector(phi)), B0)
            return m_edge * self._sum(self.ne, e, s * (self.star2 * phi)[f]) + self._sum(
                self.ne, ee, self.ec_weight * _dot(g[cc], self.edge_vec[ee]))
        return F

    def solve(self, F, m_edge, Phi, E, free, dt, tol=1e-13, steps=700):
        """(I + dt F d1) E' = E + F(Phi) on the free edges by Jacobi-preconditioned GMRES without restart."""
        d2 = self._sum(self.ne, self.e2f[0], self.star2[self.e2f[1]])
        pd = torch.where(free, 1.0 / (1.0 + dt * m_edge * d2), 0.0)
        A = lambda x: x + dt * F(self.d1(x))
        b = E + F(Phi)
        r = torch.where(free, b - A(E), 0.0)
        beta = r.norm()
        V, Hc = [r / beta], np.zeros((steps + 1, steps))
        for j in range(steps):
            w = torch.where(free, A(pd * V[j]), 0.0)
            B = torch.stack(V)
            h1 = B @ w
            w = w - h1 @ B
            h2 = B @ w
            w = w - h2 @ B
            nw = w.norm()
            Hc[:j + 1, j], Hc[j + 1, j] = (h1 + h2).cpu().numpy(), float(nw)
            V.append(w / nw)
            if j % 20 == 19 or j == steps - 1:
                e1 = np.zeros(j + 2)
                e1[0] = float(beta)
                y, res = np.linalg.lstsq(Hc[:j + 2, :j + 1], e1, rcond=None)[:2]
                if (float(res[0]) if len(res) else 0.0) ** 0.5 <= tol * float(b.norm()):
                    break
        x = torch.as_tensor(y, device="cuda") @ torch.stack(V[:len(y)])
        return E + pd * x


def exact(case, seed):
    cells = (6 if case["cells"] == "tet" else 1) * (case["n"] ** 3 if case["mesh"] == "box" else 6 * case["n"] ** 2 * case["nr"])
    if cells > 4_500_000 or case.get("steps", 1) * cells > 9_000_000:
        return None  # minutes of torch work
    if case["kind"] == "solve" and (cells > 300_000 or case["max_it"] < 300):
        return None  # a capped solve stops at an iterate of its own; a large one needs minutes
    if case["kind"] == "adjoint" and case["steps"] * cells > 2_500_000:
        return None
    h = _mesh(case)[0]
    s = _inputs(case, seed)
    x = _Exact(h)
    V = lambda v: torch.tensor(v, dtype=torch.float64, device="cuda")
    if case["kind"] == "solve":
        F = x.induction(None, s["m_edge"], s["B0"], s["ne"], 1.0)
        return {"E": x.solve(F, s["m_edge"], s["Phi"], s["E"], s["dir"] == 0, s["dt"]), "iterations": None}
    if case["kind"] == "calls":
        W = x.prims(s["U"][0])
        g = x.gradients(W, False, V(s["fs"][0]))
        B = x.cell_vector(s["Phi"])
        E = x.edge_modes(x.ideal_emf(W[:, 1:4], B, B, s["Phi"], s["Phi"]), V(s["u_inf"]), V(s["B_imf"]))
        return {"W": W.reshape(-1), "grad": g.reshape(-1), "rhs": x.flux_rhs(W, g, False, V(s["fs"][0])).reshape(-1), "B": B.reshape(-1),
                "E": E, "Phi": s["Phi"] - 1e-3 / case["n"] * x.d1(E), "J": x.current(B).reshape(-1)}
    if case["kind"] == "adjoint":
        eta = s["eta"].clone().requires_grad_()
        u = V(s["u_inf"]).requires_grad_()
        m = _Model(x, case, s, eta=eta, u_inf=u)
        U, Phi = m.shifted(s["U"], u), s["Phi"]
        dt = m.cfl(*m.prepare(s["U"], s["Phi"])[:2]).detach()
        for _ in range(case["steps"]):
            U, Phi = torch.utils.checkpoint.checkpoint(lambda a, b: m.rk2(a, b, dt), U, Phi, use_reentrant=False)
        B = x.cell_vector(Phi) + m.Badd
        J = (s["mask"].double() * _dot(B, B) * x.cell_volume).sum()
        J.backward()
        return {"J": J.detach(), "eta": eta.grad, "u_inf": u.grad}
    m = _Model(x, case, s)
    U, Phi = s["U"], s["Phi"]
    if case["kind"] == "semi":
        W, Bt, *_ = m.prepare(U, Phi)
        dt = m.cfl(W, Bt)
        hall = _semi_hall(case, s, float(dt))
        U, Phi, dt = m.semi(U, Phi, s["m_edge"], hall)
        return {"dt": dt, "iterations": None, "U": U.transpose(1, 2).contiguous(), "Phi": Phi}
    for _ in range(case["steps"]):
        U, Phi, dt = m.step(U, Phi)
    out = {"U": U.transpose(1, 2).contiguous(), "Phi": Phi}
    return {"dt": dt, **out} if case["steps"] == 1 else out


class _Model:
    """The steps of the multi-ion model on _Exact's operators."""

    def __init__(self, x, case, s, eta=None, u_inf=None):
        V = lambda v: torch.tensor(v, dtype=torch.float64, device="cuda")
        self.x, self.case, self.s = x, case, s
        self.ions, self.mass, self.src = len(s["mass"]), s["mass"], case.get("sources", "none")
        self.fs = [V(f) for f in s["fs"]]
        self.u_inf, self.B_imf, self.u0 = V(s["u_inf"]), V(s["B_imf"]), V(s["u_inf"])
        if u_inf is not None:
            self.u_inf = u_inf
            self.fs = [torch.cat([f[:1], u_inf, f[4:]]) for f in self.fs]
        self.Badd = x.cell_vector(s["PhiAdd"])
        self.absorb = [k == 1 for k in range(self.ions)]
        self.m_res = None
        if eta is not None:
            e, c = x.ec
            self.m_res = x._sum(x.ne, e, eta[c]) / x.ec_n / x.star1
        if self.src == "full":
            c, f, sg = x.c2f
            en = x.nodes[x.f2e[1]]                       # per f2e entry its edge's nodes
            fn = x.f2e[0][:, None].expand(-1, 2)
            pairs = torch.unique(torch.stack([fn.reshape(-1), en.reshape(-1)], 1), dim=0)   # face - node
            cnt = torch.bincount(pairs[:, 0], minlength=x.nf)
            ptr = torch.cat([cnt.new_zeros(1), cnt.cumsum(0)])
            nd = x._pad(ptr, pairs[:, 1])[f]
            cn = torch.stack([c[:, None].expand_as(nd)[nd >= 0], nd[nd >= 0]], 1)
            cn = torch.unique(cn, dim=0)
            self.cn = cn[x.fluid[cn[:, 0]]]              # fluid cell - node

    def shifted(self, U, u):
        W = torch.stack([self.x.prims(a) for a in U])
        W = torch.cat([W[..., :1], W[..., 1:4] + (u - self.u0), W[..., 4:]], -1)
        return torch.where(self.x.fluid[None, :, None], U + (_cons(W) - _cons(W).detach()), U)

    def numbers(self, rho):
        n = [r.clamp(min=0.0) / m for r, m in zip(rho, self.mass)]
        return n, sum(n)

    def prepare(self, U, Phi):
        W = torch.stack([self.x.prims(a) for a in U])
        n, ne = self.numbers(W[..., 0])
        up = sum((k / ne)[:, None] * w[:, 1:4] for k, w in zip(n, W))
        Bi = self.x.cell_vector(Phi)
        return W, Bi + self.Badd, Bi, torch.where(self.x.fluid[:, None], up, 0.0)

    def cfl(self, W, Bt):
        x = self.x
        c, f, _ = x.c2f
        B2, rt = _dot(Bt, Bt), W[..., 0].sum(0).clamp(min=1e-2)
        dt = math.inf
        for w in W:
            cs2 = GAMMA * w[:, 4] / w[:, 0].clamp(min=1e-30)
            term, bn = (cs2 + B2 / rt)[c], _dot(Bt[c], x.n[f])
            cf = (0.5 * (term + (term * term - 4 * cs2[c] * bn * bn / rt[c]).clamp(min=0.0).sqrt())).sqrt()
            den = x._sum(x.nc, c, (_dot(w[c, 1:4], x.n[f]).abs() + cf) * x.face_area_mag[f])
            dt = min(dt, float((0.4 * x.cell_volume / den)[x.fluid].min()))
        return V64(dt)

    def gyrate(self, U, Bt, dt):
        aH, aN = 1.0 / self.mass[0], 1.0 / self.mass[1]
        wH, wN = self.x.prims(U[0])[:, 1:4], self.x.prims(U[1])[:, 1:4]
        (nH, nN), ne = self.numbers(U[..., 0])
        den = aH * nN / ne + aN * nH / ne
        bm = Bt.norm(dim=1)
        bh = Bt / bm.clamp(min=1e-300)[:, None]
        w = wH - wN
        wp = w - _dot(w, bh)[:, None] * bh
        th = (den * bm * dt)[:, None]
        dw = (torch.cos(th) - 1.0) * wp + torch.sin(th) * _cross(wp, bh)
        out = []
        for u, v, d in ((U[0], wH, (aH * nN / ne / den)[:, None] * dw), (U[1], wN, -(aN * nH / ne / den)[:, None] * dw)):
            v2 = v + d
            e = u[:, 4] + 0.5 * u[:, 0] * (_dot(v2, v2) - _dot(v, v))
            out.append(torch.cat([u[:, :1], u[:, :1] * v2, e[:, None]], 1))
        return torch.where(self.x.fluid[None, :, None], torch.stack(out), U)

    def sources(self, W, Bt, Bi, dt):
        x, s = self.x, self.s
        (nH, nN), ne = self.numbers(W[..., 0])
        ne_eff = (ne * ne + NE_FLOOR ** 2).sqrt()
        JB = _cross(x.current(Bi), Bt)
        if self.src == "full":
            pe = W[0, :, 4] + W[1, :, 4]
            c, f, sg = x.c2f
            o = torch.where(x.L[f] == c, x.R[f], x.L[f])
            mean = (o >= 0) & x.fluid[o.clamp(min=0)]
            pf = torch.where(mean, 0.5 * (pe[c] + pe[o.clamp(min=0)]), pe[c])
            dpe = x._sum(x.nc, c, (pf * sg)[:, None] * x.face_area[f]) / x.cell_volume[:, None]
        out = []
        for k, (w, n) in enumerate(zip(W, (nH, nN))):
            ws = (n / ne_eff)[:, None]
            S = ws * JB - (ws * dpe if self.src == "full" else 0.0)
            rho, u = w[:, 0], w[:, 1:4]
            r = [torch.zeros_like(rho), S, _dot(u, S) + 0.5 * dt * _dot(S, S) / rho]
            if self.src == "full":
                v, u2, mH, mN = s["vst"], _dot(u, u), self.mass[0], self.mass[1]
                T = w[:, 4] / rho / (FULL["state_coeff_H"] if k == 0 else FULL["state_coeff_Na"]) * FULL["T_ref"]
                b1 = v * (FULL["Tn0"] - T) * (mH / (mH + mN) if k == 0 else 0.5)
                b2 = (mN / (mH + mN) if k == 0 else 0.5) * v
                r[1] = r[1] - FULL["a4"] * (rho * v)[:, None] * u
                r[2] = r[2] - FULL["a4"] * rho * u2 * v + FULL["a5"] * n * b1 + FULL["a4"] * rho * u2 * b2
                if k == 1:
                    r[0] = FULL["a1_Na"] * s["photo"]
                    r[2] = r[2] + FULL["a6"] * s["photo"] * FULL["Tn0"]
            out.append(torch.cat([r[0][:, None], r[1], r[2][:, None]], 1))
        return torch.stack(out)

    def floors(self, U):
        ke = 0.5 * (U[..., 1:4] ** 2).sum(-1) / U[..., 0].clamp(min=RHO_FLOOR)
        p = (GAMMA - 1.0) * (U[..., 4] - ke)
        low = torch.zeros_like(U)
        low[..., 0], low[..., 4] = RHO_FLOOR, P_FLOOR / (GAMMA - 1.0)
        Up = torch.cat([U[..., :4], torch.where(p < P_FLOOR, P_FLOOR / (GAMMA - 1.0) + ke, U[..., 4])[..., None]], -1)
        return torch.where((U[..., 0] >= RHO_FLOOR)[..., None], Up, low)

    def stage(self, U, Phi, dt):
        """(U + dt rhs with floors, E, B_tot)"""
        x = self.x
        W, Bt, Bi, up = self.prepare(U, Phi)
        rhs = torch.stack([x.flux_rhs(w, x.gradients(w, a, f), a, f) for w, a, f in zip(W, self.absorb, self.fs)])
        if self.src != "none":
            rhs = rhs + self.sources(W, Bt, Bi, dt)
        U1 = torch.where(x.fluid[None, :, None], self.floors(U + dt * rhs), U)
        E = x.ideal_emf(up, Bt, Bi, Phi + self.s["PhiAdd"], Phi)
        if self.src == "full":
            E = E - self.ambipolar(W)
        E = x.edge_modes(E, self.u_inf, self.B_imf)
        if self.m_res is not None:
            e, f, sg = x.e2f
            E = E + self.m_res * x._sum(x.ne, e, sg * (x.star2 * Phi)[f])
        return U1, E, Bt, W

    def ambipolar(self, W):
        x = self.x
        c, v = self.cn[:, 0], self.cn[:, 1]
        pe = W[0, :, 4] + W[1, :, 4]
        pn = x._sum(x.nn, v, x.cell_volume[c] * pe[c]) / x._sum(x.nn, v, x.cell_volume[c]).clamp(min=1e-300)
        e, cc = x.ec
        ws = x._sum(x.ne, e, x.ec_weight)
        rho = [x._sum(x.ne, e, x.ec_weight * w[cc, 0]) / ws for w in W]
        _, ne = self.numbers(rho)
        return FULL["pressure_coef"] * (pn[x.nodes[:, 1]] - pn[x.nodes[:, 0]]) / (ne * ne + NE_FLOOR ** 2).sqrt()

    def rk2(self, U, Phi, dt):
        U1, E, _, _ = self.stage(U, Phi, dt)
        Phi1 = Phi - dt * self.x.d1(E)
        U2, E, self.Bt, _ = self.stage(U1, Phi1, dt)
        return 0.5 * (U + U2), 0.5 * (Phi + Phi1 - dt * self.x.d1(E))

    def step(self, U, Phi):
        W, Bt, *_ = self.prepare(U, Phi)
        dt = self.cfl(W, Bt)
        if self.src != "none":
            U = self.gyrate(U, Bt, 0.5 * dt)
        U, Phi = self.rk2(U, Phi, dt)
        if self.src != "none":
            U = self.gyrate(U, self.Bt, 0.5 * dt)
        return U, Phi, dt

    def semi(self, U, Phi, m_edge, hall):
        x = self.x
        W, Bt, *_ = self.prepare(U, Phi)
        dt = self.cfl(W, Bt)
        U, E, Bt, W = self.stage(self.gyrate(U, Bt, 0.5 * dt), Phi, dt)
        _, ne = self.numbers(W[..., 0])
        F = x.induction(None, m_edge, Bt, torch.where(x.fluid, (ne * ne + NE_FLOOR ** 2).sqrt(), 0.0), hall)
        E = x.solve(F, m_edge, Phi, E, x.mode != 2, dt)
        return self.gyrate(U, Bt, 0.5 * dt), Phi - dt * x.d1(E), dt


def V64(v):
    return torch.tensor(float(v), dtype=torch.float64, device="cuda")
