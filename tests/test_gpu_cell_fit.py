"""The cell-field fit of a cell whose normal matrix is singular (its faces' normals in one plane) is zero, whatever the
fluxes of its faces: negative (no -0), infinite or NaN, as the oracle's."""
import numpy as np
import pytest

from helpers import MIXED_BOX_BC
from oracle import port

pytestmark = pytest.mark.gpu


class _Flattened:
    """A host mesh with the faces of one cell turned into the xy plane's normals."""

    def __init__(self, h, cell):
        self.h = h
        self.n_nodes, self.n_edges, self.n_faces, self.n_cells = h.n_nodes, h.n_edges, h.n_faces, h.n_cells
        f = np.asarray(h["c2f_idx"])[h["c2f_ptr"][cell]:h["c2f_ptr"][cell + 1]]
        A = np.array(h["face_area"])
        A[f, 2] = 0.0
        mag = np.array(h["face_area_mag"])
        mag[f] = np.sqrt((A[f] ** 2).sum(1))
        self.faces, self.over = f, {"face_area": A, "face_area_mag": mag}

    def __getitem__(self, name):
        return self.over[name] if name in self.over else self.h[name]


@pytest.mark.parametrize("tets", [True, False])
@pytest.mark.parametrize("flux", [-1.0, np.inf, -np.inf, np.nan])
def test_singular_fit_is_zero(tets, flux):
    from mpcns_uns_b200 import gpu
    from mpcns_uns_b200.mesh import HostMesh
    cell = 4
    h = _Flattened(HostMesh.box(2, 2, 3, tets=tets, jitter=0.1, seed=3).compute_geometry().boundary(*MIXED_BOX_BC), cell)
    phi = -np.random.default_rng(2).uniform(0.5, 1.0, h.n_faces)
    phi[h.faces] = flux
    want = port.PortMesh(h).cell_vector(phi)
    got = gpu.DeviceMesh(h).reconstruct_cell_vector(phi).cpu().numpy()
    assert np.array_equal(want.reshape(-1, 3)[cell], [0, 0, 0])
    assert np.array_equal(got, want, equal_nan=True)
    finite = np.isfinite(want)
    assert finite.any() and np.array_equal(np.signbit(got[finite]), np.signbit(want[finite]))
