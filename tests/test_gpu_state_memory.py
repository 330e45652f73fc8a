"""States where the device's memory is short: an FP64 state that it holds only with gradients (15 doubles per cell and
species) instead of face values (20 or 30) is still created, with the same results; one that it does not hold is refused, and
the refusal leaves neither memory nor an error behind."""
import numpy as np
import pytest

from helpers import SHELL_BC

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


class _Filled:
    """All but `left` bytes of the device's memory held (in 2 MB pages, so up to 4 MB less are left)."""

    def __init__(self, left):
        import torch
        self.held = [torch.empty(_free() - left, dtype=torch.uint8, device="cuda")]

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        import torch
        self.held.clear()
        torch.cuda.empty_cache()


@pytest.mark.parametrize("tets", [True, False])
def test_state_without_room_for_face_values(tets):
    import torch

    from mpcns_uns_b200 import gpu, workloads
    from mpcns_uns_b200.mesh import HostMesh
    n, nr = (14, 80) if tets else (28, 80)
    h = HostMesh.shell(n, nr, 1.0, 3.0, 1.02, tets=tets).compute_geometry().boundary(*SHELL_BC)
    nsp, steps = 2, 3
    rng = np.random.default_rng(3)
    W = np.empty((nsp, h.n_cells, 5))
    W[..., 0], W[..., 4] = rng.uniform(0.9, 1.1, (nsp, h.n_cells)), rng.uniform(0.09, 0.11, (nsp, h.n_cells))
    W[..., 1:4] = rng.uniform(-0.1, 0.1, (nsp, h.n_cells, 3))
    U = [workloads.to_cons(w, workloads.GAMMA).ravel() for w in W]
    Phi = workloads.d1(h, workloads.fourier_potential(h, 3, amp=0.05))
    p = gpu.step_params(nsp, workloads.GAMMA, fs=[(1.0, 0.0, 0.0, 0.0, 0.1)] * nsp, mass=[1.0, 23.0], B_imf=(0.0, 0.0, -0.5))
    dm = gpu.DeviceMesh(h)

    def run(st):
        st.set(U, Phi, np.zeros(h.n_faces))
        dts = [st.step() for _ in range(steps)]
        return dts, [st.U(s) for s in range(nsp)], st.Phi()

    want = run(gpu.ResidentState(dm, p))
    torch.cuda.empty_cache()
    extra = 8 * nsp * 5 * ((4 if tets else 6) - 3) * h.n_cells   # face values over gradients
    assert extra > 10 * MB
    with _Filled(6 << 30):      # below 8 GB no edge geometry table is kept: the size of the rest
        f = _free()
        st = gpu.ResidentState(dm, p)
        size = f - _free()
        assert run(st)[0] == want[0]
        del st
    with _Filled(size - extra // 3):
        st = gpu.ResidentState(dm, p)
        got = run(st)
    assert got[0] == want[0] and np.array_equal(got[2], want[2])
    for a, b in zip(got[1], want[1]):
        assert np.array_equal(a, b)
    if tets:                    # the differentiated run records face values: the state gets them with the function
        grads = []
        for s in (st, gpu.ResidentState(dm, p)):
            s.set(U, Phi, np.zeros(h.n_faces))
            fn = gpu.DeviceFunction(s, np.full(h.n_cells, 1e-3), np.ones(h.n_cells, np.int8), 2, 1, want[0][0])
            fn.forward()
            grads.append(fn.backward()[0])
            del fn
        # the face adjoints are summed with atomics, in any order
        assert np.max(np.abs(grads[0] - grads[1])) <= 1e-11 * np.max(np.abs(grads[1]))


def test_refused_creation_leaves_nothing():
    from mpcns_uns_b200 import gpu
    from mpcns_uns_b200.mesh import HostMesh
    h = HostMesh.shell(14, 40, 1.0, 3.0, 1.02, tets=True).compute_geometry().boundary(*SHELL_BC)
    dm = gpu.DeviceMesh(h)
    for precision in ("fp64", "mixed"):
        p = gpu.step_params(2, precision=precision)
        gpu.ResidentState(dm, p)
        with _Filled(64 * MB):   # the conservative variables alone take 2 x 2 x 40 bytes per cell (15 MB), the rest over 100 MB
            f = _free()
            with pytest.raises(gpu.MhdError, match="out of memory"):
                gpu.ResidentState(dm, p)
            assert _free() == f
        gpu.DeviceMesh(HostMesh.box(2, 2, 2, tets=False).compute_geometry().boundary("outflow"))
        gpu.ResidentState(dm, p).step(1e-6)
