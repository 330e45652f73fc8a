"""States where the device's memory is short: one that it does not hold is refused, and the refusal leaves neither memory nor an
error behind."""
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
