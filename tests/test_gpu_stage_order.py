"""A queued step on two streams keeps its place: two states stepping in turn on one mesh, the mesh's stream replaced between
steps, and a step captured in a caller's graph give the bits of the plain sequence."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
STEPS = 6


def _make(dm, wl, precision):
    from mpcns_uns_b200 import gpu
    st = gpu.ResidentState(dm, gpu.step_params(1, wl.gamma, fs=wl.fs, mass=wl.mass, u_inf=wl.u_inf, B_imf=wl.B_imf, precision=precision))
    st.set(wl.U, wl.Phi, wl.PhiAdd)
    return st


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [4, 12])
def test_queued_steps_keep_their_order(n, precision):
    import torch

    from mpcns_uns_b200 import gpu, workloads
    wl = workloads.box(n)
    plain = _make(gpu.DeviceMesh(wl.mesh), wl, precision)
    dts = [plain.step() for _ in range(STEPS)]
    want = plain.U(0), plain.Phi()

    def same(st):
        assert np.array_equal(st.U(0), want[0]) and np.array_equal(st.Phi(), want[1])

    dm = gpu.DeviceMesh(wl.mesh)
    a, b = _make(dm, wl, precision), _make(dm, wl, precision)
    for dt in dts:
        a.step(sync=False)
        b.step(dt, sync=False)
    same(a)
    same(b)

    streams = [torch.cuda.Stream() for _ in range(2)]
    dm = gpu.DeviceMesh(wl.mesh)
    st = _make(dm, wl, precision)
    for k in range(STEPS):
        if k % 2:
            torch.cuda.synchronize()   # the caller orders its own streams
            gpu.check(gpu.lib().mhd_gpu_mesh_set_stream(dm.handle, streams[k // 2 % 2].cuda_stream))
        st.step(sync=False)
    same(st)

    dm = gpu.DeviceMesh(wl.mesh)
    st = _make(dm, wl, precision)
    gpu.check(gpu.lib().mhd_gpu_mesh_set_stream(dm.handle, streams[0].cuda_stream))
    st.step(sync=False)                # modules are loaded before the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=streams[0]):
        st.step(sync=False)
    for _ in range(STEPS - 1):
        graph.replay()
    torch.cuda.synchronize()
    same(st)
