"""mesh_ctx_stage_times: the kernel launches it reports are the kernels a call launches.

The call is captured (not replayed) on a stream of its own and the captured graph's
kernel nodes are counted.  The sizes are on both sides of the rule by which the counts
scan their tiles themselves, and windows of sign words repeat the launches.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F32 = (np.float32(-1), np.float32(1))


def kernel_nodes(torch, call):
    rt = ctypes.CDLL('libcudart.so.13')  # torch's
    vp, graph, n = ctypes.c_void_p, ctypes.c_void_p(), ctypes.c_size_t()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        assert rt.cudaStreamBeginCapture(vp(s.cuda_stream), 2) == 0  # relaxed
        call()
        assert rt.cudaStreamEndCapture(vp(s.cuda_stream), ctypes.byref(graph)) == 0
    assert rt.cudaGraphGetNodes(graph, None, ctypes.byref(n)) == 0
    nodes = (vp * n.value)()
    assert rt.cudaGraphGetNodes(graph, nodes, ctypes.byref(n)) == 0
    kinds = []
    for x in nodes:
        t = ctypes.c_int()
        assert rt.cudaGraphNodeGetType(vp(x), ctypes.byref(t)) == 0
        kinds.append(t.value)
    assert rt.cudaGraphDestroy(graph) == 0
    return kinds.count(0)  # cudaGraphNodeTypeKernel


@pytest.mark.parametrize('alg', ['mc', 'mt', 'nsn'])
@pytest.mark.parametrize('shape,words', [((40, 30, 20), 0), ((300, 301, 40), 0), ((37, 11, 300), 3), ((1449, 1450, 3), 0)])
def test_reported_launches_are_the_kernels_launched(pkg, cuda, monkeypatch, alg, shape, words):
    torch = cuda
    if words:
        monkeypatch.setenv('MESHING_GB300_BITS_BYTES', str(words * 4 * shape[0] * shape[1]))
    iso = np.float32(0.1)
    m = {'mc': pkg.MarchingCubes(iso=iso), 'nsn': pkg.NaiveSurfaceNets(iso=iso),
         'mt': pkg.MarchingTetrahedra(iso=iso, eps=np.float32(1e-3))}[alg]
    g = torch.Generator(device='cuda').manual_seed(3)
    vol = torch.randn(shape[::-1], generator=g, device='cuda').permute(2, 1, 0)
    ctx = pkg.Context(0)
    v, f = pkg.isosurface(vol, m, F32, F32, F32, ctx=ctx)
    n = torch.zeros(2, dtype=torch.int64, device='cuda')

    def call():
        pkg.isosurface_device(vol, m, F32, F32, F32, verts=v, faces=f, counts=n, ctx=ctx)

    call()
    ctx.enable_timing(True)
    call()
    torch.cuda.synchronize()
    reported = sum(k for _, k in ctx.stage_times().values())
    ctx.enable_timing(False)
    assert reported == kernel_nodes(torch, call)
    ctx.close()
