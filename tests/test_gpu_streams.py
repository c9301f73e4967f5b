"""One context used on several streams, and calls between a count and its fill.

mesh_count returns when the totals are known; its offsets may still be scanned on the
stream it ran on.  Whatever the context's next stream is, the fill, and the next call
after a count without a fill, find them finished.  The volumes are flat and wide: many
pieces, so that the scan is long beside the calls around it.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F32 = (np.float32(-1), np.float32(1))
ALGS = ['mc', 'mcw', 'mt', 'nsn']


def method(pkg, alg):
    iso = np.float32(0.25)
    if alg == 'mt':
        return pkg.MarchingTetrahedra(iso=iso, eps=np.float32(1e-3))
    return pkg.NaiveSurfaceNets(iso=iso) if alg == 'nsn' else pkg.MarchingCubes(iso=iso, weld=alg == 'mcw')


def flat(torch, nx, ny, empty=False):
    # one crossing in every column (none when empty), at a height that varies with the column
    x = torch.arange(nx, device='cuda', dtype=torch.float32)
    y = torch.arange(ny, device='cuda', dtype=torch.float32)
    z = torch.arange(4, device='cuda', dtype=torch.float32)
    v = z[:, None, None] - 1.0 - 0.9 * torch.sin(0.37 * x)[None, None, :] * torch.cos(0.23 * y)[None, :, None]
    if empty:
        v = v + 9.0
    return v.contiguous().permute(2, 1, 0)


def count(pkg, ctx, vol, m):
    lib, p = ctx._lib, pkg.api.make_params(m, F32, F32, F32)
    n = (ctypes.c_int64 * 2)()
    pkg._lib.check(lib.mesh_count(ctx.handle, vol.data_ptr(), pkg._lib.MESH_DT_F32, *vol.shape, 1, ctypes.addressof(p),
                                  ctypes.addressof(n), ctypes.addressof(n) + 8), ctx.handle)
    return n[0], n[1]


@pytest.mark.parametrize('alg', ALGS)
def test_count_and_fill_on_different_streams(pkg, cuda, alg):
    torch = cuda
    vol, m = flat(torch, 2500, 1501), method(pkg, alg)
    want = pkg.isosurface(vol, m, F32, F32, F32)
    ctx = pkg.Context(0)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for k in range(6):
        ctx.set_stream((a, b)[k % 2].cuda_stream)
        nv, nf = count(pkg, ctx, vol, m)
        assert (nv, nf) == (want[0].shape[0], want[1].shape[0])
        v = torch.full((nv, 3), -7.0, device='cuda')
        f = torch.full((nf, 3), -7, dtype=torch.int64, device='cuda')
        torch.cuda.current_stream().synchronize()
        ctx.set_stream((b, a)[k % 2].cuda_stream)
        pkg._lib.check(ctx._lib.mesh_fill(ctx.handle, v.data_ptr(), f.data_ptr(), 1), ctx.handle)
        assert torch.equal(v, want[0]) and torch.equal(f, want[1]), k
    ctx.close()


@pytest.mark.parametrize('alg', ALGS)
def test_empty_mesh_then_a_call_on_another_stream(pkg, cuda, alg):
    torch = cuda
    none, some, m = flat(torch, 2500, 1501, empty=True), flat(torch, 300, 211), method(pkg, alg)
    want = pkg.isosurface(some, m, F32, F32, F32)
    host = np.asfortranarray(some.cpu().numpy())
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for k in range(6):
        with torch.cuda.stream(a):
            v, f = pkg.isosurface(none, m, F32, F32, F32)
        assert v.shape == (0, 3) and f.shape == (0, 3)
        if k % 2:  # the context's own stream
            hv, hf = pkg.isosurface(host, m, F32, F32, F32)
            assert np.array_equal(hv, want[0].cpu().numpy()) and np.array_equal(hf, want[1].cpu().numpy()), k
        else:
            with torch.cuda.stream(b):
                v, f = pkg.isosurface(some, m, F32, F32, F32)
            b.synchronize()
            assert torch.equal(v, want[0]) and torch.equal(f, want[1]), k


def test_unfilled_count_then_a_captured_call(pkg, cuda):
    # the wait for the count's offsets is no part of the capture
    torch = cuda
    big, some, m = flat(torch, 2500, 1501), flat(torch, 300, 211), method(pkg, 'mc')
    want = pkg.isosurface(some, m, F32, F32, F32)
    v, f = torch.zeros_like(want[0]), torch.zeros_like(want[1])
    n = torch.zeros(2, dtype=torch.int64, device='cuda')
    ctx = pkg.Context(0)
    pkg.isosurface_device(some, m, F32, F32, F32, verts=v, faces=f, counts=n, ctx=ctx)  # sizes the scratch
    torch.cuda.synchronize()
    a = torch.cuda.Stream()
    ctx.set_stream(a.cuda_stream)
    count(pkg, ctx, big, m)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        pkg.isosurface_device(some, m, F32, F32, F32, verts=v, faces=f, counts=n, ctx=ctx)
    v.zero_()
    f.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(v, want[0]) and torch.equal(f, want[1]) and n.tolist() == [len(want[0]), len(want[1])]
    ctx.close()
