"""The tensors that a batch and a server hand out hold the memory they look into."""
import gc
import weakref

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def sphere(torch, n):
    g = torch.linspace(-1, 1, n, device='cuda')
    r = (g[:, None, None] ** 2 + g[None, :, None] ** 2 + g[None, None, :] ** 2).sqrt()
    return r - 0.6


def test_views_of_a_dropped_batch(pkg, cuda):
    torch = cuda
    vol, m = sphere(torch, 40), pkg.MarchingCubes(iso=np.float32(0))
    want = pkg.isosurface(vol, m)
    b = pkg.Batch([vol], m)
    b.count()
    b.run()
    b.sync()
    verts, faces, _ = b.outputs()
    part = faces[3:7]
    ref = weakref.ref(b)
    del b
    gc.collect()
    assert ref() is not None
    assert torch.equal(verts, want[0]) and torch.equal(faces, want[1])
    del verts, faces, _
    gc.collect()
    assert ref() is not None  # a view of a view
    assert torch.equal(part, want[1][3:7])
    del part
    gc.collect()
    assert ref() is None


def test_views_of_a_dropped_server(pkg, cuda):
    torch = cuda
    vol, m = sphere(torch, 40), pkg.MarchingCubes(iso=np.float32(0))
    want = pkg.isosurface(vol, m)
    srv = pkg.Server(64 << 20)
    verts, faces = srv.result(srv.submit(vol, m))
    ref = weakref.ref(srv)
    del srv
    gc.collect()
    assert ref() is not None
    assert torch.equal(verts, want[0]) and torch.equal(faces, want[1])
    del verts, faces
    gc.collect()
    assert ref() is None
