"""MT and NSN on flat volumes of many columns, which take the walk instead of the sign bits.

The rule (mesh_api.cu, flat()) is at most three layers of cells and at least 2^21 columns;
the shapes are on both sides of it.  Meshes equal the oracle's, bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F32 = (np.float32(-1), np.float32(1))
IN, OUT = (1449, 1450), (1449, 1448)  # 2098152 and 2095256 columns of cells


def method(pkg, alg, iso):
    if alg == 'nsn':
        return pkg.NaiveSurfaceNets(iso=iso)
    return pkg.MarchingTetrahedra(iso=iso, eps=iso.__class__(1e-3) if isinstance(iso, np.float32) else 1e-3)


def want(oracle, A, alg, iso, r):
    return oracle.isosurface(A, alg, iso, np.float32(1e-3) if isinstance(iso, np.float32) else 1e-3, (r, r, r))


def waves(shape, dt, seed):
    rng = np.random.default_rng(seed)
    x, y, z = (np.arange(n, dtype=np.float32) * f for n, f in zip(shape, (0.31, 0.23, 0.7)))
    v = np.sin(x)[:, None, None] + np.cos(y)[None, :, None] * np.sin(z)[None, None, :]
    v += 0.01 * rng.standard_normal(shape, dtype=np.float32)
    return np.asfortranarray((v * 40 + 50).round().astype(dt) if np.issubdtype(dt, np.integer) else v.astype(dt))


def same(got, ref):
    assert np.array_equal(got[1], ref[1])
    assert got[0].dtype == ref[0].dtype and np.array_equal(got[0].view(np.uint8), ref[0].view(np.uint8))


@pytest.mark.parametrize('alg', ['mt', 'nsn'])
@pytest.mark.parametrize('xy,nz,dt,iso,r', [
    (IN, 2, np.float32, np.float32(0.1), F32), (IN, 4, np.float32, 0.1, (-1, 1)), (IN, 5, np.float32, np.float32(0.1), F32),
    (OUT, 2, np.float32, np.float32(0.1), F32), (IN, 3, np.float64, 0.05, (-1, 2)), (IN, 3, np.int16, 50, (-1.0, 1.0))])
def test_flat_volumes_match_the_oracle(pkg, oracle, cuda, alg, xy, nz, dt, iso, r):
    A = waves((*xy, nz), dt, nz)
    ref = want(oracle, A, alg, iso, r)
    t = cuda.from_numpy(np.ascontiguousarray(A.transpose(2, 1, 0))).cuda().permute(2, 1, 0)
    v, f = pkg.isosurface(t, method(pkg, alg, iso), r, r, r)
    same((v.cpu().numpy(), f.cpu().numpy()), ref)
    same(pkg.isosurface(A, method(pkg, alg, iso), r, r, r), ref)  # a host array


@pytest.mark.parametrize('alg', ['mt', 'nsn'])
def test_flat_volumes_into_kept_buffers(pkg, cuda, alg):
    torch = cuda
    A = waves((*IN, 3), np.float32, 4)
    t = torch.from_numpy(np.ascontiguousarray(A.transpose(2, 1, 0))).cuda().permute(2, 1, 0)
    m = method(pkg, alg, np.float32(0.1))
    ref = pkg.isosurface(t, m, F32, F32, F32)
    ctx = pkg.Context(0)
    n = torch.zeros(2, dtype=torch.int64, device='cuda')
    size = [len(ref[0]), len(ref[1])]
    for cut in (0, 1):  # room for all of it, then for less
        cap = [s - cut * s // 3 for s in size]
        v = torch.full((size[0], 3), 7.0, device='cuda')
        f = torch.full((size[1], 3), 7, dtype=torch.int64, device='cuda')
        pkg.isosurface_device(t, m, F32, F32, F32, verts=v[:cap[0]], faces=f[:cap[1]], counts=n, ctx=ctx)
        if cut:
            with pytest.raises(pkg.MeshError, match='capacity'):
                ctx.sync()
            assert (v[cap[0]:] == 7).all() and (f[cap[1]:] == 7).all()
        else:
            ctx.sync()
            assert torch.equal(v, ref[0]) and torch.equal(f, ref[1])
        assert n.tolist() == size
    v.zero_()
    f.zero_()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        pkg.isosurface_device(t, m, F32, F32, F32, verts=v, faces=f, counts=n, ctx=ctx)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(v, ref[0]) and torch.equal(f, ref[1]) and n.tolist() == size
    ctx.close()


@pytest.mark.parametrize('alg', ['mt', 'nsn'])
def test_flat_slabs(pkg, oracle, cuda, alg):
    # the second slab has a halo column and is on the walk too, the third is on the bits
    A = waves((3300, 1450, 3), np.float32, 6)
    m = method(pkg, alg, np.float32(0.1))
    same(pkg.isosurface_slabs(A, m, F32, F32, F32, slab_cells=1450), want(oracle, A, alg, np.float32(0.1), F32))
