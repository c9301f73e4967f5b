"""The sign-bit path (k_bits.cu and the emissions on it) where its tiles end.

A warp's item is 32 columns of one row and a word is 32 samples of z, so the
volumes here end one cell before, at and after those edges.  Their samples are
noise: every case occurs, words and batches are full, and every column crosses
the iso value many times.  Meshes equal the oracle's, bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(2, 2, 2), (33, 3, 32), (34, 9, 33), (32, 10, 34), (65, 8, 64), (5, 17, 97), (66, 2, 129)]
F32 = (np.float32(-1), np.float32(1))
TYPES = [(np.float32, np.float32(0.1), F32), (np.float32, 0.0, (-1, 1)), (np.float64, 0.05, (-1, 2)),
         (np.uint16, 500, (-1, 1)), (np.int8, 3, (-1.0, 1.0))]


def noise(shape, dt, seed):
    rng = np.random.default_rng(seed)
    if np.issubdtype(dt, np.integer):
        info = np.iinfo(dt)
        return np.asfortranarray(rng.integers(max(info.min, -100), min(info.max, 1000), shape).astype(dt))
    return np.asfortranarray(rng.standard_normal(shape).astype(dt))


def method(pkg, alg, iso):
    if alg == 'mt':
        return pkg.MarchingTetrahedra(iso=iso, eps=iso.__class__(1e-3) if isinstance(iso, np.float32) else 1e-3)
    if alg == 'nsn':
        return pkg.NaiveSurfaceNets(iso=iso)
    return pkg.MarchingCubes(iso=iso, weld=alg == 'mcw')


def want(oracle, A, alg, iso, r):
    eps = np.float32(1e-3) if isinstance(iso, np.float32) else 1e-3
    return oracle.isosurface(A, alg, iso, eps, (r, r, r))


def same(got, ref):
    assert np.array_equal(got[1], ref[1])
    assert got[0].dtype == ref[0].dtype and got[0].shape == ref[0].shape
    assert np.array_equal(got[0].view(np.uint8), ref[0].view(np.uint8))


@pytest.mark.parametrize('alg', ['mc', 'mcw', 'mt', 'nsn'])
@pytest.mark.parametrize('shape', SHAPES)
def test_edges_of_words_and_items(pkg, oracle, cuda, alg, shape):
    for k, (dt, iso, r) in enumerate(TYPES):
        A = noise(shape, dt, k)
        same(pkg.isosurface(A, method(pkg, alg, iso), r, r, r), want(oracle, A, alg, iso, r))


@pytest.mark.parametrize('alg', ['mc', 'mcw', 'mt', 'nsn'])
def test_volumes_off_16_byte_boundaries(pkg, oracle, cuda, alg):
    # a volume that starts one sample into a buffer (no 16-byte loads), and one whose
    # planes are multiples of 16 bytes while its rows are not
    torch = cuda
    for shape, skip in (((40, 24, 70), 1), ((42, 26, 65), 0), ((48, 32, 40), 0)):
        A = noise(shape, np.float32, 5)
        buf = torch.zeros(A.size + skip, device='cuda')
        t = buf[skip:].view(shape[2], shape[1], shape[0])
        t.copy_(torch.from_numpy(np.ascontiguousarray(A.transpose(2, 1, 0))))
        v, f = pkg.isosurface(t.permute(2, 1, 0), method(pkg, alg, np.float32(0.1)), F32, F32, F32)
        same((v.cpu().numpy(), f.cpu().numpy()), want(oracle, A, alg, np.float32(0.1), F32))


@pytest.mark.parametrize('alg', ['mc', 'mcw', 'mt', 'nsn'])
@pytest.mark.parametrize('words', [2, 3, 5])
def test_windows_of_sign_words(pkg, oracle, cuda, monkeypatch, alg, words):
    # sign words capped at a few words of z: the volume is classified and emitted in
    # windows of segments
    A = noise((37, 11, 300), np.float32, 9)
    monkeypatch.setenv('MESHING_GB300_BITS_BYTES', str(words * 4 * 37 * 11))
    ctx = pkg.Context(0)
    got = pkg.isosurface(A, method(pkg, alg, 0.0), (-1, 1), (-1, 1), (-1, 1), ctx=ctx)
    ctx.close()
    same(got, want(oracle, A, alg, 0.0, (-1, 1)))
