"""Segments of more than 32 words of z: several mask words to an item.

Columns of many words are cut into segments of at most the depth that leaves every SM
enough items; only long thin volumes get deep ones.  Single volumes of every algorithm,
and batches at several depths, match the oracle bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F32 = (np.float32(-1), np.float32(1))
NX, NY, NZ = 2, 1500, 65000  # 1499 rows: 52 segments of 40 words on 152 SMs


def method(pkg, alg, iso):
    if alg == 'mt':
        return pkg.MarchingTetrahedra(iso=iso, eps=np.float32(1e-3))
    return pkg.NaiveSurfaceNets(iso=iso) if alg == 'nsn' else pkg.MarchingCubes(iso=iso, weld=alg == 'mcw')


@pytest.fixture(scope='module')
def column_volume(cuda):
    # a crossing about every 500 planes, at a height that drifts with the row
    torch = cuda
    y = torch.arange(NY, device='cuda', dtype=torch.float32)[None, :, None]
    x = torch.arange(NX, device='cuda', dtype=torch.float32)[None, None, :]
    v = torch.empty((NZ, NY, NX), dtype=torch.uint8, device='cuda')
    for k in range(0, NZ, 5000):
        z = torch.arange(k, min(k + 5000, NZ), device='cuda', dtype=torch.float32)[:, None, None]
        v[k:k + 5000] = (128 + 90 * torch.sin(0.0063 * z + 0.002 * y + 0.1 * x)).round().to(torch.uint8)
    t = v.permute(2, 1, 0)
    return t, t.cpu().numpy()


@pytest.mark.parametrize('alg', ['mc', 'mcw', 'mt', 'nsn'])
def test_deep_segments_match_the_oracle(pkg, oracle, cuda, column_volume, alg):
    torch = cuda
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows, words = (NX - 1 + 31) // 32 * (NY - 1), (NZ - 1 + 31) // 32
    assert -(-words // -(-sms * 512 // rows)) > 32  # the rule of prepare_bits
    t, A = column_volume
    iso = np.float32(127.5)
    v, f = pkg.isosurface(t, method(pkg, alg, iso), F32, F32, F32)
    wv, wf = oracle.isosurface(A, alg, iso, np.float32(1e-3), (F32, F32, F32))
    assert len(wf) > 100000
    assert np.array_equal(f.cpu().numpy(), wf)
    assert np.array_equal(v.cpu().numpy().view(np.uint8), wv.view(np.uint8))


@pytest.mark.parametrize('weld', [False, True])
def test_batch_segment_depths(pkg, oracle, cuda, weld):
    # depths of one, two, three and 64 words; the longest volumes have 66
    torch = cuda
    rng = np.random.default_rng(11)
    shapes = [(5, 6, 2100), (40, 9, 200), (2, 2, 2049), (33, 17, 97), (9, 34, 2080), (1, 5, 300), (6, 5, 64)]
    vols = [np.asfortranarray(rng.standard_normal(s).astype(np.float32)) for s in shapes]
    m = pkg.MarchingCubes(iso=np.float32(0.3), weld=weld)
    b = pkg.Batch([torch.from_numpy(np.ascontiguousarray(A.transpose(2, 1, 0))).cuda().permute(2, 1, 0) for A in vols],
                  m, F32, F32, F32)
    want = [oracle.isosurface(A, 'mcw' if weld else 'mc', np.float32(0.3), np.float32(1e-3), (F32, F32, F32))
            if min(A.shape) > 1 else (np.empty((0, 3), np.float32), np.empty((0, 3), np.int64)) for A in vols]
    for zs in (0, 32, 64, 96, 2048, 2200):
        b.set_knobs(zs=zs)
        b.count()
        b.run()
        b.sync()
        for i, (wv, wf) in enumerate(want):
            v, f = b.volume(i)
            assert np.array_equal(f.cpu().numpy(), wf), (zs, i)
            assert np.array_equal(v.cpu().numpy().view(np.uint8), wv.view(np.uint8)), (zs, i)
    b.close()
