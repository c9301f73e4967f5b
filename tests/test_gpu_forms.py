"""Independent forms of the same extraction give the same mesh, and it is the oracle's.

The volume is classified and emitted whole, in windows of sign words
(MESHING_GB300_BITS_BYTES), and for Marching Cubes also through the list of active cells
(MESHING_GB300_LIST_EMIT) and in one walk (MESHING_GB300_ONE_WALK).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

R = (np.float32(0), np.float32(1))


@pytest.mark.parametrize('alg', ['mc', 'mcw', 'mt', 'nsn'])
def test_forms_agree_with_the_oracle(pkg, oracle, cuda, monkeypatch, alg):
    torch = cuda
    import meshing_gb300.fields as fields
    t = fields.gyroid(192, dtype=torch.float32)
    iso, eps = np.float32(0.05), np.float32(1e-3)
    m = {'mt': pkg.MarchingTetrahedra(iso=iso, eps=eps), 'nsn': pkg.NaiveSurfaceNets(iso=iso)}.get(
        alg, pkg.MarchingCubes(iso=iso, weld=alg == 'mcw'))
    wv, wf = oracle.isosurface(np.asfortranarray(t.cpu().numpy()), alg, iso, eps, (R, R, R))
    assert len(wf) > 100000
    forms = [{}, {'BITS_BYTES': str(3 * 4 * 192 * 192)}]
    if alg == 'mc':
        forms += [{'LIST_EMIT': '1'}, {'ONE_WALK': '1'}]
    for env in forms:
        with monkeypatch.context() as mp:
            for k, v in env.items():
                mp.setenv('MESHING_GB300_' + k, v)
            ctx = pkg.Context(0)
            v, f = pkg.isosurface(t, m, R, R, R, ctx=ctx)
            ctx.close()
        assert np.array_equal(f.cpu().numpy(), wf), env
        assert np.array_equal(v.cpu().numpy().view(np.uint8), wv.view(np.uint8)), env
