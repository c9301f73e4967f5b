"""Both load forms of the sign-bit kernel, for every volume type.

k_bits reads 16 bytes at a time (V = 16 / sample size) where the planes lie on 16-byte
boundaries and give every SM two CTAs, else sample by sample.  The volumes are above that
size; each is meshed aligned, as a copy that starts one sample into a buffer, and with
planes that are no multiple of 16 bytes, and the last word of z is a partial one.  Every
mesh equals the oracle's, bit for bit, and a batch of the three gives the same.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TYPES = [np.uint8, np.int8, np.uint16, np.int16, np.float16, np.int32, np.float32, np.int64, np.float64]
ISO = np.float32(12.25)
R = (np.float32(-1), np.float32(1))


def field(shape, dt):
    # a few waves: some crossings in every word, most cells inactive
    x, y, z = (np.linspace(-1, 1, n, dtype=np.float32) for n in shape)
    v = 60 * np.sin(7 * x)[:, None, None] + (20 * np.cos(5 * y)[:, None] + 45 * np.sin(4 * z)[None, :])[None]
    return np.asfortranarray(v.clip(0 if np.issubdtype(dt, np.unsignedinteger) else -120, 120).astype(dt))


def on_device(torch, A, skip):
    """A on the GPU, `skip` samples into a buffer."""
    raw = np.ascontiguousarray(A.transpose(2, 1, 0))
    buf = torch.zeros((A.size + skip) * A.itemsize, dtype=torch.uint8, device='cuda')
    part = buf[skip * A.itemsize:]
    part.copy_(torch.from_numpy(raw.view(np.uint8).reshape(-1)))
    dt = getattr(torch, A.dtype.name)
    if skip == 0:
        return part.view(dt).view(raw.shape).permute(2, 1, 0)
    whole = torch.zeros(A.size + skip, dtype=dt, device='cuda')
    t = whole[skip:].view(raw.shape)
    t.copy_(part.clone().view(dt).view(raw.shape))
    return t.permute(2, 1, 0)


def planes(torch, dt, nx, ny):
    """Planes of z that give k_bits its 16-byte form, with a partial last word."""
    V, sms = 16 // np.dtype(dt).itemsize, torch.cuda.get_device_properties(0).multi_processor_count
    words = -(-2 * sms // (nx * ny // (256 * V)))
    return 32 * words + 7


@pytest.mark.parametrize('dt', TYPES, ids=lambda d: np.dtype(d).name)
def test_vector_and_scalar_loads_match_the_oracle(pkg, oracle, cuda, dt):
    torch = cuda
    m, r = pkg.MarchingCubes(iso=ISO), (R, R, R)
    nz = planes(torch, dt, 512, 256)
    A = field((512, 256, nz), dt)
    odd = np.asfortranarray(A[1:, :255])  # 511 x 255 samples a plane
    assert (odd.shape[0] * odd.shape[1] * odd.itemsize) % 16
    vols = []
    for B, skip in ((A, 0), (A, 1), (odd, 0)):
        t = on_device(torch, B, skip)
        assert (t.data_ptr() % 16 == 0) == (skip == 0)
        v, f = pkg.isosurface(t, m, *r)
        wv, wf = oracle.isosurface(B, 'mc', ISO, np.float32(1e-3), r)
        assert len(wf) > 10000
        assert np.array_equal(f.cpu().numpy(), wf), skip
        assert v.cpu().numpy().dtype == wv.dtype and np.array_equal(v.cpu().numpy().view(np.uint8), wv.view(np.uint8)), skip
        vols.append((t, v, f))
    b = pkg.Batch([t for t, _, _ in vols], m, *r)
    b.count()
    b.run()
    b.sync()
    for i, (_, v, f) in enumerate(vols):
        bv, bf = b.volume(i)
        assert torch.equal(bf, f) and torch.equal(bv, v), i
    b.close()
