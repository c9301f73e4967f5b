"""The engine's work as a user's program has it do, for timing and for comparing outputs.

A case is one call (or one batch, or one burst of served requests) on a seeded synthetic
volume.  The surface (where samples cross the iso value, and so the sizes of the outputs)
belongs to the case, the samples' values to the seed.  `field` names the volume: `sphere` (signed distance), `gyroid` (dense surface),
`sines` (16 random plane waves), `ct` (noisy background with bright shells) and `sdf`
(unions of spheres and boxes).  `call` names the entry point:

  isosurface   the drop-in call on a CUDA volume: sizes its own outputs
  device       isosurface_device into buffers the program keeps, no host round trip
  host         the drop-in call on a host array, host arrays out
  batch        a Batch of uneven volumes, replayed from its CUDA graph
  serve        a burst of mixed requests to a Server, results taken as they end
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

DTYPES = {'f32': torch.float32, 'f64': torch.float64, 'i16': torch.int16, 'u16': torch.uint16}


def _pkg():
    """The package (its folder's name is no module name: loaded from its files)."""
    if 'meshing_gb300' not in sys.modules:
        d = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'meshing.jl_gb300')
        spec = importlib.util.spec_from_file_location('meshing_gb300', os.path.join(d, '__init__.py'),
                                                      submodule_search_locations=[d])
        sys.modules['meshing_gb300'] = mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
    return sys.modules['meshing_gb300']


# ---- cases ------------------------------------------------------------------

def _one(call, alg, field, dtype, nx, ny, nz, single=False):
    """`single`: iso, eps and the ranges are Float32 too, so the whole call is Float32;
    otherwise they are the defaults of a plain call (Float64 iso 0.0 and integer ranges;
    the CT volumes an integer iso of 500)."""
    return {'call': call, 'alg': alg, 'field': field, 'dtype': dtype, 'nx': nx, 'ny': ny, 'nz': nz, 'single': single}


def listed():
    return [
        # a small object meshed once: the latency of the plain call
        dict(_one('isosurface', 'mc', 'sphere', 'f64', 64, 64, 64), name='sphere_f64_64'),
        # a volume that changes every frame, meshed into kept buffers on the frame's stream
        dict(_one('device', 'mc', 'sines', 'f32', 128, 128, 128, True), name='frame_f32_128'),
        # a dense surface, the three algorithms with their default arguments
        dict(_one('isosurface', 'mc', 'gyroid', 'f32', 256, 256, 256), name='gyroid_mc_256'),
        dict(_one('isosurface', 'mt', 'gyroid', 'f32', 256, 256, 256), name='gyroid_mt_256'),
        dict(_one('isosurface', 'nsn', 'gyroid', 'f32', 256, 256, 256), name='gyroid_nsn_256'),
        # a mesh for post-processing: welded vertices, odd sizes
        dict(_one('isosurface', 'weld', 'gyroid', 'f32', 301, 187, 250, True), name='weld_f32_odd'),
        # a scan with an integer threshold
        dict(_one('isosurface', 'mc', 'ct', 'u16', 512, 512, 512), name='ct_u16_512'),
        # a simulation field of odd sizes, shared vertices, all in Float32
        dict(_one('isosurface', 'mt', 'sines', 'f32', 509, 387, 301, True), name='mt_f32_odd'),
        # the largest field
        dict(_one('isosurface', 'mc', 'sines', 'f32', 1024, 1024, 1024, True), name='sines_f32_1024'),
        # thousands of small uneven volumes (a shape data set)
        {'call': 'batch', 'volumes': 1024, 'lo': 16, 'hi': 128, 'dtype': 'f32', 'name': 'batch_1024'},
        # requests of a mixed stream, as they queue up behind a busy device
        {'call': 'serve', 'requests': 28, 'lo': 32, 'hi': 192, 'name': 'serve_28'},
        # the call of a program that keeps its volumes in host memory
        dict(_one('host', 'mc', 'sines', 'f32', 200, 180, 161), name='host_f32_odd'),
    ]


def draw(rng):
    kind = rng.choice(['small', 'frame', 'gyroid', 'weld', 'ct', 'field', 'large', 'batch', 'serve', 'host'])
    size = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    sizes = lambda lo, hi: [size(lo, hi) for _ in range(3)]
    if kind == 'small':
        return _one('isosurface', rng.choice(['mc', 'mt', 'nsn']), 'sphere', rng.choice(['f32', 'f64']), *sizes(20, 110))
    if kind == 'frame':
        return _one('device', 'mc', 'sines', rng.choice(['f32', 'f32', 'f64']), *sizes(64, 256), rng.random() < 0.7)
    if kind == 'gyroid':
        return _one('isosurface', rng.choice(['mc', 'mt', 'nsn']), 'gyroid', rng.choice(['f32', 'f64']), *sizes(100, 360),
                    rng.random() < 0.3)
    if kind == 'weld':
        return _one('isosurface', 'weld', rng.choice(['gyroid', 'sines']), 'f32', *sizes(100, 400), rng.random() < 0.5)
    if kind == 'ct':
        return _one(rng.choice(['isosurface', 'device']), 'mc', 'ct', rng.choice(['u16', 'i16']), *sizes(128, 640))
    if kind == 'field':
        return _one('isosurface', rng.choice(['mc', 'mt', 'nsn']), 'sines', rng.choice(['f32', 'f32', 'f64']),
                    *sizes(150, 600), rng.random() < 0.6)
    if kind == 'large':
        return _one('isosurface', 'mc', 'sines', 'f32', *sizes(600, 1024), rng.random() < 0.7)
    if kind == 'batch':
        lo = rng.randint(8, 40)
        return {'call': 'batch', 'volumes': size(32, 1024), 'lo': lo, 'hi': rng.randint(lo + 8, 128),
                'dtype': rng.choice(['f32', 'f32', 'f64'])}
    if kind == 'serve':
        return {'call': 'serve', 'requests': rng.randint(8, 30), 'lo': 32, 'hi': rng.randint(64, 192)}
    return _one('host', rng.choice(['mc', 'mc', 'mt']), 'sines', rng.choice(['f32', 'f64']), *sizes(64, 220),
                rng.random() < 0.5)


# ---- volumes: (nz, ny, nx) in memory, returned indexed [x, y, z] --------------

def _axes(shape, a, b):
    return [torch.linspace(a, b, n, dtype=torch.float32, device='cuda') for n in shape]


def _waves(shape, rng):
    """sum over 16 terms of a sin(2 pi w.p + phi) on [0, 1]^3, as products of x and y / z factors."""
    d = rng.standard_normal((16, 3))
    w = 2 * math.pi * rng.uniform(1, 8, (16, 1)) * d / np.linalg.norm(d, axis=1, keepdims=True)
    amp, phase = rng.standard_normal(16), rng.uniform(0, 2 * math.pi, 16)
    t = lambda v: torch.as_tensor(v, dtype=torch.float32, device='cuda')
    gx, gy, gz = _axes(shape, 0.0, 1.0)
    w, amp, phase = t(w), t(amp), t(phase)
    ax = gx[:, None] * w[:, 0] + phase
    fx = torch.cat([torch.sin(ax), torch.cos(ax)], 1).t().contiguous()  # (32, nx)
    out = torch.empty(shape[::-1], dtype=torch.float32, device='cuda')
    for k in range(0, shape[2], 64):
        ayz = gy[None, :, None] * w[:, 1] + gz[k:k + 64, None, None] * w[:, 2]
        f = torch.cat([amp * torch.cos(ayz), amp * torch.sin(ayz)], 2)
        torch.matmul(f, fx, out=out[k:k + 64])
    return out


def _solids(shape, rng):
    """Signed distance to the union of 1-8 spheres / boxes on [-1, 1]^3."""
    gx, gy, gz = _axes(shape, -1.0, 1.0)
    f = None
    for _ in range(int(rng.integers(1, 9))):
        c = rng.uniform(-0.6, 0.6, 3)
        x, y, z = gx[None, None, :] - c[0], gy[None, :, None] - c[1], gz[:, None, None] - c[2]
        if rng.integers(0, 2):
            h = rng.uniform(0.05, 0.25, 3)
            x, y, z = x.abs() - h[0], y.abs() - h[1], z.abs() - h[2]
            d = (x.clamp(min=0) ** 2 + y.clamp(min=0) ** 2 + z.clamp(min=0) ** 2).sqrt() + \
                torch.maximum(torch.maximum(x, y), z).clamp(max=0)
        else:
            d = (x * x + y * y + z * z).sqrt() - float(rng.uniform(0.05, 0.3))
        f = d if f is None else torch.minimum(f, d)
    return f


def _volume(field, dtype, shape, seed, k=0):
    """The k-th surface of this field and shape, with samples of this seed."""
    rng = np.random.default_rng((k, *shape))
    if field == 'sines':
        f = _waves(shape, rng)
    elif field == 'gyroid':
        x, y, z = (g + p for g, p in zip(_axes(shape, -3 * math.pi, 3 * math.pi), rng.uniform(0, 2 * math.pi, 3)))
        x, y, z = x[None, None, :], y[None, :, None], z[:, None, None]
        f = torch.sin(x) * torch.cos(y) + torch.sin(y) * torch.cos(z) + torch.sin(z) * torch.cos(x)
    elif field == 'sphere':
        c, r = rng.uniform(-0.1, 0.1, 3), float(rng.uniform(0.35, 0.6))
        x, y, z = (g.double() - o for g, o in zip(_axes(shape, -1.0, 1.0), c))
        f = (x[None, None, :] ** 2 + y[None, :, None] ** 2 + z[:, None, None] ** 2).sqrt() - r
    elif field == 'sdf':
        f = _solids(shape, rng)
    else:  # ct: N(100, 20) noise and three shells about 4 voxels thick of value N(1000, 50)
        f = torch.randn(shape[::-1], generator=torch.Generator(device='cuda').manual_seed(seed), device='cuda') * 20 + 100
        x, y, z = (torch.arange(n, device='cuda', dtype=torch.float32) for n in shape)
        values = np.random.default_rng(seed)
        for _ in range(3):
            c, h = rng.uniform(0.3, 0.7, 3) * shape, rng.uniform(0.1, 0.4, 3) * shape
            q = ((x[None, None, :] - c[0]) / h[0]) ** 2 + ((y[None, :, None] - c[1]) / h[1]) ** 2 + \
                ((z[:, None, None] - c[2]) / h[2]) ** 2
            f.masked_fill_((q.sqrt() - 1).abs() * float(h.min()) < 2.0, float(values.normal(1000, 50)))
        f = f.clamp_(min=0).round_().to(torch.int32)
    if field != 'ct':  # a smooth positive factor of the seed: no sample changes its side of 0
        p = np.random.default_rng(seed).uniform(1, 6, (3, 2))
        gx, gy, gz = (1 + 0.4 * torch.sin(a * g + b) for g, (a, b) in zip(_axes(shape, -1.0, 1.0), p))
        f *= gx
        f *= (gz[:, None] * gy)[..., None]
    return f.to(DTYPES[dtype]).permute(2, 1, 0)


def _params(alg, field, dtype, single):
    """(iso, eps, X range) as a program writes them."""
    if field == 'ct':
        return 500, 1e-3, (-1, 1)
    if single:
        return np.float32(0), np.float32(1e-3), (np.float32(-1), np.float32(1))
    return 0.0, 1e-3, (-1, 1)


def _method(alg, iso, eps):
    m = _pkg()
    if alg == 'mt':
        return m.MarchingTetrahedra(iso=iso, eps=eps)
    return m.NaiveSurfaceNets(iso=iso) if alg == 'nsn' else m.MarchingCubes(iso=iso, weld=alg == 'weld')


def _batch_shapes(case, seed):
    # the sizes belong to the case, the contents to the seed
    rng = np.random.default_rng(case['volumes'])
    shapes = rng.integers(case['lo'], case['hi'] + 1, (case['volumes'], 3))
    return [(tuple(int(n) for n in s), seed * 100003 + i, i) for i, s in enumerate(shapes)]


def _requests(case, seed):
    """Cubic sizes log-uniform, half Float32 and half Float64, 60 / 30 / 10 MC / MT / NSN."""
    rng = np.random.default_rng(case['requests'])
    out = []
    for i in range(case['requests']):
        n = int(round(math.exp(rng.uniform(math.log(case['lo']), math.log(case['hi'])))))
        out.append((rng.choice(['mc', 'mt', 'nsn'], p=[0.6, 0.3, 0.1]), rng.choice(['sines', 'sdf']),
                    rng.choice(['f32', 'f64']), (n, n, n), seed * 100003 + i, i))
    return out


# ---- a pass -------------------------------------------------------------------

def prepare(case, seed):
    m = _pkg()
    s = {'case': case}
    if case['call'] == 'batch':
        vols = [_volume('sdf', case['dtype'], *v) for v in _batch_shapes(case, seed)]
        s['batch'] = m.Batch(vols, m.MarchingCubes(iso=np.float32(0)))
        s['batch'].count()  # sizes the outputs
        s['batch'].set_graph(True)
        return s
    if case['call'] == 'serve':
        s['server'] = m.Server(12 << 30, slots=4)
        s['held'] = []
        s['reqs'] = []
        for alg, field, dtype, *v in _requests(case, seed):
            iso, eps, r = _params(alg, field, dtype, dtype == 'f32')
            s['reqs'].append((_volume(field, dtype, *v), _method(alg, iso, eps), r))
        return s
    shape = (case['nx'], case['ny'], case['nz'])
    iso, eps, r = _params(case['alg'], case['field'], case['dtype'], case['single'])
    A = _volume(case['field'], case['dtype'], shape, seed)
    s.update(A=A, method=_method(case['alg'], iso, eps), r=r)
    if case['call'] == 'host':
        s['A'] = np.asfortranarray(A.cpu().numpy())
    if case['call'] == 'device':  # buffers with room for this surface
        v, f = m.isosurface(A, s['method'], r, r, r)
        s['out'] = (torch.zeros_like(v), torch.zeros_like(f), torch.zeros(2, dtype=torch.int64, device='cuda'))
    return s


def _with(owner, views):
    """The views of a batch's or server's memory, holding their owner as long as they live."""
    for t in views:
        t.owner = owner
    return views


def run(state):
    m, call = _pkg(), state['case']['call']
    if call == 'batch':
        state['batch'].run()
        return _with(state['batch'], state['batch'].outputs())
    if call == 'serve':
        srv = state['server']
        for i in state['held']:  # the results of the burst before: the program is done with them
            srv.release(i)
        ids = state['held'] = [srv.submit(A, method, r, r, r) for A, method, r in state['reqs']]
        return [_with(srv, srv.result(i)) for i in ids]
    A, method, r = state['A'], state['method'], state['r']
    if call == 'device':
        v, f, counts = state['out']
        m.isosurface_device(A, method, r, r, r, verts=v, faces=f, counts=counts)
        return v, f, counts
    return m.isosurface(A, method, r, r, r)


# ---- what a pass cannot do without -------------------------------------------

# vertices and faces of one volume over (nx ny nz)^(2/3), typical of the field
DENSITY = {('mc', 'gyroid'): (57.7, 28.9), ('mt', 'gyroid'): (41.4, 82.5), ('nsn', 'gyroid'): (14.4, 27.8),
           ('weld', 'gyroid'): (14.4, 28.9), ('mc', 'sines'): (65.0, 32.5), ('mt', 'sines'): (47.0, 94.0),
           ('nsn', 'sines'): (16.3, 32.0), ('weld', 'sines'): (16.3, 32.5), ('mc', 'sphere'): (4.3, 2.1),
           ('mt', 'sphere'): (3.2, 6.4), ('nsn', 'sphere'): (1.1, 2.1), ('mc', 'ct'): (30.0, 15.0),
           ('mc', 'sdf'): (4.5, 2.2), ('mt', 'sdf'): (3.4, 6.7), ('nsn', 'sdf'): (1.1, 2.2)}


def _work(alg, field, dtype, shape, vbytes):
    n = shape[0] * shape[1] * shape[2]
    v, f = (d * n ** (2 / 3) for d in DENSITY[alg, field])
    # a comparison per sample; a quotient and a position per vertex
    return n * DTYPES[dtype].itemsize + v * 3 * vbytes + f * 24, n + 12 * v


def work(case):
    if case['call'] == 'batch':
        parts = [_work('mc', 'sdf', case['dtype'], shape, 4 if case['dtype'] == 'f32' else 8)
                 for shape, _, _ in _batch_shapes(case, 0)]
    elif case['call'] == 'serve':
        parts = [_work(alg, field, dtype, shape, 4 if dtype == 'f32' else 8)
                 for alg, field, dtype, shape, _, _ in _requests(case, 0)]
    else:
        small = case['single'] and case['dtype'] == 'f32'
        parts = [_work(case['alg'], case['field'], case['dtype'], (case['nx'], case['ny'], case['nz']), 4 if small else 8)]
    return {'bytes': int(sum(p[0] for p in parts)), 'flops': int(sum(p[1] for p in parts))}


# ---- the vertices in 64 bits, in plain torch ----------------------------------

# cube corners (x, y, z) and edges of Marching Cubes, and per cube case 1..254 its edges in
# the order their vertices are emitted (hex digits)
CORNERS = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]
EDGES = [(0, 1), (1, 2), (2, 3), (3, 0), (4, 5), (5, 6), (6, 7), (7, 4), (0, 4), (1, 5), (2, 6), (3, 7)]
CASE_EDGES = (
    '083 019 1839 12a 08312a 92a0 283a9 3b2 0b28 19023b 1b298 3a1b 0a18b 390ba 98ab 478 4307 019847 '
    '41973 12a847 347012a 92a0847 2a9734 8473b2 b4720 90184723b 47b921 3a1b784 1ba407 47890ba3 47b9a 954 '
    '954083 0541 85431 12a954 30812a495 52a40 2a5348 95423b 0b28495 054123b 2158b4 a3b1954 495081ab '
    '540ba3 548ab 9785 93057 07815 1537 9785a12 a1295037 80257a 2a537 79583b2 95720b 23b01875 b2175 '
    '9587a13b 5709b1a ba03587 ba57 a65 0835a6 9015a6 18395a6 1652 1652308 96502 598263 23ba65 b082a65 '
    '01923b5a6 5a6192b8 63b51 08b516 3b6059 659b8 5a6478 430765a 1905a6847 a6519734 6125478 12563047 '
    '84790562 7394256 3b2784a65 5a64720b 01947823b5a6 921b475a6 8473b516 51b6074 05963b847 659b47 a496 '
    '4a69083 a0164 83164a 14926 30812946 0246 83246 a496b23 082b49a6 3b20164a 641a82b 96431b 8b10694 '
    '3b604 648b 7a689 073a96 a67180 a6713 126897 2691703 78062 7326 23ba6897 207b96a 1807a623b b217a6 '
    '89671b3 091b67 78063b 7b6 76b 308b76 019b76 8193b76 a126b7 12a3086b7 290a6b7 6b72a389 7236 70862 '
    '2763019 162897 a7613 a76180 037a96 76a89 684b 36b04 86b4901 94631b 684b2a1 12a30b64 4b86029a '
    'a9324b6 82346 0426 19023468 19426 81364a a1064 4638a09 a946 49576b 083495b76 501476b b7683451 '
    '954a1276b 6b712a083495 76b54a20 34852ab76 7236549 95408627 36271504 6287145 954a1673 16a708954 '
    '40a5367 76a854 695b8 36b059 0b8516 6b351 12a95b86 0b369512a b8560a2 6b352a 589263 95602 1580632 '
    '1562 136a859 a10695 03856a a56 b5a7 b5a7830 5b7a190 a75b9813 b1275 0831275b 97520b 752b938 25a37 '
    '82057a 9015a372 98217a5 1357 08715 90357 9875 584ab 504ba3 01984ab5 ab45391 2518b4 04b3521 0259b48 '
    '9452b3 25a348 5a240 3a2584019 5a2419 84531 0451 845390 945 4b79a 083497ba 1ab407 3148a7b 4b7921 '
    '974b12083 b7420 b74283 29a734 9a74280 37a2410 1a2874 49173 491708 4037 487 9a8b 309ba 01a8b 31ab '
    '12b98 309b12 02b8 32b 238a9 9a20 238a01 1a2 1389 091 038 ').split()

# Marching Tetrahedra: corners, the six tetrahedra on them, a tetrahedron's edges and per
# tetrahedron case 1..14 its triangles' edges
T_CORNERS = [(0, 0, 0), (0, 1, 0), (1, 1, 0), (1, 0, 0), (0, 0, 1), (0, 1, 1), (1, 1, 1), (1, 0, 1)]
TETS = [(0, 2, 1, 6), (0, 7, 3, 6), (0, 3, 2, 6), (0, 1, 5, 6), (0, 4, 7, 6), (0, 5, 4, 6)]
T_EDGES = [(0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3)]
T_CASES = '023 041 241234 152 053015 045052 345 354 054025 035051 125 214243 014 032'.split()


def _mc_order():
    return [[]] + [[EDGES[int(e, 16)] for e in row] for row in CASE_EDGES] + [[]]


def _mt_order():
    """Per cube case, the edges its triangles use, in the order of their first use; an
    edge runs from its corner with the smaller coordinates to the other."""
    out = []
    for case in range(256):
        seen = []
        for tet in TETS:
            t = sum(((case >> c) & 1) << i for i, c in enumerate(tet))
            for e in ('' if t in (0, 15) else T_CASES[t - 1]):
                a, b = sorted((tet[k] for k in T_EDGES[int(e)]), key=lambda c: (sum(T_CORNERS[c]), c))
                if (a, b) not in seen:
                    seen.append((a, b))
        out.append(seen)
    return out


def _exact_points(A, alg, iso, eps, r):
    """Vertices of volume A (indexed [x, y, z]) as (V, 3) float64."""
    nx, ny, nz = A.shape
    corners = torch.tensor(T_CORNERS if alg == 'mt' else CORNERS, device='cuda')
    order = _mt_order() if alg == 'mt' else [EDGES] * 256 if alg == 'nsn' else _mc_order()
    width = max(len(o) for o in order)
    pad = lambda k: torch.tensor([[e[k] for e in o] + [0] * (width - len(o)) for o in order], device='cuda')
    start, end = pad(0), pad(1)
    used = torch.tensor([[True] * len(o) + [False] * (width - len(o)) for o in order], device='cuda')
    wrap = 65536.0 if A.dtype == torch.uint16 else None
    nodes = [torch.linspace(float(r[0]), float(r[1]), n, dtype=torch.float64, device='cuda') for n in (nx, ny, nz)]
    iso, eps = float(iso), float(eps)
    out = []
    for x0 in range(0, nx - 1, 32):
        S = A[x0:x0 + 33]
        S = (S.to(torch.int32) if wrap else S).contiguous()
        low, cells = S < iso, [n - 1 for n in S.shape]
        case = torch.zeros(cells, dtype=torch.int32, device='cuda')
        for k, (i, j, l) in enumerate(corners.tolist()):
            case |= low[i:i + cells[0], j:j + cells[1], l:l + cells[2]].int() << k
        at = torch.nonzero((case != 0) & (case != 255))  # x outermost, z fastest
        if not len(at):
            continue
        case = case[at.unbind(1)].long()
        c = at[:, None, :] + corners
        vals = S[c.unbind(2)].double()
        a, b, take = start[case], end[case], used[case]
        va, vb = vals.gather(1, a), vals.gather(1, b)
        if alg == 'nsn':
            take = (va < iso) != (vb < iso)
        den = vb - va
        if wrap:  # differences of unsigned samples wrap, as Julia's do
            den = den.remainder(wrap)
        mu = (iso - va) / den
        at = at + torch.tensor([x0, 0, 0], device='cuda')
        pa, pb = corners[a], corners[b]
        if alg in ('mt', 'weld'):
            # the vertex of an edge shared by several cells belongs to the first of them
            on_low = (pa == 0) & (pb == 0)
            take = take & (~on_low | (at == 0)[:, None, :]).all(2)
        if alg == 'mt':
            mu = mu.clamp(eps, 1 - eps)
        if alg == 'nsn':
            mu = torch.where(take, mu, torch.zeros_like(mu))
        p = []
        for k in range(3):
            qa, qb = (nodes[k][at[:, None, k] + o[..., k]] for o in (pa, pb))
            p.append(qa + mu * (qb - qa))
        p = torch.stack(p, 2)
        out.append((p * take[..., None]).sum(1) / take.sum(1)[:, None] if alg == 'nsn' else p[take])
    return torch.cat(out) if out else torch.empty((0, 3), dtype=torch.float64, device='cuda')


def exact(case, seed):
    if case['call'] == 'batch':
        pts = [_exact_points(_volume('sdf', case['dtype'], *v), 'mc', 0.0, 0.0, (-1, 1))
               for v in _batch_shapes(case, seed)]
        return torch.cat(pts), None, None
    if case['call'] == 'serve':
        out = []
        for alg, field, dtype, *v in _requests(case, seed):
            iso, eps, r = _params(alg, field, dtype, dtype == 'f32')
            out.append((_exact_points(_volume(field, dtype, *v), alg, iso, eps, r), None))
        return out
    A = _volume(case['field'], case['dtype'], (case['nx'], case['ny'], case['nz']), seed)
    iso, eps, r = _params(case['alg'], case['field'], case['dtype'], case['single'])
    pts = _exact_points(A, case['alg'], iso, eps, r)
    return (pts, None, None) if case['call'] == 'device' else (pts, None)
