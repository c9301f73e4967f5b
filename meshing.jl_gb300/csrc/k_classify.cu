// K1 -- classify: per-cell cube case and per-piece vertex/face counts, for the list
// form of Marching Cubes (k_emit_mc.cu) and the allocation-free entry.
//
// Replaces the classification half of the reference's cell loops
// (src/marching_cubes.jl:40-56, src/marching_tetrahedra.jl:144-157,
// src/common.jl:10-29).  A warp owns a tile of 31 x-cells by WY y-cells and
// walks one z segment; lane l loads sample x0+l of WY+1 sample rows per z
// plane (coalesced rows along x, Julia layout), and one ballot per row turns
// the strict `v < iso` tests of a whole row into a bit mask, from which every
// lane assembles its 8-corner case without further memory traffic.
//
// Outputs: cnt[v|f|a][seg][y][x] (u32) -- vertices first-created, faces emitted
// and active cells of column x,y inside z segment seg -- and one activity byte per
// (z chunk, x tile, y row) that lets the emit kernels skip empty chunks.
#define MESH_TBL static __device__ const
#include "mesh_internal.cuh"
#include "mesh_tables.h"
#include "mesh_case.cuh"

#include <algorithm>

namespace mesh {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int U = 4;     // z planes loaded ahead
constexpr int CWY = WY;  // cell rows per warp tile

// MC corner order (src/marching_cubes.jl:42-49) from the 2-bit (x, x+1) fields
// of rows y/y+1 in planes z/z+1.
__device__ __forceinline__ unsigned mc_case(unsigned a, unsigned b, unsigned c, unsigned d) {
    return (a & 1u) | ((a >> 1) << 1) | ((b >> 1) << 2) | ((b & 1u) << 3) | ((c & 1u) << 4) | ((c >> 1) << 5) |
           ((d >> 1) << 6) | ((d & 1u) << 7);
}
// MT corner order (src/marching_tetrahedra.jl:146-153).
__device__ __forceinline__ unsigned mt_case(unsigned a, unsigned b, unsigned c, unsigned d) {
    return (a & 1u) | ((b & 1u) << 1) | ((b >> 1) << 2) | ((a >> 1) << 3) | ((c & 1u) << 4) | ((d & 1u) << 5) |
           ((d >> 1) << 6) | ((c >> 1) << 7);
}

template <int ALG> __device__ __forceinline__ void load_tables(uint32_t *s_tab) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {
        if (ALG == MESH_ALG_MC) {
            uint64_t t = MC_CASE_VERTS[i];
            s_tab[i] = (uint32_t)((t >> 48) & 15u) | ((uint32_t)((t >> 52) & 7u) << 8);
        } else if (ALG == MESH_ALG_MT) {
            s_tab[i] = MT_TOUCHED[i] | ((uint32_t)MT_CASE_NFACES[i] << 24);
        }
    }
}

// Per-lane running counts of the NR cells (rows) a lane owns, and per-row
// activity of the current z chunk (warp-uniform).
template <int NR> struct Counts {
    uint32_t v[NR], f[NR], a[NR], act[NR];
};

// One z step: the cells between the sample planes whose row masks are mlo
// (plane z) and mhi (plane z+1).
template <int ALG, int NR>
__device__ __forceinline__ void step(const Plan &p, const uint32_t *s_tab, const uint32_t (&mlo)[NR + 1],
                                     const uint32_t (&mhi)[NR + 1], uint32_t xval, uint32_t cellm, int lane, int xs,
                                     int y0, int zc, Counts<NR> &c) {
    uint32_t all1 = xval, any1 = 0;
#pragma unroll
    for (int r = 0; r <= NR; r++) {
        all1 &= mlo[r] & mhi[r];
        any1 |= mlo[r] | mhi[r];
    }
    // warp-uniform early out: every corner of every cell in this step on one side
    if (all1 == xval || any1 == 0) return;
#pragma unroll
    for (int r = 0; r < NR; r++) {
        // bit l: cell l has corners on both sides (bits l, l+1 of the four masks)
        const uint32_t and4 = mlo[r] & mlo[r + 1] & mhi[r] & mhi[r + 1];
        const uint32_t or4 = mlo[r] | mlo[r + 1] | mhi[r] | mhi[r + 1];
        const uint32_t actm = (or4 | (or4 >> 1)) & ~(and4 & (and4 >> 1)) & cellm;
        if (actm == 0u || y0 + r >= p.cy) continue;  // warp-uniform
        c.act[r] = 1;
        if (!((actm >> lane) & 1u)) continue;
        c.a[r] += 1;
        const unsigned a = (mlo[r] >> lane) & 3u, b = (mlo[r + 1] >> lane) & 3u;
        const unsigned cc = (mhi[r] >> lane) & 3u, d = (mhi[r + 1] >> lane) & 3u;
        const unsigned cm = mc_case(a, b, cc, d);
        if (ALG == MESH_ALG_MC) {
            const uint32_t t = s_tab[cm];
            c.v[r] += t & 15u;
            c.f[r] += t >> 8;
        } else if (ALG == MESH_ALG_MT) {
            const uint32_t t = s_tab[mt_case(a, b, cc, d)];
            const int bnd = (xs + p.xg0 == 0) | ((y0 + r == 0) << 1) | ((zc == 0) << 2);
            c.v[r] += __popc(t & p.own[bnd] & 0x7ffffu);
            c.f[r] += t >> 24;
        } else {  // NSN: one vertex per active cell, a quad per crossed base edge
            c.v[r] += 1;
            const unsigned s0 = cm & 1u;
            const bool yk = y0 + r > 0, zk = zc > 0, xk = xs + p.xg0 > 0;
            unsigned q = 0;
            q += (s0 != ((cm >> 1) & 1u)) && yk && zk;  // +x edge
            q += (s0 != ((cm >> 3) & 1u)) && zk && xk;  // +y edge
            q += (s0 != ((cm >> 4) & 1u)) && xk && yk;  // +z edge
            c.f[r] += 2 * q;
        }
    }
}

// At the end of an activity chunk: publish one byte per tile row.
template <int NR>
__device__ __forceinline__ void chunk_end(const Plan &p, int lane, int tx, int y0, int seg, int zbeg, int zc,
                                          int zend, Counts<NR> &c) {
    if (((zc + 1 - zbeg) % ZC) == 0 || zc + 1 == zend) {
        const int chunk = seg * p.chunks_per_seg + (zc - zbeg) / ZC;
        uint8_t mine = 0;
#pragma unroll
        for (int r = 0; r < NR; r++) {
            if (lane == r) mine = c.act[r] != 0;  // act[] is warp-uniform
            c.act[r] = 0;
        }
        if (lane < NR && y0 + lane < p.cy) p.flags[((int64_t)chunk * p.tiles_x + tx) * p.cy + y0 + lane] = mine;
    }
}

template <int NR>
__device__ __forceinline__ void store_counts(const Plan &p, bool cellx, int xs, int y0, int seg, const Counts<NR> &c) {
    if (!cellx) return;
    const int64_t np = p.pstride;
#pragma unroll
    for (int r = 0; r < NR; r++) {
        if (y0 + r < p.cy) {
            const int64_t i = piece(p, seg, y0 + r, xs);
            p.cnt[i] = c.v[r];
            p.cnt[np + i] = c.f[r];
            p.cnt[2 * np + i] = c.a[r];
        }
    }
}

// The walk below for a warp tile inside the volume (all 32 lanes' samples and
// all WY + 1 rows exist) whose z segment spans fewer than 2^32 samples: no
// per-lane or per-row guards, 32-bit sample offsets from the segment's first
// plane, and each plane's row masks reduced once (AND / OR over the rows) for
// the one-side test of the two steps that use it.  Counts equal the walk
// below; lane 31 (no cell) is left out of the activity bytes and the counts.
template <class T>
__device__ __forceinline__ void classify_tile_mc_inner(const Plan &p, const uint32_t *s_tab, int lane, int tx,
                                                       int ty, int seg) {
    const int xs = tx * TILE_X + lane;
    const int y0 = ty * WY;
    const int zbeg = seg * p.zs;
    const int zend = min(zbeg + p.zs, p.cz);
    const uint32_t sxy = (uint32_t)(p.nx * p.ny), nx = (uint32_t)p.nx;
    const T *base = (const T *)p.vol + (int64_t)sxy * zbeg + xs + p.nx * (int64_t)y0;
    constexpr uint32_t CELLM = 0x7fffffffu;  // lanes 0..30 own cells

    uint32_t cv[WY], cf[WY], ca[WY];
#pragma unroll
    for (int r = 0; r < WY; r++) cv[r] = cf[r] = ca[r] = 0;
    uint32_t mlo[WY + 1];
#pragma unroll
    for (int r = 0; r <= WY; r++) mlo[r] = __ballot_sync(FULL, below(ldv(base + r * nx), p));
    uint32_t alo = mlo[0] & mlo[1] & mlo[2] & mlo[3] & mlo[4], olo = mlo[0] | mlo[1] | mlo[2] | mlo[3] | mlo[4];
    static_assert(WY == 4, "the plane reductions below name rows 0..4");
    uint32_t zoff = 0;  // plane zc0 relative to zbeg

    for (int zc0 = zbeg; zc0 < zend; zc0 += ZC) {
        const int n = min(ZC, zend - zc0);
        uint32_t pk[WY];
#pragma unroll
        for (int r = 0; r < WY; r++) pk[r] = 0;
        for (int u0 = 0; u0 < n; u0 += U) {
            T v[U][WY + 1];
            if (u0 + U <= n) {
#pragma unroll
                for (int u = 0; u < U; u++)
#pragma unroll
                    for (int r = 0; r <= WY; r++) v[u][r] = ldv(base + (zoff + (u + 1) * sxy + r * nx));
            } else {
#pragma unroll
                for (int u = 0; u < U; u++)
#pragma unroll
                    for (int r = 0; r <= WY; r++)
                        v[u][r] = u0 + u < n ? ldv(base + (zoff + (u + 1) * sxy + r * nx)) : T(0);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (u0 + u >= n) break;  // warp-uniform
                uint32_t mhi[WY + 1];
#pragma unroll
                for (int r = 0; r <= WY; r++) mhi[r] = __ballot_sync(FULL, below(v[u][r], p));
                const uint32_t ahi = mhi[0] & mhi[1] & mhi[2] & mhi[3] & mhi[4];
                const uint32_t ohi = mhi[0] | mhi[1] | mhi[2] | mhi[3] | mhi[4];
                if ((alo & ahi) != FULL && (olo | ohi) != 0u) {
                    uint32_t nb[WY + 1];
#pragma unroll
                    for (int r = 0; r <= WY; r++) nb[r] = row_field(mlo[r], mhi[r], lane);
#pragma unroll
                    for (int r = 0; r < WY; r++) pk[r] += s_tab[nb[r] | (nb[r + 1] << 4)];
                }
#pragma unroll
                for (int r = 0; r <= WY; r++) mlo[r] = mhi[r];
                alo = ahi;
                olo = ohi;
            }
            zoff += U * sxy;
        }
        zoff += (uint32_t)(n - (n + U - 1) / U * U) * sxy;  // back to plane zc0 + n after a short chunk
        const int chunk = seg * p.chunks_per_seg + (zc0 - zbeg) / ZC;
        uint32_t mine = 0;  // lane r: the active columns of row y0 + r
#pragma unroll
        for (int r = 0; r < WY; r++) {
            const uint32_t am = __ballot_sync(FULL, pk[r] != 0u) & CELLM;
            if (lane == r) mine = am;
            cv[r] += pk[r] & ((1u << PK_F) - 1u);
            cf[r] += (pk[r] >> PK_F) & ((1u << (PK_A - PK_F)) - 1u);
            ca[r] += pk[r] >> PK_A;
        }
        if (lane < WY) {
            p.flags[((int64_t)chunk * p.tiles_x + tx) * p.cy + y0 + lane] = mine != 0u;
        }
    }
    if (lane >= TILE_X) return;
    const int64_t np = p.pstride;
#pragma unroll
    for (int r = 0; r < WY; r++) {
        const int64_t i = piece(p, seg, y0 + r, xs);
        p.cnt[i] = cv[r];
        p.cnt[np + i] = cf[r];
        p.cnt[2 * np + i] = ca[r];
    }
}

// Marching Cubes walk of warp tile (tx, ty) through z segment seg.  Loads and
// ballots as in classify_tile; a step whose corners are not all on one side
// costs, per cell row, one lookup of the case's packed word (mesh_case.cuh)
// and one add (no branch per row or lane).  The words of an activity chunk
// (ZC planes: at most 12 * ZC vertices, 5 * ZC faces, ZC cells per field) are
// unpacked at the chunk's end, where a non-zero word marks the row active.
template <class T>
__device__ __forceinline__ void classify_tile_mc(const Plan &p, const uint32_t *s_tab, int lane, int tx, int ty,
                                                 int seg) {
    const int xs = tx * TILE_X + lane;
    const int y0 = ty * WY;
    const int zbeg = seg * p.zs;
    const int zend = min(zbeg + p.zs, p.cz);
    const bool cellx = lane < TILE_X && xs < p.cx;
    const T *vol = (const T *)p.vol;
    const int64_t sxy = p.nx * p.ny;

    bool rowok[WY + 1];
    const T *rowp[WY + 1];
#pragma unroll
    for (int r = 0; r <= WY; r++) {
        rowok[r] = xs < p.nx && y0 + r < p.ny;
        rowp[r] = rowok[r] ? vol + xs + p.nx * (int64_t)(y0 + r) : vol;
    }
    uint32_t rmask[WY];  // the lane's cell of row r exists
    uint32_t cv[WY], cf[WY], ca[WY];
#pragma unroll
    for (int r = 0; r < WY; r++) {
        rmask[r] = (cellx && y0 + r < p.cy) ? 0xffffffffu : 0u;
        cv[r] = cf[r] = ca[r] = 0;
    }
    const uint32_t xval = __ballot_sync(FULL, xs < p.nx);
    uint32_t mlo[WY + 1];
#pragma unroll
    for (int r = 0; r <= WY; r++) {
        T v = rowok[r] ? ldv(rowp[r] + sxy * zbeg) : T(0);
        mlo[r] = __ballot_sync(FULL, rowok[r] && below(v, p));
    }

    for (int zc0 = zbeg; zc0 < zend; zc0 += ZC) {
        const int zc1 = min(zc0 + ZC, zend);
        uint32_t pk[WY];
#pragma unroll
        for (int r = 0; r < WY; r++) pk[r] = 0;
        for (int z = zc0; z < zc1; z += U) {
            T v[U][WY + 1];
            const int64_t off = sxy * (int64_t)(z + 1);
            if (z + U <= zc1) {
#pragma unroll
                for (int u = 0; u < U; u++)
#pragma unroll
                    for (int r = 0; r <= WY; r++) v[u][r] = rowok[r] ? ldv(rowp[r] + off + sxy * u) : T(0);
            } else {
#pragma unroll
                for (int u = 0; u < U; u++)
#pragma unroll
                    for (int r = 0; r <= WY; r++)
                        v[u][r] = (rowok[r] && z + 1 + u <= zc1) ? ldv(rowp[r] + off + sxy * u) : T(0);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (z + u >= zc1) break;  // warp-uniform
                uint32_t mhi[WY + 1];
                uint32_t all1 = xval, any1 = 0;
#pragma unroll
                for (int r = 0; r <= WY; r++) {
                    mhi[r] = __ballot_sync(FULL, rowok[r] && below(v[u][r], p));
                    all1 &= mlo[r] & mhi[r];
                    any1 |= mlo[r] | mhi[r];
                }
                // warp-uniform early out: every corner of every cell of this step on one side
                if (all1 != xval && any1 != 0u) {
                    uint32_t nb[WY + 1];
#pragma unroll
                    for (int r = 0; r <= WY; r++) nb[r] = row_field(mlo[r], mhi[r], lane);
#pragma unroll
                    for (int r = 0; r < WY; r++) pk[r] += s_tab[nb[r] | (nb[r + 1] << 4)] & rmask[r];
                }
#pragma unroll
                for (int r = 0; r <= WY; r++) mlo[r] = mhi[r];
            }
        }
        const int chunk = seg * p.chunks_per_seg + (zc0 - zbeg) / ZC;
        uint32_t mine = 0;  // lane r: the active columns of row y0 + r (pk holds existing cells only)
#pragma unroll
        for (int r = 0; r < WY; r++) {
            const uint32_t am = __ballot_sync(FULL, pk[r] != 0u);
            if (lane == r) mine = am;
            cv[r] += pk[r] & ((1u << PK_F) - 1u);
            cf[r] += (pk[r] >> PK_F) & ((1u << (PK_A - PK_F)) - 1u);
            ca[r] += pk[r] >> PK_A;
        }
        if (lane < WY && y0 + lane < p.cy) {
            p.flags[((int64_t)chunk * p.tiles_x + tx) * p.cy + y0 + lane] = mine != 0u;
        }
    }
    if (!cellx) return;
    const int64_t np = p.pstride;
#pragma unroll
    for (int r = 0; r < WY; r++) {
        if (y0 + r < p.cy) {
            const int64_t i = piece(p, seg, y0 + r, xs);
            p.cnt[i] = cv[r];
            p.cnt[np + i] = cf[r];
            p.cnt[2 * np + i] = ca[r];
        }
    }
}

// Walk of warp tile (tx, ty) through z segment seg with one coalesced global
// load per lane, row and plane (any layout).
template <class T, int ALG>
__device__ __forceinline__ void classify_tile(const Plan &p, const uint32_t *s_tab, int lane, int tx, int ty, int seg) {
    const int xs = tx * TILE_X + lane;
    const int y0 = ty * CWY;
    const int zbeg = seg * p.zs;
    const int zend = min(zbeg + p.zs, p.cz);
    const bool cellx = lane < TILE_X && xs < p.cx;
    const T *vol = (const T *)p.vol;
    const int64_t sxy = p.nx * p.ny;

    bool rowok[CWY + 1];
    const T *rowp[CWY + 1];
#pragma unroll
    for (int r = 0; r <= CWY; r++) {
        rowok[r] = xs < p.nx && y0 + r < p.ny;
        rowp[r] = rowok[r] ? vol + xs + p.nx * (int64_t)(y0 + r) : vol;
    }
    Counts<CWY> c;
#pragma unroll
    for (int r = 0; r < CWY; r++) c.v[r] = c.f[r] = c.a[r] = c.act[r] = 0;
    // lanes whose sample exists (x < nx): only their bits take part in the uniform test
    const uint32_t xval = __ballot_sync(FULL, xs < p.nx);
    const uint32_t cellm = __ballot_sync(FULL, cellx);
    uint32_t mlo[CWY + 1];
#pragma unroll
    for (int r = 0; r <= CWY; r++) {
        T v = rowok[r] ? ldv(rowp[r] + sxy * zbeg) : T(0);
        mlo[r] = __ballot_sync(FULL, rowok[r] && below(v, p));
    }

    for (int z = zbeg; z < zend; z += U) {
        T v[U][CWY + 1];
        const int64_t off = sxy * (int64_t)(z + 1);
        if (z + U <= zend) {
#pragma unroll
            for (int u = 0; u < U; u++)
#pragma unroll
                for (int r = 0; r <= CWY; r++) v[u][r] = rowok[r] ? ldv(rowp[r] + off + sxy * u) : T(0);
        } else {
#pragma unroll
            for (int u = 0; u < U; u++)
#pragma unroll
                for (int r = 0; r <= CWY; r++)
                    v[u][r] = (rowok[r] && z + 1 + u <= zend) ? ldv(rowp[r] + off + sxy * u) : T(0);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int zc = z + u;
            if (zc >= zend) break;  // warp-uniform
            uint32_t mhi[CWY + 1];
#pragma unroll
            for (int r = 0; r <= CWY; r++) mhi[r] = __ballot_sync(FULL, rowok[r] && below(v[u][r], p));
            step<ALG, CWY>(p, s_tab, mlo, mhi, xval, cellm, lane, xs, y0, zc, c);
#pragma unroll
            for (int r = 0; r <= CWY; r++) mlo[r] = mhi[r];
            chunk_end(p, lane, tx, y0, seg, zbeg, zc, zend, c);
        }
    }
    store_counts(p, cellx, xs, y0, seg, c);
}

template <class T, int ALG>
__global__ void __launch_bounds__(256, 3) k_classify(const Plan p) {
    __shared__ uint32_t s_tab[256];
    if (ALG == MESH_ALG_MC)
        load_tables_mc_packed(s_tab);
    else
        load_tables<ALG>(s_tab);
    __syncthreads();
    const int ty = blockIdx.y * WARPS + (threadIdx.x >> 5);
    if (ty * CWY >= p.cy) return;  // warp-uniform
    if (ALG == MESH_ALG_MC) {
        if (tile_inner(p, blockIdx.x, ty, blockIdx.z))
            classify_tile_mc_inner<T>(p, s_tab, threadIdx.x & 31, blockIdx.x, ty, blockIdx.z);
        else
            classify_tile_mc<T>(p, s_tab, threadIdx.x & 31, blockIdx.x, ty, blockIdx.z);
    } else
        classify_tile<T, ALG>(p, s_tab, threadIdx.x & 31, blockIdx.x, ty, blockIdx.z);
}

template <class T> cudaError_t launch_t(const Plan &p, cudaStream_t s) {
    const int ty = (p.cy + CWY - 1) / CWY;  // warp tiles of the load walk along y
    dim3 grid(p.tiles_x, (ty + WARPS - 1) / WARPS, p.nseg);
    switch (p.alg) {
    case MESH_ALG_MC: k_classify<T, MESH_ALG_MC><<<grid, 32 * WARPS, 0, s>>>(p); break;
    case MESH_ALG_MT: k_classify<T, MESH_ALG_MT><<<grid, 32 * WARPS, 0, s>>>(p); break;
    default: k_classify<T, MESH_ALG_NSN><<<grid, 32 * WARPS, 0, s>>>(p); break;
    }
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_classify(const Plan &p, cudaStream_t s) {
    switch (p.T) {
    case MESH_DT_U16: return launch_t<uint16_t>(p, s);
    case MESH_DT_F16: return launch_t<h16>(p, s);
    case MESH_DT_I16: return launch_t<int16_t>(p, s);
    case MESH_DT_I8: return launch_t<int8_t>(p, s);
    case MESH_DT_U8: return launch_t<uint8_t>(p, s);
    case MESH_DT_F32: return launch_t<float>(p, s);
    case MESH_DT_I32: return launch_t<int32_t>(p, s);
    case MESH_DT_I64: return launch_t<int64_t>(p, s);
    default: return launch_t<double>(p, s);
    }
}

}  // namespace mesh
