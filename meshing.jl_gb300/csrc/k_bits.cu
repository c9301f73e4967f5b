// Sign bits, piece counts and piece offsets (single volumes and batches).
//
// Replaces the classification half of the reference's cell loops
// (src/marching_cubes.jl:40-56, src/marching_tetrahedra.jl:144-157,
// src/common.jl:10-29) and the running `length(vts)` that numbers their output.
//
//   k_bits     reads every sample once: a lane walks 32 z samples of its
//              column(s) and packs the strict `v < iso` tests into words
//              (mesh_bits.cuh).  4.8 warp instructions per 32 Float32 samples in
//              the 16-byte form, so the volume streams at the memory's rate.
//   k_count    a lane owns a column of cells and walks its words of z: eight
//              words (four corner columns, at z and z + 1) give the active
//              cells of 32 planes with a few logic instructions, and
//              vertices, triangles and quads of 32 cells are counted at a time
//              with population counts.  The last
//              CTA to finish scans the tiles' sums and leaves the totals.
//   k_offsets  turns the counts of a tile into offsets within it, in place.
//
// Measured (Float32 1024^3): bits 0.606 ms = 7.1 TB/s of volume, bound by HBM;
// counts 0.148 ms, bound by issue (a word of 32 x 32 cells costs about 25
// instructions when nothing crosses it, 150 when something does); tiles and offsets
// 18 us.  They replaced a walk that classified the volume step by step (0.763 ms,
// bound by issue) and a four-kernel scan of three counters (35 us; 39 us at 256^3,
// where the counts take 15 us and tiles and offsets 9).  A batch of 1024 volumes of
// 16..128 samples an axis: bits 0.243 ms (6.2 TB/s), counts 0.140, tiles and offsets
// 0.023, against 0.453 + 0.144 for the batched walk and scan.
#define MESH_TBL static constexpr
#include "mesh_internal.cuh"
#include "mesh_tables.h"
#include "mesh_bits.cuh"
#include "mesh_nodes.cuh"

#include <algorithm>

namespace mesh {

namespace {

constexpr unsigned FULL = 0xffffffffu;

// ---- sign bits ----

template <class T, int V> struct alignas(sizeof(T) * V) Vec {
    T v[V];
};
template <class T, int V> __device__ __forceinline__ Vec<T, V> load_vec(const T *p) {
    static_assert(sizeof(T) * V == 16, "16-byte loads");
    const uint4 u = __ldcs(reinterpret_cast<const uint4 *>(p));
    Vec<T, V> r;
    memcpy(&r, &u, 16);
    return r;
}
template <class T, int V> struct Loader {
    static __device__ __forceinline__ Vec<T, V> get(const T *p) { return load_vec<T, V>(p); }
};
template <class T> struct Loader<T, 1> {
    static __device__ __forceinline__ Vec<T, 1> get(const T *p) { return Vec<T, 1>{{ldv(p)}}; }
};

// Words of V consecutive samples (i .. i + V - 1 of a plane) at word zw: the
// planes 32 zw .. that exist, U loads in flight.
template <class T, int V>
__device__ __forceinline__ void pack_words(const Plan &p, const T *src, int64_t sxy, int n, uint32_t (&w)[V]) {
    constexpr int U = V == 1 ? 32 / (sizeof(T) > 4 ? 2 : 1) : 8;
#pragma unroll
    for (int k = 0; k < V; k++) w[k] = 0;
    for (int j0 = 0; j0 < n; j0 += U) {
        Vec<T, V> v[U];
        if (j0 + U <= n) {
#pragma unroll
            for (int u = 0; u < U; u++) v[u] = Loader<T, V>::get(src + u * sxy);
        } else {
#pragma unroll
            for (int u = 0; u < U; u++) v[u] = Loader<T, V>::get(src + (j0 + u < n ? u : 0) * sxy);
        }
        src += U * sxy;
#pragma unroll
        for (int k = 0; k < V; k++) {
            uint32_t b = 0;
#pragma unroll
            for (int u = 0; u < U; u++) b |= below(v[u].v[k], p) ? 1u << u : 0u;
            w[k] |= b << j0;
        }
    }
    if (n < 32) {
#pragma unroll
        for (int k = 0; k < V; k++) w[k] &= (1u << n) - 1u;
    }
}

template <int V> __device__ __forceinline__ void put_words(uint32_t *o, const uint32_t (&w)[V]) {
    if (V == 1) {
        o[0] = w[0];
    } else if (V == 2) {
        *reinterpret_cast<uint2 *>(o) = make_uint2(w[0], w[V - 1]);
    } else {
#pragma unroll
        for (int k = 0; k < V; k += 4)
            *reinterpret_cast<uint4 *>(o + k) = make_uint4(w[k], w[(k + 1) % V], w[(k + 2) % V], w[(k + 3) % V]);
    }
}

// Thread t of nt: the counters of a new extraction.
__device__ __forceinline__ void clear_counters(const Plan &p, int64_t t, int64_t nt) {
    for (int64_t k = t; k < p.ntiles; k += nt) p.tsum[k] = make_ulonglong2(0ull, 0ull);
    if (t < NCNT) p.totals[t] = 0;
    if (t < WORK_SLOTS) p.work[2 * t] = 0u;
    if (t == 0) {
        *p.err = 0u;
        *p.done = 0u;
    }
}

// CTA b < nib * nw: 256 V consecutive samples of a plane in word w0 + b / nib;
// the CTAs after those fill the coordinate tables and clear the counters.
template <class T, int V>
__global__ void __launch_bounds__(256) k_bits(const Plan p, int64_t nib, int w0, int nw, const TabArgs ta) {
    const int64_t nb = nib * nw;
    if ((int64_t)blockIdx.x >= nb) {
        const int64_t t = ((int64_t)blockIdx.x - nb) * 256 + threadIdx.x, nt = ((int64_t)gridDim.x - nb) * 256;
        clear_counters(p, t, nt);
        const int64_t ntab = ta.nx + ta.ny + ta.nz;
        for (int64_t k = t; k < ntab; k += nt)
            table_entry(ta.tabs, k, ta.nx, ta.ny, ta.nz, ta.range[0], ta.range[1], ta.range[2], ta.range[3],
                        ta.range[4], ta.range[5], ta.L32, ta.xoff, ta.nxt);
        return;
    }
    const int zw = w0 + (int)((int64_t)blockIdx.x / nib);
    const int64_t i = ((int64_t)blockIdx.x % nib) * (256 * V) + (int64_t)threadIdx.x * V;
    const int64_t sxy = p.nx * p.ny;
    if (i >= sxy) return;
    uint32_t w[V];
    pack_words<T, V>(p, (const T *)p.vol + (int64_t)zw * 32 * sxy + i, sxy, (int)min((int64_t)32, p.nz - 32 * (int64_t)zw), w);
    put_words<V>(p.bits + (int64_t)(zw - p.bw0) * sxy + i, w);
}

// Batch: the CTAs of volume v pack its planes as above (Plan::bblk_vol names the
// volume); the CTAs after all of them clear the counters.  (Tables filled here as
// well took 12 more registers and 15% of the rate.)
template <class T> __global__ void __launch_bounds__(256) k_bits_batch(const Plan p) {
    if ((int64_t)blockIdx.x >= p.nbblk) {
        clear_counters(p, ((int64_t)blockIdx.x - p.nbblk) * 256 + threadIdx.x, ((int64_t)gridDim.x - p.nbblk) * 256);
        return;
    }
    const BatchVol &b = p.bvols[p.bblk_vol[blockIdx.x]];
    constexpr int V = 16 / sizeof(T);
    const int64_t sxy = b.nx * b.ny, step = b.vec ? 256 * V : 256, nib = (sxy + step - 1) / step;
    const int64_t k = (int64_t)blockIdx.x - b.bblk0;
    const int zw = (int)(k / nib), n = (int)min((int64_t)32, b.nz - 32 * (int64_t)zw);
    const int64_t i = (k % nib) * step + (int64_t)threadIdx.x * (b.vec ? V : 1);
    if (i >= sxy) return;
    const T *src = (const T *)b.vol + (int64_t)zw * 32 * sxy + i;
    uint32_t *dst = p.bits + b.bits0 + (int64_t)zw * sxy + i;
    if (b.vec) {
        uint32_t w[V];
        pack_words<T, V>(p, src, sxy, n, w);
        put_words<V>(dst, w);
    } else {
        uint32_t w[1];
        pack_words<T, 1>(p, src, sxy, n, w);
        dst[0] = w[0];
    }
}

// ---- piece counts ----

// Marching Cubes counts without a look-up per cell.  A cell has a vertex on each
// crossed edge, and its triangles fan the closed loops through them, so it has
// vertices - 2 loops faces.  All cases but those below have one loop, so a word's
// counts are population counts; only the cells of these cases are looked up:
// a face whose diagonals are on different sides, or two opposite corners alone.
__device__ __forceinline__ uint32_t split_face(uint32_t p, uint32_t q, uint32_t r, uint32_t s) {  // cyclic order
    return ~(p ^ r) & ~(q ^ s) & (p ^ q);
}
__device__ __forceinline__ uint32_t lone_pair(uint32_t i, uint32_t j, uint32_t k, uint32_t l, uint32_t m, uint32_t n,
                                              uint32_t o, uint32_t p) {  // i, j alone against the six others
    return (i & j & ~(k | l | m | n | o | p)) | (~(i | j) & (k & l & m & n & o & p));
}
__device__ __forceinline__ uint32_t many_loops(const Corners &q) {
    return split_face(q.a, q.b, q.d, q.c) | split_face(q.as, q.bs, q.ds, q.cs) | split_face(q.a, q.b, q.bs, q.as) |
           split_face(q.c, q.d, q.ds, q.cs) | split_face(q.a, q.c, q.cs, q.as) | split_face(q.b, q.d, q.ds, q.bs) |
           lone_pair(q.a, q.ds, q.b, q.c, q.d, q.as, q.bs, q.cs) | lone_pair(q.b, q.cs, q.a, q.c, q.d, q.as, q.bs, q.ds) |
           lone_pair(q.c, q.bs, q.a, q.b, q.d, q.as, q.cs, q.ds) | lone_pair(q.d, q.as, q.a, q.b, q.c, q.bs, q.cs, q.ds);
}
// loops - 1 of a cell, by cell index (mesh_bits.cuh)
struct LoopTab {
    uint8_t extra[256];
};
constexpr int case_loops(int c) {
    const uint64_t v = MC_CASE_VERTS[c];
    return ((int)((v >> 48) & 15u) - (int)((v >> 52) & 7u)) / 2;
}
constexpr LoopTab make_loop_tab() {
    LoopTab t{};
    for (int i = 0; i < 256; i++) {
        const int l = case_loops((int)mc_case_of_bits((unsigned)i));
        t.extra[i] = (uint8_t)(l > 0 ? l - 1 : 0);
    }
    return t;
}
constexpr bool one_loop_cases_hold() {
    constexpr int F[6][4] = {{0, 1, 2, 3}, {4, 5, 6, 7}, {0, 1, 5, 4}, {1, 2, 6, 5}, {2, 3, 7, 6}, {3, 0, 4, 7}};
    constexpr int D[4] = {0, 1, 2, 3}, E[4] = {6, 7, 4, 5};
    constexpr int EA[12] = {0, 1, 2, 3, 4, 5, 6, 7, 0, 1, 2, 3}, EB[12] = {1, 2, 3, 0, 5, 6, 7, 4, 4, 5, 6, 7};
    for (int c = 1; c < 255; c++) {
        int crossed = 0;
        for (int e = 0; e < 12; e++) crossed += ((c >> EA[e]) ^ (c >> EB[e])) & 1;
        const uint64_t v = MC_CASE_VERTS[c];
        const int nv = (int)((v >> 48) & 15u), nf = (int)((v >> 52) & 7u);
        if (nv != crossed || (nv - nf) % 2 || case_loops(c) < 1) return false;
        bool many = false;
        for (int f = 0; f < 6; f++) {
            const int p = (c >> F[f][0]) & 1, q = (c >> F[f][1]) & 1, r = (c >> F[f][2]) & 1, s = (c >> F[f][3]) & 1;
            many = many || (p == r && q == s && p != q);
        }
        for (int k = 0; k < 4; k++) {
            const int m = (1 << D[k]) | (1 << E[k]);
            many = many || c == m || c == (255 ^ m);
        }
        if (!many && case_loops(c) != 1) return false;
    }
    return true;
}
static_assert(one_loop_cases_hold(), "the counts of the one-loop cases follow from their crossed edges");
__device__ const LoopTab d_loops = make_loop_tab();

// Marching Tetrahedra: the corner words of a cell in MT corner order.
struct MtWords {
    uint32_t w[8];
    __device__ __forceinline__ explicit MtWords(const Corners &c) : w{c.a, c.c, c.d, c.b, c.as, c.cs, c.ds, c.bs} {}
};
// The axes (bit 0 x, 1 y, 2 z) on which both corners of edge e sit at 0.
constexpr int mt_low_axes(int e) {
    int m = 0;
    for (int k = 0; k < 3; k++)
        if (MT_CORNER_POS[MT_EDGE_CORNERS[e][0]][k] == 0 && MT_CORNER_POS[MT_EDGE_CORNERS[e][1]][k] == 0) m |= 1 << k;
    return m;
}
struct MtEdges {
    uint8_t a[19], b[19], low[19];
};
constexpr MtEdges make_mt_edges() {
    MtEdges t{};
    for (int e = 0; e < 19; e++) {
        t.a[e] = MT_EDGE_CORNERS[e][0];
        t.b[e] = MT_EDGE_CORNERS[e][1];
        t.low[e] = (uint8_t)mt_low_axes(e);
    }
    return t;
}
constexpr MtEdges MT_E = make_mt_edges();

// The six tetrahedra (src/lut/mt.jl, subTets) on the MT corners.
constexpr uint8_t TETS[6][4] = {{0, 2, 1, 6}, {0, 7, 3, 6}, {0, 3, 2, 6}, {0, 1, 5, 6}, {0, 4, 7, 6}, {0, 5, 4, 6}};

// Triangles of tetrahedra T.. of the cells zm: one where one corner is cut off, two
// where the corners split in pairs.
template <int T> __device__ __forceinline__ uint32_t mt_triangles(const uint32_t (&w)[8], uint32_t zm) {
    constexpr int i0 = TETS[T][0], i1 = TETS[T][1], i2 = TETS[T][2], i3 = TETS[T][3];
    const uint32_t mixed = (w[i0] | w[i1] | w[i2] | w[i3]) & ~(w[i0] & w[i1] & w[i2] & w[i3]) & zm;
    const uint32_t n = __popc(mixed) + __popc(mixed & ~(w[i0] ^ w[i1] ^ w[i2] ^ w[i3]));
    if constexpr (T + 1 < 6) return n + mt_triangles<T + 1>(w, zm);
    return n;
}

// Welded Marching Cubes: the nine edges that only cells on the lower faces own, as
// pairs of corner words in MT corner order (the other three end at corner 6).
struct McLow {
    uint8_t a[9], b[9], low[9];
};
constexpr McLow make_mc_low() {
    McLow t{};
    constexpr int EA[12] = {0, 1, 3, 2, 4, 5, 7, 6, 0, 1, 3, 2}, EB[12] = {1, 3, 2, 0, 5, 7, 6, 4, 4, 5, 7, 6};
    constexpr int WORD[8] = {0, 3, 1, 2, 4, 7, 5, 6};  // corner x | y << 1 | z << 2
    int n = 0;
    for (int e = 0; e < 12; e++) {
        const int low = 7 & ~(EA[e] | EB[e]);
        if (!low) continue;
        t.a[n] = (uint8_t)WORD[EA[e]];
        t.b[n] = (uint8_t)WORD[EB[e]];
        t.low[n++] = (uint8_t)low;
    }
    return t;
}
constexpr McLow MC_LOW = make_mc_low();
template <int K> __device__ __forceinline__ uint32_t mc_boundary(const uint32_t (&w)[8], uint32_t zm, uint32_t z0, int low) {
    constexpr int la = MC_LOW.low[K], ea = MC_LOW.a[K], eb = MC_LOW.b[K];
    const uint32_t r = (la & ~low & 3) ? 0u : __popc((w[ea] ^ w[eb]) & ((la & 4) ? z0 : zm));
    if constexpr (K + 1 < 9) return r + mc_boundary<K + 1>(w, zm, z0, low);
    return r;
}

template <int E> __device__ __forceinline__ uint32_t mt_owned(const uint32_t (&w)[8], uint32_t zm, uint32_t z0, int low) {
    // edge E of the cells zm, owned when its low axes are grid boundaries
    constexpr int la = MT_E.low[E], ea = MT_E.a[E], eb = MT_E.b[E];
    if (la & ~low & 3) return 0u;
    return __popc((w[ea] ^ w[eb]) & ((la & 4) ? z0 : zm));
}
template <int E> __device__ __forceinline__ uint32_t mt_boundary(const uint32_t (&w)[8], uint32_t zm, uint32_t z0, int low) {
    constexpr bool shared = MT_E.low[E] != 0;
    const uint32_t r = shared ? mt_owned<E>(w, zm, z0, low) : 0u;
    if constexpr (E + 1 < 19) return r + mt_boundary<E + 1>(w, zm, z0, low);
    return r;
}

// The tiles' sums (and the totals), scanned by one CTA of W warps.
template <int W> __device__ __forceinline__ void scan_tiles(const Plan &p, unsigned long long (*s_w)[W]) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int per = (p.ntiles + 32 * W - 1) / (32 * W);
    const int k0 = min(p.ntiles, tid * per), k1 = min(p.ntiles, k0 + per);
    unsigned long long sv = 0, sf = 0;
    for (int k = k0; k < k1; k++) {
        sv += __ldcg(&p.tsum[k].x);
        sf += __ldcg(&p.tsum[k].y);
    }
    unsigned long long iv = sv, jf = sf;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long u = __shfl_up_sync(FULL, iv, o), t = __shfl_up_sync(FULL, jf, o);
        if (lane >= o) {
            iv += u;
            jf += t;
        }
    }
    if (lane == 31) {
        s_w[0][w] = iv;
        s_w[1][w] = jf;
    }
    __syncthreads();
    unsigned long long bv = 0, bf = 0, tv = 0, tf = 0;
#pragma unroll
    for (int k = 0; k < W; k++) {
        if (k < w) {
            bv += s_w[0][k];
            bf += s_w[1][k];
        }
        tv += s_w[0][k];
        tf += s_w[1][k];
    }
    bv += iv - sv;
    bf += jf - sf;
    for (int k = k0; k < k1; k++) {
        const unsigned long long u = __ldcg(&p.tsum[k].x), t = __ldcg(&p.tsum[k].y);
        p.tsum[k] = make_ulonglong2(bv, bf);
        bv += u;
        bf += t;
    }
    if (tid == 0) {
        p.totals[0] = (int64_t)tv;
        p.totals[1] = (int64_t)tf;
        if (p.tot_out) {
            p.tot_out[0] = (int64_t)tv;
            p.tot_out[1] = (int64_t)tf;
        }
    }
}

// Item: 32 columns (x) by BROW rows of up to gs z segments (of seg0 .. seg1 - 1; the
// batches' items are one segment each, Plan::cblk_vol names their volume); warp =
// row, lane = column; a CTA takes one item.  Where one wave of CTAs holds an
// extraction, each reports when its sums have arrived and the last of the `all`
// CTAs scans the tiles' sums; else (all 0) that is a launch of its own, since the
// wait costs every CTA of a large grid more.
template <int ALG, bool BATCH>
__global__ void __launch_bounds__(32 * BROW) k_count(const Plan p, int seg0, int seg1, int gs, unsigned all, bool vpre_only) {
    __shared__ __align__(4) uint8_t s_loops[256];
    __shared__ uint2 s_c[BCOL][BROW + 1];
    __shared__ unsigned long long s_w[2][BROW];
    __shared__ int s_last;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (ALG == MESH_ALG_MC || ALG == MESH_ALG_MC_WELDED) {
        s_loops[tid] = d_loops.extra[tid];
        static_assert(32 * BROW == 256, "one entry per thread");
        __syncthreads();
    }
    after_previous();
    BView v;
    unsigned blk = blockIdx.x;
    if constexpr (BATCH) {
        const BatchVol &b = p.bvols[p.cblk_vol[blk]];
        v = view_of(p, b);
        blk -= (unsigned)b.cblk0;
    } else {
        v = view_of(p);
    }
    const int xb = (int)(blk % v.nxb);
    const int sa = seg0 + (int)((blk / v.nxb) / v.nyb) * gs, sb = min(sa + gs, BATCH ? v.nseg : seg1);
    const int yb = (int)((blk / v.nxb) % v.nyb);
    const int x = xb * BCOL + lane, y = yb * BROW + w;
    uint32_t nv = 0, nf = 0, tv = 0, tf = 0;  // of the segment, of the item's column
    if (y < v.cy) {
        const bool xin = x < v.cx;
        const int ncw = (v.cz + 31) / 32, zw0 = sa * v.zws, zw1 = min(sb * v.zws, ncw);
        int seg = sa, zs0 = zw0, zs1 = min(zs0 + v.zws, ncw);  // the segment and its words
        const uint32_t *r0 = v.bits + (int64_t)(zw0 - v.bw0) * v.sxy + v.nx * y + min(x, v.cx - 1);
        const uint32_t *r1 = r0 + v.nx;
        uint32_t mask = 0;
        // corner columns at word zw (index 0) and the U words after it, in flight together
        constexpr int U = 4;
        uint32_t a[U + 1], b[U + 1], c[U + 1], d[U + 1];
        a[0] = r0[0];
        b[0] = r0[1];
        c[0] = r1[0];
        d[0] = r1[1];
        bool before = true;  // the word before has active cells, or is another segment's
        uint32_t *vp = ALG == MESH_ALG_MC ? nullptr : p.vpre + (int64_t)(zw0 - v.bw0) * v.sxy + v.nx * y + x;
        for (int zb = zw0; zb < zw1; zb += U) {
#pragma unroll
            for (int k = 1; k <= U; k++) {
                const bool in = zb + k < v.nzw && zb + k <= zw1;
                r0 += v.sxy;
                r1 += v.sxy;
                a[k] = in ? r0[0] : 0u;
                b[k] = in ? r0[1] : 0u;
                c[k] = in ? r1[0] : 0u;
                d[k] = in ? r1[1] : 0u;
            }
            uint32_t lo_or = a[0] | b[0] | c[0] | d[0], lo_and = a[0] & b[0] & c[0] & d[0];
#pragma unroll
            for (int k = 0; k < U; k++) {
                const int zw = zb + k;
                if (zw >= zw1) break;  // warp-uniform
                const uint32_t hi_or = a[k + 1] | b[k + 1] | c[k + 1] | d[k + 1];
                const uint32_t hi_and = a[k + 1] & b[k + 1] & c[k + 1] & d[k + 1];
                const uint32_t zm = xin ? cell_mask(v.cz, zw) : 0u;
                // cells with corners on both sides
                const uint32_t act = (lo_or | __funnelshift_r(lo_or, hi_or, 1)) &
                                     ~(lo_and & __funnelshift_r(lo_and, hi_and, 1)) & zm;
                lo_or = hi_or;
                lo_and = hi_and;
                const bool any = __any_sync(FULL, act != 0u);
                if (ALG != MESH_ALG_MC && (any || before) && xin) vp[(int64_t)(zw - zw0) * v.sxy] = nv;
                before = any;
                if (any) {
                    mask |= 1u << ((zw - zs0) & 31);
                    const Corners q{a[k], b[k], c[k], d[k], __funnelshift_r(a[k], a[k + 1], 1),
                                    __funnelshift_r(b[k], b[k + 1], 1), __funnelshift_r(c[k], c[k + 1], 1),
                                    __funnelshift_r(d[k], d[k + 1], 1)};
                    if (ALG == MESH_ALG_MC || ALG == MESH_ALG_MC_WELDED) {
                        uint32_t loops = __popc(act);
                        const uint32_t cross = __popc((q.a ^ q.b) & zm) + __popc((q.c ^ q.d) & zm) + __popc((q.a ^ q.c) & zm) +
                                               __popc((q.b ^ q.d) & zm) + __popc((q.as ^ q.bs) & zm) +
                                               __popc((q.cs ^ q.ds) & zm) + __popc((q.as ^ q.cs) & zm) +
                                               __popc((q.bs ^ q.ds) & zm) + __popc((q.a ^ q.as) & zm) +
                                               __popc((q.b ^ q.bs) & zm) + __popc((q.c ^ q.cs) & zm) + __popc((q.d ^ q.ds) & zm);
                        for (uint32_t m = many_loops(q) & zm; m; m &= m - 1)
                            loops += s_loops[cell_index(a[k], b[k], c[k], d[k], a[k + 1], b[k + 1], c[k + 1], d[k + 1],
                                                        __ffs(m) - 1)];
                        nf += cross - 2 * loops;
                        if (ALG == MESH_ALG_MC) {
                            nv += cross;
                        } else {
                            const MtWords m(q);
                            const int low = (x == 0) | ((y == 0) << 1);
                            nv += __popc((q.ds ^ q.cs) & zm) + __popc((q.ds ^ q.bs) & zm) + __popc((q.ds ^ q.d) & zm);
                            if (zw == 0 || __any_sync(FULL, low != 0))
                                nv += mc_boundary<0>(m.w, zm, zw == 0 ? zm & 1u : 0u, low);
                        }
                    } else if (ALG == MESH_ALG_MT) {
                        const MtWords m(q);
                        uint32_t own = 0;
#pragma unroll
                        for (int i = 0; i < 8; i++) own += i == 6 ? 0u : __popc((m.w[i] ^ m.w[6]) & zm);
                        const int low = (x + p.xg0 == 0) | ((y == 0) << 1);
                        if (zw == 0 || __any_sync(FULL, low != 0)) own += mt_boundary<0>(m.w, zm, zw == 0 ? zm & 1u : 0u, low);
                        nv += own;
                        nf += mt_triangles<0>(m.w, zm);
                    } else {
                        nv += __popc(act);
                        const uint32_t zk = zw == 0 ? zm & ~1u : zm;  // cells with a -z neighbour
                        const bool xk = x + p.xg0 > 0, yk = y > 0;
                        uint32_t n = 0;
                        if (yk) n += __popc((q.a ^ q.b) & zk);
                        if (xk) n += __popc((q.a ^ q.c) & zk);
                        if (xk && yk) n += __popc((q.a ^ q.as) & zm);
                        nf += 2 * n;
                    }
                }
                const bool ends = zw + 1 == zs1;
                if (((zw - zs0) & 31) == 31 || ends) {
                    if (lane == 0) p.wmask[bmask(v, seg, y, xb) + ((zw - zs0) >> 5)] = mask;
                    mask = 0;
                }
                if (ends) {
                    if (xin && !vpre_only) p.pc[bpiece(v, seg, y, x)] = make_uint2(nv, nf);
                    tv += nv;
                    tf += nf;
                    nv = nf = 0;
                    before = true;
                    seg++;
                    zs0 = zs1;
                    zs1 = min(zs0 + v.zws, ncw);
                }
            }
            a[0] = a[U];
            b[0] = b[U];
            c[0] = c[U];
            d[0] = d[U];
        }
    }
    if (ALG != MESH_ALG_MC && vpre_only) return;
    s_c[lane][w] = make_uint2(tv, tf);
    __syncthreads();
    {
        // the tiles' sums: the pieces of a column's BROW rows mostly share one
        const int xl = tid / BROW, yl = tid % BROW;
        const int X = xb * BCOL + xl, Y = yb * BROW + yl;
        const bool in = X < v.cx && Y < v.cy;
        const uint2 n = in ? s_c[xl][yl] : make_uint2(0u, 0u);
        const int64_t e0 = bpiece(v, sa, yb * BROW, X), e1 = bpiece(v, sb - 1, min(yb * BROW + BROW, v.cy) - 1, X);
        unsigned long long sv = n.x, sf = n.y;
#pragma unroll
        for (int o = BROW / 2; o; o >>= 1) {
            sv += __shfl_xor_sync(FULL, sv, o, BROW);
            sf += __shfl_xor_sync(FULL, sf, o, BROW);
        }
        if (e0 / BITS_TILE == e1 / BITS_TILE) {
            if (yl == 0 && X < v.cx && (sv | sf)) {
                atomicAdd(&p.tsum[e0 / BITS_TILE].x, sv);
                atomicAdd(&p.tsum[e0 / BITS_TILE].y, sf);
            }
        } else if (in && (n.x | n.y)) {
            for (int q = sa; q < sb; q++) {
                const int64_t e = bpiece(v, q, Y, X);
                const uint2 c = __ldcg(&p.pc[e]);
                atomicAdd(&p.tsum[e / BITS_TILE].x, (unsigned long long)c.x);
                atomicAdd(&p.tsum[e / BITS_TILE].y, (unsigned long long)c.y);
            }
        }
    }
    if (all == 0u) return;
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(p.done, 1u) == all - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    scan_tiles<BROW>(p, s_w);
}

// The tiles' sums to offsets, for grids that do not scan them themselves.
__global__ void __launch_bounds__(1024) k_scan_tiles(const Plan p) {
    __shared__ unsigned long long s_w[2][32];
    after_previous();
    scan_tiles<32>(p, s_w);
}

// ---- piece offsets ----

constexpr int OFF_T = 256, OFF_N = BITS_TILE / OFF_T;  // threads, pieces per thread
static_assert(OFF_N == 8, "four 16-byte loads per thread");

// CTA: one tile.  Offsets within a tile fit 32 bits (the host bounds the samples
// of a segment).
__global__ void __launch_bounds__(OFF_T) k_offsets(const Plan p) {
    __shared__ uint2 s_w[OFF_T / 32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int64_t e0 = (int64_t)blockIdx.x * BITS_TILE + (int64_t)tid * OFF_N;
    after_previous();
    uint4 *q = reinterpret_cast<uint4 *>(p.pc + e0);
    uint2 n[OFF_N];
    if (e0 + OFF_N <= p.npc) {
#pragma unroll
        for (int k = 0; k < OFF_N / 2; k++) {
            const uint4 u = q[k];
            n[2 * k] = make_uint2(u.x, u.y);
            n[2 * k + 1] = make_uint2(u.z, u.w);
        }
    } else {
#pragma unroll
        for (int k = 0; k < OFF_N; k++) n[k] = e0 + k < p.npc ? p.pc[e0 + k] : make_uint2(0u, 0u);
    }
    uint32_t sv = 0, sf = 0;
#pragma unroll
    for (int k = 0; k < OFF_N; k++) {
        const uint2 u = n[k];
        n[k] = make_uint2(sv, sf);
        sv += u.x;
        sf += u.y;
    }
    uint32_t iv = sv, jf = sf;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(FULL, iv, o), t = __shfl_up_sync(FULL, jf, o);
        if (lane >= o) {
            iv += u;
            jf += t;
        }
    }
    if (lane == 31) s_w[w] = make_uint2(iv, jf);
    __syncthreads();
    uint32_t bv = iv - sv, bf = jf - sf;
#pragma unroll
    for (int k = 0; k < OFF_T / 32; k++)
        if (k < w) {
            bv += s_w[k].x;
            bf += s_w[k].y;
        }
    if (e0 + OFF_N <= p.npc) {
#pragma unroll
        for (int k = 0; k < OFF_N / 2; k++)
            q[k] = make_uint4(bv + n[2 * k].x, bf + n[2 * k].y, bv + n[2 * k + 1].x, bf + n[2 * k + 1].y);
    } else {
#pragma unroll
        for (int k = 0; k < OFF_N; k++)
            if (e0 + k < p.npc) p.pc[e0 + k] = make_uint2(bv + n[k].x, bf + n[k].y);
    }
}

__global__ void k_gather_pieces(const Plan p, const GatherIdx g, int64_t *dst) {
    const int i = threadIdx.x;
    if (i >= g.n) return;
    const ulonglong2 t = p.tsum[g.idx[i] / BITS_TILE];
    const uint2 o = p.pc[g.idx[i]];
    dst[2 * i] = (int64_t)(t.x + o.x);
    dst[2 * i + 1] = (int64_t)(t.y + o.y);
}

template <class T, int V>
cudaError_t go_bits(const Plan &p, int w0, int nw, const TabArgs &ta, cudaStream_t s) {
    const int64_t sxy = p.nx * p.ny, nib = (sxy + 256 * V - 1) / (256 * V);
    const int64_t aux = ta.on ? std::min<int64_t>((std::max<int64_t>(ta.nx + ta.ny + ta.nz, p.ntiles) + 255) / 256, 256) : 0;
    const int64_t grid = nib * nw + aux;
    if (grid > 0x7fffffff) return cudaErrorInvalidConfiguration;
    if (grid < 1) return cudaSuccess;
    k_bits<T, V><<<(unsigned)grid, 256, 0, s>>>(p, nib, w0, nw, ta);
    return cudaGetLastError();
}
template <class T> cudaError_t go_bits_t(const Plan &p, int w0, int nw, const TabArgs &ta, int sms, cudaStream_t s) {
    // 16-byte loads need planes on 16-byte boundaries; volumes too small to give every
    // SM two CTAs of them take more and smaller CTAs
    constexpr int V = 16 / sizeof(T);
    const int64_t sxy = p.nx * p.ny;
    if (((uintptr_t)p.vol & 15) == 0 && (sxy * sizeof(T)) % 16 == 0 && sxy / (256 * V) * nw >= 2 * (int64_t)sms)
        return go_bits<T, V>(p, w0, nw, ta, s);
    return go_bits<T, 1>(p, w0, nw, ta, s);
}

}  // namespace

cudaError_t launch_bits(const Plan &p, int w0, int nw, const TabArgs &ta, int sms, cudaStream_t s) {
    switch (p.T) {
    case MESH_DT_U16: return go_bits_t<uint16_t>(p, w0, nw, ta, sms, s);
    case MESH_DT_F16: return go_bits_t<h16>(p, w0, nw, ta, sms, s);
    case MESH_DT_I16: return go_bits_t<int16_t>(p, w0, nw, ta, sms, s);
    case MESH_DT_I8: return go_bits_t<int8_t>(p, w0, nw, ta, sms, s);
    case MESH_DT_U8: return go_bits_t<uint8_t>(p, w0, nw, ta, sms, s);
    case MESH_DT_F32: return go_bits_t<float>(p, w0, nw, ta, sms, s);
    case MESH_DT_I32: return go_bits_t<int32_t>(p, w0, nw, ta, sms, s);
    case MESH_DT_I64: return go_bits_t<int64_t>(p, w0, nw, ta, sms, s);
    default: return go_bits_t<double>(p, w0, nw, ta, sms, s);
    }
}

// CTAs of k_count that 152 SMs hold at once: three an SM at its 70-80 registers (the
// batches' 64 allow four).
constexpr int ONE_WAVE = 456;

template <int ALG, bool BATCH>
static cudaError_t go_count(const Plan &p, int seg0, int nseg, bool vpre_only, cudaStream_t s, int *kernels) {
    const int64_t per = (int64_t)p.nxb * p.nyb;
    // segments to an item: as many as leave 2048 items
    const int gs = BATCH ? 1 : (int)std::max<int64_t>(1, std::min<int64_t>(nseg, per * nseg / 2048));
    const int64_t nitems = BATCH ? p.ncblk : per * ((nseg + gs - 1) / gs);
    const bool one = nitems <= ONE_WAVE && (BATCH || nseg == p.bseg);
    if (nitems > 0x7fffffff) return cudaErrorInvalidConfiguration;
    cudaError_t e = cudaSuccess;
    if (nitems > 0) {
        e = launch_after(k_count<ALG, BATCH>, (unsigned)nitems, 32 * BROW, 0, s, p, seg0, seg0 + nseg, gs,
                         one ? (unsigned)nitems : 0u, vpre_only);
        ++*kernels;
    }
    if (e == cudaSuccess && !one && !vpre_only && (BATCH || seg0 + nseg == p.bseg)) {
        e = launch_after(k_scan_tiles, 1, 1024, 0, s, p);
        ++*kernels;
    }
    return e;
}

cudaError_t launch_count(const Plan &p, int seg0, int nseg, cudaStream_t s, bool vpre_only, int *kernels) {
    if (p.alg == MESH_ALG_MC) return go_count<MESH_ALG_MC, false>(p, seg0, nseg, vpre_only, s, kernels);
    if (p.alg == MESH_ALG_MT) return go_count<MESH_ALG_MT, false>(p, seg0, nseg, vpre_only, s, kernels);
    if (p.alg == MESH_ALG_MC_WELDED) return go_count<MESH_ALG_MC_WELDED, false>(p, seg0, nseg, vpre_only, s, kernels);
    return go_count<MESH_ALG_NSN, false>(p, seg0, nseg, vpre_only, s, kernels);
}

template <class T> static cudaError_t go_bits_batch(const Plan &p, cudaStream_t s) {
    const int64_t grid = p.nbblk + std::min<int64_t>((p.ntiles + 255) / 256 + 1, 64);
    if (grid > 0x7fffffff) return cudaErrorInvalidConfiguration;
    k_bits_batch<T><<<(unsigned)grid, 256, 0, s>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_bits_batch(const Plan &p, cudaStream_t s) {
    switch (p.T) {
    case MESH_DT_U16: return go_bits_batch<uint16_t>(p, s);
    case MESH_DT_F16: return go_bits_batch<h16>(p, s);
    case MESH_DT_I16: return go_bits_batch<int16_t>(p, s);
    case MESH_DT_I8: return go_bits_batch<int8_t>(p, s);
    case MESH_DT_U8: return go_bits_batch<uint8_t>(p, s);
    case MESH_DT_F32: return go_bits_batch<float>(p, s);
    case MESH_DT_I32: return go_bits_batch<int32_t>(p, s);
    case MESH_DT_I64: return go_bits_batch<int64_t>(p, s);
    default: return go_bits_batch<double>(p, s);
    }
}

cudaError_t launch_count_batch(const Plan &p, cudaStream_t s) {
    int kernels = 0;
    return go_count<MESH_ALG_MC, true>(p, 0, 0, false, s, &kernels);
}

cudaError_t launch_offsets(const Plan &p, cudaStream_t s) {
    if (p.ntiles < 1) return cudaSuccess;
    return launch_after(k_offsets, (unsigned)p.ntiles, OFF_T, 0, s, p);
}

cudaError_t launch_gather_pieces(const Plan &p, const GatherIdx &g, int64_t *dst, cudaStream_t s) {
    if (g.n < 1 || 2 * g.n > GATHER_MAX) return cudaErrorInvalidValue;
    k_gather_pieces<<<1, GATHER_MAX, 0, s>>>(p, g, dst);
    return cudaGetLastError();
}

}  // namespace mesh
