// Marching Cubes emission from the sign bits (single volumes and batches).
//
// Replaces process_mc_voxel! (src/marching_cubes.jl:67-92), vertex_interp
// (:100-104) and mc_vert_points (:111-120): vertices and faces are written
// straight from the volume at the scanned offsets, and only the samples of
// active cells are read.
//
// Work item: 32 columns of one cell row through one z segment, taken by warps
// from a counter (x blocks fastest, then segments, then rows, so the write
// fronts of all columns advance together).  For each word of 32 planes with an
// active cell the warp
//   1. lists its active cells in shared memory: a lane owns a column, finds its
//      cells with logic on eight words and queues them in z order, so the list
//      is in emission order within each column;
//   2. takes the list 32 cells at a time, one cell per lane: the lane fetches
//      the words of its cell's column by shuffle, looks up the case, loads the
//      eight corner samples into shared memory and takes part in one scan of
//      (vertices | faces << 16);
//   3. maps all 32 lanes onto the vertex tasks, then onto the face tasks: the
//      cells' first tasks of a round are collected by a warp reduction, so a
//      population count finds a task's cell and a shuffle fetches its record.
// The cells of one column are consecutive in the emission order, so task t of
// column l goes to G[l] + t, G[l] being the column's next vertex (face) minus
// its first task.  A batch holds 24 to 27 cells on the fields below (the list ends with
// the word); the tasks of each round fill the warp.
//
// Measured (1024^3 Float32, 17 M cells, 1.65 GB of mesh): 0.89 ms, 0.96 for the
// form before it, which walked 8 planes of 31 columns at a time and classified
// them again; 512^3 UInt16 0.35 against 0.42, 256^3 gyroid with Float64 vertices
// 0.126 against 0.163 ms.  Of the 0.89 ms, leaving out the face stores saves 0.20,
// the vertices 0.27, the task look-ups 0.12 and the batch set-up 0.19; leaving out
// the corner loads alone 0.06 (512^3: 950 instructions per batch, 66% of issue).
// Three CTAs per SM: with four (64 registers) it is 4% slower, with five 13%.  A
// batch of 1024 volumes (1.5 GB of samples): 0.383 ms against 0.575 for listing the
// active cells and expanding the list.
#define MESH_TBL static constexpr
#include "mesh_internal.cuh"
#include "mesh_tables.h"
#include "mesh_bits.cuh"
#include "mesh_mc.cuh"

#include <algorithm>
#include <mutex>

namespace mesh {

namespace {

constexpr int EW = 8;                                // warps per CTA
constexpr int VS = 9;                                // stride of a cell's corner samples
static_assert(32 * MC_MAX_VERTS < (1 << 9) && 32 * MC_MAX_FACES < (1 << 8), "task numbers fit the cells' records");
// Node table of a warp: x nodes x0 .. x0+32, z nodes of the word 32 zw .. 32 zw + 32,
// y nodes y, y+1; the spacing of a node is stored with it.
constexpr int NX = 0, NZ = 33, NY = 66, NT = 68;

// How positions are evaluated: P (the LinRange / quotient promotion) and the output.
//   PM_F32: P Float32, Float32 output:  fl32(p1 + fl32(mu * d))
//   PM_MIX: P Float64, Float32 output:  float pairs (fast_f32_pos) for a Float32
//           quotient, FP64 when undecided or for a Float64 quotient
//   PM_F64: Float64 output:             fl64(p1 + fl64(mu * d))
constexpr int PM_F32 = 0, PM_MIX = 1, PM_F64 = 2;

template <int PM> struct Nodes;
template <> struct Nodes<PM_F32> { float p[NT], d[NT]; };
template <> struct Nodes<PM_MIX> { float p[NT], pl[NT], d[NT], dl[NT]; };
template <> struct Nodes<PM_F64> { double p[NT], d[NT]; };

template <class T, int PM> struct EmitWarp {
    long long iv[32], jf[32];    // per column: index of vertex / face task 0
    Nodes<PM> nd;
    T val[32 * VS];              // corner samples: [cell][corner x | y << 1 | z << 2]
    uint16_t queue[BCOL * 32];   // active cells of the word: column | z << 5
};

// Per case and vertex slot: the edge's start corner (x | y << 1 | z << 2) and its
// axis (bits 8-9); per case and face slot: the three vertex slots (4 bits each);
// per cell index (mesh_bits.cuh): vertices (bits 0-3), faces (4-7), case (8-15).
struct alignas(16) CaseTabs {
    uint16_t ev[256 * MC_MAX_VERTS];
    uint16_t ef[256 * MC_MAX_FACES];
    uint16_t pc[256];
};
constexpr CaseTabs make_case_tabs() {
    CaseTabs t{};
    constexpr int EA[12] = {0, 1, 2, 3, 4, 5, 6, 7, 0, 1, 2, 3}, EB[12] = {1, 2, 3, 0, 5, 6, 7, 4, 4, 5, 6, 7};
    constexpr int CO[8] = {0, 1, 3, 2, 4, 5, 7, 6};  // corner of src/marching_cubes.jl:42-49 -> x | y << 1 | z << 2
    for (int c = 0; c < 256; c++) {
        for (int k = 0; k < MC_MAX_VERTS; k++) {
            const int e = (int)((MC_CASE_VERTS[c] >> (4 * k)) & 15u);
            const int a = CO[EA[e]], m = a ^ CO[EB[e]];
            t.ev[c * MC_MAX_VERTS + k] = (uint16_t)(a | ((m == 1 ? 0 : (m == 2 ? 1 : 2)) << 8));
        }
        for (int k = 0; k < MC_MAX_FACES; k++) t.ef[c * MC_MAX_FACES + k] = (uint16_t)((MC_CASE_FACES[c] >> (12 * k)) & 0xfffu);
        const unsigned cm = mc_case_of_bits((unsigned)c);
        t.pc[c] = (uint16_t)(((MC_CASE_VERTS[cm] >> 48) & 15u) | (((MC_CASE_VERTS[cm] >> 52) & 7u) << 4) | (cm << 8));
    }
    return t;
}
__device__ const CaseTabs d_cases = make_case_tabs();
static_assert(sizeof(CaseTabs) % 16 == 0, "copied in 16-byte words");

template <class T, int PM> constexpr size_t emit_smem() { return sizeof(CaseTabs) + EW * sizeof(EmitWarp<T, PM>); }

// Table entries of node i of the warp's table: global node gi of the axis whose
// tables start at ax0.  Returns whether the node is -0.0 (its sum with mu * 0
// need not be itself).
template <int PM>
__device__ __forceinline__ bool put_node(Nodes<PM> &nd, int i, const Tabs &tb, int64_t ax0, int64_t gi) {
    if constexpr (PM == PM_F32) {
        nd.p[i] = __ldg(tb.xpf + ax0 + gi);
        nd.d[i] = __ldg(tb.dxf + ax0 + gi);
        return __float_as_uint(nd.p[i]) == 0x80000000u;
    } else if constexpr (PM == PM_MIX) {
        nd.p[i] = __ldg(tb.split + ax0 + gi);
        nd.pl[i] = __ldg(tb.split + tb.ntab + ax0 + gi);
        nd.d[i] = __ldg(tb.split + 2 * tb.ntab + ax0 + gi);
        nd.dl[i] = __ldg(tb.split + 3 * tb.ntab + ax0 + gi);
        return __float_as_uint(nd.p[i]) == 0x80000000u;
    } else {
        nd.p[i] = __ldg(tb.xp + ax0 + gi);
        nd.d[i] = __ldg(tb.dx + ax0 + gi);
        return __double_as_longlong(nd.p[i]) == (long long)0x8000000000000000ull;
    }
}

// p1 + mu * (p1 - p1) on an axis the edge does not move along, when p1 is -0.0 or
// mu is not finite (otherwise it is p1): evaluated in P, rounded to the output.
template <class P, class O> __device__ __noinline__ O still_slow(double c, double mu) {
    return (O)Ar<P>::add((P)c, Ar<P>::mul((P)mu, P(0)));
}

// The crossing on edge `ev` of cell j (column ln, plane z of the word) to `out`.
template <class T, class Q, class P, int PM>
__device__ __forceinline__ void put_vertex(const Plan &p, const Tabs &tb, const EmitWarp<T, PM> &w, uint32_t ev, int j,
                                           int ln, int z, int x0, int y, int z0, bool zero, char *out) {
    const int a = (int)(ev & 7u), ax = (int)(ev >> 8), b = a ^ (1 << ax);
    const T va = w.val[j * VS + a], vb = w.val[j * VS + b];
    const Q mu = quotient<Q>(va, vb, p);
    const bool odd = !bits_finite(mu) || zero;
    const int xi = NX + ln + (a & 1), yi = NY + ((a >> 1) & 1), zi = NZ + z + (a >> 2);
    const bool neg = a > b;                                                    // the start is the axis's upper node
    const int lo = ax == 0 ? NX + ln : (ax == 1 ? NY : NZ + z), ni = lo + neg;  // the axis's lower and start nodes
    if constexpr (PM == PM_F64) {
        double o0 = w.nd.p[xi], o1 = w.nd.p[yi], o2 = w.nd.p[zi];
        const double d = neg ? -w.nd.d[lo] : w.nd.d[lo];
        const double r = (double)Ar<P>::add((P)(ax == 0 ? o0 : (ax == 1 ? o1 : o2)), Ar<P>::mul((P)mu, (P)d));
        if (odd) {
            o0 = still_slow<P, double>(o0, (double)mu);
            o1 = still_slow<P, double>(o1, (double)mu);
            o2 = still_slow<P, double>(o2, (double)mu);
        }
        put3((double *)out, ax == 0 ? r : o0, ax == 1 ? r : o1, ax == 2 ? r : o2);
    } else {
        // p[] is the node rounded to float (PM_MIX: its high part)
        float o0 = w.nd.p[xi], o1 = w.nd.p[yi], o2 = w.nd.p[zi];
        float r;
        if constexpr (PM == PM_F32) {
            const float d = neg ? -w.nd.d[lo] : w.nd.d[lo];
            r = (float)Ar<P>::add((P)(ax == 0 ? o0 : (ax == 1 ? o1 : o2)), Ar<P>::mul((P)mu, (P)d));
        } else {
            const float dh = w.nd.d[lo], dl = w.nd.dl[lo];
            // (a Float64 quotient -- Int / Int on integer data -- has no float-pair form)
            const bool done = sizeof(Q) == 4 && bits_finite(mu) && !p.force_fp64 &&
                              fast_f32_pos((float)mu, ax == 0 ? o0 : (ax == 1 ? o1 : o2), w.nd.pl[ni], neg ? -dh : dh, neg ? -dl : dl, r);
            if (!done) {
                // the Float64 expression, from the double tables
                const int64_t ax0 = ax == 0 ? 0 : (ax == 1 ? tb.nx : tb.nx + tb.ny);
                const int64_t g = ax == 0 ? x0 + ln : (ax == 1 ? y : z0 + z);
                const double dd = __ldg(tb.dx + ax0 + g);
                r = moving_fp64<P>(__ldg(tb.xp + ax0 + g + neg), neg ? -dd : dd, (double)mu);
            }
        }
        if (odd) {
            if constexpr (PM == PM_MIX) {
                const F3 ov = still_fp64<P>(tb.xp, tb.yp, tb.zp, tb.xpf, tb.ypf, tb.zpf, x0 + ln + (a & 1),
                                            y + ((a >> 1) & 1), z0 + z + (a >> 2), (double)mu);
                o0 = ov.v[0];
                o1 = ov.v[1];
                o2 = ov.v[2];
            } else {
                o0 = still_slow<P, float>(o0, (double)mu);
                o1 = still_slow<P, float>(o1, (double)mu);
                o2 = still_slow<P, float>(o2, (double)mu);
            }
        }
        put3((float *)out, ax == 0 ? r : o0, ax == 1 ? r : o1, ax == 2 ? r : o2);
    }
}

// Where an item's mesh goes: buffers and their room, what the scanned offsets lose
// to index them (v0, f0), what vertex ids lose beyond that (id0: batches number the
// vertices of each volume from 1) and the volume's first edge key.
struct OutView {
    char *verts;
    int64_t *faces;
    long long vcap, fcap, v0, f0, id0, kbase;
};

// b: the item's volume of a batch (null: the plan's single volume); cols: the item's
// columns of the 32.
template <class T, class Q, class P, int PM, bool BATCH>
__device__ __forceinline__ void emit_item(const Plan &p, const BatchVol *b, const BView &v, const Tabs &tb,
                                          EmitWarp<T, PM> &w, const CaseTabs &ct, int lane, int xb, int y, int seg,
                                          uint32_t cols) {
    constexpr int VB = 3 * (PM == PM_F64 ? 8 : 4);  // bytes of a vertex
    const int mw = mask_words(min(v.zws, (v.cz + 31) / 32 - seg * v.zws));
    const uint32_t *mp = p.wmask + bmask(v, seg, y, xb);
    const int x0 = xb * BCOL, x = x0 + lane;
    const int zws0 = seg * v.zws;
    const bool xin = x < v.cx && (BATCH || ((cols >> lane) & 1u));
    bool ready = false;            // the item's offsets and x, y nodes are loaded
    bool zeroxy = false;
    long long gv = 0, gf = 0;      // this column's next vertex / face
    OutView out{(char *)p.verts, p.faces, p.verts_cap, p.faces_cap, 0, 0, 0, 0};
    const uint32_t *r0 = v.bits + (int64_t)(zws0 - v.bw0) * v.sxy + v.nx * y + min(x, v.cx - 1);
    const T *s0 = (const T *)v.vol + v.nx * y + x0;
    for (int q = 0; q < mw; q++) {
        uint32_t todo = mp[q];
        if (todo && !ready) {
            ready = true;
            if constexpr (BATCH) {
                const ulonglong2 t = p.tsum[v.e0 / BITS_TILE];
                const uint2 o = p.pc[v.e0];
                const long long v0 = (long long)t.x + o.x, f0 = (long long)t.y + o.y;
                if (p.vol_outputs) out = OutView{(char *)b->verts, b->faces, b->vcap, b->fcap, v0, f0, 0, 0};
                else out.id0 = v0;
                if (p.vkey) out.kbase = b->kbase;
            }
            if (xin) {
                const int64_t e = bpiece(v, seg, y, x);
                const ulonglong2 t = p.tsum[e / BITS_TILE];
                const uint2 o = p.pc[e];
                gv = (long long)t.x + o.x - out.v0;
                gf = (long long)t.y + o.y - out.f0;
            }
            __syncwarp();  // the previous item's tasks are done with the node table
            bool z = false;
            if (x < v.nx) z |= put_node<PM>(w.nd, NX + lane, tb, 0, x);
            if (lane == 0 && x0 + 32 < v.nx) z |= put_node<PM>(w.nd, NX + 32, tb, 0, x0 + 32);
            if (lane < 2) z |= put_node<PM>(w.nd, NY + lane, tb, tb.nx, y + lane);
            zeroxy = __any_sync(FULL, z);
        }
        while (todo) {
            const int k = 32 * q + __ffs(todo) - 1;
            todo &= todo - 1;
            const int zw = zws0 + k, z0 = 32 * zw;
            const uint32_t *a0 = r0 + (int64_t)k * v.sxy, *a1 = a0 + v.nx;
            const uint32_t a = a0[0], b = a0[1], c = a1[0], d = a1[1];
            uint32_t nb = 0;  // bit 0 of the next words, in the order a, b, c, d
            if (zw + 1 < v.nzw) {
                a0 += v.sxy;
                a1 += v.sxy;
                nb = (a0[0] & 1u) | ((a0[1] & 1u) << 1) | ((a1[0] & 1u) << 2) | ((a1[1] & 1u) << 3);
            }
            const Corners cn{a, b, c, d, __funnelshift_r(a, nb, 1), __funnelshift_r(b, nb >> 1, 1),
                             __funnelshift_r(c, nb >> 2, 1), __funnelshift_r(d, nb >> 3, 1)};
            uint32_t act = xin ? cn.active() & cell_mask(v.cz, zw) : 0u;
            const int n = __popc(act);
            int end = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(FULL, end, o);
                if (lane >= o) end += t;
            }
            const int total = __shfl_sync(FULL, end, 31), beg = end - n;
            __syncwarp();  // the previous word's tasks are done with the queue and the z nodes
            for (int i = beg; act; i++, act &= act - 1) w.queue[i] = (uint16_t)(lane | ((__ffs(act) - 1) << 5));
            bool z = zeroxy;
            if (z0 + lane < v.nz) z |= put_node<PM>(w.nd, NZ + lane, tb, tb.nx + tb.ny, z0 + lane);
            if (lane == 0 && z0 + 32 < v.nz) z |= put_node<PM>(w.nd, NZ + 32, tb, tb.nx + tb.ny, z0 + 32);
            const bool zero = __any_sync(FULL, z);
            const T *sw = s0 + (int64_t)z0 * v.sxy;
            __syncwarp();
            // the samples of the next batch are in flight while this one is emitted
            T s[8];
            uint32_t ent = lane < total ? w.queue[lane] : 0u;
            load_corners(s, sw, ent, v);
            for (int j0 = 0; j0 < total; j0 += 32) {
                const bool on = j0 + lane < total;
                const int ln = (int)(ent & 31u), zc = (int)(ent >> 5);
                const uint32_t wa = __shfl_sync(FULL, a, ln), wb = __shfl_sync(FULL, b, ln), wc = __shfl_sync(FULL, c, ln),
                               wd = __shfl_sync(FULL, d, ln), wn = __shfl_sync(FULL, nb, ln);
                const uint32_t pc = ct.pc[cell_index(wa, wb, wc, wd, wn, wn >> 1, wn >> 2, wn >> 3, zc)];
                const uint32_t acc = on ? (pc & 15u) | (((pc >> 4) & 15u) << 16) : 0u;
                uint32_t inc = acc;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t t = __shfl_up_sync(FULL, inc, o);
                    if (lane >= o) inc += t;
                }
                const uint32_t tot = __shfl_sync(FULL, inc, 31), exc = inc - acc;
                const int VW = (int)(tot & 0xffffu), FW = (int)(tot >> 16);
                // this column's cells of the batch are lo .. hi - 1
                const int lo = min(max(beg - j0, 0), 32), hi = min(max(end - j0, 0), 32);
                const uint32_t el = __shfl_sync(FULL, exc, lo & 31), eh = __shfl_sync(FULL, exc, hi & 31);
                const uint32_t tl = lo == 32 ? tot : el, th = hi == 32 ? tot : eh;
                const long long g0 = gv - (long long)(tl & 0xffffu), f0 = gf - (long long)(tl >> 16);
                gv = g0 + (th & 0xffffu);
                gf = f0 + (th >> 16);
                const bool fit = __all_sync(FULL, gv <= out.vcap && gf <= out.fcap);
                w.iv[lane] = g0;
                w.jf[lane] = f0;
#pragma unroll
                for (int g = 0; g < 8; g++) w.val[lane * VS + g] = s[g];
                const uint32_t cs = pc >> 8, fv = exc & 0xffffu, ff = exc >> 16;
                const uint32_t vrec = cs | ((uint32_t)ln << 8) | ((uint32_t)zc << 13) | (fv << 18);
                const uint32_t frec = cs | ((uint32_t)ln << 8) | (fv << 13) | (ff << 22);
                // first tasks: round in the high bits (none for lanes without a cell)
                const uint32_t vr = on ? fv >> 5 : 0xffu, fr = on ? ff >> 5 : 0xffu;
                if (j0 + 32 < total) {
                    ent = j0 + 32 + lane < total ? w.queue[j0 + 32 + lane] : 0u;
                    load_corners(s, sw, ent, v);
                }
                __syncwarp();
                int cb = -1;
                for (int r = 0; 32 * r < VW; r++) {
                    const uint32_t bits = __reduce_or_sync(FULL, vr == (uint32_t)r ? 1u << (fv & 31u) : 0u);
                    const int t = 32 * r + lane, j = cb + __popc(bits & lanemask_le(lane));
                    cb += __popc(bits);
                    const uint32_t rec = __shfl_sync(FULL, vrec, j);
                    if (t < VW) {
                        const int cl = (int)((rec >> 8) & 31u), cz = (int)((rec >> 13) & 31u);
                        const uint32_t ev = ct.ev[(rec & 255u) * MC_MAX_VERTS + (t - (int)(rec >> 18))];
                        const long long at = w.iv[cl] + t;
                        if (fit || at < out.vcap) {
                            put_vertex<T, Q, P, PM>(p, tb, w, ev, j, cl, cz, x0, y, z0, zero, out.verts + VB * at);
                            if (p.vkey) {
                                // the edge's lower node; the cell owns the edge when, across
                                // each other axis, the edge lies on the cell's upper side or
                                // the cell is first
                                const int ax = (int)(ev >> 8), low = (int)(ev & 7u) & ~(1 << ax);
                                const int ox = low & 1, oy = (low >> 1) & 1, oz = low >> 2;
                                const int cx = x0 + cl, cw = z0 + cz;
                                const bool own = (ax == 0 || ox || cx == 0) && (ax == 1 || oy || y == 0) &&
                                                 (ax == 2 || oz || cw == 0);
                                const long long key =
                                    out.kbase + ax +
                                    3 * ((long long)(cx + ox) + v.nx * ((long long)(y + oy) + v.ny * (long long)(cw + oz)));
                                p.vkey[at] = key | (own ? (long long)(1ull << 63) : 0ll);
                            }
                        } else {
                            *p.err = ERR_CAPACITY;
                        }
                    }
                }
                cb = -1;
                for (int r = 0; 32 * r < FW; r++) {
                    const uint32_t bits = __reduce_or_sync(FULL, fr == (uint32_t)r ? 1u << (ff & 31u) : 0u);
                    const int t = 32 * r + lane, j = cb + __popc(bits & lanemask_le(lane));
                    cb += __popc(bits);
                    const uint32_t rec = __shfl_sync(FULL, frec, j);
                    if (t < FW) {
                        const int cl = (int)((rec >> 8) & 31u);
                        const uint32_t sf = ct.ef[(rec & 255u) * MC_MAX_FACES + (t - (int)(rec >> 22))];
                        const long long at = w.jf[cl] + t;
                        const long long vb = w.iv[cl] + 1 - out.id0 + (long long)((rec >> 13) & 511u);  // 1-based
                        if (fit || at < out.fcap)
                            put3(out.faces + 3 * at, vb + (sf & 15u), vb + ((sf >> 4) & 15u), vb + ((sf >> 8) & 15u));
                        else
                            *p.err = ERR_CAPACITY;
                    }
                }
                __syncwarp();  // the next batch rewrites the records
            }
        }
    }
}

template <class T, class Q, class P, int PM>
__global__ void __launch_bounds__(32 * EW, 3) k_emit_bits_mc(const Plan p, int seg0, int nseg, int nitems, int lg) {
    extern __shared__ __align__(16) unsigned char esm[];
    CaseTabs &ct = *reinterpret_cast<CaseTabs *>(esm);
    EmitWarp<T, PM> *sw = reinterpret_cast<EmitWarp<T, PM> *>(esm + sizeof(CaseTabs));
    for (int i = threadIdx.x; i < (int)(sizeof(CaseTabs) / 16); i += blockDim.x)
        reinterpret_cast<uint4 *>(&ct)[i] = reinterpret_cast<const uint4 *>(&d_cases)[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    const BView v = view_of(p);
    const Tabs tb = tabs_of(p);
    const int nxb = p.ntx > 0 ? p.ntx : v.nxb;  // column blocks tx0 .. tx0 + ntx - 1
    after_previous();
    // the first item of a warp is its own number, spread over the CTAs
    for (int item = wi * gridDim.x + blockIdx.x; item < nitems; item = next_item(p, lane)) {
        const int q = item >> lg, width = 32 >> lg, part = item & ((1 << lg) - 1);  // 1 << lg parts of 32 columns
        const int xb = p.tx0 + q % nxb;
        const int seg = seg0 + (q / nxb) % nseg;
        const int y = q / (nxb * nseg);
        emit_item<T, Q, P, PM, false>(p, nullptr, v, tb, sw[wi], ct, lane, xb, y, seg,
                                      (FULL >> (32 - width)) << (width * part));
    }
}

// Batch: an item is `rows` rows (1, 2, 4 or 8) of an item of k_count (Plan::cblk_vol
// names its volume).  Four rows fetch the descriptor and their masks once; batches
// too small for eight such items per warp take single rows.
constexpr int BITEM = 4;
static_assert(BROW % BITEM == 0, "whole items per item of k_count");
template <class T, class Q, class P, int PM>
__global__ void __launch_bounds__(32 * EW, 3) k_emit_bits_batch(const Plan p, int64_t nitems, int rows) {
    extern __shared__ __align__(16) unsigned char esm[];
    CaseTabs &ct = *reinterpret_cast<CaseTabs *>(esm);
    EmitWarp<T, PM> *sw = reinterpret_cast<EmitWarp<T, PM> *>(esm + sizeof(CaseTabs));
    for (int i = threadIdx.x; i < (int)(sizeof(CaseTabs) / 16); i += blockDim.x)
        reinterpret_cast<uint4 *>(&ct)[i] = reinterpret_cast<const uint4 *>(&d_cases)[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    after_previous();
    // first vertex and face of every volume, then the totals
    for (int i = blockIdx.x * (32 * EW) + threadIdx.x; i <= p.nvols; i += gridDim.x * (32 * EW)) {
        const int64_t e = i < p.nvols ? p.bvols[i].e0 : p.npc;
        int64_t vo = p.totals[0], fo = p.totals[1];
        if (e < p.npc) {
            const ulonglong2 t = p.tsum[e / BITS_TILE];
            const uint2 o = p.pc[e];
            vo = (int64_t)(t.x + o.x);
            fo = (int64_t)(t.y + o.y);
        }
        p.vol_off[2 * (int64_t)i] = vo;
        p.vol_off[2 * (int64_t)i + 1] = fo;
    }
    for (;;) {
        unsigned item = 0;
        if (lane == 0) item = atomicAdd(p.work, 1u);
        item = __shfl_sync(FULL, item, 0);
        if ((int64_t)item >= nitems) break;
        const unsigned per = BROW / rows, blk = item / per;
        const BatchVol *b = p.bvols + p.cblk_vol[blk];
        const BView v = view_of(p, *b);
        const unsigned k = blk - (unsigned)b->cblk0;
        const int xb = (int)(k % v.nxb), seg = (int)((k / v.nxb) / v.nyb);
        const int y0 = (int)((k / v.nxb) % v.nyb) * BROW + (int)(item % per) * rows;
        uint32_t any = 0;
        if (lane < rows && y0 + lane < v.cy) {
            const uint32_t *mp = p.wmask + bmask(v, seg, y0 + lane, xb);
            const int mw = mask_words(min(v.zws, (v.cz + 31) / 32 - seg * v.zws));
            for (int q = 0; q < mw; q++) any |= mp[q];
        }
        const Tabs tb = tabs_at(b->tabs, v.nx, v.ny, v.nz);
        for (uint32_t todo = __ballot_sync(FULL, any != 0u); todo; todo &= todo - 1)
            emit_item<T, Q, P, PM, true>(p, b, v, tb, sw[wi], ct, lane, xb, y0 + __ffs(todo) - 1, seg, FULL);
    }
}

// Resident CTAs per SM of a kernel on the current device, with its dynamic shared
// memory allowed (one-time per device and instantiation), and the device's SMs.
template <class T, class Q, class P, int PM, bool BATCH> int emit_ctas(int *sms) {
    static std::mutex mu;
    static int ctas[64] = {0}, nsm[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return 0;
    std::lock_guard<std::mutex> lk(mu);
    if (!ctas[dev]) {
        const void *fn = BATCH ? (const void *)k_emit_bits_batch<T, Q, P, PM> : (const void *)k_emit_bits_mc<T, Q, P, PM>;
        const int smem = (int)emit_smem<T, PM>();
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        int per_sm = 0;
        cudaDeviceGetAttribute(&nsm[dev], cudaDevAttrMultiProcessorCount, dev);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 32 * EW, smem) != cudaSuccess || per_sm < 1)
            per_sm = 1;
        cudaGetLastError();
        ctas[dev] = per_sm;
    }
    *sms = nsm[dev];
    return ctas[dev];
}

// What a launch covers: segments of a single volume, or a batch (ctas per SM).
struct Range {
    int seg0, nseg, batch, ctas;
};

template <class T, class Q, class P, int PM> cudaError_t go_batch(const Plan &p, int ctas, cudaStream_t s) {
    int sms = 0;
    const int fit = emit_ctas<T, Q, P, PM, true>(&sms);
    const int64_t grid = (int64_t)sms * (ctas > 0 ? std::min(ctas, fit) : fit);
    const int rows = p.ncblk * (BROW / BITEM) >= 8 * EW * grid ? BITEM : 1;
    const int64_t nitems = p.ncblk * (BROW / rows);
    if (grid < 1) return cudaErrorInvalidDevice;
    if (nitems > 0x7fffffff) return cudaErrorInvalidConfiguration;
    return launch_after(k_emit_bits_batch<T, Q, P, PM>, (unsigned)std::max<int64_t>(1, std::min<int64_t>(grid, nitems)), 32 * EW,
                        emit_smem<T, PM>(), s, p, nitems, rows);
}

template <class T, class Q, class P, int PM> cudaError_t go(const Plan &p, const Range &r, cudaStream_t s) {
    if (r.batch) return go_batch<T, Q, P, PM>(p, r.ctas, s);
    const int seg0 = r.seg0, nseg = r.nseg;
    int sms = 0;
    const int grid = emit_ctas<T, Q, P, PM, false>(&sms) * sms;
    // volumes of few rows: items of 8 columns, so that every SM has some and dense ones
    // (a row's word of 32 x 32 active cells is 32 batches) end together (128^3 sines
    // 56 -> 44 us a call)
    const int64_t rows = (int64_t)(p.ntx > 0 ? p.ntx : p.nxb) * nseg * p.cy;
    const int lg = rows < 2 * EW * (int64_t)grid ? 2 : 0;
    const int64_t nitems = rows << lg;
    if (grid < 1) return cudaErrorInvalidDevice;
    if (nitems > 0x7fffffff - 65536) return cudaErrorInvalidConfiguration;
    if (nitems < 1) return cudaSuccess;
    return launch_after(k_emit_bits_mc<T, Q, P, PM>, (unsigned)std::min<int64_t>(grid, nitems), 32 * EW, emit_smem<T, PM>(),
                        s, p, seg0, nseg, (int)nitems, lg);
}

template <class T> cudaError_t go_t(const Plan &p, int Q64, int P64, const Range &r, cudaStream_t s) {
    if (p.out64) {
        if (Q64) return go<T, double, double, PM_F64>(p, r, s);
        return go<T, float, double, PM_F64>(p, r, s);
    }
    if (Q64) return go<T, double, double, PM_MIX>(p, r, s);  // integer data, Int iso, Float32 ranges
    if (P64) return go<T, float, double, PM_MIX>(p, r, s);
    return go<T, float, float, PM_F32>(p, r, s);
}

}  // namespace

static cudaError_t launch(const Plan &p, int Q64, int P64, const Range &r, cudaStream_t s) {
    switch (p.T) {
    case MESH_DT_U16: return go_t<uint16_t>(p, Q64, P64, r, s);
    case MESH_DT_F16: return go_t<h16>(p, Q64, P64, r, s);
    case MESH_DT_I16: return go_t<int16_t>(p, Q64, P64, r, s);
    case MESH_DT_I8: return go_t<int8_t>(p, Q64, P64, r, s);
    case MESH_DT_U8: return go_t<uint8_t>(p, Q64, P64, r, s);
    case MESH_DT_F32: return go_t<float>(p, Q64, P64, r, s);
    case MESH_DT_I32: return go_t<int32_t>(p, Q64, P64, r, s);
    case MESH_DT_I64: return go_t<int64_t>(p, Q64, P64, r, s);
    default: return go<double, double, double, PM_F64>(p, r, s);
    }
}

// Marching Cubes emission of segments seg0 .. seg0 + nseg - 1 of a single volume
// (bits, masks and offsets from k_bits.cu); column blocks tx0 .. tx0 + ntx - 1 when
// ntx > 0.  Plan::work is a cleared counter.
cudaError_t launch_emit_bits_mc(const Plan &p, int Q64, int P64, int seg0, int nseg, cudaStream_t s) {
    return launch(p, Q64, P64, Range{seg0, nseg, 0, 0}, s);
}

// Emission of a batch.
cudaError_t launch_emit_batch(const Plan &p, int Q64, int P64, int ctas, cudaStream_t s) {
    return launch(p, Q64, P64, Range{0, 0, 1, ctas}, s);
}

}  // namespace mesh
