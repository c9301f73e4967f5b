// Marching Tetrahedra, welded Marching Cubes and Naive Surface Nets emission from
// the sign bits.
//
// MT shares vertices between cells: the reference keys every lattice edge in a
// Dict and numbers a vertex when a cell first touches its edge in traversal
// order, computing its position from that first cell (getVertId/vertPos,
// src/marching_tetrahedra.jl:42-84; procVox :105-127).  Here the same numbering
// is derived without a hash table:
//   * the first cell to touch a lattice edge is the owner: the cell reached by
//     stepping -1 along every axis on which both edge corners sit at 0, as far
//     as the grid allows (traversal order is lexicographic, x slowest);
//   * a cell's new vertices are its owned crossed edges, numbered in the cell's
//     first-use order after all vertices of earlier cells;
//   * a cell that uses an edge owned by a neighbour needs the neighbour's case
//     and first vertex.
// Welded Marching Cubes (MESH_ALG_MC_WELDED) numbers the crossed lattice edges in the
// same way, in the order of the first cell's Marching Cubes vertices.
// NSN gives every active cell one vertex and connects the four cells around
// every crossed base edge, so it needs the same neighbours' first vertices.
//
// Work items, words and lists of active cells are those of k_emit_bits.cu; a
// batch is again 32 cells, one per lane.  Any cell's first vertex follows from
// bits alone: its column's offset, the vertices of the words below (left by
// k_count) and, in the word, population counts of the owned crossed edges or active
// cells (NSN) below it.  So each lane reads the 3 x 3 columns around
// its cell, at z - 1 .. z + 1, and leaves the cases and first vertices of the
// cells one step back along each set of axes in shared memory; the batch's
// vertices and faces are then dense task lists whatever the density.
//
// Measured per call against the form it replaced, which classified every sample of
// 4 + 1 rows step by step and worked on one plane's few cells at a time: 256^3
// gyroid with Float64 vertices, MT 613 -> 256 us, NSN 718 -> 243 us; 509 x 387 x 301
// Float32 sines, MT 1230 -> 523 us (this kernel 386 of them: 256 M warp
// instructions at 58% of issue, 146 MB read and 500 MB written); welded 301 x 187 x 250
// Float32 gyroid 438 -> 172 us.  The quotients and clamps run on the integer pipes
// (mesh_quot.h); what bounds it is issue and shared memory (half of its wavefronts) at
// the 16 warps per SM that 122 registers and 77-85 KB of tables and staging leave.  A
// triangle's three corners come in one word, and the neighbours' rows are padded so that
// the corners of one cell fall into different banks: MT 260 -> 256, NSN 248 -> 243,
// welded 177 -> 172, sines 528 -> 523 us.  Three CTAs per SM (80 registers, triangle
// references read through L1) are slower: MT 281 and 552 us, NSN 257.
#define MESH_TBL static constexpr
#include "mesh_internal.cuh"
#include "mesh_tables.h"
#include "mesh_bits.cuh"
#include "mesh_point.cuh"

#include <algorithm>
#include <mutex>

namespace mesh {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int SW = 8;                    // warps per CTA
constexpr int VS = 9;                    // stride of a cell's corner samples
constexpr int NX = 0, NZ = 33, NY = 66, NT = 68;  // node table, as in k_emit_bits.cu
constexpr int NC = 34;                   // columns x0 - 1 .. x0 + 32 of a window
constexpr int NPAIR = 32 * 12;           // NSN: crossed edges of a batch

// ---- tables, by cell index (mesh_bits.cuh) ----

constexpr unsigned mt_case_of_bits(unsigned u) {
    return (u & 1u) | (((u >> 4) & 1u) << 1) | (((u >> 6) & 1u) << 2) | (((u >> 2) & 1u) << 3) | (((u >> 1) & 1u) << 4) |
           (((u >> 5) & 1u) << 5) | (((u >> 7) & 1u) << 6) | (((u >> 3) & 1u) << 7);
}
// the axes (bit 0 x, 1 y, 2 z) on which both corners of MT edge e sit at 0
constexpr int low_axes(int e) {
    int m = 0;
    for (int k = 0; k < 3; k++)
        if (MT_CORNER_POS[MT_EDGE_CORNERS[e][0]][k] == 0 && MT_CORNER_POS[MT_EDGE_CORNERS[e][1]][k] == 0) m |= 1 << k;
    return m;
}
// MT edge e as the cell `dir` (+1 / -1) times the axes of s away sees it, or 31
constexpr int moved_edge(int e, int s, int dir) {
    for (int f = 0; f < 19; f++) {
        bool same = true;
        for (int k = 0; k < 3; k++) {
            const int d = ((s >> k) & 1) * dir;
            same = same && MT_CORNER_POS[MT_EDGE_CORNERS[f][0]][k] == MT_CORNER_POS[MT_EDGE_CORNERS[e][0]][k] + d &&
                   MT_CORNER_POS[MT_EDGE_CORNERS[f][1]][k] == MT_CORNER_POS[MT_EDGE_CORNERS[e][1]][k] + d;
        }
        if (same) return f;
    }
    return 31;
}
constexpr uint32_t own_mask(int bnd) {
    uint32_t m = 0;
    for (int e = 0; e < 19; e++)
        if ((low_axes(e) & ~bnd) == 0) m |= 1u << e;
    return m;
}
constexpr int bits_of(uint32_t m) {
    int n = 0;
    for (; m; m &= m - 1) n++;
    return n;
}

// The same of the Marching Cubes edges (mesh_tables.h numbering, corner bits x | y << 1 | z << 2).
constexpr int MC_A[12] = {0, 1, 3, 2, 4, 5, 7, 6, 0, 1, 3, 2}, MC_B[12] = {1, 3, 2, 0, 5, 7, 6, 4, 4, 5, 7, 6};
constexpr int mc_low_axes(int e) { return 7 & ~(MC_A[e] | MC_B[e]); }
constexpr int mc_moved_edge(int e, int s, int dir) {
    const int a = dir > 0 ? MC_A[e] | s : MC_A[e] & ~s, b = dir > 0 ? MC_B[e] | s : MC_B[e] & ~s;
    if (dir > 0 ? ((MC_A[e] | MC_B[e]) & s) != 0 : ((MC_A[e] & MC_B[e]) & s) != s) return 31;
    for (int f = 0; f < 12; f++)
        if ((MC_A[f] == a && MC_B[f] == b) || (MC_A[f] == b && MC_B[f] == a)) return f;
    return 31;
}
constexpr uint32_t mc_own_mask(int bnd) {
    uint32_t m = 0;
    for (int e = 0; e < 12; e++)
        if ((mc_low_axes(e) & ~bnd) == 0) m |= 1u << e;
    return m;
}

// Per algorithm: most triangles, edges, own edges of an interior cell, most vertices.
template <int ALG> struct EdgeDims { static constexpr int F = MT_MAX_FACES, E = 19, OWN = 8, V = MT_MAX_TOUCH; };
template <> struct EdgeDims<MESH_ALG_MC_WELDED> { static constexpr int F = MC_MAX_FACES, E = 12, OWN = 4, V = MC_MAX_VERTS; };

template <int ALG> struct alignas(16) EdgeTabs {
    using D = EdgeDims<ALG>;
    uint32_t ref[256][D::F];           // a triangle's corners, a byte each: owner's axes back << 5 | the edge in the owner
    uint8_t rank[256][D::E];           // interior cells: rank of an edge among the owned ones
    uint8_t kth[256][D::OWN];          // interior cells: the k-th owned crossed edge in first-use order
    uint8_t nvf[256];                  // interior vertices | faces << 4
    uint8_t unmoved[8][D::E];          // the edge of `ref` seen from the cells between it and the owner
    uint8_t corner[32];                // an edge's corners x | y << 1 | z << 2, start | end << 3
};
// Cells on the grid's lower faces own more edges: the full tables.
template <int ALG> struct EdgeFull {
    using D = EdgeDims<ALG>;
    uint32_t touched[256], before[256][D::E], own[8];
    uint8_t order[256][D::V];
};

constexpr EdgeTabs<MESH_ALG_MT> make_mt_tabs() {
    EdgeTabs<MESH_ALG_MT> t{};
    for (int i = 0; i < 256; i++) {
        const int c = (int)mt_case_of_bits((unsigned)i);
        for (int k = 0; k < 3 * MT_CASE_NFACES[c]; k++) {
            const int e = MT_CASE_FACES[c][k], s = low_axes(e);
            t.ref[i][k / 3] |= (uint32_t)((s << 5) | moved_edge(e, s, 1)) << (8 * (k % 3));
        }
        for (int e = 0; e < 19; e++) t.rank[i][e] = (uint8_t)bits_of(MT_BEFORE[c][e] & own_mask(0));
        int n = 0;
        for (int k = 0; k < bits_of(MT_TOUCHED[c] & 0x7ffffu); k++)
            if ((own_mask(0) >> MT_TOUCH_ORDER[c][k]) & 1u) t.kth[i][n++] = MT_TOUCH_ORDER[c][k];
        t.nvf[i] = (uint8_t)(n | (MT_CASE_NFACES[c] << 4));
    }
    for (int s = 0; s < 8; s++)
        for (int e = 0; e < 19; e++) t.unmoved[s][e] = (uint8_t)moved_edge(e, s, -1);
    for (int e = 0; e < 19; e++) {
        int c[2] = {0, 0};
        for (int q = 0; q < 2; q++)
            for (int k = 0; k < 3; k++) c[q] |= MT_CORNER_POS[MT_EDGE_CORNERS[e][q]][k] << k;
        t.corner[e] = (uint8_t)(c[0] | (c[1] << 3));
    }
    return t;
}
constexpr EdgeFull<MESH_ALG_MT> make_mt_full() {
    EdgeFull<MESH_ALG_MT> t{};
    for (int i = 0; i < 256; i++) {
        const int c = (int)mt_case_of_bits((unsigned)i);
        t.touched[i] = MT_TOUCHED[c] & 0x7ffffu;
        for (int e = 0; e < 19; e++) t.before[i][e] = MT_BEFORE[c][e];
        for (int k = 0; k < MT_MAX_TOUCH; k++) t.order[i][k] = MT_TOUCH_ORDER[c][k];
    }
    for (int b = 0; b < 8; b++) t.own[b] = own_mask(b);
    return t;
}
constexpr EdgeFull<MESH_ALG_MC_WELDED> make_mc_full() {
    EdgeFull<MESH_ALG_MC_WELDED> t{};
    for (int i = 0; i < 256; i++) {
        const uint64_t v = MC_CASE_VERTS[mc_case_of_bits((unsigned)i)];
        const int n = (int)((v >> 48) & 15u);
        for (int k = 0; k < MC_MAX_VERTS; k++) t.order[i][k] = 255;
        uint32_t m = 0;
        for (int k = 0; k < n; k++) {
            const int e = (int)((v >> (4 * k)) & 15u);
            t.order[i][k] = (uint8_t)e;
            t.before[i][e] = m;
            m |= 1u << e;
        }
        t.touched[i] = m;
    }
    for (int b = 0; b < 8; b++) t.own[b] = mc_own_mask(b);
    return t;
}
constexpr EdgeTabs<MESH_ALG_MC_WELDED> make_mc_tabs() {
    EdgeTabs<MESH_ALG_MC_WELDED> t{};
    constexpr EdgeFull<MESH_ALG_MC_WELDED> full = make_mc_full();
    for (int i = 0; i < 256; i++) {
        const unsigned c = mc_case_of_bits((unsigned)i);
        const int nf = (int)((MC_CASE_VERTS[c] >> 52) & 7u);
        for (int k = 0; k < 3 * nf; k++) {
            const int e = full.order[i][(MC_CASE_FACES[c] >> (4 * k)) & 15u], s = mc_low_axes(e);
            t.ref[i][k / 3] |= (uint32_t)((s << 5) | mc_moved_edge(e, s, 1)) << (8 * (k % 3));
        }
        for (int e = 0; e < 12; e++) t.rank[i][e] = (uint8_t)bits_of(full.before[i][e] & mc_own_mask(0));
        int n = 0;
        for (int k = 0; k < MC_MAX_VERTS; k++)
            if (full.order[i][k] < 12 && ((mc_own_mask(0) >> full.order[i][k]) & 1u)) t.kth[i][n++] = full.order[i][k];
        t.nvf[i] = (uint8_t)(n | (nf << 4));
    }
    for (int s = 0; s < 8; s++)
        for (int e = 0; e < 12; e++) t.unmoved[s][e] = (uint8_t)mc_moved_edge(e, s, -1);
    for (int e = 0; e < 12; e++) t.corner[e] = (uint8_t)(MC_A[e] | (MC_B[e] << 3));
    return t;
}
__device__ const EdgeTabs<MESH_ALG_MT> d_mt = make_mt_tabs();
__device__ const EdgeFull<MESH_ALG_MT> d_mt_full = make_mt_full();
__device__ const EdgeTabs<MESH_ALG_MC_WELDED> d_mc = make_mc_tabs();
__device__ const EdgeFull<MESH_ALG_MC_WELDED> d_mc_full = make_mc_full();
template <int ALG> __device__ __forceinline__ const EdgeFull<ALG> &full_tabs() {
    if constexpr (ALG == MESH_ALG_MT) return d_mt_full;
    else return d_mc_full;
}
static_assert(sizeof(EdgeTabs<MESH_ALG_MT>) % 16 == 0 && sizeof(EdgeTabs<MESH_ALG_MC_WELDED>) % 16 == 0,
              "copied in 16-byte words");
static_assert(MT_MAX_FACES <= 15 && bits_of(own_mask(0)) <= 8 && bits_of(mc_own_mask(0)) <= 4, "packed counts");

// NSN: a cell's crossed edges in MC edge order, start corner | axis << 3, and their number.
struct alignas(16) NsnTabs {
    uint8_t edge[256][12];
    uint8_t n[256];
};
constexpr NsnTabs make_nsn_tabs() {
    NsnTabs t{};
    constexpr int EA[12] = {0, 1, 2, 3, 4, 5, 6, 7, 0, 1, 2, 3}, EB[12] = {1, 2, 3, 0, 5, 6, 7, 4, 4, 5, 6, 7};
    constexpr int CO[8] = {0, 1, 3, 2, 4, 5, 7, 6};
    for (int i = 0; i < 256; i++) {
        const unsigned c = mc_case_of_bits((unsigned)i);
        int n = 0;
        for (int e = 0; e < 12; e++) {
            if (!(((c >> EA[e]) ^ (c >> EB[e])) & 1u)) continue;
            const int a = CO[EA[e]], m = a ^ CO[EB[e]];
            t.edge[i][n++] = (uint8_t)(a | ((m == 1 ? 0 : (m == 2 ? 1 : 2)) << 3));
        }
        t.n[i] = (uint8_t)n;
    }
    return t;
}
__device__ const NsnTabs d_nsn = make_nsn_tabs();
static_assert(sizeof(NsnTabs) % 16 == 0, "copied in 16-byte words");

template <int ALG> struct TabsOf { using type = EdgeTabs<ALG>; };
template <> struct TabsOf<MESH_ALG_NSN> { using type = NsnTabs; };

// ---- shared memory of one warp ----

template <class P, int ALG> struct Pairs {};
template <class P> struct Pairs<P, MESH_ALG_NSN> {
    P r[NPAIR];          // moving coordinate of every crossing
    uint8_t odd[NPAIR];  // 1, 2: a node may be -0.0 (mu * 0 is +0, -0); 3: mu is not finite; else 0
};
template <class T, class P, int ALG> struct SharedWarp {
    unsigned long long win[3][NC];  // rows y-1 .. y+1: bit 0 the sample below the word, 1-32 the word, 33 above
    long long col[2][NC];           // rows y-1, y, columns x0-1 ..: first vertex of the column's word
    long long nb[8][33];            // per cell: first vertex (NSN; else << 8 | cell index) of the cell back along the axes
    long long fb[32];               // per cell: first face
    P p[NT], d[NT];                 // nodes and spacings
    Pairs<P, ALG> pr;
    T val[32 * VS];                 // corner samples: [cell][corner x | y << 1 | z << 2]
    uint16_t queue[BCOL * 32];      // active cells of the word: column | z << 5
    uint8_t ov[32], of[32];         // the cells with vertex / face tasks, in order
};
template <class T, class P, int ALG> constexpr size_t shared_smem() {
    return (sizeof(typename TabsOf<ALG>::type) + 15) / 16 * 16 + SW * sizeof(SharedWarp<T, P, ALG>);
}

// ---- arithmetic ----

// a / n for a vertex's crossing count n (1..12), rounded exactly as the IEEE
// division, from one product and two fused operations (division by a small
// constant after Markstein, IBM J. Res. Develop. 34(1), 1990).  With y = RN(1/n)
// (rcp[n]) and q = RN(a*y), within 1.5 ulps of a/n and |q| <= |a|, the
// remainder a - q*n is a multiple of ulp(q) below 18 ulps: the fma computes it
// exactly.  q + r*y = a/n + r*(y - 1/n) then lies within 36 * 2^-53 ulps of
// a/n, while a/n is at least ulp/24 away from every rounding midpoint: n is
// 2^j times an odd number o, a/2^j is exact, and a - n*M for a midpoint M is a
// nonzero multiple of ulp/2.  So the one rounding of q + r*y gives RN(a/n).
// Zeros, |a| below 2^-959 (where a/2^j could round) and Inf / NaN take the
// division.
__device__ __forceinline__ double div_count(double a, int n, const double *rcp) {
    const unsigned e = (unsigned)((unsigned long long)__double_as_longlong(a) >> 52) & 0x7ffu;
    if (e < 64u || e == 0x7ffu) return __ddiv_rn(a, (double)n);
    const double y = rcp[n], q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-q, (double)n, a), y, q);
}
// The same in Float32 (24-bit significands; |a| below 2^-63 takes the division).
__device__ __forceinline__ float div_count(float a, int n, const float *rcp) {
    const unsigned e = (__float_as_uint(a) >> 23) & 0xffu;
    if (e < 64u || e == 0xffu) return __fdiv_rn(a, (float)n);
    const float y = rcp[n], q = __fmul_rn(a, y);
    return __fmaf_rn(__fmaf_rn(-q, (float)n, a), y, q);
}

// c1*b + c2*a in A, with the corner coordinates c1, c2 in {0, 1} and a, b not
// NaN: the products are b or a (times 1) and zeros carrying the sign of b or a
// (times 0), so the sum is ab = b + a (both 1), or one term plus a zero -- the
// other term, or the IEEE sum of two zeros -- with no arithmetic.
template <class A> __device__ __forceinline__ A corner_mix(int c1, int c2, A b, A a, A ab) {
    if (c1 && c2) return ab;
    const A t1 = c1 ? b : copysign(A(0), b), t2 = c2 ? a : copysign(A(0), a);
    if (!bits_zero(t1)) return t1;  // t2 is a zero
    if (!bits_zero(t2)) return t2;
    return (signbit(t1) && signbit(t2)) ? -A(0) : A(0);
}

// vertPos (src/marching_tetrahedra.jl:42-55) on the edge from corner c1 (value sv)
// to c2 (tv) of a cell whose base nodes and spacings are b3, d3.
template <class T, class Q, class A, class P>
__device__ __forceinline__ void mt_point(const Plan &p, int c1, int c2, T sv, T tv, const P (&b3)[3], const P (&d3)[3],
                                         P (&r)[3]) {
    const Q q = quotient<Q>(sv, tv, p);
    const A eps = sizeof(A) == 4 ? (A)p.eps_f : (A)p.eps_d;
    const A hi = sizeof(A) == 4 ? (A)p.hi_f : (A)p.hi_d;
    const A a = jl_min<A>(jl_max<A>((A)q, eps), hi);
    const A b = Ar<A>::sub(A(1), a);
    const A ab = Ar<A>::add(b, a);
    const bool pos = bits_positive(a) && bits_positive(b);  // the products by 0 are +0
    const bool nan = bits_nan(a);                           // then b and every weight are NaN
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int k1 = (c1 >> k) & 1, k2 = (c2 >> k) & 1;
        A w = k1 ? (k2 ? ab : b) : (k2 ? a : A(0));
        if (!pos) w = nan ? a : corner_mix<A>(k1, k2, b, a, ab);
        r[k] = Ar<P>::add(b3[k], Ar<P>::mul((P)w, d3[k]));
    }
}

template <class P> __device__ __forceinline__ void store_point(const Plan &p, long long out, P x, P y, P z) {
    if (p.out64) put3((double *)p.verts + 3 * out, (double)x, (double)y, (double)z);
    else put3((float *)p.verts + 3 * out, (float)x, (float)y, (float)z);
}

template <class P, class W>
__device__ __forceinline__ bool put_node(W &w, int i, const Tabs &tb, int64_t ax0, int64_t gi) {
    w.p[i] = tab<P>(tb.xp + ax0, tb.xpf + ax0, (int)gi);
    w.d[i] = tab<P>(tb.dx + ax0, tb.dxf + ax0, (int)gi);
    return bits_zero(w.p[i]) && signbit(w.p[i]);
}

// Vertices of a column's word below bit z (m: the lower cells that exist) that its
// cells own inside the grid, the column's corner words in MT corner order.
template <int ALG> __device__ __forceinline__ uint32_t own_below(const uint32_t (&w)[8], uint32_t m) {
    if constexpr (ALG == MESH_ALG_MC_WELDED)  // the three edges that end at the upper corner
        return __popc((w[6] ^ w[5]) & m) + __popc((w[6] ^ w[7]) & m) + __popc((w[6] ^ w[2]) & m);
    uint32_t n = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) n += k == 6 ? 0u : __popc((w[k] ^ w[6]) & m);
    return n;
}
// ... plus, for columns on the lower x / y faces (low) and the first plane (z0: the
// cells of m in it), the edges that only such cells own.
struct EdgeInfo {
    uint8_t a[19], b[19], low[19];
};
constexpr EdgeInfo make_edge_info(bool mc) {
    EdgeInfo t{};
    constexpr int WORD[8] = {0, 3, 1, 2, 4, 7, 5, 6};  // corner bits -> MT corner order
    for (int e = 0; e < (mc ? 12 : 19); e++) {
        t.a[e] = mc ? (uint8_t)WORD[MC_A[e]] : MT_EDGE_CORNERS[e][0];
        t.b[e] = mc ? (uint8_t)WORD[MC_B[e]] : MT_EDGE_CORNERS[e][1];
        t.low[e] = (uint8_t)(mc ? mc_low_axes(e) : low_axes(e));
    }
    return t;
}
constexpr EdgeInfo MT_INFO = make_edge_info(false), MC_INFO = make_edge_info(true);
template <int ALG, int E> __device__ __forceinline__ uint32_t own_extra(const uint32_t (&w)[8], uint32_t m, uint32_t z0, int low) {
    constexpr bool mc = ALG == MESH_ALG_MC_WELDED;
    constexpr int la = mc ? MC_INFO.low[E] : MT_INFO.low[E], ea = mc ? MC_INFO.a[E] : MT_INFO.a[E],
                  eb = mc ? MC_INFO.b[E] : MT_INFO.b[E];
    uint32_t r = 0;
    if constexpr (la != 0) r = (la & ~low & 3) ? 0u : __popc((w[ea] ^ w[eb]) & ((la & 4) ? z0 : m));
    if constexpr (E + 1 < EdgeDims<ALG>::E) return r + own_extra<ALG, E + 1>(w, m, z0, low);
    return r;
}

template <class T, class Q, class A, class P, int ALG>
__device__ __forceinline__ void emit_item(const Plan &p, const BView &v, const Tabs &tb, SharedWarp<T, P, ALG> &w,
                                          const typename TabsOf<ALG>::type &ct, const P *rcp, int lane, int xb, int y,
                                          int seg, uint32_t cols) {
    constexpr bool EDGES = ALG != MESH_ALG_NSN;  // vertices on lattice edges
    const int mw = mask_words(min(v.zws, (v.cz + 31) / 32 - seg * v.zws));
    const uint32_t *mp = p.wmask + bmask(v, seg, y, xb);
    const int x0 = xb * BCOL, x = x0 + lane;
    const int zws0 = seg * v.zws;
    bool ready = false;
    bool zeroxy = false;
    long long V0 = 0;           // with an x halo, its cell column's totals: every output is shifted by them
    long long gf = 0;           // this column's next face
    const bool mine = x < v.cx && !(p.xhalo && x == 0) && ((cols >> lane) & 1u);
    const T *s0 = (const T *)v.vol + v.nx * y + x0;
    auto first = [&](int yy, int xx, long long &vo, long long &fo) {
        const int64_t e = bpiece(v, seg, yy, xx);
        const ulonglong2 t = p.tsum[e / BITS_TILE];
        const uint2 o = p.pc[e];
        vo = (long long)t.x + o.x;
        fo = (long long)t.y + o.y;
    };
    long long base[2] = {0, 0}, basex = 0;  // first vertex of this lane's column in rows y-1, y; lanes 0, 1: of column x0-1
    for (int q = 0; q < mw; q++) {
        uint32_t todo = mp[q];
        if (todo && !ready) {
            ready = true;
            long long F0 = 0, f = 0;
            if (p.xhalo && p.cx > 1) {
                const int64_t e = bpiece(v, 0, 0, 1);
                const ulonglong2 t = p.tsum[e / BITS_TILE];
                const uint2 o = p.pc[e];
                V0 = (long long)t.x + o.x;
                F0 = (long long)t.y + o.y;
            }
            if (x < v.cx) {
                first(y, x, base[1], gf);
                gf -= F0;
                if (y > 0) first(y - 1, x, base[0], f);
            }
            if (lane < 2 && x0 > 0 && (lane == 1 || y > 0)) first(y - 1 + lane, x0 - 1, basex, f);
            __syncwarp();  // the previous item's tasks are done with the node table
            bool z = false;
            if (x < v.nx) z |= put_node<P>(w, NX + lane, tb, 0, x);
            if (lane == 0 && x0 + 32 < v.nx) z |= put_node<P>(w, NX + 32, tb, 0, x0 + 32);
            if (lane < 2) z |= put_node<P>(w, NY + lane, tb, tb.nx, y + lane);
            zeroxy = __any_sync(FULL, z);
        }
        while (todo) {
            const int k = 32 * q + __ffs(todo) - 1;
            todo &= todo - 1;
            const int zw = zws0 + k, z0 = 32 * zw;
            // windows of the 3 rows and 34 columns (columns outside the volume: zeros)
            const uint32_t *bw = v.bits + (int64_t)(zw - v.bw0) * v.sxy;
            auto window = [&](int yy, int xx) -> unsigned long long {
                if (yy < 0 || yy >= v.ny || xx < 0 || xx >= v.nx) return 0ull;
                const uint32_t *b = bw + v.nx * yy + xx;
                return (zw > 0 ? (unsigned long long)(b[-v.sxy] >> 31) : 0ull) | ((unsigned long long)b[0] << 1) |
                       (zw + 1 < v.nzw ? (unsigned long long)(b[v.sxy] & 1u) << 33 : 0ull);
            };
            const uint32_t *vw = p.vpre + (int64_t)(zw - v.bw0) * v.sxy;
            __syncwarp();  // the previous word's tasks are done with the windows, queue and z nodes
#pragma unroll
            for (int r = 0; r < 3; r++) w.win[r][lane + 1] = window(y - 1 + r, x);
            if (lane < 6) w.win[lane >> 1][(lane & 1) ? 33 : 0] = window(y - 1 + (lane >> 1), (lane & 1) ? x0 + 32 : x0 - 1);
            if (x < v.cx) {
                w.col[1][lane + 1] = base[1] - V0 + vw[v.nx * y + x];
                if (y > 0) w.col[0][lane + 1] = base[0] - V0 + vw[v.nx * (y - 1) + x];
            }
            if (lane < 2 && x0 > 0 && (lane == 1 || y > 0)) w.col[lane][0] = basex - V0 + vw[v.nx * (y - 1 + lane) + x0 - 1];
            bool z = zeroxy;
            if (z0 + lane < v.nz) z |= put_node<P>(w, NZ + lane, tb, tb.nx + tb.ny, z0 + lane);
            if (lane == 0 && z0 + 32 < v.nz) z |= put_node<P>(w, NZ + 32, tb, tb.nx + tb.ny, z0 + 32);
            const bool zero = __any_sync(FULL, z);
            __syncwarp();
            uint32_t act;
            {
                const unsigned long long a = w.win[1][lane + 1], b = w.win[1][lane + 2], c = w.win[2][lane + 1],
                                         d = w.win[2][lane + 2];
                const unsigned long long o = a | b | c | d, n = a & b & c & d;
                act = mine ? ((uint32_t)(o >> 1) | (uint32_t)(o >> 2)) & ~((uint32_t)(n >> 1) & (uint32_t)(n >> 2)) &
                                 cell_mask(v.cz, zw)
                           : 0u;
            }
            const int n = __popc(act);
            int end = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(FULL, end, o);
                if (lane >= o) end += t;
            }
            const int total = __shfl_sync(FULL, end, 31), beg = end - n;
            for (int i = beg; act; i++, act &= act - 1) w.queue[i] = (uint16_t)(lane | ((__ffs(act) - 1) << 5));
            const T *sw = s0 + (int64_t)z0 * v.sxy;
            __syncwarp();
            // the samples of the next batch are in flight while this one is emitted
            T s[8];
            uint32_t ent = lane < total ? w.queue[lane] : w.queue[0];
            if (total) load_corners(s, sw, ent, v);
            for (int j0 = 0; j0 < total; j0 += 32) {
                const bool on = j0 + lane < total;
                const int ln = (int)(ent & 31u), zc = (int)(ent >> 5);
                // the cell's 3 x 3 columns: t1 samples z, z+1; t0 samples z-1, z
                uint32_t t0[3][3], t1[3][3], cu[3][3], sh[3][3];
#pragma unroll
                for (int r = 0; r < 3; r++)
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        const unsigned long long l = w.win[r][ln + c];
                        const uint32_t u = (uint32_t)(l >> zc);
                        t0[r][c] = u & 3u;
                        t1[r][c] = (u >> 1) & 3u;
                        cu[r][c] = (uint32_t)(l >> 1);
                        sh[r][c] = (uint32_t)(l >> 2);
                    }
                const uint32_t low = (1u << zc) - 1u;  // cells of the word below this one
                const int cx = x0 + ln, cz = z0 + zc;
                const int gx = (int)min((int64_t)2, cx + p.xg0), gy = min(2, y), gz = min(2, cz);
                // a cell on a lower face, or with a neighbour there
                const bool edge = EDGES && __any_sync(FULL, on && (gx < 2 || gy < 2 || gz < 2));
                uint32_t idx = 0;
                long long id = 0;
#pragma unroll
                for (int dy = 0; dy < 2; dy++)
#pragma unroll
                    for (int dx = 0; dx < 2; dx++) {
                        const int r = 1 - dy, c = 1 - dx;
                        uint32_t pre;
                        if constexpr (EDGES) {
                            const uint32_t ws[8] = {cu[r][c], cu[r + 1][c], cu[r + 1][c + 1], cu[r][c + 1],
                                                    sh[r][c], sh[r + 1][c], sh[r + 1][c + 1], sh[r][c + 1]};
                            pre = own_below<ALG>(ws, low);
                            // (the first word holds cells of the first plane below this one)
                            if (edge || zw == 0)
                                pre += own_extra<ALG, 0>(ws, low, zw == 0 ? low & 1u : 0u, (gx == dx) | ((gy == dy) << 1));
                        } else {
                            const uint32_t o = cu[r][c] | cu[r][c + 1] | cu[r + 1][c] | cu[r + 1][c + 1] | sh[r][c] |
                                               sh[r][c + 1] | sh[r + 1][c] | sh[r + 1][c + 1];
                            const uint32_t a = cu[r][c] & cu[r][c + 1] & cu[r + 1][c] & cu[r + 1][c + 1] & sh[r][c] &
                                               sh[r][c + 1] & sh[r + 1][c] & sh[r + 1][c + 1];
                            pre = __popc(o & ~a & low);
                        }
                        const long long i1 = w.col[r][ln + c] + pre;  // the cell back along (dx, dy)
                        const uint32_t k1 = t1[r][c] | (t1[r][c + 1] << 2) | (t1[r + 1][c] << 4) | (t1[r + 1][c + 1] << 6);
                        const uint32_t k0 = t0[r][c] | (t0[r][c + 1] << 2) | (t0[r + 1][c] << 4) | (t0[r + 1][c + 1] << 6);
                        // and the one below it
                        uint32_t n0;
                        if constexpr (EDGES) {
                            n0 = ct.nvf[k0] & 15u;
                            if (edge)
                                n0 = __popc(full_tabs<ALG>().touched[k0] &
                                            full_tabs<ALG>().own[(gx == dx) | ((gy == dy) << 1) | ((gz == 1) << 2)]);
                            w.nb[dx | (dy << 1)][lane] = (i1 << 8) | k1;
                            if (dx + dy < 2) w.nb[4 | dx | (dy << 1)][lane] = ((i1 - n0) << 8) | k0;
                        } else {
                            n0 = k0 != 0u && k0 != 255u;
                            w.nb[dx | (dy << 1)][lane] = i1;
                            if (dx + dy < 2) w.nb[4 | dx | (dy << 1)][lane] = i1 - n0;
                        }
                        if (dx + dy == 0) {
                            idx = k1;
                            id = i1;
                        }
                    }
                // own vertices (NSN: crossings) and faces
                const int bnd = (gx == 0) | ((gy == 0) << 1) | ((gz == 0) << 2);
                uint32_t nv, nf, nverts = 1;
                if constexpr (EDGES) {
                    nv = ct.nvf[idx] & 15u;
                    nf = ct.nvf[idx] >> 4;
                    if (edge && bnd) nv = __popc(full_tabs<ALG>().touched[idx] & full_tabs<ALG>().own[bnd]);
                    nverts = nv;
                } else {
                    nv = ct.n[idx];
                    const uint32_t s = idx & 1u;
                    nf = 2u * ((s != ((idx >> 2) & 1u) && !(bnd & 6)) + (s != ((idx >> 4) & 1u) && !(bnd & 5)) +
                               (s != ((idx >> 1) & 1u) && !(bnd & 3)));
                }
                uint32_t acc = on ? nv | (nf << 16) : 0u, inc = acc;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t t = __shfl_up_sync(FULL, inc, o);
                    if (lane >= o) inc += t;
                }
                uint32_t tot = __shfl_sync(FULL, inc, 31), exc = inc - acc;
                {
                    // this column's cells of the batch are lo .. hi - 1
                    const int lo = min(max(beg - j0, 0), 32), hi = min(max(end - j0, 0), 32);
                    const uint32_t el = __shfl_sync(FULL, exc, lo & 31), eh = __shfl_sync(FULL, exc, hi & 31);
                    const long long f0 = gf - (long long)((lo == 32 ? tot : el) >> 16);
                    gf = f0 + ((hi == 32 ? tot : eh) >> 16);
                    w.fb[lane] = __shfl_sync(FULL, f0, ln) + (exc >> 16);
                }
                const bool fits = !on || (id + nverts <= p.verts_cap && w.fb[lane] + nf <= p.faces_cap);
                if (!__all_sync(FULL, fits)) {  // cells past the outputs' room are left out
                    if (!fits) {
                        *p.err = ERR_CAPACITY;
                        acc = 0;
                    }
                    inc = acc;
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t t = __shfl_up_sync(FULL, inc, o);
                        if (lane >= o) inc += t;
                    }
                    tot = __shfl_sync(FULL, inc, 31);
                    exc = inc - acc;
                }
                const int VW = (int)(tot & 0xffffu), FW = (int)(tot >> 16);
#pragma unroll
                for (int g = 0; g < 8; g++) w.val[lane * VS + g] = s[g];
                const uint32_t fv = exc & 0xffffu, ff = exc >> 16;
                const uint32_t rec = idx | ((uint32_t)ln << 8) | ((uint32_t)zc << 13);
                const uint32_t vrec = rec | (fv << 18), frec = rec | (ff << 18);
                {
                    const uint32_t bv = __ballot_sync(FULL, (acc & 0xffffu) != 0u), bf = __ballot_sync(FULL, (acc >> 16) != 0u);
                    const uint32_t lt = (1u << lane) - 1u;
                    if (acc & 0xffffu) w.ov[__popc(bv & lt)] = (uint8_t)lane;
                    if (acc >> 16) w.of[__popc(bf & lt)] = (uint8_t)lane;
                }
                const uint32_t vr = (acc & 0xffffu) ? fv >> 5 : 0xffu, fr = (acc >> 16) ? ff >> 5 : 0xffu;
                if (j0 + 32 < total) {
                    ent = j0 + 32 + lane < total ? w.queue[j0 + 32 + lane] : w.queue[0];
                    load_corners(s, sw, ent, v);
                }
                __syncwarp();
                int cb = -1;
                bool odd = false;
                for (int r = 0; 32 * r < VW; r++) {
                    const uint32_t bits = __reduce_or_sync(FULL, vr == (uint32_t)r ? 1u << (fv & 31u) : 0u);
                    const int t = 32 * r + lane, j = w.ov[cb + __popc(bits & lanemask_le(lane))];
                    cb += __popc(bits);
                    const uint32_t rc = __shfl_sync(FULL, vrec, j);
                    if (t >= VW) continue;
                    const uint32_t ci = rc & 255u;
                    const int cl = (int)((rc >> 8) & 31u), zz = (int)((rc >> 13) & 31u), i = t - (int)(rc >> 18);
                    if constexpr (EDGES) {
                        int e = ct.kth[ci][i & (EdgeDims<ALG>::OWN - 1)];
                        if (edge) {
                            const int b = (x0 + cl + p.xg0 == 0) | ((y == 0) << 1) | ((z0 + zz == 0) << 2);
                            if (b) {
                                const uint32_t om = full_tabs<ALG>().own[b] & full_tabs<ALG>().touched[ci];
                                int seen = i;
                                for (int u = 0; u < EdgeDims<ALG>::V; u++) {
                                    const int ee = full_tabs<ALG>().order[ci][u];
                                    if (ee < EdgeDims<ALG>::E && ((om >> ee) & 1u) && seen-- == 0) {
                                        e = ee;
                                        break;
                                    }
                                }
                            }
                        }
                        const int cc = ct.corner[e], c1 = cc & 7, c2 = cc >> 3;
                        P pt[3];
                        if constexpr (ALG == MESH_ALG_MT) {
                            const P b3[3] = {w.p[NX + cl], w.p[NY], w.p[NZ + zz]}, d3[3] = {w.d[NX + cl], w.d[NY], w.d[NZ + zz]};
                            mt_point<T, Q, A, P>(p, c1, c2, w.val[j * VS + c1], w.val[j * VS + c2], b3, d3, pt);
                        } else {
                            // vertex_interp (src/marching_cubes.jl:100-104) from the edge's start
                            const Q mu = quotient<Q>(w.val[j * VS + c1], w.val[j * VS + c2], p);
                            const int lo[3] = {NX + cl, NY, NZ + zz};
                            const bool lit = zero || !bits_finite(mu);
#pragma unroll
                            for (int u = 0; u < 3; u++) {
                                const int u1 = (c1 >> u) & 1;
                                const P p1 = w.p[lo[u] + u1];
                                if (u1 != ((c2 >> u) & 1))
                                    pt[u] = Ar<P>::add(p1, Ar<P>::mul((P)mu, u1 ? -w.d[lo[u]] : w.d[lo[u]]));
                                else
                                    pt[u] = lit ? Ar<P>::add(p1, Ar<P>::mul((P)mu, P(0))) : p1;
                            }
                        }
                        store_point<P>(p, (w.nb[0][j] >> 8) + i, pt[0], pt[1], pt[2]);
                    } else {
                        const int g = ct.edge[ci][i], a = g & 7, ax = g >> 3, b = a ^ (1 << ax);
                        const Q mu = quotient<Q>(w.val[j * VS + a], w.val[j * VS + b], p);
                        const int lo = ax == 0 ? NX + cl : (ax == 1 ? NY : NZ + zz);
                        const bool neg = a > b;
                        const P d = neg ? -w.d[lo] : w.d[lo];
                        w.pr.r[t] = Ar<P>::add(w.p[lo + neg], Ar<P>::mul((P)mu, d));
                        const int f = !bits_finite(mu) ? 3 : (zero ? (signbit(mu) ? 2 : 1) : 0);
                        odd |= f != 0;
                        w.pr.odd[t] = (uint8_t)f;
                    }
                }
                if constexpr (ALG == MESH_ALG_NSN) {
                    odd = __any_sync(FULL, odd);
                    __syncwarp();
                    if (acc) {
                        // the mean of the cell's crossings, summed in edge order
                        P m[3] = {P(0), P(0), P(0)};
                        for (uint32_t i = 0; i < nv; i++) {
                            const int g = ct.edge[idx][i], a = g & 7, ax = g >> 3;
                            P c[3] = {w.p[NX + ln + (a & 1)], w.p[NY + ((a >> 1) & 1)], w.p[NZ + zc + (a >> 2)]};
                            const int f = odd ? w.pr.odd[fv + i] : 0;
                            if (f) {
                                const P add = f == 3 ? (P)__longlong_as_double(0x7ff8000000000000ll) : (f == 2 ? -P(0) : P(0));
#pragma unroll
                                for (int u = 0; u < 3; u++) c[u] = Ar<P>::add(c[u], add);
                            }
                            const P mv = w.pr.r[fv + i];
#pragma unroll
                            for (int u = 0; u < 3; u++) {
                                const P cu1 = u == ax ? mv : c[u];
                                // 0 + c is c, or +0 when c is -0
                                m[u] = i ? Ar<P>::add(m[u], cu1) : (bits_zero(cu1) ? P(0) : cu1);
                            }
                        }
                        store_point<P>(p, id, div_count(m[0], (int)nv, rcp), div_count(m[1], (int)nv, rcp),
                                       div_count(m[2], (int)nv, rcp));
                    }
                }
                cb = -1;
                for (int r = 0; 32 * r < FW; r++) {
                    const uint32_t bits = __reduce_or_sync(FULL, fr == (uint32_t)r ? 1u << (ff & 31u) : 0u);
                    const int t = 32 * r + lane, j = w.of[cb + __popc(bits & lanemask_le(lane))];
                    cb += __popc(bits);
                    const uint32_t rc = __shfl_sync(FULL, frec, j);
                    if (t >= FW) continue;
                    const uint32_t ci = rc & 255u;
                    const int i = t - (int)(rc >> 18);
                    long long *out = (long long *)p.faces + 3 * (w.fb[j] + i);
                    if constexpr (EDGES) {
                        long long vid[3];
                        const uint32_t corners = ct.ref[ci][i];
#pragma unroll
                        for (int u = 0; u < 3; u++) {
                            int e = (int)(corners >> (8 * u)) & 31, m = (int)(corners >> (8 * u + 5)) & 7;
                            int b = 0;
                            if (edge) {
                                const int cl = (int)((rc >> 8) & 31u), zz = (int)((rc >> 13) & 31u);
                                const int hx = (int)min((int64_t)2, x0 + cl + p.xg0), hy = min(2, y), hz = min(2, z0 + zz);
                                const int here = (hx == 0) | ((hy == 0) << 1) | ((hz == 0) << 2);
                                e = ct.unmoved[m & here][e];  // no step back past the grid's face
                                m &= ~here;
                                b = (hx == (m & 1)) | ((hy == ((m >> 1) & 1)) << 1) | ((hz == (m >> 2)) << 2);
                            }
                            const long long nb = w.nb[m][j];
                            const uint32_t ni = (uint32_t)nb & 255u;
                            const int rank = b ? __popc(full_tabs<ALG>().before[ni][e] & full_tabs<ALG>().own[b]) : (int)ct.rank[ni][e];
                            vid[u] = (nb >> 8) + rank + 1;
                        }
                        put3((int64_t *)out, vid[0], vid[1], vid[2]);
                    } else {
                        // the (i/2)-th crossed base edge with four cells around it, triangle i%2
                        const int cl = (int)((rc >> 8) & 31u), zz = (int)((rc >> 13) & 31u);
                        const bool xk = x0 + cl + p.xg0 > 0, yk = y > 0, zk = z0 + zz > 0;
                        const uint32_t s1 = ci & 1u;
                        const bool ex = s1 != ((ci >> 2) & 1u) && yk && zk, ey = s1 != ((ci >> 4) & 1u) && zk && xk;
                        const int h = i >> 1;
                        const int kind = h == 0 ? (ex ? 0 : (ey ? 1 : 2)) : (h == 1 ? (ex && ey ? 1 : 2) : 2);
                        const int mA = kind == 0 ? 6 : (kind == 1 ? 5 : 3), mB = kind == 0 ? 4 : (kind == 1 ? 1 : 2),
                                  mD = kind == 0 ? 2 : (kind == 1 ? 4 : 1);
                        // (A, B, C), (A, C, D), reversed when the edge's start is not below iso
                        const long long vA = w.nb[mA][j] + 1, vC = w.nb[0][j] + 1, vS = w.nb[(i & 1) ? mD : mB][j] + 1;
                        const bool keep = (s1 != 0) != ((i & 1) != 0);
                        put3((int64_t *)out, vA, keep ? vS : vC, keep ? vC : vS);
                    }
                }
                __syncwarp();  // the next batch rewrites the records
            }
        }
    }
}

template <class T, class Q, class A, class P, int ALG>
__global__ void __launch_bounds__(32 * SW, 2) k_emit_shared(const Plan p, int seg0, int nseg, int nitems, int lg) {
    using Tab = typename TabsOf<ALG>::type;
    extern __shared__ __align__(16) unsigned char ssm[];
    __shared__ P s_rcp[13];  // NSN: RN(1/n) for the crossing counts n
    Tab &ct = *reinterpret_cast<Tab *>(ssm);
    SharedWarp<T, P, ALG> *sw = reinterpret_cast<SharedWarp<T, P, ALG> *>(ssm + (sizeof(Tab) + 15) / 16 * 16);
    const uint4 *src = ALG == MESH_ALG_MT    ? reinterpret_cast<const uint4 *>(&d_mt)
                       : ALG == MESH_ALG_NSN ? reinterpret_cast<const uint4 *>(&d_nsn)
                                             : reinterpret_cast<const uint4 *>(&d_mc);
    for (int i = threadIdx.x; i < (int)(sizeof(Tab) / 16); i += blockDim.x) reinterpret_cast<uint4 *>(&ct)[i] = src[i];
    if (ALG == MESH_ALG_NSN && threadIdx.x <= 12)
        s_rcp[threadIdx.x] = threadIdx.x ? Ar<P>::div(P(1), (P)(int)threadIdx.x) : P(0);
    __syncthreads();
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    const BView v = view_of(p);
    const Tabs tb = tabs_of(p);
    after_previous();
    for (;;) {
        int item = 0;
        if (lane == 0) item = (int)atomicAdd(p.work, 1u);
        item = __shfl_sync(FULL, item, 0);
        if (item >= nitems) break;
        const int q = item >> lg, width = 32 >> lg, part = item & ((1 << lg) - 1);  // 1 << lg parts of 32 columns
        const int xb = q % v.nxb;
        const int seg = seg0 + (q / v.nxb) % nseg;
        const int y = q / (v.nxb * nseg);
        emit_item<T, Q, A, P, ALG>(p, v, tb, sw[wi], ct, s_rcp, lane, xb, y, seg,
                                   (FULL >> (32 - width)) << (width * part));
    }
}

// Resident CTAs of a kernel on the current device, with its dynamic shared memory
// allowed (one-time per device and instantiation).
template <class T, class Q, class A, class P, int ALG> int shared_grid() {
    static std::mutex mu;
    static int grid[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return 0;
    std::lock_guard<std::mutex> lk(mu);
    if (!grid[dev]) {
        const void *fn = (const void *)k_emit_shared<T, Q, A, P, ALG>;
        const int smem = (int)shared_smem<T, P, ALG>();
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        int sms = 0, per_sm = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 32 * SW, smem) != cudaSuccess || per_sm < 1)
            per_sm = 1;
        cudaGetLastError();
        grid[dev] = per_sm * sms;
    }
    return grid[dev];
}

template <class T, class Q, class A, class P, int ALG> cudaError_t go(const Plan &p, int seg0, int nseg, cudaStream_t s) {
    const int grid = shared_grid<T, Q, A, P, ALG>();
    const int64_t rows = (int64_t)p.nxb * nseg * p.cy;
    const int lg = rows < 2 * SW * (int64_t)grid ? 2 : 0;  // as in k_emit_bits.cu
    const int64_t nitems = rows << lg;
    if (grid < 1) return cudaErrorInvalidDevice;
    if (nitems > 0x7fffffff - 65536) return cudaErrorInvalidConfiguration;
    if (nitems < 1) return cudaSuccess;
    return launch_after(k_emit_shared<T, Q, A, P, ALG>, (unsigned)std::min<int64_t>(grid, nitems), 32 * SW,
                        shared_smem<T, P, ALG>(), s, p, seg0, nseg, (int)nitems, lg);
}

template <class T> cudaError_t go_t(const Plan &p, int Q64, int A64, int P64, int seg0, int nseg, cudaStream_t s) {
    if (p.alg == MESH_ALG_MT) {
        if (Q64) return go<T, double, double, double, MESH_ALG_MT>(p, seg0, nseg, s);
        if (A64) return go<T, float, double, double, MESH_ALG_MT>(p, seg0, nseg, s);
        if (P64) return go<T, float, float, double, MESH_ALG_MT>(p, seg0, nseg, s);
        return go<T, float, float, float, MESH_ALG_MT>(p, seg0, nseg, s);
    }
    if (p.alg == MESH_ALG_MC_WELDED) {
        if (Q64) return go<T, double, double, double, MESH_ALG_MC_WELDED>(p, seg0, nseg, s);
        if (P64) return go<T, float, float, double, MESH_ALG_MC_WELDED>(p, seg0, nseg, s);
        return go<T, float, float, float, MESH_ALG_MC_WELDED>(p, seg0, nseg, s);
    }
    if (Q64) return go<T, double, double, double, MESH_ALG_NSN>(p, seg0, nseg, s);
    if (P64) return go<T, float, float, double, MESH_ALG_NSN>(p, seg0, nseg, s);
    return go<T, float, float, float, MESH_ALG_NSN>(p, seg0, nseg, s);
}

}  // namespace

cudaError_t launch_emit_shared(const Plan &p, int Q64, int A64, int P64, int seg0, int nseg, cudaStream_t s) {
    switch (p.T) {
    case MESH_DT_U16: return go_t<uint16_t>(p, Q64, A64, P64, seg0, nseg, s);
    case MESH_DT_F16: return go_t<h16>(p, Q64, A64, P64, seg0, nseg, s);
    case MESH_DT_I16: return go_t<int16_t>(p, Q64, A64, P64, seg0, nseg, s);
    case MESH_DT_I8: return go_t<int8_t>(p, Q64, A64, P64, seg0, nseg, s);
    case MESH_DT_U8: return go_t<uint8_t>(p, Q64, A64, P64, seg0, nseg, s);
    case MESH_DT_F32: return go_t<float>(p, Q64, A64, P64, seg0, nseg, s);
    case MESH_DT_I32: return go_t<int32_t>(p, Q64, A64, P64, seg0, nseg, s);
    case MESH_DT_I64: return go_t<int64_t>(p, Q64, A64, P64, seg0, nseg, s);
    default:
        if (p.alg == MESH_ALG_MT) return go<double, double, double, double, MESH_ALG_MT>(p, seg0, nseg, s);
        if (p.alg == MESH_ALG_MC_WELDED) return go<double, double, double, double, MESH_ALG_MC_WELDED>(p, seg0, nseg, s);
        return go<double, double, double, double, MESH_ALG_NSN>(p, seg0, nseg, s);
    }
}

}  // namespace mesh
