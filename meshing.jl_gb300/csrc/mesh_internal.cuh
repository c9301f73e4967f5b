// Internal definitions shared by the host runtime (mesh_api.cu) and the
// kernels (k_*.cu).  Not part of the public ABI.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "mesh_quot.h"
#include "meshing_gb300.h"  // include/ (on the include path)

namespace mesh {

// Tiling.  A warp tile covers 32 consecutive x samples (one per lane) and
// WY+1 consecutive y sample rows, and walks z.  Lane 31 only supplies the
// x+1 sample of lane 30, so a tile holds 31 cells in x (30 for the emit
// kernels that also need the -x neighbour cell, kept in lane 0).
constexpr int WY = 4;            // cell rows per warp tile
constexpr int WARPS = 8;         // warps per CTA
constexpr int TILE_X = 31;       // cells per tile in x (classify, MC emit)
constexpr int TILE_XH = 30;      // cells per tile in x (MT / NSN emit, with -x halo)
constexpr int ZC = 8;            // cells per activity chunk in z
constexpr int NCNT = 3;          // per-piece counters: vertices, faces, active cells
constexpr int ENT_BLOCK = 256;   // active-cell entries per expansion block
constexpr int POS_BITS = 21;     // bits per coordinate in a packed cell position

// Error bits of the device error word.
constexpr unsigned ERR_CAPACITY = 2u;
constexpr unsigned ERR_BOUNDS = 4u;
constexpr unsigned ERR_STAGE = 16u;  // the staged entry list was too short

struct BatchVol;

struct Plan {
    // volume (Julia layout: x fastest)
    const void *vol;
    int64_t nx, ny, nz;
    int32_t cx, cy, cz;  // cells = samples - 1
    int32_t T, alg;
    int32_t out64;       // output eltype is Float64
    // classification thresholds: v < iso  <=>  v < thr (exact, in the data type)
    float thr_f;
    double thr_d;
    int32_t thr_i;       // UInt16 data
    int64_t thr_l;       // Int32 / Int64 data: v < iso  <=>  v < thr_l, or every v (thr_all)
    int32_t thr_all;
    // Int64 iso on Int64 data: (iso - v1) is an Int64 difference (wrapping)
    int64_t iso_l;
    int32_t iso_int;
    int32_t iso_small, iso_s;  // iso is the integer iso_s, at most 2^30 in magnitude
    int32_t iso_zero;          // iso == 0 (tested here: a Float64 comparison is a Float64 operation)
    // iso as it enters (iso - v1)/(v2 - v1)
    float isoq_f;
    double isoq_d;
    // MT clamp bounds eps and one(T)-eps, in the clamp type
    float eps_f, hi_f;
    double eps_d, hi_d;
    uint32_t own[8];     // MT: edges owned by a cell, by (x==0)|(y==0)<<1|(z==0)<<2
    // LinRange node coordinates: exact values (L may be Float32) stored as double,
    // the same rounded to float, and the node spacings L(p[i+1]-p[i]).
    const double *xp, *yp, *zp;
    const double *dx, *dy, *dz;
    const float *xpf, *ypf, *zpf;
    const float *dxf, *dyf, *dzf;
    // float pairs hi + lo of the node coordinates and spacings (for the exact
    // float fast path of Float64 positions rounded to Float32): split[k][ntab]
    // with k = 0 p_hi, 1 p_lo, 2 d_hi, 3 d_lo, nodes of x, then y, then z
    const float *split;
    int64_t ntab;
    int32_t force_fp64;   // disable the float fast path (diagnostics)
    // z segments and activity chunks
    int32_t zs, nseg, chunks_per_seg, nchunks;
    int32_t tiles_x, tiles_y;  // classify tiling (TILE_X x WY cells)
    // scratch
    int64_t pstride;      // elements between the counters' arrays in cnt / base
    uint32_t *cnt;        // [NCNT][nseg][cy][cx] per-piece vertex / face / active-cell counts
    int64_t *base;        // [NCNT][nseg][cy][cx] exclusive prefix in traversal order
    uint8_t *flags;       // [nchunks][tiles_x][cy] 1 if the tile row has an active cell
    unsigned long long *scan_state;  // list form: run and column sums of the scan
    int64_t *totals;      // [NCNT] total vertices, faces, active cells
    unsigned int *err;    // device error word
    unsigned int *work;   // work-item counter of the persistent kernels
    // welded Marching Cubes: per emitted vertex, its lattice edge
    // (axis + 3 * linear index of the edge's lower node), bit 63 set when the
    // emitting cell is the edge's first cell in emission order (null: not written)
    long long *vkey;
    // list of active cells (Marching Cubes): packed x | y << 21 | z << 42,
    // case, the 8 corner values; in emission order with, for every 256th
    // entry, the vertex / face offsets of that entry (ent_side), or in the
    // order the walk found them with each entry's vertex / face rank inside
    // its piece (ent_rank) and *stage_next slots handed out
    unsigned long long *ent_pos;
    uint8_t *ent_cs;
    void *ent_val;
    long long *ent_side;
    uint2 *ent_rank;
    unsigned long long *stage_next;
    int64_t ent_cap;
    // outputs
    void *verts;
    int64_t *faces;
    int64_t verts_cap, faces_cap;
    // batches (Marching Cubes over many volumes in one pass): per-volume
    // descriptors, and the first vertex / face of every volume ([nvols + 1][2],
    // the last row the totals)
    const BatchVol *bvols;
    int64_t *vol_off;
    int32_t nvols;
    int32_t vol_outputs;  // 1: every volume writes to its own BatchVol::verts / faces
    // x window (mesh_set_x_window): global x of the volume's sample 0, for the
    // grid-boundary rules of MT / NSN; with xhalo, the volume's first cell column
    // is the previous slab's last one -- counted (its vertices come first in the
    // scan) but not emitted, and every emitted vertex, face and face index is
    // shifted down by that column's totals (base of piece (seg 0, y 0, x 1))
    int64_t xg0;
    int32_t xhalo;
    // emission of a range of column blocks (the pipelined host path; ntx 0: all)
    int32_t tx0, ntx;
    // sign bits (mesh_bits.cuh): words bw0 .. bw1 - 1 of z at `bits`, z segments of
    // zws words (bseg of them) and column / row blocks; per piece, the vertex and
    // face counts that the offset scan turns into offsets within their scan tile
    // (pc), per tile the sums that become the tiles' offsets (tsum), and the masks
    // of active words (wmask)
    uint32_t *bits;
    uint2 *pc;
    ulonglong2 *tsum;
    uint32_t *wmask;
    uint32_t *vpre;       // MT / NSN: vertices of a column's segment before word zw, at the words' places
    unsigned int *done;   // CTAs of k_count that have finished
    int64_t npc;
    int64_t *tot_out;     // where k_count also leaves the totals (device or pinned; null: nowhere)
    int32_t nxb, nyb, bseg, zws, nzw, bw0, bw1, ntiles;
    // batches: the volume of each CTA of the bit and count kernels, and their number
    const uint32_t *bblk_vol, *cblk_vol;
    int64_t nbblk, ncblk;
};

// One volume of a batch.  Its sign words, pieces, activity masks and CTAs of the
// bit and count kernels are ranges of the batch's arrays starting at bits0, e0, m0,
// bblk0 and cblk0 (tiling as in Plan; vec: its planes take 16-byte loads); its
// coordinate tables are a block at `tabs` (k_tables.cu layout).
// With Plan::vol_outputs its mesh goes to its own verts / faces (room for
// vcap / fcap) instead of the batch's concatenated outputs.
struct BatchVol {
    const void *vol;
    const double *tabs;
    int64_t nx, ny, nz;
    int32_t cx, cy, cz, nxb, nyb, bseg, zws, nzw, vec;
    int64_t bits0, e0, m0, bblk0, cblk0;
    void *verts;
    int64_t *faces;
    int64_t vcap, fcap;
    int64_t kbase;  // welded batches: the volume's lattice-edge keys start here
};

// Bytes per sample of a volume dtype.
inline __host__ __device__ size_t dtype_size(int T) {
    return (T == MESH_DT_I8 || T == MESH_DT_U8) ? 1
           : (T == MESH_DT_U16 || T == MESH_DT_F16 || T == MESH_DT_I16) ? 2
           : (T == MESH_DT_F32 || T == MESH_DT_I32) ? 4 : 8;
}

inline __host__ __device__ int64_t npieces(const Plan &p) { return (int64_t)p.nseg * p.cy * p.cx; }

// Coordinate tables of one volume (pointers into its table block).
struct Tabs {
    const double *xp, *yp, *zp, *dx, *dy, *dz;
    const float *xpf, *ypf, *zpf, *dxf, *dyf, *dzf, *split;
    int64_t ntab, nx, ny;
};
inline __host__ __device__ Tabs tabs_of(const Plan &p) {
    return Tabs{p.xp, p.yp, p.zp, p.dx, p.dy, p.dz, p.xpf, p.ypf, p.zpf, p.dxf, p.dyf, p.dzf, p.split,
                p.ntab, p.nx, p.ny};
}
// The tables of a block at dp (k_tables.cu layout) for nx, ny, nz nodes.
inline __host__ __device__ Tabs tabs_at(const double *dp, int64_t nx, int64_t ny, int64_t nz) {
    const int64_t ntab = nx + ny + nz;
    const double *dd = dp + ntab;
    const float *fp = (const float *)(dp + 2 * ntab), *fd = fp + ntab;
    return Tabs{dp, dp + nx, dp + nx + ny, dd, dd + nx, dd + nx + ny, fp, fp + nx, fp + nx + ny,
                fd, fd + nx, fd + nx + ny, fp + 2 * ntab, ntab, nx, ny};
}
inline __host__ __device__ void set_tabs(Plan &P, const Tabs &t) {
    P.xp = t.xp; P.yp = t.yp; P.zp = t.zp; P.dx = t.dx; P.dy = t.dy; P.dz = t.dz;
    P.xpf = t.xpf; P.ypf = t.ypf; P.zpf = t.zpf; P.dxf = t.dxf; P.dyf = t.dyf; P.dzf = t.dzf;
    P.split = t.split;
    P.ntab = t.ntab;
}
inline __host__ __device__ int64_t piece(const Plan &p, int seg, int y, int x) {
    return ((int64_t)seg * p.cy + y) * p.cx + x;
}

// Coordinate tables (k_tables.cu): bytes for ntab = nx+ny+nz nodes, and the
// Plan's pointers into a table block at dp.
inline size_t table_bytes(int64_t ntab) {
    return (size_t)ntab * 2 * (sizeof(double) + sizeof(float)) + (size_t)ntab * 4 * sizeof(float);
}
inline void bind_tables(Plan &P, const double *dp, int64_t nx, int64_t ny, int64_t nz) {
    set_tabs(P, tabs_at(dp, nx, ny, nz));
}

// Welded batches (k_weld.cu): blocks of the ownership scan and hash slots for nv
// per-cell vertices; launch_weld_batch welds verts / faces (faces in place) into
// wverts, bsum[nb] = the welded vertex count.
int64_t weld_blocks(int64_t nv);
int64_t weld_hash_slots(int64_t nv);
// The counts are read on the device (tot[0] vertices,
// tot[1] faces, at most nvmax / nfmax), faces are 1-based within their volume
// (first vertex / face of volume v at vol_off[2v], vol_off[2v + 1]; row n the
// totals) before and after, and woff receives the welded rows.
cudaError_t launch_weld_batch(const long long *vkey, int64_t nvmax, int64_t nfmax, const int64_t *tot,
                              const void *verts, int out64, int64_t *faces, const int64_t *vol_off, int n,
                              int64_t *woff, long long *bsum, void *wverts, unsigned long long *hkey, long long *hval,
                              int64_t hcap, unsigned *err, int sms, cudaStream_t s);

// Launchers (each returns cudaError_t of the launch).
// xoff / nxt: the volume is x nodes xoff .. xoff+nx-1 of an axis of nxt nodes (0, 0: the whole axis).
cudaError_t launch_tables(double *tabs, int64_t nx, int64_t ny, int64_t nz, const double *range, int L32,
                          cudaStream_t s, int64_t xoff = 0, int64_t nxt = 0);
// Tables of many volumes: job i fills the block at dst[i] (one CTA row per job).
struct TabJob {
    double *dst;
    int64_t nx, ny, nz;
    double range[6];
};
cudaError_t launch_tables_batch(const TabJob *jobs, int njobs, int64_t max_ntab, int L32, cudaStream_t s);
// Batched Marching Cubes stages (k_bits.cu, k_emit_bits.cu); ctas: CTAs per SM of
// the persistent emission (0 = as many as fit), which also leaves the first vertex
// and face of every volume in Plan::vol_off.
cudaError_t launch_bits_batch(const Plan &p, cudaStream_t s);
cudaError_t launch_count_batch(const Plan &p, cudaStream_t s);
cudaError_t launch_emit_batch(const Plan &p, int Q64, int P64, int ctas, cudaStream_t s);
cudaError_t launch_classify(const Plan &p, cudaStream_t s);
// Indices of a few pieces whose offsets the host wants.
constexpr int GATHER_MAX = 32;
struct GatherIdx {
    int64_t idx[GATHER_MAX];
    int n;
};
// First vertex and face of pieces e[0..n) (after the offset scan): dst[2 i], dst[2 i + 1].
cudaError_t launch_gather_pieces(const Plan &p, const GatherIdx &g, int64_t *dst, cudaStream_t s);
cudaError_t launch_scan(const Plan &p, cudaStream_t s);
// Sign bits of words w0 .. w0 + nw - 1 of z (k_bits.cu); with a job, the launch
// also fills its coordinate tables and clears the counters (Plan::totals, tsum).
struct TabArgs {
    double *tabs;
    int64_t nx, ny, nz, xoff, nxt;
    double range[6];
    int32_t L32, on;
};
cudaError_t launch_bits(const Plan &p, int w0, int nw, const TabArgs &ta, int sms, cudaStream_t s);
// Piece counts of segments seg0 .. seg0 + nseg - 1 from the bits; the last CTA of
// all segments' launches leaves the totals and the tiles' offsets, or a launch after
// them.  vpre_only: leave the words' vertex prefixes alone, for a window's emission.
// Adds the kernels launched to *kernels.
cudaError_t launch_count(const Plan &p, int seg0, int nseg, cudaStream_t s, bool vpre_only, int *kernels);
// Piece counts to offsets within their tile.
cudaError_t launch_offsets(const Plan &p, cudaStream_t s);
// Marching Cubes emitted from the bits (k_emit_bits.cu).
cudaError_t launch_emit_bits_mc(const Plan &p, int Q64, int P64, int seg0, int nseg, cudaStream_t s);
// Marching Tetrahedra / Naive Surface Nets from the bits (k_emit_shared.cu).
cudaError_t launch_emit_shared(const Plan &p, int Q64, int A64, int P64, int seg0, int nseg, cudaStream_t s);
// Marching Cubes in one walk: classify + stage entries, then expand them.
constexpr int STG_BLK = 128;  // staging slots a walking warp takes at a time
cudaError_t launch_walk_mc(const Plan &p, cudaStream_t s);
cudaError_t launch_expand_staged_mc(const Plan &p, int Q64, int P64, cudaStream_t s);

}  // namespace mesh

#ifdef __CUDACC__
namespace mesh {

// Round-to-nearest arithmetic that the compiler may not contract into FMA,
// matching Julia's separately rounded `+ - * /`.
template <class F> struct Ar;
template <> struct Ar<float> {
    static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
    static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
    static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
    static __device__ __forceinline__ float div(float a, float b) { return __fdiv_rn(a, b); }
};
template <> struct Ar<double> {
    static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
    static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
    static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
    static __device__ __forceinline__ double div(double a, double b) { return __ddiv_rn(a, b); }
};

// A Float16 sample, kept as its IEEE binary16 bits.  Every Float16 value is a
// Float32 value, so it converts exactly; T(0) is the zero sample.
struct h16 {
    uint16_t b;
    h16() = default;
    __host__ __device__ constexpr explicit h16(int) : b(0) {}
    __device__ __forceinline__ operator float() const { return __half2float(__ushort_as_half(b)); }
};
static_assert(sizeof(h16) == 2, "binary16 storage");

// v < iso, exact, in the data type.
__device__ __forceinline__ bool below(h16 v, const Plan &p) { return (float)v < p.thr_f; }
__device__ __forceinline__ bool below(float v, const Plan &p) { return v < p.thr_f; }
__device__ __forceinline__ bool below(double v, const Plan &p) { return v < p.thr_d; }
__device__ __forceinline__ bool below(uint16_t v, const Plan &p) { return (int32_t)v < p.thr_i; }
__device__ __forceinline__ bool below(uint8_t v, const Plan &p) { return (int32_t)v < p.thr_i; }
__device__ __forceinline__ bool below(int8_t v, const Plan &p) { return (int64_t)v < p.thr_l || p.thr_all; }
__device__ __forceinline__ bool below(int16_t v, const Plan &p) { return (int64_t)v < p.thr_l || p.thr_all; }
__device__ __forceinline__ bool below(int32_t v, const Plan &p) { return (int64_t)v < p.thr_l || p.thr_all; }
__device__ __forceinline__ bool below(int64_t v, const Plan &p) { return v < p.thr_l || p.thr_all; }

// A Float32 value widened to Q.  To Float64 the widening of a normal or zero
// value only moves bits (exponent rebiased by 1023 - 127, significand shifted
// up by 29), done here on the integer pipes; subnormals, Inf and NaN take the
// conversion instruction.
template <class Q> __device__ __forceinline__ Q widen(float v) { return (Q)v; }
template <> __device__ __forceinline__ double widen<double>(float v) {
    const uint32_t u = __float_as_uint(v), e = (u >> 23) & 0xffu;
    const unsigned long long sgn = (unsigned long long)(u & 0x80000000u) << 32;
    if (e != 0u && e != 0xffu)
        return __longlong_as_double((long long)(sgn | ((unsigned long long)(e + 896u) << 52) |
                                                ((unsigned long long)(u & 0x7fffffu) << 29)));
    if ((u << 1) == 0u) return __longlong_as_double((long long)sgn);
    return (double)v;
}

// v2 - v1 in the data type (UInt16 wraps), then converted to Q.
template <class Q> __device__ __forceinline__ Q tdiff(float v2, float v1) { return widen<Q>(__fsub_rn(v2, v1)); }
// Float16 - Float16 is a Float16: the Float32 difference of two Float16 values
// is exact, so rounding it to Float16 once gives the IEEE half subtraction.
template <class Q> __device__ __forceinline__ Q tdiff(h16 v2, h16 v1) {
    return (Q)__half2float(__float2half_rn(__fsub_rn((float)v2, (float)v1)));
}
template <class Q> __device__ __forceinline__ Q tdiff(double v2, double v1) { return (Q)__dsub_rn(v2, v1); }
template <class Q> __device__ __forceinline__ Q tdiff(uint16_t v2, uint16_t v1) { return (Q)(uint16_t)(v2 - v1); }
template <class Q> __device__ __forceinline__ Q tdiff(uint8_t v2, uint8_t v1) { return (Q)(uint8_t)(v2 - v1); }
template <class Q> __device__ __forceinline__ Q tdiff(int8_t v2, int8_t v1) {
    return (Q)(int8_t)(uint8_t)((uint8_t)v2 - (uint8_t)v1);
}
template <class Q> __device__ __forceinline__ Q tdiff(int16_t v2, int16_t v1) {
    return (Q)(int16_t)(uint16_t)((uint16_t)v2 - (uint16_t)v1);
}
// machine-integer differences wrap; the conversion to Q rounds to nearest
template <class Q> __device__ __forceinline__ Q tdiff(int32_t v2, int32_t v1) {
    return (Q)(int32_t)((uint32_t)v2 - (uint32_t)v1);
}
template <class Q> __device__ __forceinline__ Q tdiff(int64_t v2, int64_t v1) {
    return (Q)(int64_t)((unsigned long long)v2 - (unsigned long long)v1);
}

template <class Q> __device__ __forceinline__ Q isoq(const Plan &p);
template <> __device__ __forceinline__ float isoq<float>(const Plan &p) { return p.isoq_f; }
template <> __device__ __forceinline__ double isoq<double>(const Plan &p) { return p.isoq_d; }

// The Float64 division itself, out of line: the operands that mesh_quot.h leaves.
static __device__ __noinline__ double div_slow(double a, double b) { return __ddiv_rn(a, b); }

// (iso - v1) / (v2 - v1) in Float64 for samples whose difference has at most 32
// significant bits (all but Float64 and Int64), on the integer pipes (mesh_quot.h).
// The dividend too needs no Float64 operation when iso is 0 (the default), or a
// small integer on 8 / 16-bit samples.  Emission kernels, Float64 division -> this:
// Float32 256^3 gyroid MC 126 -> 91 us, UInt16 512^3 MC 350 -> 216; calls of MT 315 ->
// 294 and of NSN 299 -> 257.
__device__ __forceinline__ double quotient_f64(float v1, float diff, const Plan &p) {
    uint64_t q;
    const uint32_t d = __float_as_uint(diff);
    if (p.iso_zero) {  // 0 - v1 (a zero v1 is left to the division)
        if (quot_f32_f32(__float_as_uint(v1) ^ 0x80000000u, d, q)) return __longlong_as_double((long long)q);
        return div_slow(__dsub_rn(p.isoq_d, widen<double>(v1)), (double)diff);
    }
    const double num = __dsub_rn(p.isoq_d, widen<double>(v1));
    if (quot_f64_f32((uint64_t)__double_as_longlong(num), d, q)) return __longlong_as_double((long long)q);
    return div_slow(num, (double)diff);
}
template <bool SMALL> __device__ __forceinline__ double quotient_i64(int32_t v1, int32_t diff, const Plan &p) {
    uint64_t q;
    if (SMALL && p.iso_small) {
        if (quot_i32_i32(p.iso_s - v1, diff, q)) return __longlong_as_double((long long)q);
        return div_slow((double)(p.iso_s - v1), (double)diff);
    }
    const double num = __dsub_rn(p.isoq_d, (double)v1);
    if (quot_f64_i32((uint64_t)__double_as_longlong(num), diff, q)) return __longlong_as_double((long long)q);
    return div_slow(num, (double)diff);
}
__device__ __forceinline__ int32_t idiff(uint16_t v2, uint16_t v1) { return (uint16_t)(v2 - v1); }
__device__ __forceinline__ int32_t idiff(uint8_t v2, uint8_t v1) { return (uint8_t)(v2 - v1); }
__device__ __forceinline__ int32_t idiff(int16_t v2, int16_t v1) { return (int16_t)(uint16_t)((uint16_t)v2 - (uint16_t)v1); }
__device__ __forceinline__ int32_t idiff(int8_t v2, int8_t v1) { return (int8_t)(uint8_t)((uint8_t)v2 - (uint8_t)v1); }
__device__ __forceinline__ int32_t idiff(int32_t v2, int32_t v1) { return (int32_t)((uint32_t)v2 - (uint32_t)v1); }

// (iso - v1) / (v2 - v1) in Julia's promoted types.
template <class Q, class T> __device__ __forceinline__ Q quotient(T v1, T v2, const Plan &p) {
    if constexpr (sizeof(Q) == 8 && std::is_same<T, float>::value) return quotient_f64(v1, __fsub_rn(v2, v1), p);
    if constexpr (sizeof(Q) == 8 && std::is_same<T, h16>::value)
        return quotient_f64((float)v1, __half2float(__float2half_rn(__fsub_rn((float)v2, (float)v1))), p);
    if constexpr (sizeof(Q) == 8 && std::is_integral<T>::value && sizeof(T) <= 4)
        return quotient_i64<(sizeof(T) < 4)>((int32_t)v1, idiff(v2, v1), p);
    Q den = tdiff<Q>(v2, v1);
    Q num;
    if (std::is_integral<T>::value && sizeof(T) == 8 && p.iso_int)  // Int64 data, Int64 iso: Int64 (iso - v1)
        num = (Q)(int64_t)((unsigned long long)p.iso_l - (unsigned long long)(int64_t)v1);
    else if (std::is_same<T, float>::value)
        num = Ar<Q>::sub(isoq<Q>(p), widen<Q>((float)v1));
    else
        num = Ar<Q>::sub(isoq<Q>(p), (Q)v1);
    return Ar<Q>::div(num, den);
}

// Classification of IEEE values by their bits, so that Float64 tests stay off
// the (1/64-rate) FP64 pipe.
__device__ __forceinline__ bool bits_nan(float v) { return (__float_as_uint(v) << 1) > 0xff000000u; }
__device__ __forceinline__ bool bits_nan(double v) {
    return ((unsigned long long)__double_as_longlong(v) << 1) > 0xffe0000000000000ull;
}
__device__ __forceinline__ bool bits_finite(float v) { return (__float_as_uint(v) << 1) < 0xff000000u; }
__device__ __forceinline__ bool bits_finite(double v) {
    return ((unsigned long long)__double_as_longlong(v) << 1) < 0xffe0000000000000ull;
}
__device__ __forceinline__ bool bits_zero(float v) { return (__float_as_uint(v) << 1) == 0u; }
__device__ __forceinline__ bool bits_zero(double v) { return ((unsigned long long)__double_as_longlong(v) << 1) == 0ull; }

// signbit(x - y) for x, y that are not NaN: x before y in the order of the reals with
// -0.0 < +0.0, compared as integers.
__device__ __forceinline__ bool before(float x, float y) {
    const int32_t a = __float_as_int(x), b = __float_as_int(y);
    return (a ^ ((a >> 31) & 0x7fffffff)) < (b ^ ((b >> 31) & 0x7fffffff));
}
__device__ __forceinline__ bool before(double x, double y) {
    const long long a = __double_as_longlong(x), b = __double_as_longlong(y);
    return (a ^ ((a >> 63) & 0x7fffffffffffffffll)) < (b ^ ((b >> 63) & 0x7fffffffffffffffll));
}
// Base.max / Base.min on IEEE floats: NaN propagates, -0.0 < +0.0.
template <class A> __device__ __forceinline__ A jl_max(A x, A y) {
    if (bits_nan(x) || bits_nan(y)) return Ar<A>::sub(x, y);
    return before(x, y) ? y : x;
}
template <class A> __device__ __forceinline__ A jl_min(A x, A y) {
    if (bits_nan(x) || bits_nan(y)) return Ar<A>::sub(x, y);
    return before(x, y) ? x : y;
}
// x > 0 and not NaN, by its bits.
__device__ __forceinline__ bool bits_positive(float x) { return __float_as_uint(x) - 1u < 0x7f800000u; }
__device__ __forceinline__ bool bits_positive(double x) {
    return (unsigned long long)__double_as_longlong(x) - 1ull < 0x7ff0000000000000ull;
}

// fl32(fl64(p1 + fl64(mu * d))) for a Float32 mu and Float64 p1, d given as
// float pairs (p1 = p1h + p1l, d = dh + dl up to 2^-48 relative), without FP64
// instructions.  A float-float estimate r of p1 + mu*d is formed with
// TwoProduct / TwoSum; together with the two Float64 roundings of the
// reference it lies within E = 2^-42 (|p1| + |mu d|) of the exact value (the
// analysis gives about 2^-44).  If no Float32 rounding boundary lies within E
// of r, the reference result rounds to the same float f = fl32(r) and the
// function returns true; otherwise (or near underflow/overflow) it returns
// false and the caller evaluates the Float64 expression.
__device__ __forceinline__ bool fast_f32_pos(float mu, float p1h, float p1l, float dh, float dl, float &out) {
    const float ph = __fmul_rn(mu, dh);
    const float pe = __fmaf_rn(mu, dh, -ph);  // exact: mu*dh == ph + pe
    const float ql = __fmul_rn(mu, dl);
    const float sh = __fadd_rn(p1h, ph);      // TwoSum(p1h, ph) = sh + se
    const float bb = __fsub_rn(sh, p1h);
    const float se = __fadd_rn(__fsub_rn(p1h, __fsub_rn(sh, bb)), __fsub_rn(ph, bb));
    const float lo = __fadd_rn(se, __fadd_rn(p1l, __fadd_rn(pe, ql)));
    const float f = __fadd_rn(sh, lo);
    const float t = __fadd_rn(__fsub_rn(sh, f), lo);  // r - f
    const unsigned fb = __float_as_uint(f) & 0x7fffffffu;
    const int e = (int)(fb >> 23);
    out = f;
    if (e < 64 || e > 190) return false;
    float hu = __uint_as_float((unsigned)(e - 24) << 23);  // half ulp of |f|
    if ((fb & 0x7fffffu) == 0u) hu = __fmul_rn(hu, 0.5f);  // power of two: the gap towards zero is half
    const float E = __fmul_rn(__fadd_rn(fabsf(p1h), fabsf(ph)), 0x1p-42f);
    return __fadd_rn(__fmul_rn(fabsf(t), 1.0000002f), E) < hu;
}

template <class T> __device__ __forceinline__ T shfl_down1(T v) { return __shfl_down_sync(0xffffffffu, v, 1); }
template <> __device__ __forceinline__ int8_t shfl_down1<int8_t>(int8_t v) {
    return (int8_t)__shfl_down_sync(0xffffffffu, (int)v, 1);
}
template <> __device__ __forceinline__ uint8_t shfl_down1<uint8_t>(uint8_t v) {
    return (uint8_t)__shfl_down_sync(0xffffffffu, (unsigned)v, 1);
}
template <> __device__ __forceinline__ int16_t shfl_down1<int16_t>(int16_t v) {
    return (int16_t)__shfl_down_sync(0xffffffffu, (int)v, 1);
}
template <> __device__ __forceinline__ h16 shfl_down1<h16>(h16 v) {
    h16 r;
    r.b = (uint16_t)__shfl_down_sync(0xffffffffu, (unsigned)v.b, 1);
    return r;
}
template <> __device__ __forceinline__ uint16_t shfl_down1<uint16_t>(uint16_t v) {
    return (uint16_t)__shfl_down_sync(0xffffffffu, (unsigned)v, 1);
}

template <class T> __device__ __forceinline__ T ldv(const T *p) { return __ldg(p); }
template <> __device__ __forceinline__ h16 ldv<h16>(const h16 *p) {
    h16 r;
    r.b = __ldg(reinterpret_cast<const unsigned short *>(p));
    return r;
}
template <> __device__ __forceinline__ uint16_t ldv<uint16_t>(const uint16_t *p) {
    return __ldg(reinterpret_cast<const unsigned short *>(p));
}

}  // namespace mesh
#endif
