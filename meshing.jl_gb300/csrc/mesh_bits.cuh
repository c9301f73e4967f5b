// Sign bits of a volume and what the kernels built on them share.
//
// k_bits.cu reads the volume once and keeps one bit per sample, `v < iso`, in
// words of 32 consecutive z: bit k of word (zw, y, x) is sample (x, y, 32 zw + k).
// Words of one zw lie like the samples of one plane (x fastest), so a lane that
// owns column x reads its own four corner columns with coalesced loads and
// classifies 32 cells of the column with a few logic instructions.
#pragma once
#include "mesh_internal.cuh"

namespace mesh {

constexpr int BITS_TILE = 2048;  // pieces per tile of the offset scan
constexpr int BCOL = 32;         // cell columns (x) of a warp's item
constexpr int BROW = 8;          // cell rows (y) of a CTA of k_count
// Words of z in a segment: the vertices and faces of a tile of pieces stay below
// 2^32 (at most 12 per cell or node).
constexpr int ZWS_MAX = 4096;
constexpr int WORK_SLOTS = 8;    // work counters (8 bytes apart) that k_bits clears, one per emission launch

// One volume as the bit kernels see it: the plan's single volume or one of a batch.
struct BView {
    const void *vol;
    const uint32_t *bits;  // word (zw, y, x) at bits[(zw - bw0) * sxy + y * nx + x]
    int64_t nx, ny, nz, sxy;
    int32_t cx, cy, cz;
    int32_t nxb, nyb, nseg, zws, nzw, bw0;  // column / row blocks, z segments of zws words, words of z
    int64_t e0;            // first piece
    int64_t m0;            // first word of the activity masks
};

inline __host__ __device__ int mask_words(int zws) { return (zws + 31) / 32; }
// Piece of column (x, y) in z segment seg: emission order (x outermost, z fastest).
inline __host__ __device__ int64_t bpiece(const BView &v, int seg, int y, int x) {
    return v.e0 + ((int64_t)x * v.cy + y) * v.nseg + seg;
}
// Activity mask words of item (seg, y, xb): bit k of word q set when word
// seg * zws + 32 q + k of z has an active cell in the item's 32 columns.
inline __host__ __device__ int64_t bmask(const BView &v, int seg, int y, int xb) {
    return v.m0 + (((int64_t)seg * v.cy + y) * v.nxb + xb) * mask_words(v.zws);
}

}  // namespace mesh

#ifdef __CUDACC__
namespace mesh {

// Launch of a kernel that begins with after_previous(): its CTAs may start, and set
// up what depends on no earlier kernel, while the previous kernel of the stream
// drains (programmatic dependent launch; 256^3 gyroid 183 -> 171 us a call).
template <class... A, class... B>
inline cudaError_t launch_after(void (*k)(A...), unsigned grid, unsigned threads, size_t smem, cudaStream_t s, B... args) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    cudaLaunchAttribute a = {};
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &a;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, k, static_cast<A>(args)...);
}
// What the previous kernel writes is read with plain loads: the read-only path (__ldg)
// is for memory that nothing writes while the CTAs may be resident, here the samples and
// the coordinate tables (windows of MT, NSN and welded meshes follow k_count, which writes
// the activity masks, without a kernel between).
__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ BView view_of(const Plan &p) {
    return BView{p.vol, p.bits, p.nx, p.ny, p.nz, p.nx * p.ny, p.cx, p.cy, p.cz, p.nxb, p.nyb,
                 p.bseg, p.zws, p.nzw, p.bw0, 0, 0};
}

__device__ __forceinline__ BView view_of(const Plan &p, const BatchVol &b) {
    return BView{b.vol, p.bits + b.bits0, b.nx, b.ny, b.nz, b.nx * b.ny, b.cx, b.cy, b.cz, b.nxb, b.nyb,
                 b.bseg, b.zws, b.nzw, 0, b.e0, b.m0};
}

// The next item of a persistent warp whose first was its number in the grid.
__device__ __forceinline__ int next_item(const Plan &p, int lane) {
    int item = 0;
    if (lane == 0) item = (int)(gridDim.x * (blockDim.x >> 5) + atomicAdd(p.work, 1u));
    return __shfl_sync(0xffffffffu, item, 0);
}

// The four corner columns of column (x, y) in one word of z, and the same one
// sample up (bit k: sample z + 1).
struct Corners {
    uint32_t a, b, c, d;      // (x, y) (x+1, y) (x, y+1) (x+1, y+1)
    uint32_t as, bs, cs, ds;  // shifted
    // cells of the word with corners on both sides
    __device__ __forceinline__ uint32_t active() const {
        return (a | b | c | d | as | bs | cs | ds) & ~(a & b & c & d & as & bs & cs & ds);
    }
};

// Cells of word zw that exist.
__device__ __forceinline__ uint32_t cell_mask(int cz, int zw) {
    const int n = cz - 32 * zw;
    return n >= 32 ? 0xffffffffu : (n <= 0 ? 0u : (1u << n) - 1u);
}

// Index bits 0..7 of a cell: corners (x,y) at z, z+1, then (x+1,y), (x,y+1),
// (x+1,y+1); the cube case of src/common.jl:10-20 is a permutation of them.
__device__ __forceinline__ uint32_t cell_index(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t na, uint32_t nb,
                                               uint32_t nc, uint32_t nd, int z) {
    return (__funnelshift_r(a, na, z) & 3u) | ((__funnelshift_r(b, nb, z) & 3u) << 2) |
           ((__funnelshift_r(c, nc, z) & 3u) << 4) | ((__funnelshift_r(d, nd, z) & 3u) << 6);
}

// Three consecutive values in two stores, the pair at the address that allows it.
__device__ __forceinline__ void put3(float *o, float a, float b, float c) {
    const bool up = ((uintptr_t)o & 4) != 0;
    *reinterpret_cast<float2 *>(o + (up ? 1 : 0)) = up ? make_float2(b, c) : make_float2(a, b);
    o[up ? 0 : 2] = up ? a : c;
}
__device__ __forceinline__ void put3(double *o, double a, double b, double c) {
    const bool up = ((uintptr_t)o & 8) != 0;
    *reinterpret_cast<double2 *>(o + (up ? 1 : 0)) = up ? make_double2(b, c) : make_double2(a, b);
    o[up ? 0 : 2] = up ? a : c;
}
__device__ __forceinline__ void put3(int64_t *o, long long a, long long b, long long c) {
    const bool up = ((uintptr_t)o & 8) != 0;
    *reinterpret_cast<longlong2 *>(o + (up ? 1 : 0)) = up ? make_longlong2(b, c) : make_longlong2(a, b);
    o[up ? 0 : 2] = up ? a : c;
}
__device__ __forceinline__ uint32_t lanemask_le(int lane) { return (2u << lane) - 1u; }

// The eight corner samples of queue entry `ent`, sw at column x0 and the word's
// first plane (entry 0 is in range: the word has active cells).
template <class T> __device__ __forceinline__ void load_corners(T (&s)[8], const T *sw, uint32_t ent, const BView &v) {
    const T *s0 = sw + (ent & 31u) + (int64_t)(ent >> 5) * v.sxy, *s1 = s0 + v.sxy;
    const T *t0 = s0 + v.nx, *t1 = s1 + v.nx;
    s[0] = ldv(s0);
    s[1] = ldv(s0 + 1);
    s[2] = ldv(t0);
    s[3] = ldv(t0 + 1);
    s[4] = ldv(s1);
    s[5] = ldv(s1 + 1);
    s[6] = ldv(t1);
    s[7] = ldv(t1 + 1);
}
}  // namespace mesh
#endif

namespace mesh {
constexpr unsigned mc_case_of_bits(unsigned u) {
    return (u & 1u) | (((u >> 2) & 1u) << 1) | (((u >> 6) & 1u) << 2) | (((u >> 4) & 1u) << 3) | (((u >> 1) & 1u) << 4) |
           (((u >> 3) & 1u) << 5) | (((u >> 7) & 1u) << 6) | (((u >> 5) & 1u) << 7);
}
}  // namespace mesh
