// Host runtime behind the C ABI (include/meshing_gb300.h).
//
// Turns a reference call isosurface(A, alg, X, Y, Z) into a launch plan:
// Julia's type promotion (src/marching_cubes.jl:31, src/marching_tetrahedra.jl:131)
// picks the arithmetic and output types, the LinRange node coordinates
// (src/marching_cubes.jl:36-38) are tabulated on the device with the exact
// Base.lerpi arithmetic (k_tables.cu), and the kernels run on the context's
// stream: classify -> scan -> emit.  Nothing waits on the host between
// launches.  Device scratch grows monotonically and is reused across calls.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "mesh_host.h"
#include "mesh_internal.cuh"
#include "mesh_tables.h"

namespace mesh {
cudaError_t launch_emit_mc(const Plan &p, int Q64, int P64, int stage, cudaStream_t s);
cudaError_t launch_emit_halo(const Plan &p, int Q64, int A64, int P64, cudaStream_t s);
size_t scan_scratch_bytes(const Plan &p);
}  // namespace mesh

using namespace mesh;

namespace mesh {

constexpr double EXACT_INT = 9007199254740992.0;  // 2^53

int fail(mesh_ctx *c, int status, const char *fmt, ...) {
    if (c) {
        char buf[512];
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(buf, sizeof(buf), fmt, ap);
        va_end(ap);
        c->msg = buf;
    }
    return status;
}

int cuda_fail(mesh_ctx *c, cudaError_t e, const char *what) {
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        return fail(c, MESH_ENOMEM, "%s: %s", what, cudaGetErrorString(e));
    }
    return fail(c, MESH_ECUDA, "%s: %s", what, cudaGetErrorString(e));
}

bool is_f32_exact(double v) { return std::isnan(v) || (double)(float)v == v; }

bool valid_scalar(int ty, double v) {
    switch (ty) {
    case MESH_DT_F64: return true;
    case MESH_DT_F32: return is_f32_exact(v);
    case MESH_DT_I64: return std::isfinite(v) && std::floor(v) == v && std::fabs(v) <= EXACT_INT;
    default: return false;
    }
}

// float(FT) is Float64 unless some participating type is Float32 and none is Float64.
int out_is_f64(const int *tys, int n) {
    int any32 = 0;
    for (int i = 0; i < n; i++) {
        if (tys[i] == MESH_DT_F64) return 1;
        if (tys[i] == MESH_DT_F32) any32 = 1;
    }
    return any32 ? 0 : 1;
}

int validate(mesh_ctx *c, int T, int64_t nx, int64_t ny, int64_t nz, const mesh_params *p) {
    if (!p) return fail(c, MESH_EINVAL, "params is NULL");
    if (T != MESH_DT_U16 && T != MESH_DT_F32 && T != MESH_DT_F64 && T != MESH_DT_I32 && T != MESH_DT_I64 &&
        T != MESH_DT_F16 && T != MESH_DT_I16 && T != MESH_DT_I8 && T != MESH_DT_U8)
        return fail(c, MESH_EINVAL, "unsupported volume dtype %d", T);
    // promote(Int, Float16) is Float16: (iso - v1) / (v2 - v1) would run in Float16 arithmetic
    if (T == MESH_DT_F16 && p && p->iso_type == MESH_DT_I64)
        return fail(c, MESH_EINVAL, "Float16 volumes take a Float32 or Float64 iso");
    if (p->alg != MESH_ALG_MC && p->alg != MESH_ALG_MT && p->alg != MESH_ALG_NSN && p->alg != MESH_ALG_MC_WELDED)
        return fail(c, MESH_EINVAL, "unknown algorithm %d", p->alg);
    if (p->iso_type != MESH_DT_F32 && p->iso_type != MESH_DT_F64 && p->iso_type != MESH_DT_I64)
        return fail(c, MESH_EINVAL, "unsupported iso type %d", p->iso_type);
    if (!valid_scalar(p->iso_type, p->iso)) return fail(c, MESH_EINVAL, "iso value not representable in its type");
    if (p->alg == MESH_ALG_MT) {
        if (p->eps_type != MESH_DT_F32 && p->eps_type != MESH_DT_F64)
            return fail(c, MESH_EINVAL, "unsupported eps type %d", p->eps_type);
        if (!valid_scalar(p->eps_type, p->eps)) return fail(c, MESH_EINVAL, "eps value not representable in its type");
    }
    if (p->range_type != MESH_DT_F32 && p->range_type != MESH_DT_F64 && p->range_type != MESH_DT_I64)
        return fail(c, MESH_EINVAL, "unsupported range type %d", p->range_type);
    for (int i = 0; i < 6; i++) {
        if (!std::isfinite(p->range[i])) return fail(c, MESH_EINVAL, "range endpoints must be finite");
        if (!valid_scalar(p->range_type, p->range[i])) return fail(c, MESH_EINVAL, "range endpoint not representable");
    }
    if (nx < 0 || ny < 0 || nz < 0) return fail(c, MESH_EINVAL, "negative dimension");
    const int64_t lim = (int64_t)1 << POS_BITS;
    if (nx > lim || ny > lim || nz > lim) return fail(c, MESH_ETOOLARGE, "dimension above 2^21");
    return MESH_OK;
}

void own_masks(uint32_t own[8]) {
    for (int bnd = 0; bnd < 8; bnd++) {
        uint32_t m = 0;
        for (int e = 0; e < 19; e++) {
            const int i1 = MT_EDGE_CORNERS[e][0], i2 = MT_EDGE_CORNERS[e][1];
            int za = 0;
            for (int k = 0; k < 3; k++)
                if (MT_CORNER_POS[i1][k] == 0 && MT_CORNER_POS[i2][k] == 0) za |= 1 << k;
            if ((za & ~bnd) == 0) m |= 1u << e;
        }
        own[bnd] = m;
    }
}

void set_types(Plan &P, int T, const mesh_params *p, int *Q64, int *A64, int *P64) {
    P.T = T;
    P.alg = p->alg;
    const int I = p->iso_type, E = p->eps_type, Rt = p->range_type;
    const int mt = p->alg == MESH_ALG_MT;
    // promote(typeof(iso), T); Int / Int divides in Float64
    *Q64 = T == MESH_DT_F64 || I == MESH_DT_F64 || (T != MESH_DT_F32 && I == MESH_DT_I64);
    const int L32 = Rt == MESH_DT_F32;
    *A64 = mt ? (*Q64 || E == MESH_DT_F64) : *Q64;
    *P64 = *A64 || !L32;
    if (!mt) *P64 = *Q64 || !L32;
    const int tys[4] = {Rt, T, I, E};
    P.out64 = out_is_f64(tys, mt ? 4 : 3);

    const double iso = p->iso;
    // thresholds: v < iso  <=>  v < thr in the data type
    {
        float f = (float)iso;
        if (!std::isnan(iso) && (double)f < iso) f = std::nextafter(f, INFINITY);
        P.thr_f = f;
        P.thr_d = iso;
        double ce = std::ceil(iso);
        if (std::isnan(iso)) ce = 0;
        P.thr_i = (int32_t)std::min(65536.0, std::max(0.0, ce));  // UInt16 / UInt8 data
        // Int8 / Int16 / Int32 / Int64 data: x < iso  <=>  x < ceil(iso), exact for every Int64 x
        P.thr_all = 0;
        if (std::isnan(iso)) {
            P.thr_l = INT64_MIN;                      // nothing is below NaN
        } else if (ce >= 9223372036854775808.0) {
            P.thr_l = INT64_MAX;
            P.thr_all = 1;                            // beyond every Int64
        } else if (ce < -9223372036854775808.0) {
            P.thr_l = INT64_MIN;
        } else {
            P.thr_l = (int64_t)ce;
        }
        P.iso_int = T == MESH_DT_I64 && I == MESH_DT_I64;
        P.iso_l = I == MESH_DT_I64 ? (int64_t)iso : 0;
    }
    P.isoq_d = iso;
    P.iso_zero = iso == 0;
    P.iso_small = std::floor(iso) == iso && std::fabs(iso) <= 1073741824.0 && !(iso == 0 && std::signbit(iso));
    P.iso_s = P.iso_small ? (int32_t)iso : 0;
    P.isoq_f = (float)iso;
    if (mt) {
        const int te64 = T == MESH_DT_F64 || E == MESH_DT_F64;  // promote(T, E)
        const double hi = te64 ? 1.0 - p->eps : (double)(1.0f - (float)p->eps);
        P.eps_d = p->eps;
        P.hi_d = hi;
        P.eps_f = (float)p->eps;
        P.hi_f = (float)hi;
        own_masks(P.own);
    }
}

}  // namespace mesh

namespace {

void count_kernels(mesh_ctx *c, int stage, int n);

// Copy stream, events and split-point buffers of the pipelined host path.
int ensure_pipe(mesh_ctx *c) {
    if (c->copy) return MESH_OK;
    cudaError_t e = cudaStreamCreateWithFlags(&c->copy, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&c->ev_ready, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&c->ev_done, cudaEventDisableTiming);
    for (int g = 0; g < PIPE_MAX && e == cudaSuccess; g++) e = cudaEventCreateWithFlags(&c->ev_part[g], cudaEventDisableTiming);
    if (e == cudaSuccess) e = c->gat.ensure(GATHER_MAX * sizeof(int64_t));
    if (e == cudaSuccess && !c->h_gat) e = cudaHostAlloc((void **)&c->h_gat, GATHER_MAX * sizeof(int64_t), cudaHostAllocDefault);
    if (e != cudaSuccess) {
        // leave no half-made pipeline behind: the next call retries from scratch
        for (cudaEvent_t &ev : c->ev_part)
            if (ev) cudaEventDestroy(ev), ev = nullptr;
        if (c->ev_ready) cudaEventDestroy(c->ev_ready), c->ev_ready = nullptr;
        if (c->ev_done) cudaEventDestroy(c->ev_done), c->ev_done = nullptr;
        if (c->copy) cudaStreamDestroy(c->copy);
        c->copy = nullptr;
        return cuda_fail(c, e, "pipeline stream");
    }
    return MESH_OK;
}

bool one_walk(const mesh_ctx *c);
bool bits_path(const mesh_ctx *c);

// Buffers and tiling of the sign-bit path (mesh_bits.cuh).  The columns are cut into
// z segments until there are 512 items per SM, 20 for each warp of the emission, so
// that its last items end together (1024^3: 1.75 ms a call against 1.81 with 64).
int prepare_bits(mesh_ctx *c) {
    Plan &P = c->plan;
    P.nxb = (P.cx + BCOL - 1) / BCOL;
    P.nyb = (P.cy + BROW - 1) / BROW;
    P.nzw = (int32_t)((P.nz + 31) / 32);
    const int ncw = (P.cz + 31) / 32;
    const int64_t rows = (int64_t)P.nxb * P.cy, target = (int64_t)c->sms * 512;
    auto segments = [&](int zws) {
        P.zws = zws;
        P.bseg = (ncw + zws - 1) / zws;
    };
    const int nseg = (int)std::min<int64_t>(ncw, std::max<int64_t>(1, (target + rows - 1) / rows));
    segments(std::min(ZWS_MAX, (ncw + nseg - 1) / nseg));
    const size_t word = (size_t)P.nx * P.ny * sizeof(uint32_t);  // one word of every column
    // the whole volume's words, or windows of whole segments and the words around them
    int keep = P.nzw;
    cudaError_t e = cudaErrorMemoryAllocation;
    for (;;) {
        const size_t need = (size_t)(keep == P.nzw ? keep : keep + 2) * word;
        if (c->bits_max <= 0 || (int64_t)need <= c->bits_max || keep <= 1) {
            e = c->bits.ensure(need);
            if (e == cudaSuccess && P.alg != MESH_ALG_MC) e = c->vpre.ensure(need);
        }
        if (e == cudaSuccess) break;
        cudaGetLastError();
        if (keep <= 1) return cuda_fail(c, e, "sign words");
        keep = (keep + 1) / 2;
        e = cudaErrorMemoryAllocation;
    }
    if (keep < P.nzw) segments(std::min(P.zws, keep));
    c->win_segs = keep < P.nzw ? keep / P.zws : P.bseg;
    P.npc = (int64_t)P.cx * P.cy * P.bseg;
    const int64_t ntiles = (P.npc + BITS_TILE - 1) / BITS_TILE;
    if (ntiles > 0x7fffffff) return fail(c, MESH_ETOOLARGE, "grid too large for this volume shape");
    P.ntiles = (int32_t)ntiles;
    if ((e = c->pc.ensure((size_t)P.npc * sizeof(uint2))) != cudaSuccess) return cuda_fail(c, e, "piece counts");
    if ((e = c->tsum.ensure((size_t)ntiles * sizeof(ulonglong2))) != cudaSuccess) return cuda_fail(c, e, "tile sums");
    if ((e = c->wmask.ensure((size_t)rows * P.bseg * mask_words(P.zws) * sizeof(uint32_t))) != cudaSuccess)
        return cuda_fail(c, e, "activity masks");
    P.bits = (uint32_t *)c->bits.ptr;
    P.bw0 = 0;
    P.bw1 = P.nzw;
    P.pc = (uint2 *)c->pc.ptr;
    P.tsum = (ulonglong2 *)c->tsum.ptr;
    P.wmask = (uint32_t *)c->wmask.ptr;
    P.vpre = (uint32_t *)c->vpre.ptr;
    int64_t *m = (int64_t *)c->misc.ptr;
    P.totals = m;
    P.err = c->err_out ? c->err_out : (unsigned int *)(c->h_misc + PIN_ERR);
    P.done = (unsigned int *)(m + MISC_DONE);
    P.work = (unsigned int *)(m + MISC_WORK);
    return MESH_OK;
}

// Sign words of the window of segments s0 .. s1 - 1 (and the words around them).
cudaError_t window_bits(mesh_ctx *c, Plan &P, int s0, int s1, bool first) {
    P.bw0 = std::max(0, s0 * P.zws - 1);
    P.bw1 = std::min(P.nzw, s1 * P.zws + 1);
    TabArgs ta = c->targs;
    ta.on = first;
    return launch_bits(P, P.bw0, P.bw1 - P.bw0, ta, c->sms, c->stream);
}

// Sign words and piece counts; adds the kernels launched to *kernels.
cudaError_t count_bits(mesh_ctx *c, int *kernels) {
    Plan &P = c->plan;
    cudaError_t e = cudaSuccess;
    if (c->ngroups > 1) {
        // host volume: groups of words go up on the copy stream, each classified on
        // the compute stream as soon as its planes have arrived
        const size_t plane = (size_t)P.nx * P.ny * dtype_size(P.T);
        e = cudaEventRecord(c->ev_ready, c->stream);  // earlier work on the volume buffer
        if (e == cudaSuccess) e = cudaStreamWaitEvent(c->copy, c->ev_ready, 0);
        for (int g = 0; g < c->ngroups && e == cudaSuccess; g++) {
            const int w0 = (int)((int64_t)g * P.nzw / c->ngroups), w1 = (int)((int64_t)(g + 1) * P.nzw / c->ngroups);
            const int64_t p0 = (int64_t)w0 * 32, p1 = std::min<int64_t>((int64_t)w1 * 32, P.nz);
            e = cudaMemcpyAsync((char *)c->vol.ptr + p0 * plane, (const char *)c->upl_src + p0 * plane,
                                (size_t)(p1 - p0) * plane, cudaMemcpyHostToDevice, c->copy);
            if (e == cudaSuccess) e = cudaEventRecord(c->ev_part[g], c->copy);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(c->stream, c->ev_part[g], 0);
            TabArgs ta = c->targs;
            ta.on = g == 0;
            if (e == cudaSuccess) e = launch_bits(P, w0, w1 - w0, ta, c->sms, c->stream);
            ++*kernels;
        }
        if (e == cudaSuccess) e = launch_count(P, 0, P.bseg, c->stream, false, kernels);
    } else {
        for (int s0 = 0; s0 < P.bseg && e == cudaSuccess; s0 += c->win_segs) {
            const int s1 = std::min(P.bseg, s0 + c->win_segs);
            e = window_bits(c, P, s0, s1, s0 == 0);
            ++*kernels;
            if (e == cudaSuccess) e = launch_count(P, s0, s1 - s0, c->stream, false, kernels);
        }
    }
    return e;
}

// Emission of the column blocks of `q` (slot: its cleared work counter); adds the
// kernels launched to *kernels.
cudaError_t emit_bits(mesh_ctx *c, Plan q, int slot, int *kernels) {
    const bool mc = q.alg == MESH_ALG_MC;
    auto emit = [&](int s0, int n) {
        ++*kernels;
        return mc ? launch_emit_bits_mc(q, c->Q64, c->P64, s0, n, c->stream)
                  : launch_emit_shared(q, c->Q64, c->A64, c->P64, s0, n, c->stream);
    };
    if (c->win_segs >= q.bseg && slot < WORK_SLOTS) {
        q.work += 2 * slot;
        return emit(0, q.bseg);
    }
    cudaError_t e = cudaSuccess;
    for (int s0 = 0; s0 < q.bseg && e == cudaSuccess; s0 += c->win_segs) {
        const int s1 = std::min(q.bseg, s0 + c->win_segs);
        e = window_bits(c, q, s0, s1, false);
        ++*kernels;
        if (e == cudaSuccess) e = cudaMemsetAsync(q.work, 0, sizeof(unsigned), c->stream);
        if (e == cudaSuccess && !mc) e = launch_count(q, s0, s1 - s0, c->stream, true, kernels);
        if (e == cudaSuccess) e = emit(s0, s1 - s0);
    }
    return e;
}

int prepare(mesh_ctx *c, const void *vol, int T, int64_t nx, int64_t ny, int64_t nz, int vol_on_device,
            const mesh_params *p) {
    Plan &P = c->plan;
    P = Plan{};
    c->have_plan = 0;
    c->emitted = 0;
    c->ngroups = 1;
    P.nx = nx; P.ny = ny; P.nz = nz;
    P.cx = (int32_t)(nx - 1); P.cy = (int32_t)(ny - 1); P.cz = (int32_t)(nz - 1);
    set_types(P, T, p, &c->Q64, &c->A64, &c->P64);
    const int L32 = p->range_type == MESH_DT_F32;
    // x window: MT / NSN take the grid-boundary rules at the whole volume's x = 0; with
    // a halo, the volume's first cell column is the previous slab's last (counted, not
    // emitted)
    P.xg0 = c->win_nx && P.alg != MESH_ALG_MC_WELDED ? c->win_x0 : 0;
    P.xhalo = c->win_nx && c->win_halo;
    if (P.xhalo && P.alg != MESH_ALG_MT && P.alg != MESH_ALG_NSN)
        return fail(c, MESH_EINVAL, "a halo column is for MarchingTetrahedra / NaiveSurfaceNets slabs");

    // tiling
    P.tiles_x = (P.cx + TILE_X - 1) / TILE_X;
    P.tiles_y = (P.cy + WY - 1) / WY;
    const int64_t per_seg = (int64_t)P.tiles_x * P.tiles_y;
    const int64_t target = (int64_t)c->sms * 64;
    const int maxseg = (P.cz + ZC - 1) / ZC;
    const int nseg = (int)std::min<int64_t>(maxseg, std::max<int64_t>(1, (target + per_seg - 1) / per_seg));
    int zs = (P.cz + nseg - 1) / nseg;
    zs = (zs + ZC - 1) / ZC * ZC;
    P.zs = zs;
    P.nseg = (P.cz + zs - 1) / zs;
    P.chunks_per_seg = zs / ZC;
    P.nchunks = P.nseg * P.chunks_per_seg;
    if ((P.tiles_y + WARPS - 1) / WARPS > 65535 || P.nseg > 65535)
        return fail(c, MESH_ETOOLARGE, "grid too large for this volume shape (at most 2^21 - 31 samples on y)");

    cudaError_t e;
    const size_t es = dtype_size(T);
    const size_t vbytes = (size_t)nx * ny * nz * es;
    c->host_mapped = 0;
    cudaPointerAttributes pa;
    if (vol_on_device) {
        P.vol = vol;
    } else if (p->alg == MESH_ALG_MC && c->zerocopy && cudaPointerGetAttributes(&pa, vol) == cudaSuccess &&
               pa.type == cudaMemoryTypeHost && pa.devicePointer) {
        // pinned and mapped: the one walk reads it in place, once
        P.vol = pa.devicePointer;
        c->host_mapped = 1;
    } else {
        cudaGetLastError();
        if ((e = c->vol.ensure(vbytes)) != cudaSuccess) return cuda_fail(c, e, "volume buffer");
        P.vol = c->vol.ptr;
        if (c->pipe_bytes > 0 && (int64_t)vbytes >= c->pipe_bytes && bits_path(c) && nz > 32) {
            int rc = ensure_pipe(c);
            if (rc) return rc;
            c->ngroups = (int)std::min<int64_t>(PIPE_MAX, (nz + 31) / 32);  // the count uploads and classifies
            c->upl_src = vol;
        } else if ((e = cudaMemcpyAsync(c->vol.ptr, vol, vbytes, cudaMemcpyHostToDevice, c->stream)) != cudaSuccess) {
            return cuda_fail(c, e, "volume upload");
        }
    }

    // coordinate tables: xp yp zp dx dy dz (double), the same as float, then the
    // hi/lo float split of the nodes and spacings, computed on the device (on the
    // sign-bit path by the launch that packs the first words)
    const int64_t ntab = nx + ny + nz;
    c->bits_on = bits_path(c);
    if ((e = c->tabs.ensure(table_bytes(ntab))) != cudaSuccess) return cuda_fail(c, e, "table buffer");
    if (c->win_nx && c->win_x0 + nx > c->win_nx) return fail(c, MESH_EINVAL, "volume extends past its x window");
    const int64_t np = npieces(P);
    const size_t fb = (size_t)P.nchunks * P.tiles_x * P.cy;
    const size_t sb = (scan_scratch_bytes(P) + 255) / 256 * 256;
    if (!c->bits_on && P.alg != MESH_ALG_MC &&
        (c->cnt.ensure((size_t)np * NCNT * sizeof(uint32_t)) != cudaSuccess ||
         c->base.ensure((size_t)np * NCNT * sizeof(int64_t)) != cudaSuccess || c->flags.ensure(fb) != cudaSuccess ||
         c->scan.ensure(sb) != cudaSuccess)) {
        cudaGetLastError();  // the walk's scratch is twice that of the bits
        for (DevBuf *b : {&c->cnt, &c->base, &c->flags, &c->scan}) b->release();
        c->bits_on = 1;
    }
    if (c->bits_on) {
        c->targs = TabArgs{(double *)c->tabs.ptr, nx, ny, nz, c->win_x0, c->win_nx, {}, L32, 0};
        for (int k = 0; k < 6; k++) c->targs.range[k] = p->range[k];
    } else {
        if ((e = launch_tables((double *)c->tabs.ptr, nx, ny, nz, p->range, L32, c->stream, c->win_x0, c->win_nx)) !=
            cudaSuccess)
            return cuda_fail(c, e, "table launch");
        count_kernels(c, 0, 1);  // the coordinate tables count with the classification
    }
    bind_tables(P, (double *)c->tabs.ptr, nx, ny, nz);
    P.force_fp64 = c->force_fp64;

    if (c->bits_on) {
        const int rc = prepare_bits(c);
        if (rc == MESH_OK && c->ngroups > 1) {
            if (c->win_segs < P.bseg) {  // windows: the volume goes up first
                c->ngroups = 1;
                if ((e = cudaMemcpyAsync(c->vol.ptr, vol, vbytes, cudaMemcpyHostToDevice, c->stream)) != cudaSuccess)
                    return cuda_fail(c, e, "volume upload");
            }
        }
        return rc;
    }

    // scratch
    P.pstride = np;
    if ((e = c->cnt.ensure((size_t)np * NCNT * sizeof(uint32_t))) != cudaSuccess) return cuda_fail(c, e, "count buffer");
    if ((e = c->base.ensure((size_t)np * NCNT * sizeof(int64_t))) != cudaSuccess) return cuda_fail(c, e, "base buffer");
    if ((e = c->flags.ensure(fb)) != cudaSuccess) return cuda_fail(c, e, "flag buffer");
    if ((e = c->scan.ensure(sb)) != cudaSuccess) return cuda_fail(c, e, "scan buffer");
    P.cnt = (uint32_t *)c->cnt.ptr;
    P.base = (int64_t *)c->base.ptr;
    P.flags = (uint8_t *)c->flags.ptr;
    P.scan_state = (unsigned long long *)c->scan.ptr;
    // misc: totals[NCNT] int64, then the error word, the work counter and the
    // staging counter
    P.totals = (int64_t *)c->misc.ptr;
    P.err = (unsigned int *)((int64_t *)c->misc.ptr + NCNT);
    P.work = (unsigned int *)((int64_t *)c->misc.ptr + NCNT + 1);
    P.stage_next = (unsigned long long *)((int64_t *)c->misc.ptr + NCNT + 2);
    return MESH_OK;
}

cudaEvent_t take_event(mesh_ctx *c) {
    if (!c->ev_free.empty()) {
        cudaEvent_t e = c->ev_free.back();
        c->ev_free.pop_back();
        return e;
    }
    cudaEvent_t e = nullptr;
    if (cudaEventCreate(&e) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return e;
}

// With timing on: kernels launched in `stage` (for mesh_ctx_stage_times).
void count_kernels(mesh_ctx *c, int stage, int n) {
    if (c->timing) c->nkern[stage] += n;
}

void mark(mesh_ctx *c, int stage) {
    if (!c->timing) return;
    cudaEvent_t e = take_event(c);
    if (!e) return;
    cudaEventRecord(e, c->stream);
    c->ev_pairs[stage].push_back(e);
}

// Marching Cubes walked once, classification staging the active cells (opt-in;
// also the form that reads a mapped host volume in place).
bool one_walk(const mesh_ctx *c) {
    return c->plan.alg == MESH_ALG_MC && (c->one_walk || c->host_mapped);
}

// MT and NSN on a few layers of cells under many columns: a word of the sign bits holds
// two or three cells of a column there, and each of the emission's batches little more
// than a row's few active ones, behind a column-strided look at the piece offsets.  The walk
// over 4 rows at a time (k_classify.cu, k_emit_halo.cu) is then the faster form.  Calls on
// smooth Float32 fields, walk against bits: 4096 x 4096 x 2 MT 1264 against 2254 us, NSN
// 973 against 1942; 2048 x 2048 x 2 MT 423 against 607, NSN 335 against 518;
// 4096 x 2048 x 3 MT 993 against 1288, NSN 827 against 1021; x 4 MT 1240 against 1404, NSN
// 1110 against 1079.  With five planes, or below two million columns (where the walk's
// four-kernel scan weighs more: 1000 x 999 x 3 MT 260 against 224), the bits are no slower.
// (The walk reports errors with an atomic, which a caller's pinned word need not take.)
constexpr int FLAT_CELLS = 3;
constexpr int64_t FLAT_COLUMNS = (int64_t)1 << 21;
bool flat(const mesh_ctx *c) {
    const Plan &P = c->plan;
    return (P.alg == MESH_ALG_MT || P.alg == MESH_ALG_NSN) && P.cz <= FLAT_CELLS &&
           (int64_t)P.cx * P.cy >= FLAT_COLUMNS && !c->err_out;
}

// Classified into sign bits and emitted from them: all but flat MT / NSN volumes and the
// Marching Cubes forms kept for comparison.
bool bits_path(const mesh_ctx *c) {
    return c->plan.alg == MESH_ALG_MC ? !c->list_emit && !one_walk(c) : !flat(c);
}

int run_count(mesh_ctx *c) {
    Plan &P = c->plan;
    cudaError_t e;
    if (c->bits_on) {
        int kernels = 0;
        mark(c, 0);
        if ((e = count_bits(c, &kernels)) != cudaSuccess) return cuda_fail(c, e, "classify launch");
        mark(c, 0);
        count_kernels(c, 0, kernels);
        const bool two_phase = P.tot_out == c->h_misc + PIN_TOT;
        if (two_phase) {  // the host reads the totals while the offsets are scanned
            if (!c->ev_cnt && (e = cudaEventCreateWithFlags(&c->ev_cnt, cudaEventDisableTiming)) != cudaSuccess)
                return cuda_fail(c, e, "count event");
            if (!c->ev_off && (e = cudaEventCreateWithFlags(&c->ev_off, cudaEventDisableTiming)) != cudaSuccess)
                return cuda_fail(c, e, "count event");
            if ((e = cudaEventRecord(c->ev_cnt, c->stream)) != cudaSuccess) return cuda_fail(c, e, "count event");
        }
        mark(c, 1);
        if ((e = launch_offsets(P, c->stream)) != cudaSuccess) return cuda_fail(c, e, "scan launch");
        mark(c, 1);
        count_kernels(c, 1, 1);
        if (two_phase) {
            if ((e = cudaEventRecord(c->ev_off, c->stream)) != cudaSuccess) return cuda_fail(c, e, "count event");
            c->off_pending = 1;
        }
        return MESH_OK;
    }
    if ((e = cudaMemsetAsync(c->misc.ptr, 0, MISC_SLOTS * sizeof(int64_t), c->stream)) != cudaSuccess)
        return cuda_fail(c, e, "memset");
    mark(c, 0);
    e = one_walk(c) ? launch_walk_mc(P, c->stream) : launch_classify(P, c->stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "classify launch");
    mark(c, 0);
    count_kernels(c, 0, 1);
    mark(c, 1);
    if ((e = launch_scan(P, c->stream)) != cudaSuccess) return cuda_fail(c, e, "scan launch");
    mark(c, 1);
    count_kernels(c, 1, 4);  // reduce, column scan, column-sum scan, downsweep
    return MESH_OK;
}

int check_err(mesh_ctx *c) {
    const unsigned err = (unsigned)c->h_misc[NCNT];
    if (err & ERR_BOUNDS) return fail(c, MESH_EDEVICE, "device bounds check failed");
    if (err & (ERR_CAPACITY | ERR_STAGE)) return fail(c, MESH_ECAPACITY, "output capacity too small");
    return MESH_OK;
}

int fetch_misc(mesh_ctx *c) {
    cudaError_t e = cudaMemcpyAsync(c->h_misc, c->misc.ptr, MISC_SLOTS * sizeof(int64_t), cudaMemcpyDeviceToHost,
                                    c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "synchronize");
    c->off_pending = 0;
    if (c->bits_on) c->h_misc[NCNT] = c->h_misc[PIN_ERR];
    c->h_misc[NCNT] &= 0xffffffffll;
    return MESH_OK;
}

// Wait for the count's totals (sign-bit path: written by the kernel itself).
int fetch_totals(mesh_ctx *c) {
    if (!c->bits_on) return fetch_misc(c);
    cudaError_t e = cudaEventSynchronize(c->ev_cnt);
    if (e != cudaSuccess) return cuda_fail(c, e, "synchronize");
    c->h_misc[0] = c->h_misc[PIN_TOT];
    c->h_misc[1] = c->h_misc[PIN_TOT + 1];
    c->h_misc[2] = 0;
    c->h_misc[NCNT] = 0;
    return MESH_OK;
}

// Wait for the stream and take the error word (sign-bit path: in pinned memory).
int finish(mesh_ctx *c) {
    if (!c->bits_on) return fetch_misc(c);
    cudaError_t e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "synchronize");
    c->off_pending = 0;
    c->h_misc[NCNT] = c->h_misc[PIN_ERR] & 0xffffffffll;
    return MESH_OK;
}

// List of active cells (Marching Cubes), room for `cap` entries.
int ensure_entries(mesh_ctx *c, int64_t cap) {
    Plan &P = c->plan;
    const size_t es = dtype_size(P.T);
    const int64_t nside = cap / ENT_BLOCK + 1;
    auto up = [](size_t n) { return (n + 255) / 256 * 256; };  // every array 256-byte aligned
    const size_t o_val = up((size_t)cap * 8);
    const size_t o_side = o_val + up((size_t)cap * 8 * es);
    const size_t o_rank = o_side + up((size_t)nside * 16);
    const size_t o_cs = o_rank + up((size_t)cap * 8);
    const size_t bytes = o_cs + up((size_t)cap + 1);
    cudaError_t e = c->ent.ensure(bytes);
    if (e != cudaSuccess) return cuda_fail(c, e, "entry buffer");
    char *b = (char *)c->ent.ptr;
    P.ent_pos = (unsigned long long *)b;
    P.ent_val = b + o_val;  // 8 corner values per entry (vector stores need 16-byte alignment)
    P.ent_side = (long long *)(b + o_side);
    P.ent_rank = (uint2 *)(b + o_rank);
    P.ent_cs = (uint8_t *)(b + o_cs);
    P.ent_cap = cap;
    c->ent_cap_seen = std::max(c->ent_cap_seen, cap);
    return MESH_OK;
}

int launch_emit(mesh_ctx *c) {
    cudaError_t e;
    if (one_walk(c)) {
        mark(c, 3);
        e = launch_expand_staged_mc(c->plan, c->Q64, c->P64, c->stream);
        mark(c, 3);
        count_kernels(c, 3, 1);
        return e != cudaSuccess ? cuda_fail(c, e, "expand launch") : MESH_OK;
    }
    if (c->bits_on) {
        int kernels = 0;
        mark(c, 2);
        e = emit_bits(c, c->plan, 0, &kernels);
        mark(c, 2);
        count_kernels(c, 2, kernels);
        return e != cudaSuccess ? cuda_fail(c, e, "emit launch") : MESH_OK;
    }
    const bool mc = c->plan.alg == MESH_ALG_MC;
    mark(c, 2);
    e = mc ? launch_emit_mc(c->plan, c->Q64, c->P64, 0, c->stream)
           : launch_emit_halo(c->plan, c->Q64, c->A64, c->P64, c->stream);
    mark(c, 2);
    count_kernels(c, 2, 1);
    if (e != cudaSuccess) return cuda_fail(c, e, "emit launch");
    if (!mc) return MESH_OK;
    mark(c, 3);
    e = launch_emit_mc(c->plan, c->Q64, c->P64, 1, c->stream);
    mark(c, 3);
    count_kernels(c, 3, 1);
    return e != cudaSuccess ? cuda_fail(c, e, "expand launch") : MESH_OK;
}

// Marching Cubes emission into host buffers in K x ranges of whole x tiles.  The
// emission order is x-major, so the cells of an x range own one contiguous run of
// vertices and faces, starting at the offset of the range's first piece
// (seg 0, y 0, x0).  Range g is emitted on the compute stream; its vertices and faces go down on the copy stream while range g + 1 is
// emitted.  All launches are enqueued before the copies, so a pageable (blocking)
// destination still overlaps the copies with the emission.
int emit_pipelined(mesh_ctx *c, int K, void *verts, int64_t *faces) {
    const Plan &P = c->plan;
    const size_t vsz = (size_t)3 * (P.out64 ? 8 : 4);
    int tx[PIPE_MAX + 1];
    for (int g = 0; g <= K; g++) tx[g] = (int)((int64_t)g * P.nxb / K);
    GatherIdx gi{};
    gi.n = K - 1;
    for (int g = 1; g < K; g++) gi.idx[g - 1] = (int64_t)tx[g] * BCOL * P.cy * P.bseg;
    cudaError_t e = launch_gather_pieces(P, gi, (int64_t *)c->gat.ptr, c->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(c->h_gat, c->gat.ptr, (size_t)2 * (K - 1) * sizeof(int64_t), cudaMemcpyDeviceToHost,
                            c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "split points");
    int64_t V[PIPE_MAX + 1], F[PIPE_MAX + 1];
    V[0] = F[0] = 0;
    V[K] = c->nverts;
    F[K] = c->nfaces;
    for (int g = 1; g < K; g++) {
        V[g] = c->h_gat[2 * (g - 1)];
        F[g] = c->h_gat[2 * (g - 1) + 1];
    }
    for (int g = 0; g < K; g++)
        if (V[g] > V[g + 1] || F[g] > F[g + 1] || V[g + 1] > c->nverts || F[g + 1] > c->nfaces)
            return fail(c, MESH_EDEVICE, "inconsistent split points");
    int kernels = 0;
    mark(c, 2);
    for (int g = 0; g < K && e == cudaSuccess; g++) {
        Plan q = P;
        q.tx0 = tx[g];
        q.ntx = tx[g + 1] - tx[g];
        e = emit_bits(c, q, g, &kernels);
        if (e == cudaSuccess) e = cudaEventRecord(c->ev_part[g], c->stream);
    }
    mark(c, 2);
    count_kernels(c, 2, kernels);
    if (e != cudaSuccess) return cuda_fail(c, e, "emit launch");
    for (int g = 0; g < K && e == cudaSuccess; g++) {
        e = cudaStreamWaitEvent(c->copy, c->ev_part[g], 0);
        if (e == cudaSuccess && V[g + 1] > V[g])
            e = cudaMemcpyAsync((char *)verts + V[g] * vsz, (const char *)P.verts + V[g] * vsz,
                                (size_t)(V[g + 1] - V[g]) * vsz, cudaMemcpyDeviceToHost, c->copy);
        if (e == cudaSuccess && F[g + 1] > F[g])
            e = cudaMemcpyAsync(faces + 3 * F[g], P.faces + 3 * F[g], (size_t)(F[g + 1] - F[g]) * 24,
                                cudaMemcpyDeviceToHost, c->copy);
    }
    if (e == cudaSuccess) e = cudaEventRecord(c->ev_done, c->copy);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(c->stream, c->ev_done, 0);
    return e != cudaSuccess ? cuda_fail(c, e, "mesh download") : MESH_OK;
}

// Staging slots of the one walk beyond its active cells: at most a block per warp.
int64_t stage_slack(const Plan &P) { return (int64_t)STG_BLK * P.tiles_x * P.tiles_y * P.nseg; }

bool degenerate(int64_t nx, int64_t ny, int64_t nz) { return nx < 2 || ny < 2 || nz < 2; }

}  // namespace

extern "C" {

void mesh_params_default(mesh_params *p) {
    if (!p) return;
    memset(p, 0, sizeof(*p));
    p->alg = MESH_ALG_MC;
    p->iso_type = MESH_DT_F64;
    p->iso = 0.0;
    p->eps_type = MESH_DT_F64;
    p->eps = 1e-3;
    p->range_type = MESH_DT_I64;
    p->range[0] = p->range[2] = p->range[4] = -1.0;
    p->range[1] = p->range[3] = p->range[5] = 1.0;
}

const char *mesh_status_string(int s) {
    switch (s) {
    case MESH_OK: return "ok";
    case MESH_EINVAL: return "invalid argument";
    case MESH_ENOMEM: return "out of memory";
    case MESH_ECUDA: return "CUDA error";
    case MESH_EDEVICE: return "device-side error";
    case MESH_ESTATE: return "mesh_fill called without a successful mesh_count";
    case MESH_ECAPACITY: return "output capacity too small";
    case MESH_ETOOLARGE: return "volume too large";
    case MESH_ESCRATCH: return "needs more scratch than the no-allocation limit";
    case MESH_EBUDGET: return "worst case exceeds the memory budget";
    case MESH_EBUSY: return "queue full";
    default: return "unknown status";
    }
}

const char *mesh_ctx_last_error(const mesh_ctx *c) { return c ? c->msg.c_str() : ""; }

int mesh_ctx_create(int device, mesh_ctx **out) {
    if (!out) return MESH_EINVAL;
    *out = nullptr;
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess || device < 0 || device >= n) {
        cudaGetLastError();
        return e != cudaSuccess ? MESH_ECUDA : MESH_EINVAL;
    }
    if ((e = cudaSetDevice(device)) != cudaSuccess) return MESH_ECUDA;
    mesh_ctx *c = new (std::nothrow) mesh_ctx();
    if (!c) return MESH_ENOMEM;
    c->device = device;
    cudaDeviceGetAttribute(&c->sms, cudaDevAttrMultiProcessorCount, device);
    if (cudaStreamCreateWithFlags(&c->own, cudaStreamNonBlocking) != cudaSuccess ||
        c->misc.ensure(MISC_WORDS * sizeof(int64_t)) != cudaSuccess ||
        cudaHostAlloc((void **)&c->h_misc, PIN_WORDS * sizeof(int64_t), cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        mesh_ctx_destroy(c);
        return MESH_ENOMEM;
    }
    c->stream = c->own;
    memset(c->h_misc, 0, PIN_WORDS * sizeof(int64_t));
    const char *bb = getenv("MESHING_GB300_BITS_BYTES");
    if (bb && bb[0]) c->bits_max = strtoll(bb, nullptr, 10);
    const char *ff = getenv("MESHING_GB300_FORCE_FP64");
    c->force_fp64 = ff && ff[0] == '1';
    const char *ow = getenv("MESHING_GB300_ONE_WALK");
    c->one_walk = ow && ow[0] == '1';
    const char *le = getenv("MESHING_GB300_LIST_EMIT");
    c->list_emit = le && le[0] == '1';
    const char *zc = getenv("MESHING_GB300_ZEROCOPY");
    c->zerocopy = zc && zc[0] == '1';
    const char *pb = getenv("MESHING_GB300_PIPELINE_BYTES");  // <= 0: never pipelined
    if (pb && pb[0]) c->pipe_bytes = strtoll(pb, nullptr, 10);
    *out = c;
    return MESH_OK;
}

void mesh_ctx_destroy(mesh_ctx *c) {
    if (!c) return;
    cudaSetDevice(c->device);
    if (c->stream) cudaStreamSynchronize(c->stream);
    if (c->copy) cudaStreamSynchronize(c->copy);
    DevBuf *bufs[] = {&c->vol,   &c->tabs,  &c->cnt, &c->base, &c->flags,    &c->scan,   &c->misc,
                      &c->out_v, &c->out_f, &c->ent, &c->nrm,  &c->gat,
                      &c->bits, &c->pc,   &c->tsum, &c->wmask,
                      &c->vpre};
    for (DevBuf *b : bufs) b->release();
    for (cudaEvent_t e : c->ev_part)
        if (e) cudaEventDestroy(e);
    if (c->ev_ready) cudaEventDestroy(c->ev_ready);
    if (c->ev_done) cudaEventDestroy(c->ev_done);
    if (c->ev_cnt) cudaEventDestroy(c->ev_cnt);
    if (c->ev_off) cudaEventDestroy(c->ev_off);
    if (c->copy) cudaStreamDestroy(c->copy);
    if (c->h_gat) cudaFreeHost(c->h_gat);
    for (auto &v : c->ev_pairs)
        for (cudaEvent_t e : v) cudaEventDestroy(e);
    for (cudaEvent_t e : c->ev_free) cudaEventDestroy(e);
    if (c->h_misc) cudaFreeHost(c->h_misc);
    if (c->own) cudaStreamDestroy(c->own);
    delete c;
}

int mesh_ctx_set_stream(mesh_ctx *c, void *stream) {
    if (!c) return MESH_EINVAL;
    // A count's offsets may still be scanned on the old stream (an empty mesh, a fill that
    // follows or never came): they end before anything is issued on the new one.  The host
    // waits: the new stream may be capturing, and the old one destroyed by now.
    if (c->off_pending) {
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        // (fails only when the device has failed, or for a count that was refused because its
        // stream was capturing, whose offsets were never launched)
        if (cudaEventSynchronize(c->ev_off) != cudaSuccess) cudaGetLastError();
        cudaThreadExchangeStreamCaptureMode(&mode);
        c->off_pending = 0;
    }
    c->stream = stream ? (cudaStream_t)stream : c->own;
    return MESH_OK;
}

int mesh_set_x_window(mesh_ctx *c, int64_t x_first, int64_t nx_total, int halo) {
    if (!c) return MESH_EINVAL;
    if (x_first < 0 || nx_total < 0 || (nx_total == 0 && (x_first != 0 || halo)) ||
        nx_total > ((int64_t)1 << POS_BITS) || (halo != 0 && halo != 1))
        return fail(c, MESH_EINVAL, "invalid x window");
    c->win_x0 = x_first;
    c->win_nx = nx_total;
    c->win_halo = halo;
    c->have_plan = 0;
    return MESH_OK;
}

int mesh_output_float_bits(int T, const mesh_params *p, int *bits) {
    if (!p || !bits) return MESH_EINVAL;
    int rc = validate(nullptr, T, 0, 0, 0, p);
    if (rc) return rc;
    const int tys[4] = {p->range_type, T, p->iso_type, p->eps_type};
    *bits = out_is_f64(tys, p->alg == MESH_ALG_MT ? 4 : 3) ? 64 : 32;
    return MESH_OK;
}

}  // extern "C"

namespace {
// An x window with a halo column (MT / NSN slab after the first): the halo
// column's vertices and faces come first in the scan and are not emitted, so
// the counts lose its totals (the first vertex and face of piece (x 1, y 0, seg 0)).
int drop_halo_counts(mesh_ctx *c) {
    const Plan &P = c->plan;
    int64_t v0 = c->nverts, f0 = c->nfaces;  // a window of the halo column alone emits nothing
    if (P.cx > 1) {
        int64_t h[2] = {0, 0};
        cudaError_t e;
        if (c->bits_on) {
            GatherIdx gi{};
            gi.n = 1;
            gi.idx[0] = (int64_t)P.cy * P.bseg;
            e = c->gat.ensure(GATHER_MAX * sizeof(int64_t));
            if (e == cudaSuccess) e = launch_gather_pieces(P, gi, (int64_t *)c->gat.ptr, c->stream);
            if (e == cudaSuccess) e = cudaMemcpyAsync(h, c->gat.ptr, sizeof(h), cudaMemcpyDeviceToHost, c->stream);
        } else {
            const int64_t *b = P.base + piece(P, 0, 0, 1);  // the walk's prefixes
            e = cudaMemcpyAsync(h, b, 8, cudaMemcpyDeviceToHost, c->stream);
            if (e == cudaSuccess) e = cudaMemcpyAsync(h + 1, b + P.pstride, 8, cudaMemcpyDeviceToHost, c->stream);
        }
        if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
        if (e != cudaSuccess) return cuda_fail(c, e, "halo counts");
        v0 = h[0];
        f0 = h[1];
    }
    if (v0 < 0 || v0 > c->nverts || f0 < 0 || f0 > c->nfaces) return fail(c, MESH_EDEVICE, "inconsistent halo counts");
    c->nverts -= v0;
    c->nfaces -= f0;
    return MESH_OK;
}
}  // namespace

extern "C" {

int mesh_count(mesh_ctx *c, const void *vol, int T, int64_t nx, int64_t ny, int64_t nz, int vol_on_device,
               const mesh_params *p, int64_t *nverts, int64_t *nfaces) {
    if (!c || !nverts || !nfaces) return fail(c, MESH_EINVAL, "NULL argument");
    c->have_plan = 0;
    c->msg.clear();
    int rc = validate(c, T, nx, ny, nz, p);
    if (rc) return rc;
    if (cudaSetDevice(c->device) != cudaSuccess) return fail(c, MESH_ECUDA, "cudaSetDevice");
    if (degenerate(nx, ny, nz)) {
        c->nverts = c->nfaces = 0;
        c->plan = Plan{};
        c->plan.alg = p->alg;
        c->have_plan = 2;  // empty mesh
        *nverts = *nfaces = 0;
        return MESH_OK;
    }
    if (!vol) return fail(c, MESH_EINVAL, "volume is NULL");
    if ((rc = prepare(c, vol, T, nx, ny, nz, vol_on_device, p))) return rc;
    if (c->bits_on) c->plan.tot_out = c->h_misc + PIN_TOT;
    if (one_walk(c)) {
        // the list of active cells is filled during the count: start from a
        // guess (or the context's earlier list), and if the walk ran out of
        // slots walk again with the exact number it reported
        const int64_t cells = (int64_t)c->plan.cx * c->plan.cy * c->plan.cz;
        const int64_t guess = std::max<int64_t>(c->ent_cap_seen, cells / 48 + stage_slack(c->plan));
        if ((rc = ensure_entries(c, guess))) return rc;
    }
    if ((rc = run_count(c))) return rc;
    if ((rc = fetch_totals(c))) return rc;
    if (one_walk(c) && ((unsigned)c->h_misc[NCNT] & ERR_STAGE)) {
        if ((rc = ensure_entries(c, c->h_misc[NCNT + 2]))) return rc;
        if ((rc = run_count(c))) return rc;
        if ((rc = fetch_misc(c))) return rc;
    }
    if ((rc = check_err(c))) return rc;
    c->nverts = c->h_misc[0];
    c->nfaces = c->h_misc[1];
    c->nactive = c->h_misc[2];
    if (c->plan.xhalo && (rc = drop_halo_counts(c))) return rc;
    *nverts = c->nverts;
    *nfaces = c->nfaces;
    c->have_plan = 1;
    return MESH_OK;
}

int mesh_fill(mesh_ctx *c, void *verts, int64_t *faces, int out_on_device) {
    if (!c) return MESH_EINVAL;
    if (!c->have_plan) return fail(c, MESH_ESTATE, "mesh_fill without mesh_count");
    if (c->have_plan == 2 || (c->nverts == 0 && c->nfaces == 0)) return MESH_OK;
    if ((c->nverts && !verts) || (c->nfaces && !faces)) return fail(c, MESH_EINVAL, "NULL output");
    if (cudaSetDevice(c->device) != cudaSuccess) return fail(c, MESH_ECUDA, "cudaSetDevice");
    Plan &P = c->plan;
    const size_t vb = (size_t)c->nverts * 3 * (P.out64 ? 8 : 4), fbytes = (size_t)c->nfaces * 3 * 8;
    cudaError_t e;
    if (out_on_device) {
        P.verts = verts;
        P.faces = faces;
    } else {
        if ((e = c->out_v.ensure(vb + 16)) != cudaSuccess) return cuda_fail(c, e, "vertex staging");
        if ((e = c->out_f.ensure(fbytes + 16)) != cudaSuccess) return cuda_fail(c, e, "face staging");
        P.verts = c->out_v.ptr;
        P.faces = (int64_t *)c->out_f.ptr;
    }
    P.verts_cap = c->nverts;
    P.faces_cap = c->nfaces;
    int rc;
    if (P.alg == MESH_ALG_MC && !one_walk(c) && !c->bits_on && (rc = ensure_entries(c, c->nactive))) return rc;
    if (!c->bits_on && (e = cudaMemsetAsync(P.err, 0, sizeof(unsigned), c->stream)) != cudaSuccess)
        return cuda_fail(c, e, "memset");
    // a fill whose download failed may be called again
    if (c->bits_on && c->emitted &&
        (e = cudaMemsetAsync(P.work, 0, WORK_SLOTS * 2 * sizeof(unsigned), c->stream)) != cudaSuccess)
        return cuda_fail(c, e, "memset");
    c->emitted = 1;
    int parts = 1;
    if (!out_on_device && P.alg == MESH_ALG_MC && c->bits_on && c->pipe_bytes > 0 &&
        (int64_t)(vb + fbytes) >= c->pipe_bytes && P.nxb >= 2) {
        if ((rc = ensure_pipe(c))) return rc;
        parts = std::min(PIPE_MAX, P.nxb);
    }
    if (parts > 1) {
        if ((rc = emit_pipelined(c, parts, verts, faces))) return rc;
    } else {
        if ((rc = launch_emit(c))) return rc;
        if (!out_on_device) {
            if (vb && (e = cudaMemcpyAsync(verts, P.verts, vb, cudaMemcpyDeviceToHost, c->stream)) != cudaSuccess)
                return cuda_fail(c, e, "vertex download");
            if (fbytes &&
                (e = cudaMemcpyAsync(faces, P.faces, fbytes, cudaMemcpyDeviceToHost, c->stream)) != cudaSuccess)
                return cuda_fail(c, e, "face download");
        }
    }
    if ((rc = finish(c))) return rc;
    c->have_plan = 0;  // a plan may reference a caller's device volume: one fill per count
    return check_err(c);
}

int mesh_extract_device(mesh_ctx *c, const void *vol, int T, int64_t nx, int64_t ny, int64_t nz,
                        const mesh_params *p, void *verts, int64_t verts_cap, int64_t *faces, int64_t faces_cap,
                        int64_t *counts) {
    if (!c || !counts) return fail(c, MESH_EINVAL, "NULL argument");
    c->msg.clear();
    int rc = validate(c, T, nx, ny, nz, p);
    if (rc) return rc;
    if (cudaSetDevice(c->device) != cudaSuccess) return fail(c, MESH_ECUDA, "cudaSetDevice");
    cudaError_t e;
    if (degenerate(nx, ny, nz)) {
        if ((e = cudaMemsetAsync(counts, 0, 2 * sizeof(int64_t), c->stream)) != cudaSuccess)
            return cuda_fail(c, e, "memset");
        return MESH_OK;
    }
    if (!vol) return fail(c, MESH_EINVAL, "volume is NULL");
    if (p->alg == MESH_ALG_MC_WELDED) return fail(c, MESH_EINVAL, "welded meshes are built by mesh_count / mesh_fill");
    if ((rc = prepare(c, vol, T, nx, ny, nz, 1, p))) return rc;
    Plan &P = c->plan;
    if (P.xhalo) return fail(c, MESH_EINVAL, "an x window with a halo column is meshed by mesh_count / mesh_fill");
    P.verts = verts;
    P.faces = faces;
    P.verts_cap = verts ? verts_cap : 0;
    P.faces_cap = faces ? faces_cap : 0;
    if (c->bits_on) P.tot_out = counts;
    // an active Marching Cubes cell emits at least 3 vertices; the one walk
    // also leaves up to a block of slots per warp unused
    if (P.alg == MESH_ALG_MC && !c->bits_on &&
        (rc = ensure_entries(c, P.verts_cap / 3 + (one_walk(c) ? stage_slack(P) : 0))))
        return rc;
    if ((rc = run_count(c))) return rc;
    if ((rc = launch_emit(c))) return rc;
    if (!c->bits_on &&
        (e = cudaMemcpyAsync(counts, P.totals, 2 * sizeof(int64_t), cudaMemcpyDeviceToDevice, c->stream)) !=
        cudaSuccess)
        return cuda_fail(c, e, "count copy");
    c->have_plan = 0;
    return MESH_OK;
}

int mesh_ctx_sync(mesh_ctx *c) {
    if (!c) return MESH_EINVAL;
    if (cudaSetDevice(c->device) != cudaSuccess) return fail(c, MESH_ECUDA, "cudaSetDevice");
    int rc = fetch_misc(c);
    if (rc) return rc;
    return check_err(c);
}

int mesh_ctx_enable_timing(mesh_ctx *c, int enable) {
    if (!c) return MESH_EINVAL;
    c->timing = enable ? 1 : 0;
    return MESH_OK;
}

int mesh_ctx_stage_times(mesh_ctx *c, double *ms, int64_t *launches) {
    if (!c || !ms || !launches) return MESH_EINVAL;
    if (cudaSetDevice(c->device) != cudaSuccess) return fail(c, MESH_ECUDA, "cudaSetDevice");
    int rc = MESH_OK;
    for (int s = 0; s < NSTAGE; s++) {
        ms[s] = 0;
        launches[s] = 0;
        auto &v = c->ev_pairs[s];
        for (size_t i = 0; i + 1 < v.size(); i += 2) {
            float t = 0;
            cudaError_t e = cudaEventSynchronize(v[i + 1]);
            if (e == cudaSuccess) e = cudaEventElapsedTime(&t, v[i], v[i + 1]);
            if (e != cudaSuccess) rc = cuda_fail(c, e, "stage timing");
            ms[s] += t;
        }
        launches[s] = c->nkern[s];
        c->nkern[s] = 0;
        for (cudaEvent_t e : v) c->ev_free.push_back(e);
        v.clear();
    }
    return rc;
}

}  // extern "C"
