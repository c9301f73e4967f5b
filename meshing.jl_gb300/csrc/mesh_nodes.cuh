// One entry of a volume's coordinate tables (layout: k_tables.cu), for the
// kernels that fill them.
#pragma once
#include "mesh_internal.cuh"

namespace mesh {

namespace {

// LinRange node coordinates, spacings and their float forms, computed on the
// device with the host path's arithmetic: L((1 - t)*a + t*b), t = i/(n-1), every
// operation rounded separately.
// Entry k of the table block at `tabs` for nx, ny, nz nodes.  The x nodes are
// nodes xoff .. xoff+nx-1 of an x axis of nxt nodes (a slab of a larger volume;
// xoff = 0, nxt = nx for a whole volume).
__device__ __forceinline__ void table_entry(double *tabs, int64_t k, int64_t nx, int64_t ny, int64_t nz, double x0,
                                            double x1, double y0, double y1, double z0, double z1, int L32,
                                            int64_t xoff = 0, int64_t nxt = 0) {
    const int64_t ntab = nx + ny + nz;
    double *hp = tabs, *hd = tabs + ntab;
    float *hpf = (float *)(tabs + 2 * ntab), *hdf = hpf + ntab, *hs = hdf + ntab;
    int64_t i = k + xoff, n = nxt > 0 ? nxt : nx;
    double a = x0, b = x1;
    if (k >= nx + ny) {
        i = k - nx - ny; n = nz; a = z0; b = z1;
    } else if (k >= nx) {
        i = k - nx; n = ny; a = y0; b = y1;
    }
    if (L32) {
        a = (double)(float)a;
        b = (double)(float)b;
    }
    const double dn = (double)(n > 1 ? n - 1 : 1);
    auto node = [&](int64_t j) {
        const double t = __ddiv_rn((double)j, dn);
        const double v = __dadd_rn(__dmul_rn(__dsub_rn(1.0, t), a), __dmul_rn(t, b));
        return L32 ? (double)(float)v : v;
    };
    const double v = node(i);
    double d = 0;
    if (i + 1 < n) {
        const double v1 = node(i + 1);
        d = L32 ? (double)__fsub_rn((float)v1, (float)v) : __dsub_rn(v1, v);
    }
    hp[k] = v;
    hd[k] = d;
    hpf[k] = (float)v;
    hdf[k] = (float)d;
    hs[k] = (float)v;
    hs[ntab + k] = (float)__dsub_rn(v, (double)(float)v);
    hs[2 * ntab + k] = (float)d;
    hs[3 * ntab + k] = (float)__dsub_rn(d, (double)(float)d);
}

}  // namespace

}  // namespace mesh
