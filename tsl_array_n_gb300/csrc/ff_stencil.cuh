// Level geometry and the cell stencils shared by the fused level kernels
// (ff_fused.cu) and the resident solver (ff_resident.cu).
#pragma once
#include "ff_device.cuh"

namespace {

// a brick is BRICK_X x BRICK_Y x 8 cells (regular-brick flags)
constexpr int BRICK_X = 32, BRICK_Y = 16;

struct Geo {
    Dims d;
    float h2x, h2y, h2z;
    float dreg;          // diagonal of a regular interior cell: -2(h2x+h2y+h2z)
    long long sy, sz;
    int bnx, bny;        // bricks per row / column
};

struct Coef {
    float kx, ky, kz, e, ux, uy, uz;
};
__device__ __forceinline__ Coef coef_at(const Geo &g, const float4 *coef, bool regular, int i, int j,
                                        int k, long long c) {
    Coef q;
    if (regular) {
        q.kx = i > 0 ? g.h2x : 0.f;
        q.ky = j > 0 ? g.h2y : 0.f;
        q.kz = k > 0 ? g.h2z : 0.f;
        q.e = 0.f;
        q.ux = i < g.d.nx - 1 ? g.h2x : 0.f;
        q.uy = j < g.d.ny - 1 ? g.h2y : 0.f;
        q.uz = k < g.d.nz - 1 ? g.h2z : 0.f;
    } else {
        float4 a = __ldg(coef + c);
        q.kx = i > 0 ? a.x : 0.f;
        q.ky = j > 0 ? a.y : 0.f;
        q.kz = k > 0 ? a.z : 0.f;
        q.e = a.w;
        q.ux = i < g.d.nx - 1 ? __ldg(&coef[c + 1].x) : 0.f;
        q.uy = j < g.d.ny - 1 ? __ldg(&coef[c + g.sy].y) : 0.f;
        q.uz = k < g.d.nz - 1 ? __ldg(&coef[c + g.sz].z) : 0.f;
    }
    return q;
}

// (A v)_c, difference form; absent faces carry zero coefficients and their
// staged neighbour values are zero-filled (finite).
__device__ __forceinline__ float apply_q(const Coef &q, float vc, float xm, float xp, float ym, float yp,
                                         float zm, float zp) {
    float s = -q.e * vc;
    s += q.kx * (xm - vc);
    s += q.ux * (xp - vc);
    s += q.ky * (ym - vc);
    s += q.uy * (yp - vc);
    s += q.kz * (zm - vc);
    s += q.uz * (zp - vc);
    return s;
}
__device__ __forceinline__ float diag_q(const Coef &q) {
    return -(q.e + q.kx + q.ux + q.ky + q.uy + q.kz + q.uz);
}
// regular interior cell: second differences per axis
__device__ __forceinline__ float apply_reg(const Geo &g, float vc, float xm, float xp, float ym, float yp,
                                           float zm, float zp) {
    float s = g.h2x * ((xm - vc) + (xp - vc));
    s = __fmaf_rn(g.h2y, (ym - vc) + (yp - vc), s);
    s = __fmaf_rn(g.h2z, (zm - vc) + (zp - vc), s);
    return s;
}
__device__ __forceinline__ bool interior(const Geo &g, int i, int j, int k) {
    return i > 0 && i < g.d.nx - 1 && j > 0 && j < g.d.ny - 1 && k > 0 && k < g.d.nz - 1;
}

__device__ __forceinline__ unsigned long long globaltimer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// One relaxation of a cell with the plain couplings (class 0 or 2).  With
// S the h^-2-weighted sum of the six neighbours (the tensor maps zero-fill
// those across the domain edge, which drops the absent faces from S) and
// d = dreg + corr the cell's diagonal (corr = h^-2 summed over the absent
// faces), the row is (A v) = S + d v and the relaxation
// v + sor (b - A v) / d = (1 - sor) v + (b - S) rd, rd = sor / d.
__device__ __forceinline__ float relax_plain(const Geo &g, float omsor, float vc, float xm, float xp, float ym,
                                             float yp, float zm, float zp, float bval, float rd) {
    const float s = __fmaf_rn(g.h2z, zm + zp, __fmaf_rn(g.h2y, ym + yp, g.h2x * (xm + xp)));
    return __fmaf_rn(bval - s, rd, omsor * vc);
}

__device__ __forceinline__ void rtap4(int c, int nc, int *idx) {
    idx[0] = c > 0 ? 2 * c - 1 : 2 * c;
    idx[1] = 2 * c;
    idx[2] = 2 * c + 1;
    idx[3] = c + 1 < nc ? 2 * c + 2 : 2 * c + 1;
}

__device__ __forceinline__ void ptaps2(int f, int nc, int *idx, float *w) {
    const int ci = f >> 1;
    if ((f & 1) == 0) {
        idx[0] = ci > 0 ? ci - 1 : ci; w[0] = 0.25f;
        idx[1] = ci; w[1] = 0.75f;
    } else {
        idx[0] = ci; w[0] = 0.75f;
        idx[1] = ci < nc - 1 ? ci + 1 : ci; w[1] = 0.25f;
    }
}

inline Geo make_geo(const Level &L) {
    Geo g;
    g.d = L.d;
    g.h2x = L.h2inv[0];
    g.h2y = L.h2inv[1];
    g.h2z = L.d.nz > 1 ? L.h2inv[2] : 0.f;
    g.dreg = -2.f * (g.h2x + g.h2y + g.h2z);
    g.sy = L.d.nx;
    g.sz = (long long)L.d.nx * L.d.ny;
    g.bnx = (L.d.nx + BRICK_X - 1) / BRICK_X;
    g.bny = (L.d.ny + BRICK_Y - 1) / BRICK_Y;
    return g;
}

}  // namespace
