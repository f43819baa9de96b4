// FP32 grid sampling, trace and extrapolation helpers shared by the
// grid-velocity (ff_grid.cu) and FLIP (ff_flip.cu) kernels.  Both files are
// compiled with -fmad=false: every operation rounds on its own, in the
// evaluation order of the reference's expressions (fluxflow
// src/grid/grid_math3.js, advection_solver3.js, array_utils3.js).
#pragma once
#include "ff_internal.h"

// private to each translation unit that includes it
namespace {
namespace ffg {

struct G3 {
    int nx, ny, nz;
    float hx, hy, hz, ox, oy, oz;
};
struct F3 {
    float x, y, z;
};

__device__ __forceinline__ int iclamp(int v, int lo, int hi) { return max(lo, min(v, hi)); }
// keeps the float->int conversion defined for absurd or non-finite positions
__device__ __forceinline__ float gclamp(float g) { return fminf(fmaxf(g, -1.0e8f), 1.0e8f); }

__host__ __device__ __forceinline__ void comp_shape(const G3 &g, int a, int &sx, int &sy, int &sz) {
    sx = g.nx + (a == 0);
    sy = g.ny + (a == 1);
    sz = g.nz + (a == 2);
}
// dataOriginU/V/W (grid_data3.js:131-133); a == 3: cell centres (:208)
__device__ __forceinline__ F3 comp_origin(const G3 &g, int a) {
    F3 o;
    o.x = g.ox + (a == 0 ? 0.0f : g.hx * 0.5f);
    o.y = g.oy + (a == 1 ? 0.0f : g.hy * 0.5f);
    o.z = g.oz + (a == 2 ? 0.0f : g.hz * 0.5f);
    return o;
}
__device__ __forceinline__ F3 index_pos(const G3 &g, F3 o, int i, int j, int k) {
    return F3{o.x + g.hx * (float)i, o.y + g.hy * (float)j, o.z + g.hz * (float)k};
}

// collocatedValueAtPosition3 (grid_math3.js:61-117): clamped corners,
// weights (1-f) products in x, y, z order, summed corner by corner
__device__ float trilinear(const float *__restrict__ d, int sx, int sy, int sz, const G3 &g, F3 o, F3 p) {
    const float gx = gclamp((p.x - o.x) / g.hx), gy = gclamp((p.y - o.y) / g.hy), gz = gclamp((p.z - o.z) / g.hz);
    const int i0 = (int)floorf(gx), j0 = (int)floorf(gy), k0 = (int)floorf(gz);
    const float fx = gx - (float)i0, fy = gy - (float)j0, fz = gz - (float)k0;
    const int i0c = iclamp(i0, 0, sx - 1), i1c = iclamp(i0 + 1, 0, sx - 1);
    const int j0c = iclamp(j0, 0, sy - 1), j1c = iclamp(j0 + 1, 0, sy - 1);
    const int k0c = iclamp(k0, 0, sz - 1), k1c = iclamp(k0 + 1, 0, sz - 1);
    const float ux = 1.0f - fx, uy = 1.0f - fy, uz = 1.0f - fz;
    // 32-bit offsets: the entry points keep every array below 2^31 elements
    const int r00 = sx * (j0c + sy * k0c), r10 = sx * (j1c + sy * k0c);
    const int r01 = sx * (j0c + sy * k1c), r11 = sx * (j1c + sy * k1c);
    float s = __ldg(d + r00 + i0c) * (ux * uy * uz);
    s = s + __ldg(d + r00 + i1c) * (fx * uy * uz);
    s = s + __ldg(d + r10 + i0c) * (ux * fy * uz);
    s = s + __ldg(d + r10 + i1c) * (fx * fy * uz);
    s = s + __ldg(d + r01 + i0c) * (ux * uy * fz);
    s = s + __ldg(d + r01 + i1c) * (fx * uy * fz);
    s = s + __ldg(d + r11 + i0c) * (ux * fy * fz);
    s = s + __ldg(d + r11 + i1c) * (fx * fy * fz);
    return s;
}

// monotonicCubic1d3 (grid_math3.js:137-160)
__device__ __forceinline__ float mono_cubic(float f0, float f1, float f2, float f3, float f) {
    const float D1 = f2 - f1;
    const float rawD1 = (f2 - f0) * 0.5f, rawD2 = (f3 - f1) * 0.5f;
    const bool flat = fabsf(D1) < 1e-12f;
    const float d1 = (flat || rawD1 * D1 < 0.0f) ? 0.0f : rawD1;
    const float d2 = (flat || rawD2 * D1 < 0.0f) ? 0.0f : rawD2;
    const float a3 = (d1 + d2) - D1 * 2.0f;
    const float a2 = (D1 * 3.0f - d1 * 2.0f) - d2;
    float t = a3 * f * f * f;
    t = t + a2 * f * f;
    t = t + d1 * f;
    return t + f1;
}

__device__ __forceinline__ void cubic_idx(float coord, int n, int idx[4], float &f) {
    const int i0 = (int)floorf(coord);
    f = coord - (float)i0;
    idx[0] = iclamp(i0 - 1, 0, n - 1);
    idx[1] = iclamp(i0, 0, n - 1);
    idx[2] = iclamp(i0 + 1, 0, n - 1);
    idx[3] = iclamp(i0 + 2, 0, n - 1);
}

// collocatedCubicValueAtPosition3 (grid_math3.js:174-199): cubic in x for
// each (y, z) tap, then y per z tap, then z
__device__ float tricubic(const float *__restrict__ d, int sx, int sy, int sz, const G3 &g, F3 o, F3 p) {
    const float gx = gclamp((p.x - o.x) / g.hx), gy = gclamp((p.y - o.y) / g.hy), gz = gclamp((p.z - o.z) / g.hz);
    int xi[4], yi[4], zi[4];
    float fx, fy, fz;
    cubic_idx(gx, sx, xi, fx);
    cubic_idx(gy, sy, yi, fy);
    cubic_idx(gz, sz, zi, fz);
    float zv[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        float row[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const float *r = d + sx * (yi[b] + sy * zi[c]);
            row[b] = mono_cubic(__ldg(r + xi[0]), __ldg(r + xi[1]), __ldg(r + xi[2]), __ldg(r + xi[3]), fx);
        }
        zv[c] = mono_cubic(row[0], row[1], row[2], row[3], fy);
    }
    return mono_cubic(zv[0], zv[1], zv[2], zv[3], fz);
}

typedef unsigned long long f32x2;   // two packed floats

// what one axis of the grid gives the samples of the trace (trace_field)
struct TraceAxis {
    float h, r;      // spacing, reciprocal
    float o[2];      // origin of the face grid (0) and of the centre grid (1)
    int end[2];      // below it an index has both linear taps inside
};
struct VelField {
    G3 g;
    const float *u, *v, *w;   // velocity the trace follows
    const float *phi;         // collider SDF (cell centred) or null
    // for the trace and the samples along it (trace_field)
    TraceAxis ax[3];
    f32x2 nzero;              // (-0, -0), see prod2
    int pow2;                 // all three spacings are powers of two
};
inline VelField trace_field(VelField F) {
    const float h[3] = {F.g.hx, F.g.hy, F.g.hz}, o[3] = {F.g.ox, F.g.oy, F.g.oz};
    const int n[3] = {F.g.nx, F.g.ny, F.g.nz};
    F.nzero = 0x8000000080000000ull;
    F.pow2 = 1;
    for (int a = 0; a < 3; ++a) {
        int e;
        F.pow2 = F.pow2 && frexpf(h[a], &e) == 0.5f;
        // (split() takes coordinates below 2^22)
        const int end = std::min(n[a], 1 << 22);
        F.ax[a] = TraceAxis{h[a], 1.0f / h[a], {o[a], o[a] + h[a] * 0.5f}, {end, end - 1}};
    }
    return F;
}

__device__ __forceinline__ F3 sample_vel(const VelField &F, F3 p) {
    int sx, sy, sz;
    F3 r;
    comp_shape(F.g, 0, sx, sy, sz);
    r.x = trilinear(F.u, sx, sy, sz, F.g, comp_origin(F.g, 0), p);
    comp_shape(F.g, 1, sx, sy, sz);
    r.y = trilinear(F.v, sx, sy, sz, F.g, comp_origin(F.g, 1), p);
    comp_shape(F.g, 2, sx, sy, sz);
    r.z = trilinear(F.w, sx, sy, sz, F.g, comp_origin(F.g, 2), p);
    return r;
}
__device__ __forceinline__ float sample_phi(const VelField &F, const float *phi, F3 p) {
    if (!phi) return 1.0f;
    return trilinear(phi, F.g.nx, F.g.ny, F.g.nz, F.g, comp_origin(F.g, 3), p);
}

// ---- samples away from the array ends -----------------------------------
// (of grids of two planes and more: see advect_form and point_form)
// The trace and the tricubic sample are bound by issue and by instruction
// fetch (about 2300 instructions a face in the straightforward form), so where
// no tap needs clamping they run in a shorter form of the same operations: the
// six coordinates that the three face grids and the cell grid share are formed
// once, the division by h is a multiplication where h is a power of two (P2) and
// a corrected product elsewhere, floor is an addition, taps of a row share an
// address, and two samples run in one packed FP32 pair (add, sub and mul round
// each half as the scalar instruction does).  A point with a tap past an end
// takes the functions above.

// a / h, correctly rounded: with r the correctly rounded 1 / h, one Newton
// correction makes the product faithful and a second, by Markstein's theorem
// (1990), correct; exact for a power of two.  For quotients from 1e-20 to 2e8,
// where the remainders are exact.
template <bool P2>
__device__ __forceinline__ float div_in(float a, float h, float r) {
    const float q = a * r;
    if (P2) return q;
    const float q1 = __fmaf_rn(__fmaf_rn(-q, h, a), r, q);
    return __fmaf_rn(__fmaf_rn(-q1, h, a), r, q1);
}
__device__ __noinline__ float div_any(float a, float h) { return a / h; }
template <bool P2>
__device__ __forceinline__ float div_h(float a, float h, float r) {
    const float q = div_in<P2>(a, h, r);
    if (P2) return q;
    return q < 2.0e8f && q > 1.0e-20f ? q : div_any(a, h);
}
// index and fraction of a coordinate in [0, 2^22): 1.5 * 2^23 added rounding
// down leaves the floor in the low bits of the significand (floorf and the
// conversion run at a quarter of the rate).  As an unsigned number the index is
// 2^22 or more for a larger or negative coordinate and for a NaN.
__device__ __forceinline__ void split(float q, int &i, float &f) {
    const float t = __fadd_rd(q, 12582912.0f);
    i = __float_as_int(t) - 0x4b400000;
    f = q - (t - 12582912.0f);
}
// one axis: index and fraction of a point on the face (0) or centre (1) grid;
// false where a tap is outside, or the coordinate below div_in's range
template <bool P2>
__device__ __forceinline__ bool axis_at(const TraceAxis &A, int c, float p, int &i, float &f) {
    const float q = div_in<P2>(p - A.o[c], A.h, A.r);
    split(q, i, f);
    return (unsigned)i < (unsigned)A.end[c] && (P2 || q > 1.0e-20f);
}

__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ void unpack2(f32x2 d, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(d));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// a product that is an operand of a sum: the compiler contracts add2(c, mul2(a,
// b)) to one rounding whatever -fmad says.  A fused a b + (-0) is the rounded
// product, sign of zero included, and where the compiler cannot see that the
// addend z is -0 it stays two operations; z therefore comes with the arguments.
__device__ __forceinline__ f32x2 prod2(f32x2 a, f32x2 b, f32x2 z) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(z));
    return d;
}
struct Axis6 {
    int i[2];
    float f[2];
};
struct Point6 {
    Axis6 x, y, z;
};
template <bool P2>
__device__ __forceinline__ bool point6(const VelField &F, F3 p, Point6 &q) {
    bool in = true;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        in &= axis_at<P2>(F.ax[0], c, p.x, q.x.i[c], q.x.f[c]);
        in &= axis_at<P2>(F.ax[1], c, p.y, q.y.i[c], q.y.f[c]);
        in &= axis_at<P2>(F.ax[2], c, p.z, q.z.i[c], q.z.f[c]);
    }
    return in;
}
// trilinear() at index (i, j, k) with all taps inside
__device__ __forceinline__ float lin1(const float *__restrict__ d, int sx, int sy, int i, int j, int k, float fx, float fy,
                                      float fz) {
    const float *r0 = d + (i + sx * (j + sy * k)), *r1 = r0 + sx, *r2 = r0 + sx * sy, *r3 = r2 + sx;
    const float ux = 1.0f - fx, uy = 1.0f - fy, uz = 1.0f - fz;
    const float w00 = ux * uy, w10 = fx * uy, w01 = ux * fy, w11 = fx * fy;
    float s = __ldg(r0) * (w00 * uz);
    s = s + __ldg(r0 + 1) * (w10 * uz);
    s = s + __ldg(r1) * (w01 * uz);
    s = s + __ldg(r1 + 1) * (w11 * uz);
    s = s + __ldg(r2) * (w00 * fz);
    s = s + __ldg(r2 + 1) * (w10 * fz);
    s = s + __ldg(r3) * (w01 * fz);
    return s + __ldg(r3 + 1) * (w11 * fz);
}
// two of them, u and v
__device__ __forceinline__ void lin_uv(const VelField &F, const Point6 &q, float &u, float &v) {
    const int nx = F.g.nx, ny = F.g.ny;
    const float *a0 = F.u + (q.x.i[0] + (nx + 1) * (q.y.i[1] + ny * q.z.i[1]));
    const float *b0 = F.v + (q.x.i[1] + nx * (q.y.i[0] + (ny + 1) * q.z.i[1]));
    const float *a1 = a0 + (nx + 1), *a2 = a0 + (nx + 1) * ny, *a3 = a2 + (nx + 1);
    const float *b1 = b0 + nx, *b2 = b0 + nx * (ny + 1), *b3 = b2 + nx;
    const f32x2 one = pack2(1.0f, 1.0f);
    const f32x2 fx = pack2(q.x.f[0], q.x.f[1]), fy = pack2(q.y.f[1], q.y.f[0]), fz = pack2(q.z.f[1], q.z.f[1]);
    const f32x2 ux = sub2(one, fx), uy = sub2(one, fy), uz = sub2(one, fz);
    const f32x2 w00 = mul2(ux, uy), w10 = mul2(fx, uy), w01 = mul2(ux, fy), w11 = mul2(fx, fy);
    auto d = [](const float *a, const float *b) { return pack2(__ldg(a), __ldg(b)); };
    f32x2 s = prod2(d(a0, b0), mul2(w00, uz), F.nzero);
    s = add2(s, prod2(d(a0 + 1, b0 + 1), mul2(w10, uz), F.nzero));
    s = add2(s, prod2(d(a1, b1), mul2(w01, uz), F.nzero));
    s = add2(s, prod2(d(a1 + 1, b1 + 1), mul2(w11, uz), F.nzero));
    s = add2(s, prod2(d(a2, b2), mul2(w00, fz), F.nzero));
    s = add2(s, prod2(d(a2 + 1, b2 + 1), mul2(w10, fz), F.nzero));
    s = add2(s, prod2(d(a3, b3), mul2(w01, fz), F.nzero));
    s = add2(s, prod2(d(a3 + 1, b3 + 1), mul2(w11, fz), F.nzero));
    unpack2(s, u, v);
}
// Lanes that are together here take one path: the other's results are the same, and
// both one after the other cost more than the straightforward form alone (which
// showed on small grids, where most warps touch an end: one of 39 us took 63).
__device__ __forceinline__ bool warp_any(bool p) { return __any_sync(__activemask(), p); }
__device__ __noinline__ F3 sample_vel_ends(const VelField &F, F3 p) { return sample_vel(F, p); }
__device__ __noinline__ float sample_phi_ends(const VelField &F, F3 p) { return sample_phi(F, F.phi, p); }
template <bool P2>
__device__ __forceinline__ F3 trace_vel(const VelField &F, F3 p) {
    Point6 q;
    if (warp_any(!point6<P2>(F, p, q))) return sample_vel_ends(F, p);
    F3 r;
    lin_uv(F, q, r.x, r.y);
    r.z = lin1(F.w, F.g.nx, F.g.ny, q.x.i[1], q.y.i[1], q.z.i[0], q.x.f[1], q.y.f[1], q.z.f[0]);
    return r;
}
template <bool P2>
__device__ __forceinline__ float trace_phi(const VelField &F, F3 p) {
    if (!F.phi) return 1.0f;
    int i, j, k;
    float fx, fy, fz;
    bool in = axis_at<P2>(F.ax[0], 1, p.x, i, fx);
    in &= axis_at<P2>(F.ax[1], 1, p.y, j, fy);
    in &= axis_at<P2>(F.ax[2], 1, p.z, k, fz);
    if (warp_any(!in)) return sample_phi_ends(F, p);
    return lin1(F.phi, F.g.nx, F.g.ny, i, j, k, fx, fy, fz);
}

// mono_cubic on two rows of taps at once
__device__ __forceinline__ f32x2 mono_cubic2(f32x2 f0, f32x2 f1, f32x2 f2, f32x2 f3, f32x2 f, f32x2 z) {
    const f32x2 half = pack2(0.5f, 0.5f);
    const f32x2 D1 = sub2(f2, f1), r1 = mul2(sub2(f2, f0), half), r2 = mul2(sub2(f3, f1), half);
    float Da, Db, r1a, r1b, r2a, r2b, p1a, p1b, p2a, p2b;
    unpack2(D1, Da, Db);
    unpack2(r1, r1a, r1b);
    unpack2(r2, r2a, r2b);
    unpack2(mul2(r1, D1), p1a, p1b);
    unpack2(mul2(r2, D1), p2a, p2b);
    const bool fa = fabsf(Da) < 1e-12f, fb = fabsf(Db) < 1e-12f;
    const f32x2 d1 = pack2((fa || p1a < 0.0f) ? 0.0f : r1a, (fb || p1b < 0.0f) ? 0.0f : r1b);
    const f32x2 d2 = pack2((fa || p2a < 0.0f) ? 0.0f : r2a, (fb || p2b < 0.0f) ? 0.0f : r2b);
    const f32x2 three = pack2(3.0f, 3.0f);
    const f32x2 a3 = sub2(add2(d1, d2), add2(D1, D1));
    const f32x2 a2 = sub2(sub2(prod2(D1, three, z), add2(d1, d1)), d2);
    f32x2 t = prod2(mul2(mul2(a3, f), f), f, z);
    t = add2(t, prod2(mul2(a2, f), f, z));
    t = add2(t, prod2(d1, f, z));
    return add2(t, f1);
}
__device__ __noinline__ float tricubic_ends(const float *__restrict__ d, int sx, int sy, int sz, const G3 &g, F3 o, F3 p) {
    return tricubic(d, sx, sy, sz, g, o, p);
}
// tricubic() on component a (3: cells): rows of two z taps at a time
template <bool P2>
__device__ __forceinline__ float trace_cubic(const VelField &F, int a, const float *__restrict__ d, int sx, int sy, int sz,
                                             F3 o, F3 p) {
    int i, j, k;
    float fx, fy, fz;
    bool in = axis_at<P2>(F.ax[0], a != 0, p.x, i, fx);
    in &= axis_at<P2>(F.ax[1], a != 1, p.y, j, fy);
    in &= axis_at<P2>(F.ax[2], a != 2, p.z, k, fz);
    const int dz = sx * sy;
    if (warp_any(!(in && i >= 1 && i <= sx - 3 && j >= 1 && j <= sy - 3 && k >= 1 && k <= sz - 3)))
        return tricubic_ends(d, sx, sy, sz, F.g, o, p);
    const f32x2 fx2 = pack2(fx, fx), fy2 = pack2(fy, fy);
    const float *r = d + ((i - 1) + sx * ((j - 1) + sy * (k - 1)));
    float z[4];
#pragma unroll 1
    for (int c = 0; c < 2; ++c) {
        f32x2 row[4];
        const float *ra = r, *rb = r + dz;
#pragma unroll
        for (int b = 0; b < 4; ++b, ra += sx, rb += sx)
            row[b] = mono_cubic2(pack2(__ldg(ra), __ldg(rb)), pack2(__ldg(ra + 1), __ldg(rb + 1)),
                                 pack2(__ldg(ra + 2), __ldg(rb + 2)), pack2(__ldg(ra + 3), __ldg(rb + 3)), fx2, F.nzero);
        z[0] = z[2], z[1] = z[3];
        unpack2(mono_cubic2(row[0], row[1], row[2], row[3], fy2, F.nzero), z[2], z[3]);
        r += 2 * dz;
    }
    return mono_cubic(z[0], z[1], z[2], z[3], fz);
}

// backTrace (advection_solver3.js:20-62): RK2 midpoint substeps of at most
// one cell, stopping on the collider with a linear blend of the last step.  The
// straightforward form.
__device__ inline F3 back_trace_plain(const VelField &F, F3 pos, float dt, float dirn, int max_substeps) {
    const float h = fminf(F.g.hx, fminf(F.g.hy, F.g.hz));
    F3 pt = pos;
    float T = dt;
    for (int s = 0; s < max_substeps; ++s) {
        if (T <= 1e-6f) break;
        const F3 v0 = sample_vel(F, pt);
        const float len = sqrtf(v0.x * v0.x + v0.y * v0.y + v0.z * v0.z);
        const float nsub = fmaxf(ceilf(len * T / h), 1.0f);
        const float sdt = T / nsub;
        const float hs = sdt * 0.5f;
        const F3 mid{pt.x - v0.x * hs * dirn, pt.y - v0.y * hs * dirn, pt.z - v0.z * hs * dirn};
        const F3 mv = sample_vel(F, mid);
        const F3 nxt{pt.x - mv.x * sdt * dirn, pt.y - mv.y * sdt * dirn, pt.z - mv.z * sdt * dirn};
        const float phi1 = sample_phi(F, F.phi, nxt);
        if (phi1 <= 0.0f) {
            const float phi0 = sample_phi(F, F.phi, pt);   // (here: few paths end at the collider)
            const float w = fabsf(phi1) / (fabsf(phi0) + fabsf(phi1));
            const float wm = 1.0f - w;
            pt = F3{pt.x * w + nxt.x * wm, pt.y * w + nxt.y * wm, pt.z * w + nxt.z * wm};
            break;
        }
        T = T - sdt;
        pt = nxt;
    }
    return pt;
}

// back_trace_plain in the short form.
// phi0: the collider's value at pos, if the caller has it (else a NaN); a
// substep's end is the next one's start, with its value.
template <bool P2>
__device__ __forceinline__ F3 back_trace(const VelField &F, F3 pos, float dt, float dirn, int max_substeps, float phi0) {
    const float h = fminf(F.g.hx, fminf(F.g.hy, F.g.hz));
    const float rh = h == F.g.hx ? F.ax[0].r : (h == F.g.hy ? F.ax[1].r : F.ax[2].r);
    F3 pt = pos;
    float T = dt;
#pragma unroll 1
    for (int s = 0; s < max_substeps; ++s) {
        if (T <= 1e-6f) break;
        F3 at = pt;
        float sdt = 0.0f;
        // one copy of the sample's code for the start and the midpoint
#pragma unroll 1
        for (int mid = 0; mid < 2; ++mid) {
            const F3 v = trace_vel<P2>(F, at);
            float step;
            if (mid == 0) {
                const float len = sqrtf(v.x * v.x + v.y * v.y + v.z * v.z);
                const float nsub = fmaxf(ceilf(div_h<P2>(len * T, h, rh)), 1.0f);
                sdt = nsub == 1.0f ? T : T / nsub;
                step = sdt * 0.5f;
            } else {
                step = sdt;
            }
            at = F3{pt.x - v.x * step * dirn, pt.y - v.y * step * dirn, pt.z - v.z * step * dirn};
        }
        const F3 nxt = at;
        const float phi1 = trace_phi<P2>(F, nxt);
        if (phi1 <= 0.0f) {
            if (s == 0 && isnan(phi0)) phi0 = trace_phi<P2>(F, pt);
            const float w = fabsf(phi1) / (fabsf(phi0) + fabsf(phi1));
            const float wm = 1.0f - w;
            pt = F3{pt.x * w + nxt.x * wm, pt.y * w + nxt.y * wm, pt.z * w + nxt.z * wm};
            break;
        }
        phi0 = phi1;
        T = T - sdt;
        pt = nxt;
    }
    return pt;
}

// the forms of the trace and the samples: the straightforward one, and the short one
// for any spacing and for powers of two
enum { FORM_PLAIN, FORM_SHORT, FORM_SHORT_P2 };
template <int FORM>
__device__ __forceinline__ F3 trace_back(const VelField &F, F3 pos, float dt, float dirn, int max_substeps, float phi0) {
    if constexpr (FORM == FORM_PLAIN) return back_trace_plain(F, pos, dt, dirn, max_substeps);
    else return back_trace<FORM == FORM_SHORT_P2>(F, pos, dt, dirn, max_substeps, phi0);
}

// The form for a list of n points.  A point takes a trace and no tricubic sample, and
// lanes of one warp can have points anywhere: the short form pays for lists that keep
// the GPU full, in cell order from about a million points (128^3, straightforward over
// short: 1M points 0.91-1.03, 2M 1.00-1.18, 8M 1.25-1.36), in random
// order from about eight (4M 0.95-0.98, 8M 1.00); in a grid one cell thick it never does
// (1024 x 256, a million points: 0.62-0.69).
constexpr long long POINTS_SHORT = 1LL << 23;
inline int point_form(const VelField &F, long long n) {
    if (F.g.nz == 1 || n < POINTS_SHORT) return FORM_PLAIN;
    return F.pow2 ? FORM_SHORT_P2 : FORM_SHORT;
}

// (i, j, k) of a flat index; below 2^31 in 32-bit unsigned arithmetic (a
// 64-bit division is a long software sequence on the GPU)
__device__ __forceinline__ void unflatten(long long f, int sx, int sy, int &i, int &j, int &k) {
    if (f < 0x7fffffffLL) {
        const unsigned u = (unsigned)f, r = u / (unsigned)sx, q = r / (unsigned)sy;
        i = (int)(u - r * (unsigned)sx);
        j = (int)(r - q * (unsigned)sy);
        k = (int)q;
        return;
    }
    i = (int)(f % sx);
    long long r = f / sx;
    j = (int)(r % sy);
    k = (int)(r / sy);
}

// ---------------------------------------------------- velocity constraint --
// fractionInsideSdf (level_set_utils.js:24-40)
__device__ __forceinline__ float frac_inside_sdf(float p0, float p1) {
    const bool a = p0 < 0.0f, b = p1 < 0.0f;
    if (a && b) return 1.0f;
    if (a) return p0 / (p0 - p1);
    if (b) return p1 / (p1 - p0);
    return 0.0f;
}

// Division of face indices (below 2^31) by a grid extent as a multiply, an
// add and a shift: q = (hi(n m) + n) >> s with s = ceil(log2 d) and
// m = floor(2^32 (2^s - d) / d) + 1 (Granlund and Montgomery 1994).
struct FastDiv {
    unsigned d, m, s;
    __device__ __forceinline__ unsigned div(unsigned n) const { return (__umulhi(n, m) + n) >> s; }
};
inline FastDiv fast_div(int d) {
    unsigned s = 0;
    while ((1u << s) < (unsigned)d) ++s;
    const unsigned long long m = ((1ull << 32) * ((1ull << s) - (unsigned)d)) / (unsigned)d + 1;
    return FastDiv{(unsigned)d, (unsigned)m, s};
}

// One face component's array extents, and up to three components for one
// launch (blockIdx.z picks the component).
struct CompDims {
    int sx, sy, sz;
    unsigned n;
    FastDiv dx, dy;
    __device__ __forceinline__ void at(unsigned f, int &i, int &j, int &k) const {
        const unsigned r = dx.div(f), q = dy.div(r);
        i = (int)(f - r * (unsigned)sx);
        j = (int)(r - q * (unsigned)sy);
        k = (int)q;
    }
};
inline CompDims comp_dims(const G3 &g, int a) {
    CompDims c;
    comp_shape(g, a, c.sx, c.sy, c.sz);
    c.n = (unsigned)((long long)c.sx * c.sy * c.sz);
    c.dx = fast_div(c.sx);
    c.dy = fast_div(c.sy);
    return c;
}
struct Comps3 {
    CompDims c[3];
    float *d[3];
};

// createExtrapolateToRegion3's Jacobi steps (array_utils3.js:88-150) in
// place.  A face carries one byte: 0 valid from the start, t made valid by
// step t, LAYER_OPEN not valid yet.  Step t gives a face that is not valid
// the mean of its neighbours with a byte below t, which no thread of the
// step writes; a face that the step itself makes valid reads as t or as
// LAYER_OPEN, and neither is below t.  So one value array and one byte array
// do for the two value and two marker arrays of the double-buffered form.
constexpr unsigned LAYER_OPEN = 255;
constexpr int LAYER_STEPS = 254;   // steps before the bytes are folded back to 0

__device__ __forceinline__ bool extend_face(const CompDims &c, const float *d, const uint8_t *lay, unsigned f, int t,
                                            float &out) {
    int i, j, k;
    c.at(f, i, j, k);
    const int sy = c.sx, sz = c.sx * c.sy;
    float total = 0.0f;
    int count = 0;
    if (i + 1 < c.sx && lay[f + 1] < t) { total = total + d[f + 1]; ++count; }
    if (i > 0 && lay[f - 1] < t) { total = total + d[f - 1]; ++count; }
    if (j + 1 < c.sy && lay[f + sy] < t) { total = total + d[f + sy]; ++count; }
    if (j > 0 && lay[f - sy] < t) { total = total + d[f - sy]; ++count; }
    if (k + 1 < c.sz && lay[f + sz] < t) { total = total + d[f + sz]; ++count; }
    if (k > 0 && lay[f - sz] < t) { total = total + d[f - sz]; ++count; }
    if (count == 0) return false;
    out = total / (float)count;
    return true;
}

// trilinearGradientAtPosition3 (grid_math3.js:295-352)
__device__ F3 trilinear_gradient(const float *__restrict__ d, const G3 &g, F3 o, F3 pos) {
    const int n[3] = {g.nx, g.ny, g.nz};
    const float coord[3] = {gclamp((pos.x - o.x) / g.hx), gclamp((pos.y - o.y) / g.hy), gclamp((pos.z - o.z) / g.hz)};
    int lo[3], hi[3];
    float t[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int idx = (int)floorf(coord[a]);
        lo[a] = max(0, min(idx, n[a] - 2));
        hi[a] = min(lo[a] + 1, n[a] - 1);
        t[a] = fminf(fmaxf(coord[a] - (float)lo[a], 0.0f), 1.0f);
    }
    auto V = [&](int i, int j, int k) { return __ldg(d + i + g.nx * (j + g.ny * k)); };
    const float v000 = V(lo[0], lo[1], lo[2]), v100 = V(hi[0], lo[1], lo[2]), v010 = V(lo[0], hi[1], lo[2]);
    const float v110 = V(hi[0], hi[1], lo[2]), v001 = V(lo[0], lo[1], hi[2]), v101 = V(hi[0], lo[1], hi[2]);
    const float v011 = V(lo[0], hi[1], hi[2]), v111 = V(hi[0], hi[1], hi[2]);
    const float tx = t[0], ty = t[1], tz = t[2];
    F3 r;
    float s = (1.0f - ty) * (1.0f - tz) * (v100 - v000);
    s = s + ty * (1.0f - tz) * (v110 - v010);
    s = s + (1.0f - ty) * tz * (v101 - v001);
    s = s + ty * tz * (v111 - v011);
    r.x = s / g.hx;
    s = (1.0f - tx) * (1.0f - tz) * (v010 - v000);
    s = s + tx * (1.0f - tz) * (v110 - v100);
    s = s + (1.0f - tx) * tz * (v011 - v001);
    s = s + tx * tz * (v111 - v101);
    r.y = s / g.hy;
    s = (1.0f - tx) * (1.0f - ty) * (v001 - v000);
    s = s + tx * (1.0f - ty) * (v101 - v100);
    s = s + (1.0f - tx) * ty * (v011 - v010);
    s = s + tx * ty * (v111 - v110);
    r.z = s / g.hz;
    return r;
}


}  // namespace ffg
}  // namespace
