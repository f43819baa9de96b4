// Level geometry and the cell stencils shared by the fused level kernels
// (ff_fused.cu) and the resident solver (ff_resident.cu).
#pragma once
#include "ff_device.cuh"

namespace {

using namespace ffd;

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
    float s = __fmul_rn(-q.e, vc);
    s = __fmaf_rn(q.kx, xm - vc, s);
    s = __fmaf_rn(q.ux, xp - vc, s);
    s = __fmaf_rn(q.ky, ym - vc, s);
    s = __fmaf_rn(q.uy, yp - vc, s);
    s = __fmaf_rn(q.kz, zm - vc, s);
    return __fmaf_rn(q.uz, zp - vc, s);
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

// The sums of products below are shared by the launch-per-pass kernels and the one-launch
// ones, whose results are equal bit for bit: which product is rounded before it enters a
// fused multiply-add is written out, not left to the compiler (it chose by what else a
// product is used for, differently for the two cells of a thread).
// x taps of the restriction; first: the first product is the rounded one (even coarse
// cells of level 0), else the second
__device__ __forceinline__ float x_taps(bool first, float r0, float r1, float r2, float r3) {
    const float s = first ? __fmaf_rn(0.375f, r1, __fmul_rn(0.125f, r0)) : __fmaf_rn(0.125f, r0, __fmul_rn(0.375f, r1));
    return __fmaf_rn(0.125f, r3, __fmaf_rn(0.375f, r2, s));
}
// the two x taps of the prolongation
__device__ __forceinline__ float two_taps(float wa, float a, float wb, float b) {
    return __fmaf_rn(wa, a, __fmul_rn(wb, b));
}

// compensated (TwoSum) FP32 accumulation, folded into FP64 once
struct Acc {
    float s = 0.f, e = 0.f;
    __device__ __forceinline__ void add(float v) {
        float t, err;
        two_sum(s, v, t, err);
        s = t;
        e = __fadd_rn(e, err);
    }
    __device__ __forceinline__ double value() const { return (double)s + (double)e; }
};

// A neighbour across the domain edge stands in as the cell itself, so the
// absent face's difference is an exact zero.  (Adding h^-2 v back to a
// zero-filled neighbour's -h^-2 v cancels to within a rounding of h^-2 |v|:
// near a wall under a hydrostatic pressure that is far above the residual
// the solve has to reach.)
__device__ __forceinline__ void edge_self(const Geo &g, int i, int j, int k, float vc, float &xm, float &xp,
                                          float &ym, float &yp, float &zm, float &zp) {
    if (i == 0) xm = vc;
    if (i == g.d.nx - 1) xp = vc;
    if (j == 0) ym = vc;
    if (j == g.d.ny - 1) yp = vc;
    if (k == 0) zm = vc;
    if (k == g.d.nz - 1) zp = vc;
}

// the couplings of class-3 cell ci
__device__ __forceinline__ Coef general_coef(const float4 *coef, const float4 *gco, int i, int j, int k, long long ci) {
    const float4 lo = __ldg(coef + ci), hi = __ldg(gco + ci);
    return Coef{i > 0 ? lo.x : 0.f, j > 0 ? lo.y : 0.f, k > 0 ? lo.z : 0.f, lo.w, hi.x, hi.y, hi.z};
}
// (A v)_c of one cell by class; general(): a class-3 cell's couplings
template <class Q>
__device__ __forceinline__ float ap_by_class(const Geo &g, unsigned c, int i, int j, int k, float vc, float xm, float xp,
                                             float ym, float yp, float zm, float zp, Q general) {
    if (c == 2u) edge_self(g, i, j, k, vc, xm, xp, ym, yp, zm, zp);
    const float ar = apply_reg(g, vc, xm, xp, ym, yp, zm, zp);
    if (c == 0u || c == 2u) return ar;
    if (c == 1u) return -vc;
    return apply_q(general(), vc, xm, xp, ym, yp, zm, zp);
}
__device__ __forceinline__ float ap_cell(const Geo &g, const float4 *coef, const float4 *gco, unsigned c, int i,
                                         int j, int k, long long ci, float vc, float xm, float xp, float ym, float yp,
                                         float zm, float zp) {
    return ap_by_class(g, c, i, j, k, vc, xm, xp, ym, yp, zm, zp,
                       [&] { return general_coef(coef, gco, i, j, k, ci); });
}

// r = b - A x in double-single for one cell of class 1 or 3: each coupling
// term K (x_n - x_c) formed from (hi, lo) with an error-free difference and
// product, summed with TwoSum (the general path of the cp.async kernel).
__device__ __forceinline__ float resid_ds_general(const Coef &q, float bc, float chv, float clv, float xmh,
                                                  float xml, float xph, float xpl, float ymh, float yml, float yph,
                                                  float ypl, float zmh, float zml, float zph, float zpl) {
    float S = 0.f, Se = 0.f;
    auto term = [&](float K, float hn, float ln) {
        float dh, de;
        two_sum(hn, -chv, dh, de);
        de = __fadd_rn(de, __fsub_rn(ln, clv));
        float pr, pe;
        two_prod(K, dh, pr, pe);
        pe = __fmaf_rn(K, de, pe);
        float s2, e2;
        two_sum(S, pr, s2, e2);
        S = s2;
        Se = __fadd_rn(Se, __fadd_rn(e2, pe));
    };
    term(q.kx, xmh, xml);
    term(q.ux, xph, xpl);
    term(q.ky, ymh, yml);
    term(q.uy, yph, ypl);
    term(q.kz, zmh, zml);
    term(q.uz, zph, zpl);
    {
        float pr, pe;
        two_prod(-q.e, chv, pr, pe);
        pe = __fmaf_rn(-q.e, clv, pe);
        float s2, e2;
        two_sum(S, pr, s2, e2);
        S = s2;
        Se = __fadd_rn(Se, __fadd_rn(e2, pe));
    }
    float r0, e0;
    two_sum(bc, -S, r0, e0);
    return __fadd_rn(r0, __fsub_rn(e0, Se));
}

// One cell's residual by class (hi/lo of the cell and its six neighbours);
// general(): a class-3 cell's couplings.
template <bool DS, class Q>
__device__ __forceinline__ float resid_by_class(const Geo &g, unsigned c, int i, int j, int k, float bc, float ch, float cl,
                                                float xmh, float xml, float xph, float xpl, float ymh, float yml,
                                                float yph, float ypl, float zmh, float zml, float zph, float zpl,
                                                Q general) {
    if (!(c & 1u)) {
        if (c == 2u) {
            edge_self(g, i, j, k, ch, xmh, xph, ymh, yph, zmh, zph);
            if (DS) edge_self(g, i, j, k, cl, xml, xpl, yml, ypl, zml, zpl);
        }
        float ax = apply_reg(g, ch, xmh, xph, ymh, yph, zmh, zph);
        if (DS) ax += apply_reg(g, cl, xml, xpl, yml, ypl, zml, zpl);
        return bc - ax;
    }
    Coef q{0.f, 0.f, 0.f, 1.f, 0.f, 0.f, 0.f};
    if (c != 1u) q = general();
    if (DS)
        return resid_ds_general(q, bc, ch, cl, xmh, xml, xph, xpl, ymh, yml, yph, ypl, zmh, zml, zph, zpl);
    return bc - apply_q(q, ch, xmh, xph, ymh, yph, zmh, zph);
}
template <bool DS>
__device__ __forceinline__ float resid_cell(const Geo &g, const float4 *coef, const float4 *gco, unsigned c, int i,
                                            int j, int k, long long ci, float bc, float ch, float cl, float xmh,
                                            float xml, float xph, float xpl, float ymh, float yml, float yph,
                                            float ypl, float zmh, float zml, float zph, float zpl) {
    return resid_by_class<DS>(g, c, i, j, k, bc, ch, cl, xmh, xml, xph, xpl, ymh, yml, yph, ypl, zmh, zml, zph, zpl,
                              [&] { return general_coef(coef, gco, i, j, k, ci); });
}

// The order in which the level-0 CG kernels and the last sweep sum a dot product:
// work items of 64 x 16 cells by zc planes, in an item 256 threads that each add
// up one x-quad's products (rounded to FP32) plane by plane, the threads by
// warps, the items dealt out over 256 threads again.
constexpr int DOT_TX = 64, DOT_TY = 16, DOT_THREADS = 256;
struct DotOrder {
    int gx, gy, zc, items;
    int first;   // place of the items' sums among the solver's
};
// quad and row in its tile of a thread of an item
__device__ __forceinline__ int dot_quad(int tid) { return tid & (DOT_TX / 4 - 1); }
__device__ __forceinline__ int dot_row(int tid) { return 4 * (tid >> 6) + ((tid >> 5) & 1) + 2 * ((tid >> 4) & 1); }

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
