// Cooperative kernels for the parts of a projection that are too small for
// one launch per pass: the coarse levels of a V-cycle (k_vcycle_tail), and,
// where level 0 itself is small, the whole PCG solve (k_pcg_resident).
//
// Phases over one level are separated by grid-wide barriers; values that
// another block wrote in this launch are read through L2 (ld.global.cg).  A
// phase on such a level is bound by latency, a barrier plus one or two L2
// round trips, and not by bandwidth or issue, so
//  - the work of a phase is dealt out a warp at a time over all blocks: a
//    level of a few thousand cells then keeps one or two warps busy on every
//    SM instead of all warps on a few;
//  - levels of up to HELD_CELLS cells, and the coarsest level's sweeps, run in
//    block 0 with their arrays in shared memory: a phase there costs a block
//    barrier and a shared-memory round trip.
// Per cell the arithmetic is that of the level kernels in ff_fused.cu: the
// sweep's relaxation by class, the residual by class followed by the x, y and
// z taps of the restriction, k_coarse_direct's row products, k_prolong4's
// correction; the CG phases are k_update_p_pap's and k_update_x_residual's.
#include "ff_stencil.cuh"
#include <algorithm>
#include <type_traits>

using namespace ffd;

namespace {

constexpr int NT = 512;
constexpr int MAXL = 12;
constexpr int HELD_CELLS = 8192;        // level held in block 0's shared memory
constexpr int COARSE_CELLS = 8192;      // coarsest level swept in block 0
constexpr int SMEM_BYTES = 192 * 1024;

struct RLevel {
    Geo g;
    float *x, *b, *r;              // r: residual scratch of the level
    // a held level's x and b in shared memory (offsets in floats, one zero
    // cell around the level on every axis) and its pair table
    int xo, bo, to;
    // t / (nx / 2), t / nx and t / ny as (t m) >> 40 with m = ceil(2^40 /
    // divisor) (exact for every t below 2^22 and divisor below 2^18)
    unsigned long long mhx, mnx, mny;
    const float4 *coef, *gco;
    const uint8_t *cls, *mask;     // class bytes (cpitch bytes per row), Dirichlet mask (may be null)
    int cpitch;
    float rdreg_sor;               // sor / dreg
};
struct VArgs {
    RLevel lv[MAXL];
    int nl;                        // levels, the last one the coarsest
    int held;                      // first held level (nl - 1: none)
    int down, up, final;           // sweeps before and after the correction, and after it on lv[0]
    float sor, omsor;
    const double *G;               // coarsest inverse, nG x nG, row-major (direct mode)
    int nG;
    int coarse_sweeps;             // > 0: that many sweeps on the coarsest level instead of G b
    unsigned *bar;                 // grid barrier: arrivals, blocks done, abort
    int ro, cxo, cbo;              // shared memory: held levels' residual, the coarsest x and b
};

// The arguments as the phases read them: a phase is a function of its own
// (inlined into one body they need more registers than there are, and spilled
// in every pass), takes a level by its index and copies what it uses.
__shared__ VArgs SA;
struct Relax {
    float sor, omsor;
};
__device__ __forceinline__ Relax relax_of() { return Relax{SA.sor, SA.omsor}; }

__device__ __forceinline__ int tdiv(int t, unsigned long long m) {
    return (int)(((unsigned long long)(unsigned)t * m) >> 40);
}

// Grid-wide barrier of a cooperative launch over three words: a count of
// arrivals that only grows within a launch (barrier k completes when it
// reaches k x blocks), the number of blocks done with the launch (the last
// one clears both counts, once no block polls them), and an abort flag.  A
// block that waits more than 0.5 s raises the abort flag, which releases
// every waiting block; all then return false.  The arrival is a release and
// the poll an acquire, so no separate fence orders the phases.
__device__ bool grid_sync(unsigned *bar, unsigned &passed) {
    __shared__ int ok_s;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned target = (passed + 1) * gridDim.x;
        int ok = 1, spins = 0;
        unsigned long long t0 = 0;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        while (true) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            if ((int)(v - target) >= 0) break;
            if ((++spins & 127) == 0) {
                unsigned ab;
                asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(ab) : "l"(bar + 2) : "memory");
                const unsigned long long t = globaltimer_ns();
                if (t0 == 0) t0 = t;
                if (ab || t - t0 > 500000000ull) {
                    atomicExch(bar + 2, 1u);
                    ok = 0;
                    break;
                }
            }
        }
        ok_s = ok;
    }
    __syncthreads();
    ++passed;
    return ok_s != 0;
}

// after a block's last barrier: the last block to get here clears the counts
__device__ void grid_done(unsigned *bar) {
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&bar[1], 1u) == gridDim.x - 1) {
            atomicExch(&bar[0], 0u);
            atomicExch(&bar[1], 0u);
        }
    }
}

// this thread's first item and the stride of a grid-wide phase: warps dealt
// out over the blocks in turn
struct Deal {
    int t0, stride;
};
__device__ __forceinline__ Deal deal() {
    return Deal{(int)(((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32 + (threadIdx.x & 31)),
                (int)(gridDim.x * NT)};
}

__device__ __forceinline__ unsigned class_at(const RLevel &L, int i, int j, int k) {
    return (__ldg(L.cls + L.cpitch * (j + L.g.d.ny * k) + (i >> 2)) >> (2 * (i & 3))) & 3u;
}
// sor over the diagonal of a plain cell (class 0 or 2)
template <bool D3>
__device__ __forceinline__ float plain_scale(const Relax &a, const RLevel &L, int i, int j, int k) {
    const Geo &g = L.g;
    float corr = g.h2x * (float)((i == 0) + (i == g.d.nx - 1)) + g.h2y * (float)((j == 0) + (j == g.d.ny - 1));
    if (D3) corr += g.h2z * (float)((k == 0) + (k == g.d.nz - 1));
    return corr == 0.f ? L.rdreg_sor : a.sor / (g.dreg + corr);
}
template <bool D3>
__device__ __forceinline__ float plain_sum(const Geo &g, float xm, float xp, float ym, float yp, float zm, float zp) {
    const float s = __fmaf_rn(g.h2y, ym + yp, g.h2x * (xm + xp));
    return D3 ? __fmaf_rn(g.h2z, zm + zp, s) : s;
}
__device__ __forceinline__ float general_sum(const float4 &lo, const float4 &hi, float xm, float xp, float ym, float yp,
                                             float zm, float zp) {
    float s = lo.x * xm;
    s = __fmaf_rn(hi.x, xp, s);
    s = __fmaf_rn(lo.y, ym, s);
    s = __fmaf_rn(hi.y, yp, s);
    s = __fmaf_rn(lo.z, zm, s);
    return __fmaf_rn(hi.z, zp, s);
}
// the relaxation of one cell by class, neighbours across the domain edge 0
template <bool D3>
__device__ __forceinline__ float relax_cell(const Relax &a, const RLevel &L, unsigned cl, int c, int i, int j, int k,
                                            float vc, float xm, float xp, float ym, float yp, float zm, float zp,
                                            float bval) {
    if (cl == 3u) {
        const float4 lo = __ldg(L.coef + c), hi = __ldg(L.gco + c);
        return __fmaf_rn(bval - general_sum(lo, hi, xm, xp, ym, yp, zm, zp), a.sor * hi.w, a.omsor * vc);
    }
    if (cl == 1u) return __fmaf_rn(bval, -a.sor, a.omsor * vc);
    return __fmaf_rn(bval - plain_sum<D3>(L.g, xm, xp, ym, yp, zm, zp), plain_scale<D3>(a, L, i, j, k), a.omsor * vc);
}
// the same from x = 0
template <bool D3>
__device__ __forceinline__ float relax_zero(const Relax &a, const RLevel &L, unsigned cl, int c, int i, int j, int k,
                                            float bval) {
    return relax_cell<D3>(a, L, cl, c, i, j, k, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, bval);
}
// a cell's couplings (zero across the domain edge)
template <bool D3>
__device__ __forceinline__ Coef cell_coef(const RLevel &L, unsigned cl, int c, bool xlo, bool xhi, bool ylo, bool yhi,
                                          bool zlo, bool zhi) {
    Coef q;
    if (cl == 3u) {
        const float4 lo = __ldg(L.coef + c), hi = __ldg(L.gco + c);
        q.kx = lo.x; q.ky = lo.y; q.kz = lo.z; q.e = lo.w;
        q.ux = hi.x; q.uy = hi.y; q.uz = hi.z;
    } else {
        const Geo &g = L.g;
        q.e = 0.f;
        q.kx = xlo ? 0.f : g.h2x; q.ux = xhi ? 0.f : g.h2x;
        q.ky = ylo ? 0.f : g.h2y; q.uy = yhi ? 0.f : g.h2y;
        q.kz = !D3 || zlo ? 0.f : g.h2z; q.uz = !D3 || zhi ? 0.f : g.h2z;
    }
    return q;
}
// A v by class; a neighbour across the domain edge is any finite value
template <bool D3>
__device__ __forceinline__ float apply_cell(const RLevel &L, unsigned cl, int c, int i, int j, int k, float vc, float xm,
                                            float xp, float ym, float yp, float zm, float zp) {
    if (cl == 0u) return apply_reg(L.g, vc, xm, xp, ym, yp, zm, zp);
    if (cl == 1u) return -vc;
    const Dims &d = L.g.d;
    return apply_q(cell_coef<D3>(L, cl, c, i == 0, i == d.nx - 1, j == 0, j == d.ny - 1, k == 0, k == d.nz - 1), vc, xm,
                   xp, ym, yp, zm, zp);
}

// ------------------------------------------------------ grid-wide phases --
// one colour pass (colour col = (i + j + k) & 1) in place, one thread per
// cell of the colour (nx is even: nx / 2 of them per row); `first`: x is 0
// on entry and the thread also writes 0 to the row neighbour of the other
// colour.  RZ: also sums b x of the cell and that neighbour (the level's
// last pass: the other colour is final).
template <bool D3, bool RZ>
__device__ __noinline__ double g_colour(int l, int col, bool first) {
    const RLevel L = SA.lv[l];
    const Relax a = relax_of();
    double rz = 0.0;
    const int nx = L.g.d.nx, ny = L.g.d.ny, nz = L.g.d.nz, hx = nx >> 1;
    const int sy = nx, sz = nx * ny, n = hx * ny * nz;
    float *x = L.x;
    const Deal w = deal();
    for (int t = w.t0; t < n; t += w.stride) {
        const int rr = tdiv(t, L.mhx), m = t - rr * hx;
        const int k = D3 ? tdiv(rr, L.mny) : 0, j = rr - k * ny;
        const int par = (j + k + col) & 1, i = 2 * m + par, c = i + sy * j + sz * k;
        const float bv = __ldcg(L.b + c);
        const unsigned cl = class_at(L, i, j, k);
        if (first) {
            x[c + (par ? -1 : 1)] = 0.f;
            x[c] = relax_zero<D3>(a, L, cl, c, i, j, k, bv);
            continue;
        }
        float xm = 0.f, xp = 0.f, ym = 0.f, yp = 0.f, zm = 0.f, zp = 0.f;
        const float vc = __ldcg(x + c);
        if (i > 0) xm = __ldcg(x + c - 1);
        if (i < nx - 1) xp = __ldcg(x + c + 1);
        if (j > 0) ym = __ldcg(x + c - sy);
        if (j < ny - 1) yp = __ldcg(x + c + sy);
        if (D3) {
            if (k > 0) zm = __ldcg(x + c - sz);
            if (k < nz - 1) zp = __ldcg(x + c + sz);
        }
        const float v = relax_cell<D3>(a, L, cl, c, i, j, k, vc, xm, xp, ym, yp, zm, zp, bv);
        x[c] = v;
        if (RZ) {
            rz += (double)bv * (double)v;
            rz += (double)__ldcg(L.b + c + (par ? -1 : 1)) * (double)(par ? xm : xp);
        }
    }
    return rz;
}

// r = b - A x (0 on Dirichlet cells); xzero: x is taken as 0 and cleared
template <bool D3>
__device__ __noinline__ void g_residual(int l, bool xzero) {
    const RLevel L = SA.lv[l];
    const int nx = L.g.d.nx, ny = L.g.d.ny, nz = L.g.d.nz, sy = nx, sz = nx * ny, n = nx * ny * nz;
    float *x = L.x;
    const Deal w = deal();
    for (int c = w.t0; c < n; c += w.stride) {
        const int rr = tdiv(c, L.mnx), i = c - rr * nx;
        const int k = D3 ? tdiv(rr, L.mny) : 0, j = rr - k * ny;
        const unsigned cl = class_at(L, i, j, k);
        const float bv = __ldcg(L.b + c);
        if (xzero) {
            L.r[c] = cl == 1u ? 0.f : bv;
            x[c] = 0.f;
            continue;
        }
        const float vc = __ldcg(x + c);
        const float xm = i > 0 ? __ldcg(x + c - 1) : vc, xp = i < nx - 1 ? __ldcg(x + c + 1) : vc;
        const float ym = j > 0 ? __ldcg(x + c - sy) : vc, yp = j < ny - 1 ? __ldcg(x + c + sy) : vc;
        const float zm = D3 && k > 0 ? __ldcg(x + c - sz) : vc, zp = D3 && k < nz - 1 ? __ldcg(x + c + sz) : vc;
        L.r[c] = cl == 1u ? 0.f : bv - apply_cell<D3>(L, cl, c, i, j, k, vc, xm, xp, ym, yp, zm, zp);
    }
}

// the 1/8, 3/8, 3/8, 1/8 taps per axis on the fine residual around coarse
// cell (I, J, K)
template <bool D3, class LD>
__device__ __forceinline__ float restrict_cell(const Dims &fd, const Dims &cd, int I, int J, int K, LD ldr) {
    const float w4[4] = {0.125f, 0.375f, 0.375f, 0.125f};
    int ix[4], jy[4], kz[4];
    rtap4(I, cd.nx, ix);
    rtap4(J, cd.ny, jy);
    if (D3) rtap4(K, cd.nz, kz);
    else kz[0] = K;
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < (D3 ? 4 : 1); ++q) {
        const float wz = D3 ? w4[q] : 1.0f;
        float part = 0.f;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const int row = fd.nx * (jy[p] + fd.ny * kz[q]);
            const float rx = 0.125f * ldr(row + ix[0]) + 0.375f * ldr(row + ix[1]) + 0.375f * ldr(row + ix[2]) +
                             0.125f * ldr(row + ix[3]);
            part += rx * w4[p];
        }
        s += part * wz;
    }
    return s;
}
// coarse b = R r, 0 on coarse Dirichlet cells; relax0: also the coarse
// level's first colour-0 pass (from x = 0 a cell needs only its own b;
// colour-1 cells get 0)
template <bool D3>
__device__ __noinline__ void g_restrict(int l, bool relax0) {
    const RLevel F = SA.lv[l], C = SA.lv[l + 1];
    const Relax a = relax_of();
    const Dims fd = F.g.d, cd = C.g.d;
    const int n = cd.nx * cd.ny * cd.nz;
    const Deal w = deal();
    for (int c = w.t0; c < n; c += w.stride) {
        const int rr = tdiv(c, C.mnx), I = c - rr * cd.nx;
        const int K = D3 ? tdiv(rr, C.mny) : 0, J = rr - K * cd.ny;
        float s = 0.f;
        if (!(C.mask && __ldg(C.mask + c)))
            s = restrict_cell<D3>(fd, cd, I, J, K, [&](int f) { return __ldcg(F.r + f); });
        C.b[c] = s;
        if (relax0) C.x[c] = ((I + J + K) & 1) ? 0.f : relax_zero<D3>(a, C, class_at(C, I, J, K), c, I, J, K, s);
    }
}

// P x_c at fine cell (i, j, k)
template <bool D3, class LD>
__device__ __forceinline__ float prolong_cell(const Dims &cd, int i, int j, int k, LD ldx) {
    int ii[2], jj[2], kk[2];
    float wi[2], wj[2], wk[2];
    ptaps2(i, cd.nx, ii, wi);
    ptaps2(j, cd.ny, jj, wj);
    if (D3) ptaps2(k, cd.nz, kk, wk);
    else { kk[0] = 0; wk[0] = 1.f; }
    float acc = 0.f;
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int q = 0; q < (D3 ? 2 : 1); ++q) {
            const float w = wj[b] * wk[q];
            acc += (wi[0] * ldx(ii[0], jj[b], kk[q]) + wi[1] * ldx(ii[1], jj[b], kk[q])) * w;
        }
    return acc;
}
// fine x += P coarse x, skipped on fine Dirichlet cells
template <bool D3>
__device__ __noinline__ void g_prolong(int l) {
    const RLevel C = SA.lv[l + 1], F = SA.lv[l];
    const Dims fd = F.g.d, cd = C.g.d;
    const int n = fd.nx * fd.ny * fd.nz;
    const Deal w = deal();
    for (int c = w.t0; c < n; c += w.stride) {
        if (F.mask && __ldg(F.mask + c)) continue;
        const int rr = tdiv(c, F.mnx), i = c - rr * fd.nx;
        const int k = D3 ? tdiv(rr, F.mny) : 0, j = rr - k * fd.ny;
        const float v = __ldcg(F.x + c);
        F.x[c] = v + prolong_cell<D3>(cd, i, j, k, [&](int I, int J, int K) {
                     return __ldcg(C.x + I + cd.nx * (J + cd.ny * K));
                 });
    }
}

// coarsest x = G b, one warp per row (FP64)
__device__ __noinline__ void g_direct() {
    const RLevel C = SA.lv[SA.nl - 1];
    const double *G = SA.G;
    const int nG = SA.nG;
    const int lane = threadIdx.x & 31, nw = gridDim.x * (NT / 32);
    for (int row = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; row < nG; row += nw) {
        const double *gr = G + (long long)row * nG;
        double s = 0.0;
        for (int j = lane; j < nG; j += 32) s += __ldg(gr + j) * (double)__ldcg(C.b + j);
        s = warp_sum(s);
        if (lane == 0) C.x[row] = (float)s;
    }
}

// one colour pass on a coarsest level too large for one block, from the
// stored coefficients (k_coarse_sweeps' arithmetic: x += sor (b - A x) / diag)
__device__ __noinline__ void g_coarse_colour(int col) {
    const RLevel C = SA.lv[SA.nl - 1];
    const float sor = SA.sor;
    const Dims d = C.g.d;
    const int sy = d.nx, sz = d.nx * d.ny, n = (int)d.n();
    float *x = C.x;
    const Deal w = deal();
    for (int c = w.t0; c < n; c += w.stride) {
        const int rr = tdiv(c, C.mnx), i = c - rr * d.nx, k = tdiv(rr, C.mny), j = rr - k * d.ny;
        if (((i + j + k) & 1) != col) continue;
        const float xc = __ldcg(x + c);
        const float4 kc = __ldg(C.coef + c);
        float s = -kc.w * xc;
        float D = -(kc.w + kc.x + kc.y + kc.z);
        if (i > 0) s += kc.x * (__ldcg(x + c - 1) - xc);
        if (i < d.nx - 1) { const float k1 = __ldg(&C.coef[c + 1].x); s += k1 * (__ldcg(x + c + 1) - xc); D -= k1; }
        if (j > 0) s += kc.y * (__ldcg(x + c - sy) - xc);
        if (j < d.ny - 1) { const float k1 = __ldg(&C.coef[c + sy].y); s += k1 * (__ldcg(x + c + sy) - xc); D -= k1; }
        if (k > 0) s += kc.z * (__ldcg(x + c - sz) - xc);
        if (k < d.nz - 1) { const float k1 = __ldg(&C.coef[c + sz].z); s += k1 * (__ldcg(x + c + sz) - xc); D -= k1; }
        x[c] = xc + ((__ldcg(C.b + c) - s) / D) * sor;
    }
}

// ------------------------------------- held levels (block 0, shared memory) --
extern __shared__ __align__(16) float rsm[];

// A held level's arrays: cell (i, j, k) at x[i + py j + pz k], zeros around.
struct Held {
    float *x, *b;
    int py, pz;
};
template <bool D3>
__device__ __forceinline__ Held held_arrays(const RLevel &L) {
    Held h;
    h.py = L.g.d.nx + 2;
    h.pz = h.py * (L.g.d.ny + 2);
    const int first = 1 + h.py + (D3 ? h.pz : 0);
    h.x = rsm + L.xo + first;
    h.b = rsm + L.bo + first;
    return h;
}
__host__ __device__ inline int held_floats(const Dims &d, bool d3) {
    return (d.nx + 2) * (d.ny + 2) * (d3 ? d.nz + 2 : 1);
}
// Two neighbouring cells of a row, one of each colour: pair t of a level holds
// its cells 2 t and 2 t + 1 (nx is even).  What the passes need of a pair sits
// in one word of a table in shared memory, built once per launch: its place p
// in the held arrays (14 bits), (j + k) & 1, the two classes (2 bits each) and
// two indices (5 bits each) into the level's relaxation scales: sor / diagonal
// of a plain cell by its faces across the domain edge, -sor of a Dirichlet
// cell.  (Kept per thread in registers instead, the pairs of a level of
// HELD_CELLS cells spilled in every pass.)
constexpr int SCALES = 28, SCALE_DIRICHLET = 27;
struct HeldTable {
    const unsigned *word;
    const float *scale;
};
__device__ __forceinline__ HeldTable held_table(const RLevel &L) {
    return HeldTable{reinterpret_cast<const unsigned *>(rsm + L.to) + SCALES, rsm + L.to};
}
template <bool D3>
__device__ __noinline__ void held_build(int l) {
    const RLevel L = SA.lv[l];
    const float sor = SA.sor;
    const Dims d = L.g.d;
    const Held h = held_arrays<D3>(L);
    float *scale = rsm + L.to;
    unsigned *word = reinterpret_cast<unsigned *>(rsm + L.to) + SCALES;
    for (int q = threadIdx.x; q < SCALES; q += NT) {
        const float corr = L.g.h2x * (float)(q % 3) + L.g.h2y * (float)(q / 3 % 3) + L.g.h2z * (float)(q / 9);
        scale[q] = q == SCALE_DIRICHLET ? -sor : (corr == 0.f ? L.rdreg_sor : sor / (L.g.dreg + corr));
    }
    const int hx = d.nx >> 1, n = hx * d.ny * d.nz;
    for (int t = threadIdx.x; t < n; t += NT) {
        const int rr = tdiv(t, L.mhx), i = 2 * (t - rr * hx);
        const int k = D3 ? tdiv(rr, L.mny) : 0, j = rr - k * d.ny;
        const unsigned cb = (__ldg(L.cls + L.cpitch * (j + d.ny * k) + (i >> 2)) >> (2 * (i & 3))) & 15u;
        const unsigned yz = 3u * (unsigned)((j == 0) + (j == d.ny - 1)) +
                            (D3 ? 9u * (unsigned)((k == 0) + (k == d.nz - 1)) : 0u);
        const unsigned s0 = (cb & 3u) == 1u ? SCALE_DIRICHLET : yz + (i == 0);
        const unsigned s1 = (cb >> 2) == 1u ? SCALE_DIRICHLET : yz + (i + 2 == d.nx);
        word[t] = (unsigned)(i + h.py * j + h.pz * k) | ((unsigned)((j + k) & 1) << 14) | (cb << 15) | (s0 << 19) |
                  (s1 << 24);
    }
    __syncthreads();
}
// one colour pass; FIRST: from x = 0, the other colour set to 0
template <bool D3, bool FIRST>
__device__ __forceinline__ void held_colour(const Relax &a, const RLevel &L, const Held &h, const HeldTable &T, int n,
                                            int col) {
#pragma unroll 2
    for (int t = threadIdx.x; t < n; t += NT) {
        const unsigned w = T.word[t];
        const int o = (int)((w >> 14 ^ (unsigned)col) & 1u), p = (int)(w & 0x3fffu) + o;
        const unsigned cl = (w >> (o ? 17 : 15)) & 3u;
        const float bv = h.b[p], rd = T.scale[(w >> (o ? 24 : 19)) & 31u];
        float vc = 0.f, xm = 0.f, xp = 0.f, ym = 0.f, yp = 0.f, zm = 0.f, zp = 0.f;
        if (!FIRST) {
            vc = h.x[p];
            xm = h.x[p - 1];
            xp = h.x[p + 1];
            ym = h.x[p - h.py];
            yp = h.x[p + h.py];
            if (D3) {
                zm = h.x[p - h.pz];
                zp = h.x[p + h.pz];
            }
        }
        float v;
        if (cl == 3u) {
            const float4 lo = __ldg(L.coef + 2 * t + o), hi = __ldg(L.gco + 2 * t + o);
            v = __fmaf_rn(bv - general_sum(lo, hi, xm, xp, ym, yp, zm, zp), a.sor * hi.w, a.omsor * vc);
        } else {
            const float sum = cl == 1u ? 0.f : plain_sum<D3>(L.g, xm, xp, ym, yp, zm, zp);
            v = __fmaf_rn(bv - sum, rd, a.omsor * vc);
        }
        h.x[p] = v;
        if (FIRST) h.x[p + (o ? -1 : 1)] = 0.f;
    }
}
// r = b - A x (0 on Dirichlet cells), flat as in global memory; xzero: x is
// taken as 0 and cleared
template <bool D3>
__device__ __forceinline__ void held_residual(float *r, const RLevel &L, const Held &h, const HeldTable &T, int n,
                                              bool xzero) {
    const Dims d = L.g.d;
#pragma unroll 1
    for (int t = threadIdx.x; t < n; t += NT) {
        const unsigned w = T.word[t];
#pragma unroll
        for (int o = 0; o < 2; ++o) {
            const int p = (int)(w & 0x3fffu) + o, c = 2 * t + o;
            const unsigned cl = (w >> (o ? 17 : 15)) & 3u;
            float res = h.b[p];
            if (xzero) {
                h.x[p] = 0.f;
            } else if (cl != 1u) {
                const float vc = h.x[p], xm = h.x[p - 1], xp = h.x[p + 1], ym = h.x[p - h.py], yp = h.x[p + h.py];
                const float zm = D3 ? h.x[p - h.pz] : vc, zp = D3 ? h.x[p + h.pz] : vc;
                float ax;
                if (cl == 0u) {
                    ax = apply_reg(L.g, vc, xm, xp, ym, yp, zm, zp);
                } else {
                    const int rr = tdiv(c, L.mnx), i = c - rr * d.nx;
                    const int k = D3 ? tdiv(rr, L.mny) : 0, j = rr - k * d.ny;
                    ax = apply_q(cell_coef<D3>(L, cl, c, i == 0, i == d.nx - 1, j == 0, j == d.ny - 1, k == 0,
                                               k == d.nz - 1),
                                 vc, xm, xp, ym, yp, zm, zp);
                }
                res = res - ax;
            }
            r[c] = cl == 1u ? 0.f : res;
        }
    }
}
// x += P e, e from `cx` with the strides of its array
template <bool D3>
__device__ __forceinline__ void held_prolong(const RLevel &L, const Held &h, const HeldTable &T, int n, const Dims &cd,
                                             const float *cx, int cpy, int cpz) {
    const Dims d = L.g.d;
    const int hx = d.nx >> 1;
#pragma unroll 1
    for (int t = threadIdx.x; t < n; t += NT) {
        const int p = (int)(T.word[t] & 0x3fffu);
        const int rr = tdiv(t, L.mhx), i = 2 * (t - rr * hx);
        const int k = D3 ? tdiv(rr, L.mny) : 0, j = rr - k * d.ny;
#pragma unroll
        for (int o = 0; o < 2; ++o) {
            if (L.mask && __ldg(L.mask + 2 * t + o)) continue;
            h.x[p + o] += prolong_cell<D3>(cd, i + o, j, k, [&](int I, int J, int K) {
                return cx[I + cpy * J + (D3 ? cpz * K : 0)];
            });
        }
    }
}

// All sweeps of a coarsest level of up to COARSE_CELLS cells, x in shared
// memory from the first pass to the last (through L2 a colour pass is two
// dependent round trips).  A cell's operator as the passes use it: the six
// couplings (0 across the domain edge, where the neighbour index is the cell
// itself), E, the diagonal and b.
// The quotient (b - s) / D by the correctly rounded reciprocal r of D: with
// q = t r and the remainder t - q D formed in one rounding, fma(rem, r, q) is
// the correctly rounded quotient (Markstein 1990), as the division gives it,
// at a third of its latency.
template <bool D3>
struct CoarseCell {
    float k[D3 ? 6 : 4], e, D, r, b;
    int c, n[D3 ? 6 : 4];
};
template <bool D3>
__device__ __forceinline__ CoarseCell<D3> coarse_cell(const RLevel &C, const float *b, int i, int j, int k) {
    const Dims d = C.g.d;
    const int sy = d.nx, sz = d.nx * d.ny;
    CoarseCell<D3> q;
    q.c = i + sy * j + sz * k;
    const float4 kc = __ldg(C.coef + q.c);
    q.e = kc.w;
    q.D = -(kc.w + kc.x + kc.y + kc.z);
    const bool in[6] = {i > 0, i < d.nx - 1, j > 0, j < d.ny - 1, k > 0, k < d.nz - 1};
    const int st[3] = {1, sy, sz};
#pragma unroll
    for (int f = 0; f < (D3 ? 6 : 4); ++f) {
        const int a = f >> 1;
        q.n[f] = in[f] ? q.c + (f & 1 ? st[a] : -st[a]) : q.c;
        float kf = 0.f;
        if (in[f]) {
            const int cc = f & 1 ? q.n[f] : q.c;
            kf = a == 0 ? __ldg(&C.coef[cc].x) : (a == 1 ? __ldg(&C.coef[cc].y) : __ldg(&C.coef[cc].z));
            if (f & 1) q.D -= kf;
        }
        q.k[f] = kf;
    }
    q.r = 1.f / q.D;
    q.b = b[q.c];
    return q;
}
template <bool D3>
__device__ __forceinline__ void coarse_relax(const CoarseCell<D3> &q, float *x, float sor) {
    const float xc = x[q.c];
    float s = -q.e * xc;
#pragma unroll
    for (int f = 0; f < (D3 ? 6 : 4); ++f) s += q.k[f] * (x[q.n[f]] - xc);
    const float t = q.b - s, u = __fmul_rn(t, q.r);
    x[q.c] = xc + __fmaf_rn(__fmaf_rn(-u, q.D, t), q.r, u) * sor;
}
__device__ __forceinline__ void bar_sync_n(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
template <bool D3>
__device__ __noinline__ void coarse_sweeps() {
    const RLevel C = SA.lv[SA.nl - 1];
    const float sor = SA.sor;
    const int sweeps = SA.coarse_sweeps;
    float *x = rsm + SA.cxo;
    const float *b = rsm + SA.cbo;
    const Dims d = C.g.d;
    const int n = (int)d.n(), hx = (d.nx + 1) >> 1, pairs = hx * d.ny * d.nz, tid = threadIdx.x;
    for (int c = tid; c < n; c += NT) x[c] = 0.f;
    __syncthreads();
    // cell of colour col of a pair (two neighbours of a row, one of each colour)
    auto cell_of = [&](int t, int col, int &i, int &j, int &k) {
        const int r = t / hx;
        k = r / d.ny;
        j = r - k * d.ny;
        i = 2 * (t - r * hx) + ((j + k + col) & 1);
        return i < d.nx;
    };
    if (pairs <= NT) {
        // one pair a thread, its operator in registers; only the warps with
        // pairs take part in the passes' barriers
        const int nthr = (pairs + 31) & ~31;
        if (tid < nthr) {
            CoarseCell<D3> q[2];
            bool has[2] = {false, false};
#pragma unroll
            for (int col = 0; col < 2; ++col) {
                int i, j, k;
                if (tid < pairs && cell_of(tid, col, i, j, k)) {
                    q[col] = coarse_cell<D3>(C, b, i, j, k);
                    has[col] = true;
                }
            }
            for (int it = 0; it < sweeps; ++it) {
#pragma unroll
                for (int col = 0; col < 2; ++col) {
                    if (has[col]) coarse_relax<D3>(q[col], x, sor);
                    bar_sync_n(1, nthr);
                }
            }
        }
    } else {
        for (int it = 0; it < 2 * sweeps; ++it) {
            for (int t = tid; t < pairs; t += NT) {
                int i, j, k;
                if (cell_of(t, it & 1, i, j, k)) coarse_relax<D3>(coarse_cell<D3>(C, b, i, j, k), x, sor);
            }
            __syncthreads();
        }
    }
    __syncthreads();
}

// block 0: from a held level's b (in shared memory) down to the coarsest b
template <bool D3>
__device__ __noinline__ void held_down(int l) {
    const RLevel L = SA.lv[l], C = SA.lv[l + 1];
    const Relax a = relax_of();
    const int down = SA.down, sweeps = SA.coarse_sweeps;
    const bool last = l + 1 == SA.nl - 1;
    float *r = rsm + SA.ro, *cb = rsm + SA.cbo;
    const Held h = held_arrays<D3>(L);
    const HeldTable T = held_table(L);
    const int np = (int)L.g.d.n() >> 1;
    for (int pass = 0; pass < 2 * down; ++pass) {
        if (pass == 0) held_colour<D3, true>(a, L, h, T, np, 0);
        else held_colour<D3, false>(a, L, h, T, np, pass & 1);
        __syncthreads();
    }
    held_residual<D3>(r, L, h, T, np, down == 0);
    __syncthreads();
    const Held hc = held_arrays<D3>(C);
    const Dims cd = C.g.d;
    const int n = cd.nx * cd.ny * cd.nz;
    for (int c = threadIdx.x; c < n; c += NT) {
        const int rr = tdiv(c, C.mnx), I = c - rr * cd.nx;
        const int K = D3 ? tdiv(rr, C.mny) : 0, J = rr - K * cd.ny;
        float s = 0.f;
        if (!(C.mask && __ldg(C.mask + c))) s = restrict_cell<D3>(L.g.d, cd, I, J, K, [&](int f) { return r[f]; });
        if (!last) hc.b[I + hc.py * J + hc.pz * K] = s;
        else if (sweeps > 0) cb[c] = s;
        else C.b[c] = s;
    }
    __syncthreads();
}
// block 0: correction from the level below (held, or the coarsest x in
// shared memory) and the post-smoothing
template <bool D3>
__device__ __noinline__ void held_up(int l) {
    const RLevel L = SA.lv[l], C = SA.lv[l + 1];
    const Relax a = relax_of();
    const int up = l > 0 ? SA.up : SA.final;
    const bool last = l + 1 == SA.nl - 1;
    const float *cx = rsm + SA.cxo;
    const Held h = held_arrays<D3>(L), hc = held_arrays<D3>(C);
    const HeldTable T = held_table(L);
    const int np = (int)L.g.d.n() >> 1;
    held_prolong<D3>(L, h, T, np, C.g.d, last ? cx : hc.x, last ? C.g.d.nx : hc.py,
                     last ? C.g.d.nx * C.g.d.ny : hc.pz);
    __syncthreads();
    for (int pass = 0; pass < 2 * up; ++pass) {
        held_colour<D3, false>(a, L, h, T, np, ~pass & 1);
        __syncthreads();
    }
}
// block 0: a held level's b from global memory, or its x there
template <bool D3>
__device__ __noinline__ void held_copy(int l, bool in) {
    const RLevel L = SA.lv[l];
    const Dims d = L.g.d;
    const Held h = held_arrays<D3>(L);
    const int n = (int)d.n();
    for (int c = threadIdx.x; c < n; c += NT) {
        const int rr = tdiv(c, L.mnx), i = c - rr * d.nx;
        const int k = D3 ? tdiv(rr, L.mny) : 0, j = rr - k * d.ny, e = i + h.py * j + h.pz * k;
        if (in) h.b[e] = __ldcg(L.b + c);
        else L.x[c] = h.x[e];
    }
}

// the held levels' tables and the zeros around them, once per launch
template <bool D3>
__device__ void held_init() {
    if (blockIdx.x != 0 || SA.held >= SA.nl - 1) return;
    const int lo = SA.lv[SA.held].xo, hi = SA.lv[SA.nl - 2].bo + held_floats(SA.lv[SA.nl - 2].g.d, D3);
    for (int e = lo + (int)threadIdx.x; e < hi; e += NT) rsm[e] = 0.f;
    for (int l = SA.held; l < SA.nl - 1; ++l) held_build<D3>(l);
}

// ---------------------------------------------------------------- V-cycle --
// z = M r on lv[0] (x = z, b = r).  first_done: the caller made the first
// colour-0 pass.  RZ: *rz gets this thread's share of r.z, and the caller
// takes the last barrier.  Every block takes the same sequence of barriers
// (it depends only on the levels).  False when a barrier gave up.
template <bool D3, bool RZ>
__device__ bool vcycle(unsigned &passed, bool first_done, double *rz) {
    const int nl = SA.nl, held = SA.held, down = SA.down, sweeps = SA.coarse_sweeps, nc = (int)SA.lv[nl - 1].g.d.n();
    unsigned *bar = SA.bar;
    const bool solo = blockIdx.x == 0;
    for (int l = 0; l < held; ++l) {
        for (int it = 0; it < down; ++it) {
            if (!(first_done && it == 0)) {
                g_colour<D3, false>(l, 0, it == 0);
                if (!grid_sync(bar, passed)) return false;
            }
            g_colour<D3, false>(l, 1, false);
            if (!grid_sync(bar, passed)) return false;
        }
        g_residual<D3>(l, down == 0);
        if (!grid_sync(bar, passed)) return false;
        first_done = l + 1 < held && down > 0;
        g_restrict<D3>(l, first_done);
        if (!grid_sync(bar, passed)) return false;
    }
    if (solo && held < nl - 1) {
        held_copy<D3>(held, true);
        __syncthreads();
        for (int l = held; l < nl - 1; ++l) held_down<D3>(l);
    }
    if (sweeps > 0 && nc <= COARSE_CELLS) {
        if (solo) {
            const bool io = held == nl - 1;
            float *cb = rsm + SA.cbo, *cx = rsm + SA.cxo, *gb = SA.lv[nl - 1].b, *gx = SA.lv[nl - 1].x;
            if (io) {
                for (int c = threadIdx.x; c < nc; c += NT) cb[c] = __ldcg(gb + c);
                __syncthreads();
            }
            coarse_sweeps<D3>();
            if (io)
                for (int c = threadIdx.x; c < nc; c += NT) gx[c] = cx[c];
        }
    } else if (sweeps > 0) {
        const Deal w = deal();
        float *gx = SA.lv[nl - 1].x;
        for (int c = w.t0; c < nc; c += w.stride) gx[c] = 0.f;
        if (!grid_sync(bar, passed)) return false;
        for (int it = 0; it < 2 * sweeps; ++it) {
            g_coarse_colour(it & 1);
            if (it + 1 < 2 * sweeps && !grid_sync(bar, passed)) return false;
        }
    } else {
        if (held < nl - 1 && !grid_sync(bar, passed)) return false;
        g_direct();
        if (held < nl - 1) {
            if (!grid_sync(bar, passed)) return false;
            if (solo) {
                float *cx = rsm + SA.cxo;
                const float *gx = SA.lv[nl - 1].x;
                for (int c = threadIdx.x; c < nc; c += NT) cx[c] = __ldcg(gx + c);
                __syncthreads();
            }
        }
    }
    if (solo && held < nl - 1) {
        for (int l = nl - 2; l >= held; --l) held_up<D3>(l);
        held_copy<D3>(held, false);
        if (RZ && held == 0) {
            // x of every cell of lv[0] was final at the last block barrier
            const RLevel L = SA.lv[0];
            const Held h = held_arrays<D3>(L);
            for (int c = threadIdx.x; c < (int)L.g.d.n(); c += NT) {
                const int rr = tdiv(c, L.mnx), i = c - rr * L.g.d.nx;
                const int k = D3 ? tdiv(rr, L.mny) : 0, j = rr - k * L.g.d.ny, e = i + h.py * j + h.pz * k;
                *rz += (double)h.b[e] * (double)h.x[e];
            }
        }
    }
    for (int l = held - 1; l >= 0; --l) {
        if (!grid_sync(bar, passed)) return false;
        g_prolong<D3>(l);
        const int up = l > 0 ? SA.up : SA.final;
        for (int it = 0; it < up; ++it) {
            if (!grid_sync(bar, passed)) return false;
            g_colour<D3, false>(l, 1, false);
            if (!grid_sync(bar, passed)) return false;
            if (RZ && l == 0 && it == up - 1) *rz += g_colour<D3, true>(l, 0, false);
            else g_colour<D3, false>(l, 0, false);
        }
    }
    return true;
}

__device__ __forceinline__ void load_args(const VArgs &a) {
    static_assert(sizeof(VArgs) % 4 == 0, "copied by words");
    for (int w = threadIdx.x; w < (int)(sizeof(VArgs) / 4); w += NT)
        reinterpret_cast<unsigned *>(&SA)[w] = reinterpret_cast<const unsigned *>(&a)[w];
    __syncthreads();
}

// the V-cycle from one level of a larger hierarchy down and back, its x in
// lv[0].x
template <bool D3>
__global__ void __launch_bounds__(NT, 1) k_vcycle_tail(const __grid_constant__ VArgs a, PcgState *st) {
    if (st && (st->stop || st->err)) return;
    unsigned passed = 0;
    load_args(a);
    held_init<D3>();
    if (vcycle<D3, false>(passed, false, nullptr)) grid_done(SA.bar);
    else if (threadIdx.x == 0 && st) atomicOr(&st->err, 2);
}

// -------------------------------------------------------------- PCG solve --
// One solve of the reference's GPU-resident PCG (fluxflow src/linalg/linalg.js:
// 1147-1311, 1627-1911) in one launch, for a level 0 of at most
// PCG_RESIDENT_CELLS cells: there a launch per pass costs 4 to 12 us for work
// of about one, and the passes' own latency is a barrier and an L2 round trip.
// Every block keeps the solver's scalars in shared memory and forms each dot
// product from the blocks' partial sums in the same order, so all blocks
// take the same decisions; block 0 writes the state back at the end.
constexpr double MAX_BETA_MAGNITUDE = 10.0;     // linalg.js:226
constexpr double MAX_ALPHA_MAGNITUDE = 1e6;     // linalg.js:244
constexpr double MAX_PAP_GROWTH_FACTOR = 1e8;   // linalg.js:284
constexpr double PAP_BASELINE_FLOOR = 1e-12;    // linalg.js:1052
constexpr double MAX_RESIDUAL_GROWTH = 100.0;   // linalg.js:1095

struct PcgArgs {
    const float *b;                // right-hand side
    float *p[2], *xh[2], *xl[2];   // search direction and iterate, ping-pong
    double *partials;              // 8 sums of gridDim.x partials
    PcgState *st;
};

// the block's sum of a value a thread into slot `slot` of the partials.  FP64
// adds run at two lanes a clock and SM here, so 16 warps of shuffles would take
// 250 cycles a step: warp 0 adds up the warps that had cells (n items dealt
// out) from shared memory instead, lane by lane.
__device__ __noinline__ void put_partial(double v, double *partials, int slot, int n) {
    __shared__ double sred[NT];
    sred[threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        double s = 0.0;
        for (int w = 0; w < NT / 32 && (w * (int)gridDim.x + (int)blockIdx.x) * 32 < n; ++w) s += sred[w * 32 + threadIdx.x];
        s = warp_sum(s);
        if (threadIdx.x == 0) partials[slot * gridDim.x + blockIdx.x] = s;
    }
}
// after the barrier: the sum of slot `slot` (warp 0)
__device__ __forceinline__ double get_sum(const double *partials, int slot) {
    double s = 0.0;
    for (unsigned b = threadIdx.x & 31; b < gridDim.x; b += 32) s += __ldcg(partials + slot * gridDim.x + b);
    return warp_sum(s);
}

// p = z + beta p (FIRST: z itself), A p; returns this thread's share of p.Ap.
// A neighbour across the domain edge is the cell itself: its difference is an
// exact zero, and no load waits on a branch.
template <bool D3, bool FIRST>
__device__ __noinline__ double pcg_p(const float *pold, float *pnew, float beta) {
    const RLevel L = SA.lv[0];
    const int nx = L.g.d.nx, ny = L.g.d.ny, nz = L.g.d.nz, sy = nx, sz = nx * ny, n = nx * ny * nz;
    const float *z = L.x;
    auto P = [&](int c) {
        const float zc = __ldcg(z + c);
        return FIRST ? zc : __fmaf_rn(beta, __ldcg(pold + c), zc);
    };
    double acc = 0.0;
    const Deal w = deal();
#pragma unroll 2
    for (int c = w.t0; c < n; c += w.stride) {
        const int rr = tdiv(c, L.mnx), i = c - rr * nx;
        const int k = D3 ? tdiv(rr, L.mny) : 0, j = rr - k * ny;
        const unsigned cl = class_at(L, i, j, k);
        const float pc = P(c);
        const float xm = P(c - (i > 0)), xp = P(c + (i < nx - 1));
        const float ym = P(j > 0 ? c - sy : c), yp = P(j < ny - 1 ? c + sy : c);
        const float zm = D3 ? P(k > 0 ? c - sz : c) : pc, zp = D3 ? P(k < nz - 1 ? c + sz : c) : pc;
        const float ap = apply_cell<D3>(L, cl, c, i, j, k, pc, xm, xp, ym, yp, zm, zp);
        pnew[c] = pc;
        acc += (double)pc * (double)ap;
    }
    return acc;
}

// x + alpha p (SETUP: x as it is), r = b - A x, and z's first colour-0 pass
// from zero; v gets this thread's shares of r.r and (SETUP) b.b.  DS: x as a
// hi + lo pair, the residual formed with compensated products and sums.
template <bool D3, bool DS, bool SETUP>
__device__ __noinline__ double2 pcg_x(const float *b, const float *xh, const float *xl, const float *p, float *oh, float *ol,
                                      double alpha) {
    const RLevel L = SA.lv[0];
    const Relax a = relax_of();
    double2 v = make_double2(0.0, 0.0);
    const int nx = L.g.d.nx, ny = L.g.d.ny, nz = L.g.d.nz, sy = nx, sz = nx * ny, n = nx * ny * nz;
    const float ahi = (float)alpha, alo = (float)(alpha - (double)ahi);
    auto X = [&](int c, float &h, float &l) {
        h = __ldcg(xh + c);
        l = DS ? __ldcg(xl + c) : 0.f;
        if (SETUP) return;
        const float pv = __ldcg(p + c);
        if (DS) ds_axpy(h, l, ahi, alo, pv, h, l);
        else h = __fmaf_rn(ahi, pv, h);
    };
    const Deal w = deal();
    for (int c = w.t0; c < n; c += w.stride) {
        const int rr = tdiv(c, L.mnx), i = c - rr * nx;
        const int k = D3 ? tdiv(rr, L.mny) : 0, j = rr - k * ny;
        const unsigned cl = class_at(L, i, j, k);
        const float bc = __ldg(b + c);
        const bool in[6] = {i > 0, i < nx - 1, j > 0, j < ny - 1, D3 && k > 0, D3 && k < nz - 1};
        const int nb[6] = {c - 1, c + 1, c - sy, c + sy, c - sz, c + sz};
        float hc, lc, hn[6], ln[6];
        X(c, hc, lc);
#pragma unroll
        for (int f = 0; f < (D3 ? 6 : 4); ++f) X(in[f] ? nb[f] : c, hn[f], ln[f]);
        float rc;
        if (!DS) {
            rc = bc - apply_cell<D3>(L, cl, c, i, j, k, hc, hn[0], hn[1], hn[2], hn[3], D3 ? hn[4] : hc, D3 ? hn[5] : hc);
        } else {
            // b - A (hi + lo) as k_update_x_residual forms it
            Coef q;
            if (cl == 1u) {
                q.kx = q.ky = q.kz = q.ux = q.uy = q.uz = 0.f;
                q.e = 1.f;
            } else {
                q = cell_coef<D3>(L, cl, c, !in[0], !in[1], !in[2], !in[3], !in[4], !in[5]);
            }
            const float K[6] = {q.kx, q.ux, q.ky, q.uy, q.kz, q.uz};
            float S = 0.f, Se = 0.f;
#pragma unroll
            for (int f = 0; f < (D3 ? 6 : 4); ++f) {
                float dh, de, pr, pe, t, e;
                two_sum(hn[f], -hc, dh, de);
                de = __fadd_rn(de, __fsub_rn(ln[f], lc));
                two_prod(K[f], dh, pr, pe);
                pe = __fmaf_rn(K[f], de, pe);
                two_sum(S, pr, t, e);
                S = t;
                Se = __fadd_rn(Se, __fadd_rn(e, pe));
            }
            if (q.e != 0.f) {
                float pr, pe, t, e;
                two_prod(-q.e, hc, pr, pe);
                pe = __fmaf_rn(-q.e, lc, pe);
                two_sum(S, pr, t, e);
                S = t;
                Se = __fadd_rn(Se, __fadd_rn(e, pe));
            }
            float r0, e0;
            two_sum(bc, -S, r0, e0);
            rc = __fadd_rn(r0, __fsub_rn(e0, Se));
        }
        if (!SETUP) {
            oh[c] = hc;
            if (DS) ol[c] = lc;
        }
        L.b[c] = rc;
        L.x[c] = ((i + j + k) & 1) ? 0.f : relax_zero<D3>(a, L, cl, c, i, j, k, rc);
        v.x += (double)rc * (double)rc;
        if (SETUP) v.y += (double)bc * (double)bc;
    }
    return v;
}

template <bool D3, bool DS>
__global__ void __launch_bounds__(NT, 1) k_pcg_resident(const __grid_constant__ VArgs a, const __grid_constant__ PcgArgs A) {
    __shared__ PcgState S;
    unsigned passed = 0;
    if (threadIdx.x == 0) S = *A.st;   // as k_state_init left it
    load_args(a);
    held_init<D3>();
    bool ok = true;
    // items of the phases that sum: cells, and pairs of the last colour pass
    // (all of block 0's threads when it holds lv[0])
    const int n0 = (int)SA.lv[0].g.d.n(), nz = SA.held == 0 ? NT * (int)gridDim.x : n0 / 2;
    auto x_phase = [&](auto setup) {
        const int c = S.x_cur;
        return pcg_x<D3, DS, decltype(setup)::value>(A.b, c ? A.xh[1] : A.xh[0], c ? A.xl[1] : A.xl[0],
                                                     S.p_cur ? A.p[1] : A.p[0], c ? A.xh[0] : A.xh[1],
                                                     c ? A.xl[0] : A.xl[1], S.alpha);
    };
    // setup (linalg.js:1627-1637): r = b - A x, its norm and b's, z = M r, r.z
    {
        const double2 w = x_phase(std::true_type());
        put_partial(w.x, A.partials, 0, n0);
        __syncthreads();
        put_partial(w.y, A.partials, 1, n0);
        ok = grid_sync(SA.bar, passed);
        if (ok && threadIdx.x < 32) {
            const double rr = get_sum(A.partials, 0), bb = get_sum(A.partials, 1);
            if (threadIdx.x == 0) {
                S.rr = rr;
                S.bb = bb;
                S.thr = S.relative ? fmax(S.tol * sqrt(fabs(bb)), S.tol) : S.tol;
                // the start already meets the tolerance (linalg.js:1695-1699)
                if (sqrt(fabs(rr)) < S.thr) {
                    S.stop = FF_STOP_CONVERGED;
                    S.stop_iter = 0;
                }
            }
        }
        __syncthreads();
    }
    if (ok && S.stop == 0) {
        double v = 0.0;
        ok = vcycle<D3, true>(passed, true, &v);
        if (ok) {
            put_partial(v, A.partials, 2, nz);
            ok = grid_sync(SA.bar, passed);
        }
        if (ok && threadIdx.x < 32) {
            const double rz = get_sum(A.partials, 2);
            if (threadIdx.x == 0) {
                // seedScalarsKernel (linalg.js:1259-1267)
                S.rz = S.rz_old = rz;
                S.pap_baseline = fmax(fabs(S.rr), PAP_BASELINE_FLOOR);
                S.first = 1;
                S.best_rr = -1.0;
            }
        }
        __syncthreads();
    }
    while (ok && S.stop == 0 && S.iter < S.maxiter) {
        {
            const float *po = S.p_cur ? A.p[1] : A.p[0];
            float *pn = S.p_cur ? A.p[0] : A.p[1];
            put_partial(S.first ? pcg_p<D3, true>(po, pn, 0.f) : pcg_p<D3, false>(po, pn, (float)S.beta), A.partials, 3, n0);
            if (!(ok = grid_sync(SA.bar, passed))) break;
            if (threadIdx.x < 32) {
                const double pAp = get_sum(A.partials, 3);
                if (threadIdx.x == 0) {
                    // alphaKernel (linalg.js:1147-1199)
                    const double value = S.rz_old / pAp;
                    int code = 0;
                    if (nonfinite_d(pAp) || pAp == 0.0) code = FF_STOP_DEGENERATE_PAP;
                    else if (fabs(pAp) > S.pap_baseline * MAX_PAP_GROWTH_FACTOR) code = FF_STOP_PAP_GROWTH;
                    else if (nonfinite_or_above(value, MAX_ALPHA_MAGNITUDE)) code = FF_STOP_ALPHA_MAGNITUDE;
                    S.pAp = pAp;
                    S.alpha = code != 0 ? 0.0 : value;
                    S.stop = code;
                    S.p_cur ^= 1;
                    S.first = 0;
                    S.launched += 1;
                }
            }
            __syncthreads();
            if (S.stop) break;
        }
        {
            put_partial(x_phase(std::false_type()).x, A.partials, 4, n0);
            if (!(ok = grid_sync(SA.bar, passed))) break;
            if (threadIdx.x < 32) {
                const double rr = get_sum(A.partials, 4);
                if (threadIdx.x == 0) {
                    S.rr = rr;
                    S.x_cur ^= 1;
                    S.iter += 1;
                    // residual-growing (linalg.js:1864-1882), sampled where
                    // the reference's host reads the residual
                    if (!nonfinite_d(rr) && S.iter >= S.guard_next) {
                        S.guard_next += GROWTH_SAMPLE;
                        if (S.best_rr < 0.0 || fabs(rr) < S.best_rr) S.best_rr = fabs(rr);
                        else if (S.best_rr > 0.0 && fabs(rr) > S.best_rr * MAX_RESIDUAL_GROWTH) S.growth_stop = 1;
                    }
                    // convergenceKernel (linalg.js:1283-1311)
                    if (!nonfinite_or_above(sqrt(fabs(rr)), S.thr)) {
                        S.stop = FF_STOP_CONVERGED;
                        S.stop_iter = S.iter;
                    } else if (S.growth_stop) {
                        S.stop = FF_STOP_RESIDUAL_GROWING;
                    }
                }
            }
            __syncthreads();
            if (S.stop) break;
        }
        {
            double v = 0.0;
            if (!(ok = vcycle<D3, true>(passed, true, &v))) break;
            put_partial(v, A.partials, 5, nz);
            if (!(ok = grid_sync(SA.bar, passed))) break;
            if (threadIdx.x < 32) {
                const double rz = get_sum(A.partials, 5);
                if (threadIdx.x == 0) {
                    // betaKernel (linalg.js:1201-1240)
                    const double rz_old = S.rz_old, value = rz / rz_old;
                    const bool degenerate = nonfinite_d(rz_old) || rz_old == 0.0;
                    const bool restart = (rz_old * rz < 0.0) || nonfinite_or_above(value, MAX_BETA_MAGNITUDE);
                    S.rz = rz;
                    S.beta = restart ? 0.0 : value;
                    if (degenerate) S.stop = FF_STOP_DEGENERATE_OLD_RZ;
                    S.rz_old = rz;
                }
            }
            __syncthreads();
        }
    }
    if (ok) grid_done(SA.bar);
    else if (threadIdx.x == 0) atomicOr(&A.st->err, 2);
    if (ok && blockIdx.x == 0 && threadIdx.x == 0) {
        if (S.maxiter > 0) {
            // the count the next solve's first chunk is sized by (linalg.js:1839-1905)
            S.last_iters = S.stop == FF_STOP_CONVERGED ? S.stop_iter : S.iter;
            S.last_valid = 1;
        }
        *A.st = S;
    }
}

VArgs make_args(const Level *lv, const SweepMaps *sm, int nl, int dims, int down, int up, int fin, float sor,
                const double *G, int nG, int coarse_sweeps, unsigned *bar, int &smem) {
    VArgs a{};
    a.nl = nl;
    a.down = down;
    a.up = up;
    a.final = fin;
    a.sor = sor;
    a.omsor = 1.f - sor;
    a.G = G;
    a.nG = nG;
    a.coarse_sweeps = coarse_sweeps;
    a.bar = bar;
    auto magic = [](long long d) { return ((1ULL << 40) + (unsigned long long)d - 1) / (unsigned long long)d; };
    for (int l = 0; l < nl; ++l) {
        RLevel &t = a.lv[l];
        const Level &L = lv[l];
        t.g = make_geo(L);
        t.x = (float *)L.x;
        t.b = (float *)L.b;
        t.r = (float *)L.buf;
        t.coef = L.coef;
        t.mask = L.mask;
        t.rdreg_sor = sor / t.g.dreg;
        t.xo = t.bo = t.to = 0;
        t.mhx = magic(std::max(1, L.d.nx / 2));
        t.mnx = magic(L.d.nx);
        t.mny = magic(L.d.ny);
        if (l < nl - 1) {
            t.cls = sm[l].cls_ptr;
            t.cpitch = sm[l].cls_pitch;
            t.gco = sm[l].gco;
        }
    }
    // shared memory: the coarsest x and b, the held levels' residual and
    // arrays.  Levels are held from the last but one upward while they have
    // at most HELD_CELLS cells and the arrays fit.
    const int nc = lv[nl - 1].d.n() <= COARSE_CELLS ? (int)lv[nl - 1].d.n() : 0;
    a.cxo = 0;
    a.cbo = nc;
    int used = 2 * nc;
    a.held = nl - 1;
    a.ro = used;
    long long arrays = 0, most = 0;
    for (int l = nl - 2; l >= 0; --l) {
        const long long n = lv[l].d.n(), more = 2LL * held_floats(lv[l].d, dims == 3) + SCALES + n / 2;
        // (a place in the held arrays takes 14 bits of a pair's word)
        if (n > HELD_CELLS || held_floats(lv[l].d, dims == 3) > 0x3fff || 4 * (used + std::max(most, n) + arrays + more) > SMEM_BYTES) break;
        most = std::max(most, n);
        arrays += more;
        a.held = l;
    }
    used += (int)most;
    for (int l = a.held; l < nl - 1; ++l) {
        a.lv[l].xo = used;
        used += held_floats(lv[l].d, dims == 3);
        a.lv[l].bo = used;
        used += held_floats(lv[l].d, dims == 3);
    }
    for (int l = a.held; l < nl - 1; ++l) {
        a.lv[l].to = used;
        used += SCALES + (int)(lv[l].d.n() / 2);
    }
    smem = 4 * used;
    return a;
}

int launch_coop(const void *kernel, int blocks, int smem, cudaStream_t s, void **args) {
    FF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    FF_CUDA(cudaLaunchKernelExC(&cfg, kernel, args));
    return FF_OK;
}

int check_levels(const Level *lv, const SweepMaps *sm, int nl, const double *G, int nG, int coarse_sweeps, unsigned *bar) {
    FF_CHECK(nl >= 2 && nl <= MAXL, FF_E_ARG, "coarse V-cycle: %d levels (2..%d)", nl, MAXL);
    FF_CHECK(bar, FF_E_ARG, "coarse V-cycle: no barrier words");
    FF_CHECK(coarse_sweeps > 0 || (G && nG == lv[nl - 1].d.n()), FF_E_STATE, "coarse V-cycle: no coarsest inverse");
    for (int l = 0; l < nl - 1; ++l)
        FF_CHECK(sm[l].cls_ptr && sm[l].gco && lv[l].buf, FF_E_STATE, "coarse V-cycle: level %d lacks classes", l);
    return FF_OK;
}

}  // namespace

namespace ffk {

int vcycle_tail(const Level *lv, const SweepMaps *sm, int nl, int dims, int down, int up, float sor, const double *G,
                int nG, int coarse_sweeps, PcgState *st, unsigned *bar, int sm_count, cudaStream_t s) {
    FF_TRY(check_levels(lv, sm, nl, G, nG, coarse_sweeps, bar));
    int smem = 0;
    VArgs a = make_args(lv, sm, nl, dims, down, up, up, sor, G, nG, coarse_sweeps, bar, smem);
    void *args[] = {&a, &st};
    // a hierarchy that block 0 holds whole needs no other block
    const bool alone = a.held == 0 && coarse_sweeps > 0;
    return launch_coop(dims == 3 ? (const void *)k_vcycle_tail<true> : (const void *)k_vcycle_tail<false>,
                       alone ? 1 : sm_count, smem, s, args);
}

int pcg_resident(const Level *lv, const SweepMaps *sm, int nl, int dims, int down, int up, int fin, float sor,
                 const double *G, int nG, int coarse_sweeps, const float *b, float *p0, float *p1, float *xh0, float *xl0,
                 float *xh1, float *xl1, int ds, PcgState *st, double *partials, unsigned *bar, int sm_count,
                 cudaStream_t s) {
    FF_TRY(check_levels(lv, sm, nl, G, nG, coarse_sweeps, bar));
    int smem = 0;
    VArgs a = make_args(lv, sm, nl, dims, down, up, fin, sor, G, nG, coarse_sweeps, bar, smem);
    PcgArgs A{b, {p0, p1}, {xh0, xh1}, {xl0, xl1}, partials, st};
    void *args[] = {&a, &A};
    const void *k = dims == 3 ? (ds ? (const void *)k_pcg_resident<true, true> : (const void *)k_pcg_resident<true, false>)
                              : (ds ? (const void *)k_pcg_resident<false, true> : (const void *)k_pcg_resident<false, false>);
    return launch_coop(k, sm_count, smem, s, args);
}

}  // namespace ffk
