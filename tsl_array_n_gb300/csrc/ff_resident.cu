// Kernels for the parts of a projection that are too small for one launch per
// pass: the coarse levels of a V-cycle (k_vcycle_tail), and, where level 0 itself is
// small, the whole PCG solve, over the grid (k_pcg_resident) or, smaller still, on
// one thread-block cluster (k_pcg_cluster).
//
// In the cooperative ones phases over one level are separated by grid-wide
// barriers; values that
// another block wrote in this launch are read through L2 (ld.global.cg).  A
// phase on such a level is bound by latency, a barrier plus one or two L2
// round trips, and not by bandwidth or issue, so
//  - the work of a phase is dealt out a warp at a time over all blocks: a
//    level of a few thousand cells then keeps one or two warps busy on every
//    SM instead of all warps on a few;
//  - levels of up to HELD_CELLS cells, and the coarsest level's sweeps, run in
//    block 0 with their arrays in shared memory: a phase there costs a block
//    barrier and a shared-memory round trip.
// Per cell the arithmetic is that of the level kernels in ff_fused.cu, bit for bit
// (sums of two products are rounded as ff_stencil.cuh writes them out): the
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
constexpr int SMEM_BYTES = 220 * 1024;

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
    // a level spread over a cluster: rows (j + ny k) a block owns, q / rows as
    // above, its x and b in shared memory (floats; x has one row of zeros after
    // the rows), its tables of rows (8 words each) and of pairs, and room for the
    // couplings of `cap` cells (8 floats each)
    int rows, cx, cb, rt, pt, co, cap;
    unsigned long long mrows;
};
struct VArgs {
    RLevel lv[MAXL];
    int nl;                        // levels, the last one the coarsest
    int clu;                       // first level spread over the cluster (held: none)
    int held;                      // first held level (nl - 1: none)
    int csize;                     // blocks of a cluster
    int ccoarse;                   // the coarsest level is swept over the cluster
    int down, up, final;           // sweeps before and after the correction, and after it on lv[0]
    float sor, omsor;
    const double *G;               // coarsest inverse, nG x nG, row-major (direct mode)
    int nG;
    int coarse_sweeps;             // > 0: that many sweeps on the coarsest level instead of G b
    unsigned *bar;                 // grid barrier: arrivals, blocks done, abort
    int ro, cxo, cbo;              // shared memory: held levels' residual, the coarsest x and b
    int cr, crx, cop, cow, cok;    // cluster levels' residual and its x taps; the swept coarsest's diagonals, pair words and couplings
    int p, xh, xl, rhs;            // k_pcg_cluster's search direction, iterate (lv[0]'s x layout) and right-hand side
    int floats;                    // shared memory in use
    DotOrder dot[3];               // of p.Ap, r.r and r.z
    int pairs;                     // lv[0] is the solver's level 0 (see EDGE_KEEP)
    float *alt;                    // and its first colour's values at tile edges, as x
    int parts;                     // k_pcg_cluster: the items' sums (2 x items doubles)
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

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
// the same place in block `rank` of the cluster
__device__ __forceinline__ unsigned in_block(unsigned addr, unsigned rank) {
    unsigned d;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(addr), "r"(rank));
    return d;
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

__device__ __forceinline__ void bar_sync_n(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
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
__device__ __forceinline__ float4 plain_couplings(const Geo &g) { return make_float4(g.h2x, g.h2y, g.h2z, 0.f); }
// the relaxation of one cell by class, neighbours across the domain edge 0;
// coupled: a plain cell in the general form
template <bool D3>
__device__ __forceinline__ float relax_cell(const Relax &a, const RLevel &L, unsigned cl, int c, int i, int j, int k,
                                            float vc, float xm, float xp, float ym, float yp, float zm, float zp,
                                            float bval, bool coupled = false) {
    if (cl == 3u) {
        const float4 lo = __ldg(L.coef + c), hi = __ldg(L.gco + c);
        return __fmaf_rn(bval - general_sum(lo, hi, xm, xp, ym, yp, zm, zp), a.sor * hi.w, a.omsor * vc);
    }
    if (cl == 1u) return __fmaf_rn(bval, -a.sor, a.omsor * vc);
    const float s = coupled ? general_sum(plain_couplings(L.g), plain_couplings(L.g), xm, xp, ym, yp, zm, zp)
                            : plain_sum<D3>(L.g, xm, xp, ym, yp, zm, zp);
    return __fmaf_rn(bval - s, plain_scale<D3>(a, L, i, j, k), a.omsor * vc);
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
// Level 0's sweeps round as the launch-per-pass sweep does, which decides two
// things by its layout: a plain cell takes the general form where the other cell of
// its colour in its quad is a Dirichlet or general one, and the second colour of a
// sweep sees, across the edge of a 64-cell tile, the first colour's value in the
// general form (it is recomputed there).  The first colour's pass keeps that value
// (EDGE_KEEP), the second's uses it (EDGE_USE).
enum { EDGE_NONE, EDGE_KEEP, EDGE_USE };

// one colour pass (colour col = (i + j + k) & 1) in place, one thread per
// cell of the colour (nx is even: nx / 2 of them per row); `first`: x is 0
// on entry and the thread also writes 0 to the row neighbour of the other
// colour.  RZ: also leaves b x of the cell and that neighbour in L.r (the level's
// last pass: the other colour is final).
template <bool D3, bool RZ>
__device__ __noinline__ void g_colour(int l, int col, bool first, int edge = EDGE_NONE) {
    const RLevel L = SA.lv[l];
    const Relax a = relax_of();
    const int nx = L.g.d.nx, ny = L.g.d.ny, nz = L.g.d.nz, hx = nx >> 1;
    const int sy = nx, sz = nx * ny, n = hx * ny * nz;
    float *x = L.x, *alt = SA.alt;
    const Deal w = deal();
    for (int t = w.t0; t < n; t += w.stride) {
        const int rr = tdiv(t, L.mhx), m = t - rr * hx;
        const int k = D3 ? tdiv(rr, L.mny) : 0, j = rr - k * ny;
        const int par = (j + k + col) & 1, i = 2 * m + par, c = i + sy * j + sz * k;
        const float bv = __ldcg(L.b + c);
        const unsigned cb = __ldg(L.cls + L.cpitch * (j + ny * k) + (i >> 2)), cl = cb >> (2 * (i & 3)) & 3u;
        if (first) {
            x[c + (par ? -1 : 1)] = 0.f;
            x[c] = relax_zero<D3>(a, L, cl, c, i, j, k, bv);
            continue;
        }
        float xm = 0.f, xp = 0.f, ym = 0.f, yp = 0.f, zm = 0.f, zp = 0.f;
        const float vc = __ldcg(x + c);
        const bool tile_lo = (i & (DOT_TX - 1)) == 0, tile_hi = (i & (DOT_TX - 1)) == DOT_TX - 1;
        if (i > 0) xm = __ldcg((edge == EDGE_USE && tile_lo ? alt : x) + c - 1);
        if (i < nx - 1) xp = __ldcg((edge == EDGE_USE && tile_hi ? alt : x) + c + 1);
        if (j > 0) ym = __ldcg(x + c - sy);
        if (j < ny - 1) yp = __ldcg(x + c + sy);
        if (D3) {
            if (k > 0) zm = __ldcg(x + c - sz);
            if (k < nz - 1) zp = __ldcg(x + c + sz);
        }
        const bool coupled = l == 0 && SA.pairs && (cb >> (2 * ((i & 3) ^ 2)) & 1u);
        const float v = relax_cell<D3>(a, L, cl, c, i, j, k, vc, xm, xp, ym, yp, zm, zp, bv, coupled);
        x[c] = v;
        if (edge == EDGE_KEEP && (tile_lo || tile_hi))
            alt[c] = relax_cell<D3>(a, L, cl, c, i, j, k, vc, xm, xp, ym, yp, zm, zp, bv, true);
        if (RZ) {
            const float o = par ? __ldcg(x + c - 1) : __ldcg(x + c + 1);   // (not the tile edge's other value)
            L.r[c] = bv * v;
            L.r[c + (par ? -1 : 1)] = __ldcg(L.b + c + (par ? -1 : 1)) * o;
        }
    }
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
// cell (I, J, K); level0: F is the solver's level 0, whose x taps k_resid_rx rounds
template <bool D3, class LD>
__device__ __forceinline__ float restrict_cell(const Dims &fd, const Dims &cd, int I, int J, int K, LD ldr,
                                               bool level0 = false) {
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
            const float r0 = ldr(row + ix[0]), r1 = ldr(row + ix[1]), r2 = ldr(row + ix[2]), r3 = ldr(row + ix[3]);
            const float rx = x_taps(level0 && !(I & 1), r0, r1, r2, r3);
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
            s = restrict_cell<D3>(fd, cd, I, J, K, [&](int f) { return __ldcg(F.r + f); }, l == 0 && SA.pairs);
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
            acc = __fmaf_rn(two_taps(wi[0], ldx(ii[0], jj[b], kk[q]), wi[1], ldx(ii[1], jj[b], kk[q])), w, acc);
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
        float s = __fmul_rn(-kc.w, xc);
        float D = -(kc.w + kc.x + kc.y + kc.z);
        if (i > 0) s = __fmaf_rn(kc.x, __ldcg(x + c - 1) - xc, s);
        if (i < d.nx - 1) { const float k1 = __ldg(&C.coef[c + 1].x); s = __fmaf_rn(k1, __ldcg(x + c + 1) - xc, s); D -= k1; }
        if (j > 0) s = __fmaf_rn(kc.y, __ldcg(x + c - sy) - xc, s);
        if (j < d.ny - 1) { const float k1 = __ldg(&C.coef[c + sy].y); s = __fmaf_rn(k1, __ldcg(x + c + sy) - xc, s); D -= k1; }
        if (k > 0) s = __fmaf_rn(kc.z, __ldcg(x + c - sz) - xc, s);
        if (k < d.nz - 1) { const float k1 = __ldg(&C.coef[c + sz].z); s = __fmaf_rn(k1, __ldcg(x + c + sz) - xc, s); D -= k1; }
        x[c] = xc + ((__ldcg(C.b + c) - s) / D) * sor;
    }
}

// ------------------------------------- held levels (block 0, shared memory) --
extern __shared__ __align__(16) float rsm[];

// the couplings of a class-3 cell, lower and upper: those kept in shared memory at
// `slot`, or (slot < 0) of cell c.  A level's lower ones come first, then the upper
// ones (16 bytes apart, as the lanes of a pass read them).
__device__ __forceinline__ void couplings(const RLevel &L, int c, int slot, float4 &lo, float4 &hi) {
    if (slot >= 0) {
        const float4 *q = reinterpret_cast<const float4 *>(rsm + L.co);
        lo = q[slot];
        hi = q[L.cap + slot];
    } else {
        lo = __ldg(L.coef + c);
        hi = __ldg(L.gco + c);
    }
}
__device__ __forceinline__ Coef kept_coef(const RLevel &L, int c, int slot) {
    float4 lo, hi;
    couplings(L, c, slot, lo, hi);
    return Coef{lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z};
}
// a held level keeps the couplings of all its cells or of none
__device__ __forceinline__ int held_slot(const RLevel &L, int c) {
    return L.cap > 0 ? (c >> 1) + (c & 1) * (L.cap >> 1) : -1;
}
template <bool D3>
__device__ __forceinline__ Coef c_coef(const RLevel &L, unsigned cl, int c, int slot, const bool (&in)[6]) {
    const Geo &g = L.g;
    if (cl == 3u) return kept_coef(L, c, slot);
    return Coef{in[0] ? g.h2x : 0.f, in[2] ? g.h2y : 0.f, D3 && in[4] ? g.h2z : 0.f, 0.f,
                in[1] ? g.h2x : 0.f, in[3] ? g.h2y : 0.f, D3 && in[5] ? g.h2z : 0.f};
}
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
__device__ __forceinline__ void keep_couplings(const RLevel &L, int c, int slot) {
    float4 *q = reinterpret_cast<float4 *>(rsm + L.co);
    q[slot] = __ldg(L.coef + c);
    q[L.cap + slot] = __ldg(L.gco + c);
}
__device__ __forceinline__ void held_scales(const RLevel &L) {
    const float sor = SA.sor;
    for (int q = threadIdx.x; q < SCALES; q += NT) {
        const float corr = L.g.h2x * (float)(q % 3) + L.g.h2y * (float)(q / 3 % 3) + L.g.h2z * (float)(q / 9);
        rsm[L.to + q] = q == SCALE_DIRICHLET ? -sor : (corr == 0.f ? L.rdreg_sor : sor / (L.g.dreg + corr));
    }
}
template <bool D3>
__device__ __noinline__ void held_build(int l) {
    const RLevel L = SA.lv[l];
    const Dims d = L.g.d;
    const Held h = held_arrays<D3>(L);
    unsigned *word = reinterpret_cast<unsigned *>(rsm + L.to) + SCALES;
    held_scales(L);
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
        for (int o = 0; o < 2 && L.cap > 0; ++o)
            if (((cb >> (2 * o)) & 3u) == 3u) keep_couplings(L, 2 * t + o, held_slot(L, 2 * t + o));
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
            float4 lo, hi;
            couplings(L, 2 * t + o, held_slot(L, 2 * t + o), lo, hi);
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
                    const bool in[6] = {i > 0, i < d.nx - 1, j > 0, j < d.ny - 1, k > 0, k < d.nz - 1};
                    ax = apply_q(c_coef<D3>(L, cl, c, held_slot(L, c), in), vc, xm, xp, ym, yp, zm, zp);
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
        const unsigned w = T.word[t];
        const int p = (int)(w & 0x3fffu);
        const int rr = tdiv(t, L.mhx), i = 2 * (t - rr * hx);
        const int k = D3 ? tdiv(rr, L.mny) : 0, j = rr - k * d.ny;
#pragma unroll
        for (int o = 0; o < 2; ++o) {
            if ((w >> (o ? 17 : 15) & 3u) == 1u) continue;
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
// t / D, correctly rounded, by the correctly rounded reciprocal r of D: one
// correction by the exact remainder makes t r faithful, a second correct (Markstein
// 1990), at half the division's latency.
__device__ __forceinline__ float quotient(float t, float D, float r) {
    const float u = __fmul_rn(t, r), v = __fmaf_rn(__fmaf_rn(-u, D, t), r, u);
    return __fmaf_rn(__fmaf_rn(-v, D, t), r, v);
}
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
    float s = __fmul_rn(-q.e, xc);
#pragma unroll
    for (int f = 0; f < (D3 ? 6 : 4); ++f) s = __fmaf_rn(q.k[f], x[q.n[f]] - xc, s);
    x[q.c] = xc + quotient(q.b - s, q.D, q.r) * sor;
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

// block 0, above a held level: the coarsest x of the direct solve
__device__ __forceinline__ void held_coarse_in() {
    const RLevel &C = SA.lv[SA.nl - 1];
    if (blockIdx.x != 0 || SA.held >= SA.nl - 1) return;
    for (int c = threadIdx.x; c < (int)C.g.d.n(); c += NT) rsm[SA.cxo + c] = __ldcg(C.x + c);
    __syncthreads();
}

// ------------------------------------ levels spread over a cluster's blocks --
// A level's rows (j + ny k) in equal runs over the blocks of a cluster, each
// block's x, b and residual rows in its shared memory; y and z neighbours of
// another block's rows are read there through the cluster.  A phase costs a
// cluster barrier (480 cycles) and a remote round trip (240) where a grid-wide
// phase costs a grid barrier (3000) and L2 round trips.
constexpr int CLUSTER_CELLS = 1 << 16;  // level spread over a cluster
constexpr int CLUSTER_SOLVE_2D = 3 << 14;   // level 0 of a 2D solve on one cluster
constexpr int BLOCK_CELLS = 2048;       // level held in one block of a cluster
constexpr int CLUSTER_DIRECT = 384;     // unknowns of a direct coarsest solve on one cluster
constexpr int ROW_WORDS = 8;
constexpr int PAIR_ROWS = 1 << 10, PAIR_CELLS = 1 << 14, NO_SLOT = 0x3fff;

// (volatile: ordered with the barriers; not a barrier to plain accesses, which no
// phase makes to cells that it reads this way)
__device__ __forceinline__ float ld_cluster(unsigned addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ float2 ld_cluster2(unsigned addr) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ void st_cluster(unsigned addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(unsigned addr, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}

// this block's rows of a level
struct Rows {
    int q0, n;
};
__device__ __forceinline__ Rows rows_of(const RLevel &L) {
    const int all = L.g.d.ny * L.g.d.nz, q0 = min((int)cluster_rank() * L.rows, all);
    return Rows{q0, min(L.rows, all - q0)};
}
// address of row q of an array `off` of a level, in the block that owns it
__device__ __forceinline__ unsigned row_addr(const RLevel &L, int off, int q) {
    const int o = tdiv(q, L.mrows);
    return in_block(smem_addr(rsm + off + (q - o * L.rows) * L.g.d.nx), (unsigned)o);
}
// A row of the table: the addresses of x's rows y-, y+, z- and z+ of it (the
// row of zeros across the domain edge), j, k, parity of j + k, and the row's part
// of the index into the relaxation scales.
struct RowRef {
    unsigned ym, yp, zm, zp;
    int j, k;
    unsigned par, yz;
};
__device__ __forceinline__ RowRef row_ref(const RLevel &L, int lr) {
    const uint4 *p = reinterpret_cast<const uint4 *>(rsm + L.rt + ROW_WORDS * lr);
    const uint4 a = p[0], b = p[1];
    return RowRef{a.x, a.y, a.z, a.w, (int)b.x, (int)b.y, b.z, b.w};
}
// Pair t of a block's rows (cells 2 t and 2 t + 1, one of each colour): its row
// (10 bits), (j + k) & 1, the two classes, and the place of its couplings among
// those of each colour (14 bits).
struct PairRef {
    int e, lr, place, half;
    unsigned par, cls;
    __device__ __forceinline__ int slot(int o) const {
        return place == NO_SLOT ? -1 : place + (((unsigned)o ^ par) ? half : 0);
    }
};
__device__ __forceinline__ PairRef pair_ref(const RLevel &L, int t) {
    const unsigned w = reinterpret_cast<const unsigned *>(rsm + L.pt)[t];
    return PairRef{2 * t, (int)(w >> 14 & 0x3ffu), (int)(w & 0x3fffu), L.cap >> 1, w >> 24 & 1u, w >> 25};
}
template <bool D3>
__device__ __noinline__ void c_build(int l) {
    const RLevel L = SA.lv[l];
    const Dims d = L.g.d;
    const Rows R = rows_of(L);
    const unsigned zero = smem_addr(rsm + L.cx + L.rows * d.nx);
    for (int lr = threadIdx.x; lr < R.n; lr += NT) {
        const int q = R.q0 + lr, k = D3 ? tdiv(q, L.mny) : 0, j = q - k * d.ny;
        auto at = [&](bool in, int t) {
            if (!in) return zero;
            return t >= R.q0 && t < R.q0 + R.n ? smem_addr(rsm + L.cx + (t - R.q0) * d.nx) : row_addr(L, L.cx, t);
        };
        uint4 *p = reinterpret_cast<uint4 *>(rsm + L.rt + ROW_WORDS * lr);
        p[0] = make_uint4(at(j > 0, q - 1), at(j < d.ny - 1, q + 1), at(D3 && k > 0, q - d.ny),
                          at(D3 && k < d.nz - 1, q + d.ny));
        p[1] = make_uint4((unsigned)j, (unsigned)k, (unsigned)(j + k) & 1u,
                          3u * (unsigned)((j == 0) + (j == d.ny - 1)) +
                              (D3 ? 9u * (unsigned)((k == 0) + (k == d.nz - 1)) : 0u));
    }
    if (l == SA.nl - 1) return;
    held_scales(L);
    // (the couplings that fit are kept, whichever cells come first)
    __shared__ int kept;
    if (threadIdx.x == 0) kept = 0;
    __syncthreads();
    const int hx = d.nx >> 1, n = hx * R.n;
    unsigned *word = reinterpret_cast<unsigned *>(rsm + L.pt);
    for (int t = threadIdx.x; t < n; t += NT) {
        const int lr = tdiv(t, L.mhx), i = 2 * (t - lr * hx), q = R.q0 + lr, k = D3 ? tdiv(q, L.mny) : 0, j = q - k * d.ny;
        const unsigned cb = (__ldg(L.cls + L.cpitch * q + (i >> 2)) >> (2 * (i & 3))) & 15u;
        // a pair takes a place among each colour's
        const bool any = (cb & 3u) == 3u || cb >> 2 == 3u;
        int slot = any && L.cap > 0 ? atomicAdd(&kept, 1) : NO_SLOT;
        if (slot >= L.cap >> 1) slot = NO_SLOT;
        word[t] = (unsigned)slot | (unsigned)lr << 14 | (unsigned)((j + k) & 1) << 24 | cb << 25;
        const PairRef pr = pair_ref(L, t);
        for (int o = 0; o < 2 && slot != NO_SLOT; ++o)
            if ((cb >> (2 * o) & 3u) == 3u) keep_couplings(L, R.q0 * d.nx + 2 * t + o, pr.slot(o));
    }
    __syncthreads();
}
// A v at a cell from its neighbours x-, x+, y-, y+, z-, z+ as apply_cell
template <bool D3>
__device__ __forceinline__ float c_apply(const RLevel &L, unsigned cl, int c, int slot, const bool (&in)[6], float vc,
                                         const float (&n)[6]) {
    if (cl == 0u) return apply_reg(L.g, vc, n[0], n[1], n[2], n[3], n[4], n[5]);
    if (cl == 1u) return -vc;
    return apply_q(c_coef<D3>(L, cl, c, slot, in), vc, n[0], n[1], n[2], n[3], n[4], n[5]);
}
// An array's values at a pair and around it: cell o has neighbours nb[o].  rows:
// the array's place relative to x's.  (Across the domain edge: zeros, and in x
// the cell itself.)
struct PairVals {
    float2 c;
    float nb[2][6];
};
template <bool D3>
__device__ __forceinline__ PairVals pair_vals(const float *v, const RowRef &w, int rows, int e, int i, int nx) {
    PairVals q;
    const int o = rows + 4 * i;
    const float2 ym = ld_cluster2(w.ym + o), yp = ld_cluster2(w.yp + o);
    float2 zm = make_float2(0.f, 0.f), zp = zm;
    if (D3) {
        zm = ld_cluster2(w.zm + o);
        zp = ld_cluster2(w.zp + o);
    }
    q.c = *reinterpret_cast<const float2 *>(v + e);
    const float lo = v[i > 0 ? e - 1 : e], hi = v[i + 2 < nx ? e + 2 : e + 1];
    q.nb[0][0] = lo, q.nb[0][1] = q.c.y, q.nb[1][0] = q.c.x, q.nb[1][1] = hi;
    q.nb[0][2] = ym.x, q.nb[0][3] = yp.x, q.nb[0][4] = D3 ? zm.x : q.c.x, q.nb[0][5] = D3 ? zp.x : q.c.x;
    q.nb[1][2] = ym.y, q.nb[1][3] = yp.y, q.nb[1][4] = D3 ? zm.y : q.c.y, q.nb[1][5] = D3 ? zp.y : q.c.y;
    return q;
}
template <bool D3>
__device__ __forceinline__ void inside(const RLevel &L, const RowRef &w, int i, bool (&in)[6]) {
    const Dims &d = L.g.d;
    in[0] = i > 0, in[1] = i < d.nx - 1, in[2] = w.j > 0, in[3] = w.j < d.ny - 1;
    in[4] = D3 && w.k > 0, in[5] = D3 && w.k < d.nz - 1;
}

// the relaxation from x = 0 of a cell with right-hand side b
__device__ __forceinline__ float c_relax_zero(const Relax &a, const RLevel &L, unsigned cl, int c, int slot, int i,
                                              unsigned yz, float b) {
    if (cl == 3u) {
        float4 lo, hi;
        couplings(L, c, slot, lo, hi);
        return b * (a.sor * hi.w);
    }
    return b * rsm[L.to + (cl == 1u ? SCALE_DIRICHLET : yz + (i == 0) + (i == L.g.d.nx - 1))];
}

// one colour pass, as g_colour
template <bool D3, bool RZ>
__device__ __noinline__ void c_colour(int l, int col, bool first, int edge = EDGE_NONE) {
    const RLevel L = SA.lv[l];
    const Relax a = relax_of();
    const Rows R = rows_of(L);
    const int nx = L.g.d.nx, n = (nx >> 1) * R.n;
    float *x = rsm + L.cx, *alt = rsm + SA.crx;
    const float *b = rsm + L.cb, *scale = rsm + L.to;
#pragma unroll 2
    for (int t = threadIdx.x; t < n; t += NT) {
        const PairRef q = pair_ref(L, t);
        const RowRef w = row_ref(L, q.lr);
        const int o = (int)((q.par ^ (unsigned)col) & 1u), e = q.e + o, i = e - q.lr * nx;
        const unsigned cl = q.cls >> (2 * o) & 3u;
        const float bv = b[e];
        const bool tile_lo = (i & (DOT_TX - 1)) == 0, tile_hi = (i & (DOT_TX - 1)) == DOT_TX - 1;
        float vc = 0.f, xm = 0.f, xp = 0.f, ym = 0.f, yp = 0.f, zm = 0.f, zp = 0.f;
        if (!first) {
            ym = ld_cluster(w.ym + 4 * i);
            yp = ld_cluster(w.yp + 4 * i);
            if (D3) {
                zm = ld_cluster(w.zm + 4 * i);
                zp = ld_cluster(w.zp + 4 * i);
            }
            vc = x[e];
            if (i > 0) xm = edge == EDGE_USE && tile_lo ? alt[(e - 1) >> 1] : x[e - 1];
            if (i < nx - 1) xp = edge == EDGE_USE && tile_hi ? alt[(e + 1) >> 1] : x[e + 1];
        }
        float v;
        if (cl == 3u) {
            float4 lo, hi;
            couplings(L, R.q0 * nx + e, q.slot(o), lo, hi);
            v = __fmaf_rn(bv - general_sum(lo, hi, xm, xp, ym, yp, zm, zp), a.sor * hi.w, a.omsor * vc);
        } else {
            const float4 h2 = plain_couplings(L.g);
            const bool coupled = l == 0 && SA.pairs && pair_ref(L, t ^ 1).cls >> (2 * o) & 1u;
            const float rd = scale[cl == 1u ? SCALE_DIRICHLET : w.yz + (i == 0) + (i == nx - 1)];
            float sum = coupled ? general_sum(h2, h2, xm, xp, ym, yp, zm, zp) : plain_sum<D3>(L.g, xm, xp, ym, yp, zm, zp);
            if (cl == 1u) sum = 0.f;
            v = __fmaf_rn(bv - sum, rd, a.omsor * vc);
            if (edge == EDGE_KEEP && (tile_lo || tile_hi))
                alt[e >> 1] = cl == 1u ? v : __fmaf_rn(bv - general_sum(h2, h2, xm, xp, ym, yp, zm, zp), rd, a.omsor * vc);
        }
        if (cl == 3u && edge == EDGE_KEEP) alt[e >> 1] = v;
        x[e] = v;
        if (first) x[e + (o ? -1 : 1)] = 0.f;
        if (RZ) {
            rsm[SA.cr + e] = bv * v;
            rsm[SA.cr + e + (o ? -1 : 1)] = b[e + (o ? -1 : 1)] * x[e + (o ? -1 : 1)];
        }
    }
}

// r = b - A x, as g_residual
template <bool D3>
__device__ __noinline__ void c_residual(int l, bool xzero) {
    const RLevel L = SA.lv[l];
    const Rows R = rows_of(L);
    const int nx = L.g.d.nx, n = (nx >> 1) * R.n;
    float *x = rsm + L.cx, *r = rsm + SA.cr;
    const float *b = rsm + L.cb;
    for (int t = threadIdx.x; t < n; t += NT) {
        const PairRef q = pair_ref(L, t);
        const RowRef w = row_ref(L, q.lr);
        const int i = q.e - q.lr * nx;
        const float2 bv = *reinterpret_cast<const float2 *>(b + q.e);
        PairVals v;
        if (!xzero) v = pair_vals<D3>(x, w, 0, q.e, i, nx);
        else *reinterpret_cast<float2 *>(x + q.e) = make_float2(0.f, 0.f);
#pragma unroll
        for (int o = 0; o < 2; ++o) {
            const unsigned cl = q.cls >> (2 * o) & 3u;
            float res = o ? bv.y : bv.x;
            if (!xzero) {
                bool in[6];
                inside<D3>(L, w, i + o, in);
                res -= c_apply<D3>(L, cl, R.q0 * nx + q.e + o, q.slot(o), in, o ? v.c.y : v.c.x, v.nb[o]);
            }
            r[q.e + o] = cl == 1u ? 0.f : res;
        }
    }
    // the x taps of the restriction, row by row: its y and z taps then read one
    // value of a (mostly remote) row each
    __syncthreads();
    const int hx = nx >> 1;
    for (int t = threadIdx.x; t < n; t += NT) {
        const int lr = tdiv(t, L.mhx);
        int ix[4];
        rtap4(t - lr * hx, hx, ix);
        const float *row = r + lr * nx;
        rsm[SA.crx + t] = x_taps(l == 0 && SA.pairs && !((t - lr * hx) & 1), row[ix[0]], row[ix[1]], row[ix[2]], row[ix[3]]);
    }
}

// where a level's values are, seen from the level above
enum { AT_CLUSTER, AT_BLOCK, AT_COARSE, AT_GLOBAL };
__device__ __forceinline__ int place_of(int l) {
    if (l < SA.held && l < SA.nl - 1) return AT_CLUSTER;
    if (l < SA.nl - 1) return AT_BLOCK;
    return SA.coarse_sweeps > 0 ? (SA.ccoarse ? AT_CLUSTER : AT_COARSE) : AT_GLOBAL;
}

// coarse b = R r, as g_restrict, in 3D a lane per z tap; the rows of a level
// that is not spread are dealt out all the same and go to block 0 (or global
// memory)
template <bool D3>
__device__ __noinline__ void c_restrict(int l, bool relax0) {
    const RLevel F = SA.lv[l], C = SA.lv[l + 1];
    const Relax a = relax_of();
    const Dims cd = C.g.d;
    const int place = place_of(l + 1), fny = F.g.d.ny, crx = SA.crx;
    const Rows R = rows_of(C);
    constexpr int LANES = D3 ? 4 : 1;
    const int n = cd.nx * R.n;
    const Held hc = held_arrays<D3>(C);
    // (whole warps go round: the lanes of a cell meet in a shuffle)
    for (int t = threadIdx.x; t < ((LANES * n + 31) & ~31); t += NT) {
        const int e = t / LANES, q = t % LANES;
        const int lr = tdiv(e, C.mnx), I = e - lr * cd.nx, Q = R.q0 + lr;
        const int K = D3 ? tdiv(Q, C.mny) : 0, J = Q - K * cd.ny, c = Q * cd.nx + I;
        const float w4[4] = {0.125f, 0.375f, 0.375f, 0.125f};
        float s = 0.f;
        unsigned cl = 0u;
        int slot = -1;
        if (e < n) {
            if (place == AT_CLUSTER && l + 2 < SA.nl) {
                const PairRef pr = pair_ref(C, e >> 1);
                cl = pr.cls >> (2 * (e & 1)) & 3u;
                slot = pr.slot(e & 1);
            } else {
                cl = C.mask && __ldg(C.mask + c);
            }
            int jy[4], kz[4] = {0, 0, 0, 0};
            rtap4(J, cd.ny, jy);
            if (D3) rtap4(K, cd.nz, kz);
            const int k = q == 0 ? kz[0] : q == 1 ? kz[1] : q == 2 ? kz[2] : kz[3];
            float v[4];
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                const int fq = jy[p] + fny * k, o = tdiv(fq, F.mrows);
                v[p] = ld_cluster(in_block(smem_addr(rsm + crx + (fq - o * F.rows) * cd.nx + I), (unsigned)o));
            }
#pragma unroll
            for (int p = 0; p < 4; ++p) s += v[p] * w4[p];
        }
        if (D3) {
            float z[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) z[m] = __shfl_sync(0xffffffffu, s, (threadIdx.x & 28) + m);
            s = 0.f;
#pragma unroll
            for (int m = 0; m < 4; ++m) s += z[m] * w4[m];
        }
        if (e >= n || q != 0) continue;
        if (cl == 1u) s = 0.f;
        if (place == AT_CLUSTER) {
            rsm[C.cb + e] = s;
            if (relax0)
                rsm[C.cx + e] = (I + J + K) & 1 ? 0.f : c_relax_zero(a, C, cl, c, slot, I, row_ref(C, lr).yz, s);
        } else if (place == AT_BLOCK) {
            st_cluster(in_block(smem_addr(hc.b + I + hc.py * J + (D3 ? hc.pz * K : 0)), 0), s);
        } else if (place == AT_COARSE) {
            st_cluster(in_block(smem_addr(rsm + SA.cbo + c), 0), s);
        } else {
            C.b[c] = s;
        }
    }
}

// fine x += P coarse x, as g_prolong; a pair of cells has three coarse columns
template <bool D3>
__device__ __noinline__ void c_prolong(int l) {
    const RLevel F = SA.lv[l], C = SA.lv[l + 1];
    const Dims cd = C.g.d;
    const int nx = F.g.d.nx, place = place_of(l + 1), cxo = SA.cxo;
    const Rows R = rows_of(F);
    const int n = (nx >> 1) * R.n;
    const Held hc = held_arrays<D3>(C);
    float *x = rsm + F.cx;
    for (int t = threadIdx.x; t < n; t += NT) {
        const PairRef q = pair_ref(F, t);
        const RowRef w = row_ref(F, q.lr);
        const int i = q.e - q.lr * nx;
        int ia[2], ib[2], jj[2], kk[2] = {0, 0};
        float wa[2], wb[2], wj[2], wk[2] = {1.f, 1.f};
        ptaps2(i, cd.nx, ia, wa);
        ptaps2(i + 1, cd.nx, ib, wb);
        ptaps2(w.j, cd.ny, jj, wj);
        if (D3) ptaps2(w.k, cd.nz, kk, wk);
        // (ia[1] == ib[0])
        float v[2][D3 ? 2 : 1][3];
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int z = 0; z < (D3 ? 2 : 1); ++z) {
                const int Q = jj[b] + cd.ny * kk[z];
                if (place == AT_GLOBAL) {
                    const float *g = C.x + Q * cd.nx;
                    v[b][z][0] = __ldcg(g + ia[0]), v[b][z][1] = __ldcg(g + ia[1]), v[b][z][2] = __ldcg(g + ib[1]);
                } else {
                    const unsigned row = place == AT_CLUSTER ? row_addr(C, C.cx, Q)
                                         : in_block(smem_addr(place == AT_BLOCK
                                                                  ? hc.x + hc.py * jj[b] + (D3 ? hc.pz * kk[z] : 0)
                                                                  : rsm + cxo + Q * cd.nx), 0);
                    v[b][z][0] = ld_cluster(row + 4 * ia[0]);
                    v[b][z][1] = ld_cluster(row + 4 * ia[1]);
                    v[b][z][2] = ld_cluster(row + 4 * ib[1]);
                }
            }
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int z = 0; z < (D3 ? 2 : 1); ++z) {
                const float wt = wj[b] * wk[z];
                s0 = __fmaf_rn(two_taps(wa[0], v[b][z][0], wa[1], v[b][z][1]), wt, s0);
                s1 = __fmaf_rn(two_taps(wb[0], v[b][z][1], wb[1], v[b][z][2]), wt, s1);
            }
        if ((q.cls & 3u) != 1u) x[q.e] += s0;
        if (q.cls >> 2 != 1u) x[q.e + 1] += s1;
    }
}

// Sweeps of a coarsest level spread over the cluster, coarse_relax's
// arithmetic.  A pair of neighbours of a row is a word: its first cell (14
// bits), its row (10), (j + k) & 1, and for each cell whether its couplings are
// the plain ones on all sides (then nothing else is loaded); the diagonals, their
// reciprocals and, where they fit, the couplings of the others are kept (through L2,
// after a cluster barrier, they cost more than the rest of a pass).
template <bool D3>
__device__ __forceinline__ void coarse_couplings(const RLevel &C, int c, int i, int j, int k, float (&kf)[6], float &e) {
    const Dims d = C.g.d;
    const int sy = d.nx, sz = d.nx * d.ny;
    const float4 kc = __ldg(C.coef + c);
    kf[0] = i > 0 ? kc.x : 0.f;
    kf[1] = i < d.nx - 1 ? __ldg(&C.coef[c + 1].x) : 0.f;
    kf[2] = j > 0 ? kc.y : 0.f;
    kf[3] = j < d.ny - 1 ? __ldg(&C.coef[c + sy].y) : 0.f;
    kf[4] = D3 && k > 0 ? kc.z : 0.f;
    kf[5] = D3 && k < d.nz - 1 ? __ldg(&C.coef[c + sz].z) : 0.f;
    e = kc.w;
}
template <bool D3>
__device__ __noinline__ void c_coarse_build() {
    const RLevel C = SA.lv[SA.nl - 1];
    const Dims d = C.g.d;
    const Rows R = rows_of(C);
    const int hx = (d.nx + 1) >> 1, n = hx * R.n;
    unsigned *word = reinterpret_cast<unsigned *>(rsm + SA.cow);
    float2 *diag = reinterpret_cast<float2 *>(rsm + SA.cop);
    for (int t = threadIdx.x; t < n; t += NT) {
        const int lr = t / hx, i0 = 2 * (t - lr * hx), q = R.q0 + lr, k = q / d.ny, j = q - k * d.ny;
        unsigned w = (unsigned)(lr * d.nx + i0) | ((unsigned)lr << 14) | ((unsigned)((j + k) & 1) << 24);
#pragma unroll
        for (int o = 0; o < 2; ++o) {
            const int i = i0 + o, e = lr * d.nx + i, c = q * d.nx + i;
            if (i >= d.nx) continue;
            const float4 kc = __ldg(C.coef + c);
            float kf[6], E;
            coarse_couplings<D3>(C, c, i, j, k, kf, E);
            float D = -(kc.w + kc.x + kc.y + kc.z);
            if (i < d.nx - 1) D -= kf[1];
            if (j < d.ny - 1) D -= kf[3];
            if (D3 && k < d.nz - 1) D -= kf[5];
            diag[e] = make_float2(D, 1.f / D);
            if (SA.cok >= 0) {
                float4 *q8 = reinterpret_cast<float4 *>(rsm + SA.cok + 8 * e);
                q8[0] = make_float4(kf[0], kf[1], kf[2], kf[3]);
                q8[1] = make_float4(kf[4], kf[5], E, 0.f);
            }
            const bool plain = E == 0.f && kf[0] == C.g.h2x && kf[1] == C.g.h2x && kf[2] == C.g.h2y && kf[3] == C.g.h2y &&
                               (!D3 || (kf[4] == C.g.h2z && kf[5] == C.g.h2z));
            if (plain) w |= 1u << (25 + o);
        }
        word[t] = w;
    }
}
template <bool D3>
__device__ __noinline__ void c_coarse() {
    const RLevel C = SA.lv[SA.nl - 1];
    const Dims d = C.g.d;
    const float sor = SA.sor;
    const int passes = 2 * SA.coarse_sweeps;
    const Rows R = rows_of(C);
    const int nx = d.nx, n = ((nx + 1) >> 1) * R.n;
    const unsigned *word = reinterpret_cast<const unsigned *>(rsm + SA.cow);
    const float2 *diag = reinterpret_cast<const float2 *>(rsm + SA.cop);
    float *x = rsm + C.cx;
    const float *b = rsm + C.cb;
    // a plain cell's diagonal, summed as c_coarse_build sums it
    float2 plain;
    plain.x = -(0.f + C.g.h2x + C.g.h2y + C.g.h2z) - C.g.h2x - C.g.h2y;
    if (D3) plain.x -= C.g.h2z;
    plain.y = 1.f / plain.x;
    for (int e = threadIdx.x; e < nx * R.n; e += NT) x[e] = 0.f;
    cluster_sync();
    for (int pass = 0; pass < passes; ++pass) {
#pragma unroll 2
        for (int t = threadIdx.x; t < n; t += NT) {
            const unsigned w = word[t];
            const int o = (int)((w >> 24 ^ (unsigned)pass) & 1u), e = (int)(w & 0x3fffu) + o, lr = (int)(w >> 14 & 0x3ffu);
            const int i = e - lr * nx;
            if (i >= nx) continue;
            const uint4 nb = *reinterpret_cast<const uint4 *>(rsm + C.rt + ROW_WORDS * lr);
            const float xc = x[e];
            const float ym = ld_cluster(nb.x + 4 * i), yp = ld_cluster(nb.y + 4 * i);
            const float zm = D3 ? ld_cluster(nb.z + 4 * i) : 0.f, zp = D3 ? ld_cluster(nb.w + 4 * i) : 0.f;
            // (a row's end: any finite value, its coupling is 0)
            const float xm = x[i > 0 ? e - 1 : e], xp = x[i < nx - 1 ? e + 1 : e];
            float kf[6] = {C.g.h2x, C.g.h2x, C.g.h2y, C.g.h2y, C.g.h2z, C.g.h2z}, E = 0.f;
            float2 D = plain;
            if (!(w >> (25 + o) & 1u)) {
                D = diag[e];
                if (SA.cok >= 0) {
                    const float4 *q8 = reinterpret_cast<const float4 *>(rsm + SA.cok + 8 * e);
                    const float4 k0 = q8[0], k1 = q8[1];
                    kf[0] = k0.x, kf[1] = k0.y, kf[2] = k0.z, kf[3] = k0.w, kf[4] = k1.x, kf[5] = k1.y, E = k1.z;
                } else {
                    const int q = R.q0 + lr, k = D3 ? tdiv(q, C.mny) : 0, j = q - k * d.ny;
                    coarse_couplings<D3>(C, R.q0 * nx + e, i, j, k, kf, E);
                }
            }
            float s = __fmul_rn(-E, xc);
            s = __fmaf_rn(kf[0], xm - xc, s);
            s = __fmaf_rn(kf[1], xp - xc, s);
            s = __fmaf_rn(kf[2], ym - xc, s);
            s = __fmaf_rn(kf[3], yp - xc, s);
            if (D3) {
                s = __fmaf_rn(kf[4], zm - xc, s);
                s = __fmaf_rn(kf[5], zp - xc, s);
            }
            x[e] = xc + quotient(b[e] - s, D.x, D.y) * sor;
        }
        cluster_sync();
    }
}

// tables and zeros of the placed levels, once per launch
template <bool D3, bool CL>
__device__ void low_init() {
    for (int e = threadIdx.x; e < SA.floats; e += NT) rsm[e] = 0.f;
    __syncthreads();
    if (CL) {
        for (int l = SA.clu; l < SA.held && l < SA.nl - 1; ++l) c_build<D3>(l);
        if (SA.ccoarse) {
            c_build<D3>(SA.nl - 1);
            c_coarse_build<D3>();
        }
    }
    if (!CL || cluster_rank() == 0)
        for (int l = SA.held; l < SA.nl - 1; ++l) held_build<D3>(l);
    if (CL) cluster_sync();
    else __syncthreads();
}
// From the first placed level down, through the swept coarsest one.
// first_done: the first colour-0 pass is done.
template <bool D3, bool CL>
__device__ void low_down(bool first_done) {
    const int nl = SA.nl, held = SA.held, down = SA.down;
    for (int l = SA.clu; CL && l < min(held, nl - 1); ++l) {
        for (int it = 0; it < down; ++it) {
            const bool edges = it > 0 && l == 0 && SA.pairs && SA.lv[0].g.d.nx > DOT_TX;
            if (!(first_done && it == 0)) {
                c_colour<D3, false>(l, 0, it == 0, edges ? EDGE_KEEP : EDGE_NONE);
                cluster_sync();
            }
            c_colour<D3, false>(l, 1, false, edges ? EDGE_USE : EDGE_NONE);
            cluster_sync();
        }
        c_residual<D3>(l, down == 0);
        cluster_sync();
        first_done = l + 1 < min(held, nl - 1) && down > 0;
        c_restrict<D3>(l, first_done);
        cluster_sync();
    }
    const bool first = !CL || cluster_rank() == 0;
    if (first)
        for (int l = held; l < nl - 1; ++l) held_down<D3>(l);
    if (CL && SA.ccoarse) c_coarse<D3>();
    else if (SA.coarse_sweeps > 0 && first) coarse_sweeps<D3>();
}
// and back up to it; RZ: the last pass leaves the products of r.z (lv[0] is the first)
template <bool D3, bool CL, bool RZ>
__device__ void low_up() {
    const int nl = SA.nl, held = SA.held;
    if (!CL || cluster_rank() == 0)
        for (int l = nl - 2; l >= held; --l) held_up<D3>(l);
    for (int l = min(held, nl - 1) - 1; CL && l >= SA.clu; --l) {
        cluster_sync();
        c_prolong<D3>(l);
        const int up = l > 0 ? SA.up : SA.final;
        for (int it = 0; it < up; ++it) {
            const bool edges = l == 0 && SA.pairs && SA.lv[0].g.d.nx > DOT_TX;
            const int keep = edges ? EDGE_KEEP : EDGE_NONE, use = edges ? EDGE_USE : EDGE_NONE;
            cluster_sync();
            c_colour<D3, false>(l, 1, false, keep);
            cluster_sync();
            if (RZ && l == 0 && it == up - 1) c_colour<D3, true>(l, 0, false, use);
            else c_colour<D3, false>(l, 0, false, use);
        }
    }
}

// ------------------------------------------------------------ dot products --
// A thread's share of an item's sum: the products of its quad on the item's planes;
// ld gives the four products of a quad.  `any`: whether any lane of the warp has
// cells (a warp without adds exact zeros).
template <class LD>
__device__ __forceinline__ double item_share(const DotOrder &o, const Dims &d, int item, int tid, bool &any, LD ld) {
    const int i = (item % o.gx) * DOT_TX + 4 * dot_quad(tid), j = ((item / o.gx) % o.gy) * DOT_TY + dot_row(tid);
    const int k0 = (item / (o.gx * o.gy)) * o.zc, k1 = min(k0 + o.zc, d.nz);
    const bool in = i < d.nx && j < d.ny;
    Acc acc;
    if (in)
#pragma unroll 4
        for (int k = k0; k < k1; ++k) {
            const float4 v = ld(i, j, k);
            acc.add(v.x);
            acc.add(v.y);
            acc.add(v.z);
            acc.add(v.w);
        }
    any = __any_sync(0xffffffffu, in);
    return any ? acc.value() : 0.0;
}
// the item's sum, in thread 0 of the DOT_THREADS threads of half `half` of the block
__device__ __forceinline__ double item_sum(double v, bool any, int half) {
    __shared__ double sred[NT / 32];
    const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) & 7;
    const double w = any ? warp_sum(v) : 0.0;
    bar_sync_n(2 + half, DOT_THREADS);   // (the last item's sums are read)
    if (lane == 0) sred[8 * half + warp] = w;
    bar_sync_n(2 + half, DOT_THREADS);
    double t = 0.0;
    if (warp == 0) {
        // warp_sum over 32 lanes of which eight hold a sum
        t = lane < 8 ? sred[8 * half + lane] : 0.0;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    return t;
}
// the items' sums added up, in warp 0
template <class LD>
__device__ __forceinline__ double items_total(int items, LD ld) {
    __shared__ double sred[DOT_THREADS / 32];
    const int tid = threadIdx.x, lane = tid & 31;
    if (items <= 32) return tid < 32 ? warp_sum(lane < items ? ld(lane) : 0.0) : 0.0;
    if (tid < DOT_THREADS) {
        double s = 0.0;
        for (int b = tid; b < items; b += DOT_THREADS) s += ld(b);
        s = warp_sum(s);
        if (lane == 0) sred[tid >> 5] = s;
    }
    __syncthreads();
    double t = 0.0;
    if (tid < 32) {
        t = lane < DOT_THREADS / 32 ? sred[lane] : 0.0;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    __syncthreads();
    return t;
}
// the barrier after the items' sums, and their totals in thread 0 of every block
// (the dots have places of their own: a block may write the next one's sums while
// another still reads the last one's)
__device__ __noinline__ bool grid_total(int which, bool two, const double *partials, unsigned &passed, double &sum,
                                        double &sum2) {
    if (!grid_sync(SA.bar, passed)) return false;
    const int items = SA.dot[which].items;
    const double *at = partials + SA.dot[which].first;
    sum = items_total(items, [&](int b) { return __ldcg(at + b); });
    if (two) sum2 = items_total(items, [&](int b) { return __ldcg(at + items + b); });
    return true;
}
// Grid-wide: the sum of the products q that the phase before left (q2: of another
// set too), in thread 0 of every block, in the order of `which`.  Two barriers.
__device__ __noinline__ bool grid_dot(int which, const float *q, const float *q2, double *partials, unsigned &passed,
                                      double &sum, double &sum2) {
    if (!grid_sync(SA.bar, passed)) return false;
    const DotOrder o = SA.dot[which];
    const Dims d = SA.lv[0].g.d;
    const int half = threadIdx.x >> 8, tid = threadIdx.x & (DOT_THREADS - 1);
    for (int item = blockIdx.x + half * gridDim.x; item < o.items; item += 2 * gridDim.x) {
        for (int set = 0; set < (q2 ? 2 : 1); ++set) {
            const float *src = set ? q2 : q;
            bool any;
            const double v = item_share(o, d, item, tid, any, [&](int i, int j, int k) {
                return __ldcg(reinterpret_cast<const float4 *>(src + i + d.nx * (j + d.ny * k)));
            });
            const double t = item_sum(v, any, half);
            if (tid == 0) partials[o.first + set * o.items + item] = t;
        }
    }
    return grid_total(which, q2 != nullptr, partials, passed, sum, sum2);
}


// In 2D an item is one plane: its 256 threads have the quads of the phase itself,
// and the sums need no products in memory and one barrier less.  (In 3D a thread
// would march an item's planes, 16 cells or more each: 64^3 2.13 ms against 1.85,
// 80^3 4.57 against 4.19; 2D 1024 x 768 18.9 against 20.4 for the products.)
// quad(i, j, acc) adds up the products of the quad at (i, j).
template <int SETS, class F>
__device__ __forceinline__ void quad_items(int which, double *partials, F quad) {
    const DotOrder o = SA.dot[which];
    const Dims d = SA.lv[0].g.d;
    const int half = threadIdx.x >> 8, tid = threadIdx.x & (DOT_THREADS - 1);
    for (int item = blockIdx.x + half * gridDim.x; item < o.items; item += 2 * gridDim.x) {
        const int i = (item % o.gx) * DOT_TX + 4 * dot_quad(tid), j = (item / o.gx) * DOT_TY + dot_row(tid);
        const bool in = i < d.nx && j < d.ny, any = __any_sync(0xffffffffu, in);
        Acc acc[SETS];
        if (in) quad(i, j, acc);
#pragma unroll
        for (int q = 0; q < SETS; ++q) {
            const double t = item_sum(any ? acc[q].value() : 0.0, any, half);
            if (tid == 0) partials[o.first + q * o.items + item] = t;
        }
    }
}
__device__ __forceinline__ float4 ldcg4(const float *p) { return __ldcg(reinterpret_cast<const float4 *>(p)); }
__device__ __forceinline__ void st4(float *p, const float4 &v) { *reinterpret_cast<float4 *>(p) = v; }
__device__ __forceinline__ float at4(const float4 &v, int o) { return o == 0 ? v.x : o == 1 ? v.y : o == 2 ? v.z : v.w; }
__device__ __forceinline__ unsigned quad_class(const RLevel &L, int i, int j) {
    return __ldg(L.cls + L.cpitch * j + (i >> 2));
}
// 2D: the last colour pass of level 0 (colour 0), and the items' sums of r.z
__device__ __noinline__ void quad_last_colour(int edge, double *partials) {
    const RLevel L = SA.lv[0];
    const Relax a = relax_of();
    const int nx = L.g.d.nx, ny = L.g.d.ny;
    float *x = L.x;
    const float *alt = SA.alt;
    quad_items<1>(2, partials, [&](int i, int j, Acc (&acc)[1]) {
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        const int c = i + nx * j, P = j & 1, t = i & (DOT_TX - 1);   // cells P and P + 2 are of colour 0
        const unsigned cb = quad_class(L, i, j);
        const float4 bq = ldcg4(L.b + c), q = ldcg4(x + c);
        const float4 ym = j > 0 ? ldcg4(x + c - nx) : zero, yp = j < ny - 1 ? ldcg4(x + c + nx) : zero;
        float s = 0.f;   // the neighbour outside the quad
        if (P == 0 && i > 0) s = __ldcg((edge == EDGE_USE && t == 0 ? alt : x) + c - 1);
        if (P == 1 && i + 4 < nx) s = __ldcg((edge == EDGE_USE && t == DOT_TX - 4 ? alt : x) + c + 4);
        const unsigned cl0 = cb >> (2 * P) & 3u, cl1 = cb >> (2 * P + 4) & 3u;
        const bool pair = (cl0 | cl1) & 1u;
        const float n0 = relax_cell<false>(a, L, cl0, c + P, i + P, j, 0, P ? q.y : q.x, P ? q.x : s, P ? q.z : q.y,
                                           P ? ym.y : ym.x, P ? yp.y : yp.x, 0.f, 0.f, P ? bq.y : bq.x, pair);
        const float n1 = relax_cell<false>(a, L, cl1, c + P + 2, i + P + 2, j, 0, P ? q.w : q.z, P ? q.z : q.y,
                                           P ? s : q.w, P ? ym.w : ym.z, P ? yp.w : yp.z, 0.f, 0.f, P ? bq.w : bq.z, pair);
        x[c + P] = n0;
        x[c + P + 2] = n1;
        acc[0].add(bq.x * (P ? q.x : n0));
        acc[0].add(bq.y * (P ? n0 : q.y));
        acc[0].add(bq.z * (P ? q.z : n1));
        acc[0].add(bq.w * (P ? n1 : q.w));
    });
}

// ---------------------------------------------------------------- V-cycle --
// block 0, the first level below the grid-wide ones: its b from global memory, or
// its x back there
template <bool D3>
__device__ __noinline__ void tier_copy(int l, bool in) {
    const int place = place_of(l);
    const RLevel L = SA.lv[l];
    if (place == AT_BLOCK) {
        held_copy<D3>(l, in);
    } else if (place == AT_COARSE) {
        for (int c = threadIdx.x; c < (int)L.g.d.n(); c += NT) {
            if (in) rsm[SA.cbo + c] = __ldcg(L.b + c);
            else L.x[c] = rsm[SA.cxo + c];
        }
    }
    __syncthreads();
}

// z = M r on lv[0] (x = z, b = r).  first_done: the caller made the first
// colour-0 pass.  RZ: the last pass leaves the products of r.z in lv[0].r, in 2D
// the items' sums (lv[0] is one of the grid-wide levels).  The caller takes the last
// barrier.  Every block takes the same sequence of barriers
// (it depends only on the levels).  False when a barrier gave up.
template <bool D3, bool RZ>
__device__ bool vcycle(unsigned &passed, bool first_done, double *partials) {
    const int nl = SA.nl, clu = SA.clu, down = SA.down, sweeps = SA.coarse_sweeps, nc = (int)SA.lv[nl - 1].g.d.n();
    unsigned *bar = SA.bar;
    const bool low = blockIdx.x == 0;   // this block has the levels from clu down
    for (int l = 0; l < clu; ++l) {
        for (int it = 0; it < down; ++it) {
            const bool edges = it > 0 && l == 0 && SA.pairs && SA.lv[0].g.d.nx > DOT_TX;
            if (!(first_done && it == 0)) {
                g_colour<D3, false>(l, 0, it == 0, edges ? EDGE_KEEP : EDGE_NONE);
                if (!grid_sync(bar, passed)) return false;
            }
            g_colour<D3, false>(l, 1, false, edges ? EDGE_USE : EDGE_NONE);
            if (!grid_sync(bar, passed)) return false;
        }
        g_residual<D3>(l, down == 0);
        if (!grid_sync(bar, passed)) return false;
        first_done = l + 1 < clu && down > 0;
        g_restrict<D3>(l, first_done);
        if (!grid_sync(bar, passed)) return false;
    }
    if (clu == nl - 1 && sweeps > 0 && !SA.ccoarse && nc > COARSE_CELLS) {
        const Deal w = deal();
        float *gx = SA.lv[nl - 1].x;
        for (int c = w.t0; c < nc; c += w.stride) gx[c] = 0.f;
        if (!grid_sync(bar, passed)) return false;
        for (int it = 0; it < 2 * sweeps; ++it) {
            g_coarse_colour(it & 1);
            if (it + 1 < 2 * sweeps && !grid_sync(bar, passed)) return false;
        }
    } else {
        if (low) {
            tier_copy<D3>(clu, true);
            low_down<D3, false>(false);
        }
        if (sweeps == 0) {
            if (clu < nl - 1 && !grid_sync(bar, passed)) return false;
            g_direct();
            if (clu < nl - 1) {
                if (!grid_sync(bar, passed)) return false;
                held_coarse_in();
            }
        }
        if (low) {
            low_up<D3, false, false>();
            __syncthreads();
            tier_copy<D3>(clu, false);
        }
    }
    for (int l = clu - 1; l >= 0; --l) {
        if (!grid_sync(bar, passed)) return false;
        g_prolong<D3>(l);
        const int up = l > 0 ? SA.up : SA.final;
        for (int it = 0; it < up; ++it) {
            const bool edges = l == 0 && SA.pairs && SA.lv[0].g.d.nx > DOT_TX;
            const int keep = edges ? EDGE_KEEP : EDGE_NONE, use = edges ? EDGE_USE : EDGE_NONE;
            if (!grid_sync(bar, passed)) return false;
            g_colour<D3, false>(l, 1, false, keep);
            if (!grid_sync(bar, passed)) return false;
            if (RZ && l == 0 && it == up - 1) {
                if (D3) g_colour<D3, true>(l, 0, false, use);
                else quad_last_colour(use, partials);
            } else {
                g_colour<D3, false>(l, 0, false, use);
            }
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
    if (blockIdx.x == 0) low_init<D3, false>();
    if (vcycle<D3, false>(passed, false, nullptr)) grid_done(SA.bar);
    else if (threadIdx.x == 0 && st) atomicOr(&st->err, 2);
}

// The same with every level on one cluster, from a first level of up to CLUSTER_CELLS
// cells: 64 x 32 x 32 and below with variable density (every cell's couplings its own)
// 94 us over the grid, 73 here.
template <bool D3>
__global__ void __launch_bounds__(NT, 1) k_vcycle_cluster(const __grid_constant__ VArgs a, const PcgState *st) {
    if (st && (st->stop || st->err)) return;
    load_args(a);
    low_init<D3, true>();
    const RLevel &L = SA.lv[0];
    const Rows R = rows_of(L);
    const int n = L.g.d.nx * R.n, c0 = R.q0 * L.g.d.nx;
    for (int e = threadIdx.x; e < n; e += NT) rsm[L.cb + e] = __ldcg(L.b + c0 + e);
    __syncthreads();
    low_down<D3, true>(false);
    if (SA.coarse_sweeps == 0) {
        cluster_sync();
        g_direct();
        cluster_sync();
        held_coarse_in();
    }
    low_up<D3, true, false>();
    __syncthreads();
    for (int e = threadIdx.x; e < n; e += NT) L.x[c0 + e] = rsm[L.cx + e];
    cluster_sync();   // no block leaves while another may read its memory
}

// The sweeps of a coarsest level alone, from x = 0: its rows over the blocks of a
// cluster (up to 2 NT cells: in one block), the operator in tables, x in shared memory
// from the first pass to the last.  Bound by latency, a pass being a cluster barrier
// and a remote round trip.  45 x 27 x 33 with 40 passes: 55 us, 90 with one launch a
// pass (projection of 90 x 54 x 66: 7.03 -> 6.20 ms).
template <bool D3>
__global__ void __launch_bounds__(NT, 1) k_coarse_cluster(const __grid_constant__ VArgs a, const PcgState *st) {
    if (st && st->stop) return;
    load_args(a);
    low_init<D3, true>();
    const RLevel &C = SA.lv[0];
    if (SA.ccoarse) {
        const Rows R = rows_of(C);
        const int n = C.g.d.nx * R.n, c0 = R.q0 * C.g.d.nx;
        for (int e = threadIdx.x; e < n; e += NT) rsm[C.cb + e] = __ldg(C.b + c0 + e);
        __syncthreads();
        c_coarse<D3>();
        for (int e = threadIdx.x; e < n; e += NT) C.x[c0 + e] = rsm[C.cx + e];
    } else {
        tier_copy<D3>(0, true);
        coarse_sweeps<D3>();
        tier_copy<D3>(0, false);
    }
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
    double *partials;              // the work items' sums
    PcgState *st;
};

// The solver's decisions, by thread 0 of every block from the same sums.
__device__ void after_setup(PcgState &S, double rr, double bb) {
    S.rr = rr;
    S.bb = bb;
    S.thr = S.relative ? fmax(S.tol * sqrt(fabs(bb)), S.tol) : S.tol;
    // the start already meets the tolerance (linalg.js:1695-1699)
    if (sqrt(fabs(rr)) < S.thr) {
        S.stop = FF_STOP_CONVERGED;
        S.stop_iter = 0;
    }
}
// seedScalarsKernel (linalg.js:1259-1267)
__device__ void after_first_rz(PcgState &S, double rz) {
    S.rz = S.rz_old = rz;
    S.pap_baseline = fmax(fabs(S.rr), PAP_BASELINE_FLOOR);
    S.first = 1;
    S.best_rr = -1.0;
}
// alphaKernel (linalg.js:1147-1199)
__device__ void after_pap(PcgState &S, double pAp) {
    const double value = S.rz_old / pAp;
    int code = 0;
    if (nonfinite_d(pAp) || pAp == 0.0) code = FF_STOP_DEGENERATE_PAP;
    else if (fabs(pAp) > S.pap_baseline * MAX_PAP_GROWTH_FACTOR) code = FF_STOP_PAP_GROWTH;
    else if (nonfinite_or_above(value, MAX_ALPHA_MAGNITUDE)) code = FF_STOP_ALPHA_MAGNITUDE;
    S.pAp = pAp;
    S.alpha = code != 0 ? 0.0 : value;
    S.stop = code;
    S.first = 0;
    S.launched += 1;
}
__device__ void after_rr(PcgState &S, double rr) {
    S.rr = rr;
    S.iter += 1;
    // residual-growing (linalg.js:1864-1882), sampled where the reference's host
    // reads the residual
    if (!nonfinite_d(rr) && S.iter >= S.guard_next) {
        S.guard_next += GROWTH_SAMPLE;
        if (S.best_rr < 0.0 || fabs(rr) < S.best_rr) S.best_rr = fabs(rr);
        else if (S.best_rr > 0.0 && fabs(rr) > S.best_rr * MAX_RESIDUAL_GROWTH) S.growth_stop = 1;
    }
    // convergenceKernel (linalg.js:1283-1311); well above the threshold's square no
    // root is needed to see that it is not met
    if (!(fabs(rr) > S.thr * S.thr * 1.0001) && !nonfinite_or_above(sqrt(fabs(rr)), S.thr)) {
        S.stop = FF_STOP_CONVERGED;
        S.stop_iter = S.iter;
    } else if (S.growth_stop) {
        S.stop = FF_STOP_RESIDUAL_GROWING;
    }
}
// betaKernel (linalg.js:1201-1240)
__device__ void after_rz(PcgState &S, double rz) {
    const double rz_old = S.rz_old, value = rz / rz_old;
    const bool degenerate = nonfinite_d(rz_old) || rz_old == 0.0;
    const bool restart = (rz_old * rz < 0.0) || nonfinite_or_above(value, MAX_BETA_MAGNITUDE);
    S.rz = rz;
    S.beta = restart ? 0.0 : value;
    if (degenerate) S.stop = FF_STOP_DEGENERATE_OLD_RZ;
    S.rz_old = rz;
}
// what the next solve's first chunk is sized by (linalg.js:1839-1905)
__device__ void after_solve(PcgState &S) {
    if (S.maxiter <= 0) return;
    S.last_iters = S.stop == FF_STOP_CONVERGED ? S.stop_iter : S.iter;
    S.last_valid = 1;
}

// p = z + beta p (FIRST: z itself); leaves p Ap in lv[0].r.
// A neighbour across the domain edge is the cell itself: its difference is an
// exact zero, and no load waits on a branch.
template <bool D3, bool FIRST>
__device__ __noinline__ void pcg_p(const float *pold, float *pnew, float beta) {
    const RLevel L = SA.lv[0];
    const int nx = L.g.d.nx, ny = L.g.d.ny, nz = L.g.d.nz, sy = nx, sz = nx * ny, n = nx * ny * nz;
    const float *z = L.x;
    auto P = [&](int c) {
        const float zc = __ldcg(z + c);
        return FIRST ? zc : __fmaf_rn(beta, __ldcg(pold + c), zc);
    };
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
        const float ap = ap_cell(L.g, L.coef, L.gco, cl, i, j, k, c, pc, xm, xp, ym, yp, zm, zp);
        pnew[c] = pc;
        L.r[c] = pc * ap;
    }
}

// x + alpha p (SETUP: x as it is), r = b - A x, and z's first colour-0 pass
// from zero; leaves r r in lv[0].r and (SETUP) b b in bb.
template <bool D3, bool DS, bool SETUP>
__device__ __noinline__ void pcg_x(const float *b, const float *xh, const float *xl, const float *p, float *oh, float *ol,
                                      double alpha, float *bb) {
    const RLevel L = SA.lv[0];
    const Relax a = relax_of();
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
        const float rc = resid_by_class<DS>(L.g, cl, i, j, k, bc, hc, lc, hn[0], ln[0], hn[1], ln[1], hn[2], ln[2], hn[3],
                                            ln[3], D3 ? hn[4] : hc, D3 ? ln[4] : lc, D3 ? hn[5] : hc, D3 ? ln[5] : lc,
                                            [&] { return general_coef(L.coef, L.gco, i, j, k, c); });
        if (!SETUP) {
            oh[c] = hc;
            if (DS) ol[c] = lc;
        }
        L.b[c] = rc;
        L.x[c] = ((i + j + k) & 1) ? 0.f : relax_zero<D3>(a, L, cl, c, i, j, k, rc);
        L.r[c] = rc * rc;
        if (SETUP) bb[c] = bc * bc;
    }
}

// The 2D forms of pcg_p and pcg_x: a thread has an x-quad, and the items' sums come
// out of the phase.  A neighbour across the domain edge is any finite value.
template <bool FIRST>
__device__ __noinline__ void quad_p(const float *pold, float *pnew, float beta, double *partials) {
    const RLevel L = SA.lv[0];
    const int nx = L.g.d.nx, ny = L.g.d.ny;
    const float *z = L.x;
    auto P1 = [&](int c) {
        const float zc = __ldcg(z + c);
        return FIRST ? zc : __fmaf_rn(beta, __ldcg(pold + c), zc);
    };
    auto P4 = [&](int c) {
        const float4 zq = ldcg4(z + c);
        if (FIRST) return zq;
        const float4 q = ldcg4(pold + c);
        return make_float4(__fmaf_rn(beta, q.x, zq.x), __fmaf_rn(beta, q.y, zq.y), __fmaf_rn(beta, q.z, zq.z),
                           __fmaf_rn(beta, q.w, zq.w));
    };
    quad_items<1>(0, partials, [&](int i, int j, Acc (&acc)[1]) {
        const int c = i + nx * j;
        const unsigned cb = quad_class(L, i, j);
        const float4 q = P4(c), ym = P4(j > 0 ? c - nx : c), yp = P4(j < ny - 1 ? c + nx : c);
        const float xl = P1(i > 0 ? c - 1 : c), xr = P1(i + 4 < nx ? c + 4 : c + 3);
        st4(pnew + c, q);
        auto add = [&](int o, float pc, float xm, float xp) {
            const float v = ap_cell(L.g, L.coef, L.gco, cb >> (2 * o) & 3u, i + o, j, 0, c + o, pc, xm, xp, at4(ym, o),
                                    at4(yp, o), pc, pc);
            acc[0].add(pc * v);
        };
        add(0, q.x, xl, q.y);
        add(1, q.y, q.x, q.z);
        add(2, q.z, q.y, q.w);
        add(3, q.w, q.z, xr);
    });
}
template <bool DS, bool SETUP>
__device__ __noinline__ void quad_x(const float *b, const float *xh, const float *xl, const float *p, float *oh, float *ol,
                                    double alpha, double *partials) {
    const RLevel L = SA.lv[0];
    const Relax a = relax_of();
    const int nx = L.g.d.nx, ny = L.g.d.ny;
    const float ahi = (float)alpha, alo = (float)(alpha - (double)ahi);
    struct Quad {
        float4 h, l;
    };
    auto form = [&](float pv, float &h, float &l) {
        if (DS) ds_axpy(h, l, ahi, alo, pv, h, l);
        else h = __fmaf_rn(ahi, pv, h);
    };
    auto X1 = [&](int c, float &h, float &l) {
        h = __ldcg(xh + c);
        l = DS ? __ldcg(xl + c) : 0.f;
        if (!SETUP) form(__ldcg(p + c), h, l);
    };
    auto X4 = [&](int c) {
        Quad q{ldcg4(xh + c), DS ? ldcg4(xl + c) : make_float4(0.f, 0.f, 0.f, 0.f)};
        if (!SETUP) {
            const float4 pv = ldcg4(p + c);
            form(pv.x, q.h.x, q.l.x);
            form(pv.y, q.h.y, q.l.y);
            form(pv.z, q.h.z, q.l.z);
            form(pv.w, q.h.w, q.l.w);
        }
        return q;
    };
    quad_items<SETUP ? 2 : 1>(1, partials, [&](int i, int j, Acc (&acc)[SETUP ? 2 : 1]) {
        const int c = i + nx * j;
        const unsigned cb = quad_class(L, i, j);
        const float4 bq = __ldg(reinterpret_cast<const float4 *>(b + c));
        const Quad q = X4(c), ym = X4(j > 0 ? c - nx : c), yp = X4(j < ny - 1 ? c + nx : c);
        float xlh, xll, xrh, xrl;
        X1(i > 0 ? c - 1 : c, xlh, xll);
        X1(i + 4 < nx ? c + 4 : c + 3, xrh, xrl);
        if (!SETUP) {
            st4(oh + c, q.h);
            if (DS) st4(ol + c, q.l);
        }
        auto res = [&](int o, float bc, float h, float l, float xmh, float xml, float xph, float xpl) {
            const float r = resid_by_class<DS>(L.g, cb >> (2 * o) & 3u, i + o, j, 0, bc, h, l, xmh, xml, xph, xpl,
                                               at4(ym.h, o), at4(ym.l, o), at4(yp.h, o), at4(yp.l, o), h, l, h, l,
                                               [&] { return general_coef(L.coef, L.gco, i + o, j, 0, c + o); });
            acc[0].add(r * r);
            if (SETUP) acc[SETUP ? 1 : 0].add(bc * bc);
            return r;
        };
        float4 r;
        r.x = res(0, bq.x, q.h.x, q.l.x, xlh, xll, q.h.y, q.l.y);
        r.y = res(1, bq.y, q.h.y, q.l.y, q.h.x, q.l.x, q.h.z, q.l.z);
        r.z = res(2, bq.z, q.h.z, q.l.z, q.h.y, q.l.y, q.h.w, q.l.w);
        r.w = res(3, bq.w, q.h.w, q.l.w, q.h.z, q.l.z, xrh, xrl);
        st4(L.b + c, r);
        auto first = [&](int o, float rc) { return relax_zero<false>(a, L, cb >> (2 * o) & 3u, c + o, i + o, j, 0, rc); };
        st4(L.x + c, j & 1 ? make_float4(0.f, first(1, r.y), 0.f, first(3, r.w))
                           : make_float4(first(0, r.x), 0.f, first(2, r.z), 0.f));
    });
}

template <bool D3, bool DS>
__global__ void __launch_bounds__(NT, 1) k_pcg_resident(const __grid_constant__ VArgs a, const __grid_constant__ PcgArgs A) {
    __shared__ PcgState S;
    unsigned passed = 0;
    if (threadIdx.x == 0) S = *A.st;   // as k_state_init left it
    load_args(a);
    if (blockIdx.x == 0) low_init<D3, false>();
    bool ok = true;
    double sum = 0.0, sum2 = 0.0;
    const float *products = a.lv[0].r;
    // a phase and its sum (3D: the phase leaves products; 2D: the items' sums)
    auto total = [&](int which, const float *second = nullptr) {
        if constexpr (D3) return grid_dot(which, products, second, A.partials, passed, sum, sum2);
        else return grid_total(which, second != nullptr, A.partials, passed, sum, sum2);
    };
    auto x_phase = [&](auto setup) {
        constexpr bool SETUP = decltype(setup)::value;
        const int c = S.x_cur;
        const float *xh = c ? A.xh[1] : A.xh[0], *xl = c ? A.xl[1] : A.xl[0], *p = S.p_cur ? A.p[1] : A.p[0];
        float *oh = c ? A.xh[0] : A.xh[1], *ol = c ? A.xl[0] : A.xl[1];
        if constexpr (D3) pcg_x<D3, DS, SETUP>(A.b, xh, xl, p, oh, ol, S.alpha, A.p[0]);
        else quad_x<DS, SETUP>(A.b, xh, xl, p, oh, ol, S.alpha, A.partials);
        return total(1, SETUP ? A.p[0] : nullptr);
    };
    auto p_phase = [&](auto first) {
        constexpr bool FIRST = decltype(first)::value;
        const float *po = S.p_cur ? A.p[1] : A.p[0];
        const float beta = FIRST ? 0.f : (float)S.beta;
        float *pn = S.p_cur ? A.p[0] : A.p[1];
        if constexpr (D3) pcg_p<D3, FIRST>(po, pn, beta);
        else quad_p<FIRST>(po, pn, beta, A.partials);
        return total(0);
    };
    // setup (linalg.js:1627-1637): r = b - A x, its norm and b's, z = M r, r.z
    ok = x_phase(std::true_type());
    if (ok && threadIdx.x == 0) after_setup(S, sum, sum2);
    __syncthreads();
    if (ok && S.stop == 0) {
        ok = vcycle<D3, true>(passed, true, A.partials) && total(2);
        if (ok && threadIdx.x == 0) after_first_rz(S, sum);
        __syncthreads();
    }
    while (ok && S.stop == 0 && S.iter < S.maxiter) {
        if (!(ok = S.first ? p_phase(std::true_type()) : p_phase(std::false_type()))) break;
        if (threadIdx.x == 0) {
            after_pap(S, sum);
            S.p_cur ^= 1;
        }
        __syncthreads();
        if (S.stop) break;
        if (!(ok = x_phase(std::false_type()))) break;
        if (threadIdx.x == 0) {
            S.x_cur ^= 1;
            after_rr(S, sum);
        }
        __syncthreads();
        if (S.stop) break;
        if (!(ok = vcycle<D3, true>(passed, true, A.partials) && total(2))) break;
        if (threadIdx.x == 0) after_rz(S, sum);
        __syncthreads();
    }
    if (ok) grid_done(SA.bar);
    else if (threadIdx.x == 0) atomicOr(&A.st->err, 2);
    if (ok && blockIdx.x == 0 && threadIdx.x == 0) {
        after_solve(S);
        *A.st = S;
    }
}

// ------------------------------------------- PCG solve on one cluster ------
// The same solve with level 0 spread over the blocks of one cluster: every
// array in shared memory, phases one cluster barrier apart.  Bound by latency: a
// phase of one pair a thread takes about 1100 cycles with its barrier, where a
// grid-wide one takes 5000; a dot product 3000 to 4000 (FP64 runs at two lanes a
// clock here), the coarsest level's 40 passes in one block 8000 to 13000.
// Whole projections, over the grid and here: 48 x 32 x 32 0.91 and 0.72 ms, 64 x 32 x
// 24 1.18 and 1.04, 192 x 128 2.43 and 1.85.  The line lies where both meet (64 x 32 x
// 32 0.83 and 0.77; 256 x 192 3.66 and 3.41, 256^2 3.52 and 3.78) and where the arrays
// still fit.
// A cluster in a launch over the whole GPU, for the lower levels of larger solves,
// was slower: 8 blocks a cluster leave 120 of 152 SMs to the grid-wide phases, and a
// spread phase of eight pairs a thread takes as long as a grid-wide one.

// The sum of the products at `q` (shared memory, lv[0]'s rows; q2: of another set
// too) that the phase before left, in thread 0 of every block, in the order of
// `which`.  Two cluster barriers.
__device__ __noinline__ void cluster_dot(int which, int q, int q2, double &sum, double &sum2) {
    cluster_sync();
    const DotOrder o = SA.dot[which];
    const RLevel &L = SA.lv[0];
    const Dims d = L.g.d;
    const int half = threadIdx.x >> 8, tid = threadIdx.x & (DOT_THREADS - 1), n = SA.csize;
    double *parts = reinterpret_cast<double *>(rsm + SA.parts);
    for (int item = (int)cluster_rank() + half * n; item < o.items; item += 2 * n) {
        for (int set = 0; set < (q2 >= 0 ? 2 : 1); ++set) {
            bool any;
            const double v = item_share(o, d, item, tid, any, [&](int i, int j, int k) {
                float4 w;
                asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(w.x), "=f"(w.y), "=f"(w.z), "=f"(w.w)
                             : "r"(row_addr(L, set ? q2 : q, j + d.ny * k) + 4 * i));
                return w;
            });
            const double t = item_sum(v, any, half);
            if (tid < 32) {
                const double all = __shfl_sync(0xffffffffu, t, 0);
                if (tid < n) st_cluster(in_block(smem_addr(parts + set * o.items + item), (unsigned)tid), all);
            }
        }
    }
    cluster_sync();
    sum = items_total(o.items, [&](int b) { return parts[b]; });
    if (q2 >= 0) sum2 = items_total(o.items, [&](int b) { return parts[o.items + b]; });
}

// p = z + beta p of this block's rows
template <bool FIRST>
__device__ __forceinline__ void c_direction(float beta) {
    const RLevel &L = SA.lv[0];
    const int n = L.g.d.nx * rows_of(L).n;
    float *p = rsm + SA.p;
    const float *z = rsm + L.cx;
    for (int e = threadIdx.x; e < n; e += NT) p[e] = FIRST ? z[e] : __fmaf_rn(beta, p[e], z[e]);
}
// p Ap of this block's rows into the scratch rows
template <bool D3>
__device__ __noinline__ void c_pap() {
    const RLevel L = SA.lv[0];
    const Rows R = rows_of(L);
    const int nx = L.g.d.nx, n = (nx >> 1) * R.n, dp = 4 * (SA.p - L.cx);
    const float *p = rsm + SA.p;
#pragma unroll 2
    for (int t = threadIdx.x; t < n; t += NT) {
        const PairRef q = pair_ref(L, t);
        const RowRef w = row_ref(L, q.lr);
        const int i = q.e - q.lr * nx;
        const PairVals v = pair_vals<D3>(p, w, dp, q.e, i, nx);
        float2 out;
#pragma unroll
        for (int o = 0; o < 2; ++o) {
            const float pc = o ? v.c.y : v.c.x;
            const float ap = ap_by_class(L.g, q.cls >> (2 * o) & 3u, i + o, w.j, w.k, pc, v.nb[o][0], v.nb[o][1], v.nb[o][2],
                                         v.nb[o][3], v.nb[o][4], v.nb[o][5],
                                         [&] { return kept_coef(L, R.q0 * nx + q.e + o, q.slot(o)); });
            (o ? out.y : out.x) = pc * ap;
        }
        *reinterpret_cast<float2 *>(rsm + SA.cr + q.e) = out;
    }
}
// x += alpha p of this block's rows
template <bool DS>
__device__ __forceinline__ void c_step(double alpha) {
    const RLevel &L = SA.lv[0];
    const int n = L.g.d.nx * rows_of(L).n;
    const float ahi = (float)alpha, alo = (float)(alpha - (double)ahi);
    const float *p = rsm + SA.p;
    float *xh = rsm + SA.xh, *xl = rsm + SA.xl;
    for (int e = threadIdx.x; e < n; e += NT) {
        if (DS) ds_axpy(xh[e], xl[e], ahi, alo, p[e], xh[e], xl[e]);
        else xh[e] = __fmaf_rn(ahi, p[e], xh[e]);
    }
}
// r = b - A x and z's first colour-0 pass; r r into the scratch rows and (SETUP) b b
// into p's
template <bool D3, bool DS, bool SETUP>
__device__ __noinline__ void c_new_residual() {
    const RLevel L = SA.lv[0];
    const Relax a = relax_of();
    const Rows R = rows_of(L);
    const int nx = L.g.d.nx, n = (nx >> 1) * R.n, dh = 4 * (SA.xh - L.cx), dl = 4 * (SA.xl - L.cx);
    float *r = rsm + L.cb, *z = rsm + L.cx;
#pragma unroll 1
    for (int t = threadIdx.x; t < n; t += NT) {
        const PairRef q = pair_ref(L, t);
        const RowRef w = row_ref(L, q.lr);
        const int i = q.e - q.lr * nx, c0 = R.q0 * nx;
        const float2 bc = *reinterpret_cast<const float2 *>(rsm + SA.rhs + q.e);
        const PairVals h = pair_vals<D3>(rsm + SA.xh, w, dh, q.e, i, nx);
        PairVals lo;
        if (DS) lo = pair_vals<D3>(rsm + SA.xl, w, dl, q.e, i, nx);
#pragma unroll
        for (int o = 0; o < 2; ++o) {
            const unsigned cl = q.cls >> (2 * o) & 3u;
            const int e = q.e + o;
            const float hc = o ? h.c.y : h.c.x, bo = o ? bc.y : bc.x;
            const float (&H)[6] = h.nb[o], (&G)[6] = lo.nb[o];
            const float rc = resid_by_class<DS>(L.g, cl, i + o, w.j, w.k, bo, hc, o ? lo.c.y : lo.c.x, H[0], G[0], H[1],
                                                G[1], H[2], G[2], H[3], G[3], H[4], G[4], H[5], G[5],
                                                [&] { return kept_coef(L, c0 + e, q.slot(o)); });
            r[e] = rc;
            z[e] = (unsigned)o ^ q.par ? 0.f : c_relax_zero(a, L, cl, c0 + e, q.slot(o), i + o, w.yz, rc);
            rsm[SA.cr + e] = rc * rc;
            if (SETUP) rsm[SA.p + e] = bo * bo;
        }
    }
}
template <bool D3>
__device__ void cluster_vcycle() {
    low_down<D3, true>(true);
    if (SA.coarse_sweeps == 0) {
        cluster_sync();
        g_direct();
        cluster_sync();
        held_coarse_in();
    }
    low_up<D3, true, true>();
}

template <bool D3, bool DS>
__global__ void __launch_bounds__(NT, 1) k_pcg_cluster(const __grid_constant__ VArgs a, const __grid_constant__ PcgArgs A) {
    __shared__ PcgState S;
    if (threadIdx.x == 0) S = *A.st;   // as k_state_init left it: x in slot 0
    load_args(a);
    low_init<D3, true>();
    const Rows R = rows_of(SA.lv[0]);
    const int nx = SA.lv[0].g.d.nx, n = nx * R.n;
    float *xh = rsm + SA.xh, *xl = rsm + SA.xl;
    for (int e = threadIdx.x; e < n; e += NT) {
        xh[e] = __ldcg(A.xh[0] + R.q0 * nx + e);
        if (DS) xl[e] = __ldcg(A.xl[0] + R.q0 * nx + e);
        rsm[SA.rhs + e] = __ldg(A.b + R.q0 * nx + e);
    }
    double sum = 0.0, sum2 = 0.0;
    cluster_sync();
    c_new_residual<D3, DS, true>();
    cluster_dot(1, SA.cr, SA.p, sum, sum2);
    if (threadIdx.x == 0) after_setup(S, sum, sum2);
    __syncthreads();
    if (S.stop == 0) {
        cluster_vcycle<D3>();
        cluster_dot(2, SA.cr, -1, sum, sum2);
        if (threadIdx.x == 0) after_first_rz(S, sum);
        __syncthreads();
    }
    while (S.stop == 0 && S.iter < S.maxiter) {
        if (S.first) c_direction<true>(0.f);
        else c_direction<false>((float)S.beta);
        cluster_sync();
        c_pap<D3>();
        cluster_dot(0, SA.cr, -1, sum, sum2);
        if (threadIdx.x == 0) after_pap(S, sum);
        __syncthreads();
        if (S.stop) break;
        c_step<DS>(S.alpha);
        cluster_sync();
        c_new_residual<D3, DS, false>();
        cluster_dot(1, SA.cr, -1, sum, sum2);
        if (threadIdx.x == 0) after_rr(S, sum);
        __syncthreads();
        if (S.stop) break;
        cluster_vcycle<D3>();
        cluster_dot(2, SA.cr, -1, sum, sum2);
        if (threadIdx.x == 0) after_rz(S, sum);
        __syncthreads();
    }
    for (int e = threadIdx.x; e < n; e += NT) {
        A.xh[0][R.q0 * nx + e] = xh[e];
        if (DS) A.xl[0][R.q0 * nx + e] = xl[e];
        SA.lv[0].b[R.q0 * nx + e] = rsm[SA.lv[0].cb + e];   // the residual, for the diagnostics
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        after_solve(S);
        *A.st = S;
    }
    cluster_sync();   // no block leaves while another may read its memory
}

// Places levels in shared memory, from the last but one upward: in block 0 up to
// BLOCK_CELLS cells (HELD_CELLS without a cluster), above them spread over the
// cluster up to CLUSTER_CELLS, as far as they fit; `solver`: lv[0] is spread or not
// placed, with the solver's vectors.  The coarsest level, if it is swept, in block 0
// or spread.  a.clu says how far it went; returns the bytes a block needs.
int place(VArgs &a, bool d3, bool solver) {
    const int nl = a.nl;
    int used = 0;
    auto take = [&](long long floats) {
        const int at = used;
        used += (int)((floats + 3) & ~3LL);
        return at;
    };
    auto fits = [&](long long floats) { return 4 * (used + floats) <= SMEM_BYTES; };
    const bool clusters = a.csize > 1;
    const long long items = std::max(a.dot[0].items, std::max(a.dot[1].items, a.dot[2].items));
    RLevel &C = a.lv[nl - 1];
    const long long nc = C.g.d.n(), ccells = (long long)C.rows * C.g.d.nx;
    a.held = a.clu = nl - 1;
    if (clusters && a.coarse_sweeps > 0 && nc > 2 * NT && nc <= CLUSTER_CELLS && C.rows <= PAIR_ROWS && ccells <= PAIR_CELLS) {
        const long long tables = ccells + C.g.d.nx + ccells + (long long)C.rows * ROW_WORDS + 2 * ccells +
                                 (long long)C.rows * ((C.g.d.nx + 1) / 2) + 64;
        if (fits(tables)) {
            a.ccoarse = 1;
            C.cx = take(ccells + C.g.d.nx);
            C.cb = take(ccells);
            C.rt = take((long long)C.rows * ROW_WORDS);
            a.cop = take(2 * ccells);
            a.cow = take((long long)C.rows * ((C.g.d.nx + 1) / 2));
        }
    }
    if (!a.ccoarse) {
        // (a coarsest level swept over the grid leaves nothing for block 0)
        if (a.coarse_sweeps > 0 && nc > COARSE_CELLS) return 0;
        if (nc <= COARSE_CELLS) {
            a.cxo = take(nc);
            a.cbo = take(nc);
        }
        long long most = 0;
        for (int l = nl - 2; l >= (solver ? 1 : 0); --l) {
            RLevel &L = a.lv[l];
            const long long n = L.g.d.n(), arr = held_floats(L.g.d, d3);
            // (a place in the held arrays takes 14 bits of a pair's word)
            if (n > (clusters ? BLOCK_CELLS : HELD_CELLS) || arr > 0x3fff ||
                !fits(std::max(most, n) + 2 * arr + SCALES + n / 2 + 64))
                break;
            L.xo = take(arr);
            L.bo = take(arr);
            L.to = take(SCALES + n / 2);
            most = std::max(most, n);
            a.held = a.clu = l;
        }
        a.ro = take(most);
    }
    for (int l = a.held - 1; clusters && l >= 0; --l) {
        RLevel &L = a.lv[l];
        const long long n = L.g.d.n(), cells = (long long)L.rows * L.g.d.nx, padded = cells + L.g.d.nx;
        const bool vectors = solver && l == 0;
        // (with the residual scratch, as large as the level farthest up)
        const long long more = 2 * padded + 3 * cells / 2 + (vectors ? 4 * padded + 4 * items : 0) + (long long)L.rows * ROW_WORDS +
                               cells / 2 + SCALES + 64;
        if (n > CLUSTER_CELLS || L.rows > PAIR_ROWS || cells > PAIR_CELLS || !fits(more)) break;
        L.cx = take(padded);
        L.cb = take(cells);
        L.rt = take((long long)L.rows * ROW_WORDS);
        L.pt = take(cells / 2);
        L.to = take(SCALES);
        if (vectors) {
            a.p = take(padded);
            a.xh = take(padded);
            a.xl = take(padded);
            a.rhs = take(cells);
            a.parts = take(4 * items);
        }
        a.clu = l;
    }
    if (a.clu < a.held) {
        const long long cells = (long long)a.lv[a.clu].rows * a.lv[a.clu].g.d.nx;
        a.cr = take(cells);
        a.crx = take(cells / 2);
    }
    // couplings, of the lowest levels first: a held level's whole or none, a spread
    // one's as many as there is room for
    for (int l = nl - 2; l >= a.clu; --l) {
        RLevel &L = a.lv[l];
        const bool held = l >= a.held;
        const long long cells = held ? L.g.d.n() : (long long)L.rows * L.g.d.nx, room = (SMEM_BYTES / 4 - used) / 8;
        L.cap = (int)std::max(0LL, std::min(std::min(cells, room), 2LL * NO_SLOT - 2)) & ~1;
        if (held && L.cap < cells) L.cap = 0;
        L.co = take(8LL * L.cap);
    }
    a.cok = a.ccoarse && fits(8 * ccells) ? take(8 * ccells) : -1;
    a.floats = used;
    return 4 * used;
}

VArgs make_args(const Level *lv, const SweepMaps *sm, int nl, int dims, int down, int up, int fin, float sor,
                const double *G, int nG, int coarse_sweeps, unsigned *bar, int csize, bool solver, int sm_count, int &smem) {
    VArgs a{};
    a.csize = csize;
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
        t.rows = (L.d.ny * L.d.nz + csize - 1) / csize;
        t.mrows = magic(t.rows);
        t.mhx = magic(std::max(1, L.d.nx / 2));
        t.mnx = magic(L.d.nx);
        t.mny = magic(L.d.ny);
        if (l < nl - 1 && sm) {
            t.cls = sm[l].cls_ptr;
            t.cpitch = sm[l].cls_pitch;
            t.gco = sm[l].gco;
        }
    }
    for (int w = 0; w < 3 && sm_count > 0; ++w) {
        const Dims &d = lv[0].d;
        const int zc = ffk::cg_tma_planes(d, sm_count, w);
        DotOrder &o = a.dot[w];
        o.gx = (d.nx + DOT_TX - 1) / DOT_TX;
        o.gy = (d.ny + DOT_TY - 1) / DOT_TY;
        o.zc = zc;
        o.items = o.gx * o.gy * ((d.nz + zc - 1) / zc);
        o.first = w == 0 ? 0 : a.dot[w - 1].first + w * a.dot[w - 1].items;   // (r.r comes with b.b)
    }
    a.pairs = solver;
    smem = place(a, dims == 3, solver);
    return a;
}

// one cluster of csize blocks, or (csize 1) blocks that all run at once
int launch(const void *kernel, int blocks, int csize, int smem, cudaStream_t s, void **args) {
    FF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
    if (csize > 8) FF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    if (csize > 1) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim = {(unsigned)csize, 1, 1};
    } else {
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    FF_CUDA(cudaLaunchKernelExC(&cfg, kernel, args));
    return FF_OK;
}

// clusters of c blocks that run at once
int clusters_of(const void *kernel, int c) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim = {(unsigned)c, 1, 1};
    cfg.gridDim = dim3((unsigned)c);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int most = 0;
    const bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) == cudaSuccess &&
                    (c <= 8 || cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) &&
                    cudaOccupancyMaxActiveClusters(&most, kernel, &cfg) == cudaSuccess;
    if (!ok) (void)cudaGetLastError();
    return ok ? most : 0;
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

int cluster_blocks() {
    const void *k = (const void *)k_pcg_cluster<true, true>;
    return clusters_of(k, 16) > 0 ? 16 : clusters_of(k, 8) > 0 ? 8 : 0;
}

int vcycle_tail(const Level *lv, const SweepMaps *sm, int nl, int dims, int down, int up, float sor, const double *G,
                int nG, int coarse_sweeps, PcgState *st, unsigned *bar, int sm_count, int cluster, cudaStream_t s) {
    FF_TRY(check_levels(lv, sm, nl, G, nG, coarse_sweeps, bar));
    int smem = 0;
    if (cluster > 0 && lv[0].d.n() > BLOCK_CELLS && lv[0].d.n() <= CLUSTER_CELLS &&
        (coarse_sweeps > 0 || nG <= CLUSTER_DIRECT)) {
        VArgs a = make_args(lv, sm, nl, dims, down, up, up, sor, G, nG, coarse_sweeps, bar, cluster, false, 0, smem);
        void *args[] = {&a, &st};
        if (a.clu == 0 && a.held > 0)
            return launch(dims == 3 ? (const void *)k_vcycle_cluster<true> : (const void *)k_vcycle_cluster<false>, cluster,
                          cluster, smem, s, args);
    }
    VArgs a = make_args(lv, sm, nl, dims, down, up, up, sor, G, nG, coarse_sweeps, bar, 1, false, 0, smem);
    void *args[] = {&a, &st};
    // a hierarchy that block 0 holds whole needs no other block
    const bool alone = a.clu == 0 && coarse_sweeps > 0;
    return launch(dims == 3 ? (const void *)k_vcycle_tail<true> : (const void *)k_vcycle_tail<false>, alone ? 1 : sm_count, 1,
                  smem, s, args);
}

// (up to 2 NT cells: one block)
static int coarse_blocks(const Level &L, int cluster) { return L.d.n() <= 2 * NT ? 1 : cluster; }

bool coarse_cluster_fits(const Level &L, int dims, int sweeps, int cluster) {
    int smem = 0;
    const int csize = coarse_blocks(L, cluster);
    return csize == 1 ||
           make_args(&L, nullptr, 1, dims, 0, 0, 0, 1.f, nullptr, 0, sweeps, nullptr, csize, false, 0, smem).ccoarse;
}

int coarse_cluster(const Level &L, int dims, int sweeps, float sor, const PcgState *st, int cluster, cudaStream_t s) {
    int smem = 0;
    const int csize = coarse_blocks(L, cluster);
    VArgs a = make_args(&L, nullptr, 1, dims, 0, 0, 0, sor, nullptr, 0, sweeps, nullptr, csize, false, 0, smem);
    FF_CHECK(sweeps > 0 && (csize == 1 || a.ccoarse), FF_E_STATE, "coarsest sweeps: the level does not fit a cluster");
    void *args[] = {&a, &st};
    return launch(dims == 3 ? (const void *)k_coarse_cluster<true> : (const void *)k_coarse_cluster<false>, csize, csize, smem,
                  s, args);
}

int pcg_resident(const Level *lv, const SweepMaps *sm, int nl, int dims, int down, int up, int fin, float sor,
                 const double *G, int nG, int coarse_sweeps, const float *b, float *p0, float *p1, float *xh0, float *xl0,
                 float *xh1, float *xl1, int ds, PcgState *st, double *partials, unsigned *bar, int sm_count,
                 int cluster, float *alt, cudaStream_t s) {
    FF_TRY(check_levels(lv, sm, nl, G, nG, coarse_sweeps, bar));
    int smem = 0;
    PcgArgs A{b, {p0, p1}, {xh0, xh1}, {xl0, xl1}, partials, st};
    VArgs a;
    void *args[] = {&a, &A};
    // on one cluster, if level 0 fits it
    if (cluster > 0 && lv[0].d.n() <= (dims == 3 ? CLUSTER_CELLS : CLUSTER_SOLVE_2D) && (coarse_sweeps > 0 || nG <= CLUSTER_DIRECT)) {
        a = make_args(lv, sm, nl, dims, down, up, fin, sor, G, nG, coarse_sweeps, bar, cluster, true, sm_count, smem);
        const void *k = dims == 3 ? (ds ? (const void *)k_pcg_cluster<true, true> : (const void *)k_pcg_cluster<true, false>)
                                  : (ds ? (const void *)k_pcg_cluster<false, true> : (const void *)k_pcg_cluster<false, false>);
        if (a.clu == 0) return launch(k, cluster, cluster, smem, s, args);
    }
    a = make_args(lv, sm, nl, dims, down, up, fin, sor, G, nG, coarse_sweeps, bar, 1, true, sm_count, smem);
    a.alt = alt;
    const void *k = dims == 3 ? (ds ? (const void *)k_pcg_resident<true, true> : (const void *)k_pcg_resident<true, false>)
                              : (ds ? (const void *)k_pcg_resident<false, true> : (const void *)k_pcg_resident<false, false>);
    return launch(k, sm_count, 1, smem, s, args);
}

}  // namespace ffk
