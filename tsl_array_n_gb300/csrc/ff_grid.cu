// Grid-velocity kernels around the projection: semi-Lagrangian advection of
// the MAC velocity and of cell scalars (fluxflow src/grid/advection_solver3.js),
// the blocked-boundary velocity constraint
// (src/grid/grid_blocked_boundary_condition_solver3.js) and explicit viscosity
// (no reference counterpart; src/grid/grid_solver3.js:104 leaves it a no-op).
//
// Arithmetic is FP32 as in the reference's WGSL, one IEEE operation at a
// time: this file is compiled with -fmad=false so no multiply-add is fused,
// and every expression keeps the reference's evaluation order.  That makes
// the results reproducible operation for operation on any IEEE FP32 machine.
//
// Advection is bound by issue (a tricubic sample reads 64 taps of one component,
// mostly L1/L2 hits), the constraint by the bytes of the faces that its stages can
// change, which lists keep; one thread per face or cell, or four for a pass over all.
#include "ff_grid.cuh"
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <utility>

namespace {
using namespace ffg;

// The constraint's work outside the obstacle is one read of the weights and
// one of the values: a 256^3 grid has 50M faces, of which the collider
// closes 0.2M, and only those change before the clamp.  So the marking pass
// lists them, the extension steps, the no-flux projection and its write-back
// run over the list, and the last pass writes a face only when it changes.
// Measured at 256^3 around a sphere of radius 24 cells, back to back: 0.18 ms
// a call (mark 52 us, clamp 39 us and solid cells 17 us with cold caches, at
// 4.8, 5.2 and 3.9 TB/s; the list kernels 2-10 us each), against 2.43 ms for
// passes over every face with int32 markers (five extension passes of 88 us a
// component, no-flux 118 us, copies).
struct FaceLists {
    uint8_t *layer[3];   // extension bytes (extend_face)
    int *list[3];        // listed faces, in no fixed order
    float *temp[3];      // the no-flux result, by list position
    unsigned *count;     // entries per component
    const float *cw[3];  // collider face weights, or null
};

// appends this lane's faces (`keep` bit m: face f0 + m) to the list; every
// lane of the warp takes part
__device__ __forceinline__ void list_append(unsigned keep, unsigned f0, int *__restrict__ list, unsigned *count) {
    if (!__ballot_sync(0xffffffffu, keep != 0)) return;
    const int lane = threadIdx.x & 31, mine = __popc(keep);
    int s = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += t;
    }
    unsigned base = 0;
    if (lane == 31) base = atomicAdd(count, (unsigned)s);
    base = __shfl_sync(0xffffffffu, base, 31) + (unsigned)(s - mine);
#pragma unroll
    for (int m = 0; m < 4; ++m)
        if (keep >> m & 1) list[base++] = (int)(f0 + m);
}

// makeMarkAndProject (grid_blocked_boundary_condition_solver3.js:196-249):
// open faces are valid; closed faces take the collider's velocity (a static
// collider: 0) and are listed.  Four faces a thread (16-byte weights, one
// word of layer bytes; every array is 256-byte aligned and padded).
__global__ void __launch_bounds__(256) k_mark(Comps3 C, FaceLists L) {
    const int a = blockIdx.z;
    const CompDims &c = C.c[a];
    const float *__restrict__ cw = L.cw[a];
    const unsigned nq = (c.n + 3) / 4, step = gridDim.x * blockDim.x;
    // whole warps step together (list_append shuffles), two quads' loads in flight a thread
    for (unsigned q0 = blockIdx.x * blockDim.x + threadIdx.x; (q0 & ~31u) < nq; q0 += 2 * step) {
        const float4 one = make_float4(1.f, 1.f, 1.f, 1.f);
        const float4 w4[2] = {q0 < nq ? __ldg(reinterpret_cast<const float4 *>(cw) + q0) : one,
                              q0 + step < nq ? __ldg(reinterpret_cast<const float4 *>(cw) + q0 + step) : one};
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const unsigned q = q0 + p * step, f0 = 4 * q;
            const float wv[4] = {w4[p].x, w4[p].y, w4[p].z, w4[p].w};
            unsigned keep = 0, bytes = 0;
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if (f0 + m < c.n && !(wv[m] > 0.0f)) {
                    keep |= 1u << m;
                    bytes |= LAYER_OPEN << (8 * m);
                    C.d[a][f0 + m] = 0.0f;
                }
            if (q < nq) reinterpret_cast<unsigned *>(L.layer[a])[q] = bytes;
            list_append(keep, f0, L.list[a], L.count + a);
        }
    }
}

// whether the no-flux projection replaces a face (makeNoFluxProjection, :251-286)
__device__ __forceinline__ bool face_blocked(const VelField &F, const float *cw, unsigned f, F3 pt) {
    return cw ? (cw[f] <= 0.0f) : (sample_phi(F, F.phi, pt) < 0.0f);
}

// k_mark without collider weights: the open fraction from the SDF on the
// two sides of the face; listed when closed or blocked
__global__ void __launch_bounds__(256, 6) k_mark_sdf(VelField F, Comps3 C, FaceLists L) {
    const int a = blockIdx.z;
    const CompDims &c = C.c[a];
    const F3 o = comp_origin(F.g, a);
    const F3 off{a == 0 ? F.g.hx * 0.5f : 0.0f, a == 1 ? F.g.hy * 0.5f : 0.0f, a == 2 ? F.g.hz * 0.5f : 0.0f};
    for (unsigned f0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); f0 < c.n; f0 += gridDim.x * blockDim.x) {
        const unsigned f = f0 + (threadIdx.x & 31u);
        unsigned keep = 0;
        if (f < c.n) {
            int i, j, k;
            c.at(f, i, j, k);
            const F3 pt = index_pos(F.g, o, i, j, k);
            const float fr = frac_inside_sdf(sample_phi(F, F.phi, F3{pt.x - off.x, pt.y - off.y, pt.z - off.z}),
                                             sample_phi(F, F.phi, F3{pt.x + off.x, pt.y + off.y, pt.z + off.z}));
            const bool open = 1.0f - fminf(fmaxf(fr, 0.0f), 1.0f) > 0.0f;
            if (!open) C.d[a][f] = 0.0f;
            L.layer[a][f] = open ? 0 : LAYER_OPEN;
            keep = (!open || face_blocked(F, nullptr, f, pt)) ? 1u : 0u;
        }
        list_append(keep, f, L.list[a], L.count + a);
    }
}

// extension step t over the listed faces
__global__ void __launch_bounds__(256) k_extend_list(Comps3 C, FaceLists L, int t) {
    const int a = blockIdx.z;
    const unsigned n = L.count[a];
    for (unsigned q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        const unsigned f = (unsigned)L.list[a][q];
        float v;
        if (L.layer[a][f] == LAYER_OPEN && extend_face(C.c[a], C.d[a], L.layer[a], f, t, v)) {
            C.d[a][f] = v;
            L.layer[a][f] = (uint8_t)t;
        }
    }
}

// folds the bytes of the listed faces: valid ones to 0 (steps then count from 1 again)
__global__ void __launch_bounds__(256) k_fold_list(FaceLists L) {
    const int a = blockIdx.z;
    const unsigned n = L.count[a];
    for (unsigned q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        uint8_t &b = L.layer[a][L.list[a][q]];
        if (b != LAYER_OPEN) b = 0;
    }
}

// The faces (or cells) of a component as blocks of 256 take them: tiles of 32 x 8
// on one plane, whose taps share rows in L1 (a run of 256 faces of one row reads
// four times the lines), and the last columns, fewer than 32, as runs over (x, y).
struct TileMap {
    int sx, sy, tiles_x, full;   // full tiles a row of them and a plane
    __host__ __device__ TileMap(int x, int y) : sx(x), sy(y), tiles_x(x / 32), full(x / 32 * ((y + 7) / 8)) {}
    int blocks() const { return full + (int)(((long long)(sx - 32 * tiles_x) * sy + 255) / 256); }
    __device__ __forceinline__ bool at(int &i, int &j) const {
        const int t = threadIdx.x;
        if ((int)blockIdx.x < full) {
            i = (int)(blockIdx.x % (unsigned)tiles_x) * 32 + (t & 31);
            j = (int)(blockIdx.x / (unsigned)tiles_x) * 8 + (t >> 5);
            return j < sy;
        }
        const unsigned w = (unsigned)(sx - 32 * tiles_x), e = (blockIdx.x - full) * 256u + t;
        if (w == 0) return false;
        i = 32 * tiles_x + (int)(e % w);
        j = (int)(e / w);
        return j < sy;
    }
};

// Advection stages, blockIdx.y a component (three faces, or one cell scalar):
//   0 order 1: out = cubic(src @ trace(+1)) where the position is open
//   1 MacCormack forward:  aux = open ? cubic(src @ trace(+1)) : src
//   2 MacCormack backward: aux = open ? cubic(fwd @ trace(-1)) : fwd
//   3 MacCormack correct:  out = clamp(fwd + (src - bwd)/2) where open
// (one kernel per stage: a smaller body for the instruction cache).
struct AdvectIO {
    const float *src[3], *fwd[3], *bwd[3];
    float *out[3];
};
template <int FORM>
__device__ __forceinline__ float advect_phi(const VelField &F, F3 p) {
    if constexpr (FORM == FORM_PLAIN) return sample_phi(F, F.phi, p);
    else return trace_phi<FORM == FORM_SHORT_P2>(F, p);
}
template <int FORM>
__device__ __forceinline__ float advect_cubic(const VelField &F, int a, const float *d, int sx, int sy, int sz, F3 o, F3 p) {
    if constexpr (FORM == FORM_PLAIN) return tricubic(d, sx, sy, sz, F.g, o, p);
    else return trace_cubic<FORM == FORM_SHORT_P2>(F, a, d, sx, sy, sz, o, p);
}
template <int stage, int FORM>
__device__ __forceinline__ void advect_at(const VelField &F, int a, const AdvectIO &io, int q, int sx, int sy, int sz, F3 o,
                                          long long f, int i, int j, int k, float dt, int max_substeps) {
    const float *src = io.src[q], *fwd = io.fwd[q], *bwd = io.bwd[q];
    float *out = io.out[q];
    const F3 pos = index_pos(F.g, o, i, j, k);
    const float phi = advect_phi<FORM>(F, pos);
    const bool open = phi > 0.0f;
    auto traced = [&](const float *d, float dirn) {
        return advect_cubic<FORM>(F, a, d, sx, sy, sz, o, trace_back<FORM>(F, pos, dt, dirn, max_substeps, phi));
    };
    if constexpr (stage == 0) {
        if (open) out[f] = traced(src, 1.0f);
    } else if constexpr (stage == 1) {
        out[f] = open ? traced(src, 1.0f) : src[f];
    } else if constexpr (stage == 2) {
        out[f] = open ? traced(fwd, -1.0f) : fwd[f];
    } else if (open) {
        // clampCorrection (stage 3): min/max over the 8 trilinear corners of the
        // traced point whose own positions are open
        const F3 tr = trace_back<FORM>(F, pos, dt, 1.0f, max_substeps, phi);
        const float fv = fwd[f];
        const float corr = fv + (src[f] - bwd[f]) * 0.5f;
        const float gx = gclamp((tr.x - o.x) / F.g.hx), gy = gclamp((tr.y - o.y) / F.g.hy),
                    gz = gclamp((tr.z - o.z) / F.g.hz);
        const int i0 = (int)floorf(gx), j0 = (int)floorf(gy), k0 = (int)floorf(gz);
        const int ic[2] = {iclamp(i0, 0, sx - 1), iclamp(i0 + 1, 0, sx - 1)};
        const int jc[2] = {iclamp(j0, 0, sy - 1), iclamp(j0 + 1, 0, sy - 1)};
        const int kc[2] = {iclamp(k0, 0, sz - 1), iclamp(k0 + 1, 0, sz - 1)};
        float mn = 1e30f, mx = -1e30f;
        bool have = false;
        auto corner = [&](int c) {
            const int ni = ic[c & 1], nj = jc[(c >> 1) & 1], nk = kc[(c >> 2) & 1];
            const bool valid = advect_phi<FORM>(F, index_pos(F.g, o, ni, nj, nk)) > 0.0f;
            const float val = src[ni + (long long)sx * (nj + (long long)sy * nk)];
            if (valid) {
                mn = fminf(mn, val);
                mx = fmaxf(mx, val);
                have = true;
            }
        };
        if constexpr (FORM == FORM_PLAIN) {
#pragma unroll
            for (int c = 0; c < 8; ++c) corner(c);
        } else {
#pragma unroll 1
            for (int c = 0; c < 8; ++c) corner(c);
        }
        out[f] = (have && corr >= mn && corr <= mx) ? corr : fv;
    }
}
// The short form: bound by issue (78% of the slots, 2100 instructions a face at two to
// three substeps; DRAM 4%): order 1 on the 16.8M faces of one component of a 256^3
// grid takes 1.08 ms, 1.55 ms in the straightforward form.  Of that 0.1 ms is the
// short form itself; the rest came with one copy of the trace's sample and of the
// tricubic's plane pair in the code (a third of all issue slots had waited for
// instructions), arguments read in place instead of from a local copy, and floor
// as an addition.
template <int stage, int FORM>
__global__ void __launch_bounds__(256) k_advect(const __grid_constant__ VelField F, int a0, const __grid_constant__ AdvectIO io,
                                                float dt, int max_substeps, int z0) {
    const int a = a0 + (int)blockIdx.y, k = z0 + (int)blockIdx.z;
    int sx, sy, sz, i, j;
    if (a < 3) comp_shape(F.g, a, sx, sy, sz);
    else sx = F.g.nx, sy = F.g.ny, sz = F.g.nz;
    if (k >= sz || !TileMap(sx, sy).at(i, j)) return;
    advect_at<stage, FORM>(F, a, io, blockIdx.y, sx, sy, sz, comp_origin(F.g, a), i + (long long)sx * (j + (long long)sy * k), i,
                           j, k, dt, max_substeps);
}
// The straightforward form, runs of 256 faces, where the short one does not pay.  64
// registers, as a small grid is bound by one warp's latency (48, the compiler's choice:
// 32^3 with a collider 13.2 us, 12.1 so).  In the short form a warp that touches an end of
// the arrays takes the straightforward sample there, so its gain goes with the share of
// the warps (32 faces of a row) that touch none, and a spacing that is no power of two
// costs it the corrected quotients.  Straightforward over short, all faces and a scalar,
// both orders, 0.3 and 1.6 cells a step, with and without a collider (least and most):
//   power of two:  112^3 (share 0.41) 1.03-1.23, 128^3 1.03-1.23, 256 x 256 x 16 1.08-1.21,
//                  160^3 1.12-1.32, 256^3 1.24-1.56; 64 x 1024 x 64 (share 0) 0.93-1.09,
//                  512 x 512 x 4 (0.22) 0.97-1.14, 2048 x 1024 x 2 (0) 0.87-1.08
//   any spacing:   112^3 0.92-1.02, 144^3 (0.53) 0.99-1.14, 256 x 256 x 16 (0.60, 1.05M
//                  cells) 0.96-1.10, 160^3 (0.58) 1.00-1.14, 200^3 1.10-1.29, 256^3 1.14-1.39;
//                  64 x 1024 x 64 0.81-0.93, 2048 x 1024 x 2 0.79-0.90
// and below a million cells it was slower throughout (33 x 43 x 49 41 us against 32).
int advect_form(const VelField &F) {
    const double nx = F.g.nx, ny = F.g.ny, nz = F.g.nz;
    const double share = std::max(0.0, nx - 64) / nx * std::max(0.0, ny - 3) / ny * std::max(0.0, nz - 3) / nz;
    const double cells = nx * ny * nz;
    if (F.pow2) return cells >= 1 << 20 && share >= 0.4 ? FORM_SHORT_P2 : FORM_PLAIN;
    return cells >= 1 << 21 && share >= 0.55 ? FORM_SHORT : FORM_PLAIN;
}
template <int stage>
__global__ void __launch_bounds__(256, 4) k_advect_plain(const __grid_constant__ VelField F, int a0, const __grid_constant__ AdvectIO io, float dt,
                               int max_substeps) {
    const int a = a0 + (int)blockIdx.y;
    int sx, sy, sz, i, j, k;
    if (a < 3) comp_shape(F.g, a, sx, sy, sz);
    else sx = F.g.nx, sy = F.g.ny, sz = F.g.nz;
    const long long n = (long long)sx * sy * sz;
    const F3 o = comp_origin(F.g, a);
    for (long long f = blockIdx.x * (long long)blockDim.x + threadIdx.x; f < n; f += (long long)gridDim.x * blockDim.x) {
        unflatten(f, sx, sy, i, j, k);
        advect_at<stage, FORM_PLAIN>(F, a, io, blockIdx.y, sx, sy, sz, o, f, i, j, k, dt, max_substeps);
    }
}

// trace(start, direction) of a list of points (float3 per point)
template <int FORM>
__global__ void __launch_bounds__(256, 4) k_trace(const __grid_constant__ VelField F, long long n, const float *__restrict__ pin,
                                                  float *__restrict__ pout, float dt, float dirn, int max_substeps) {
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const F3 r = trace_back<FORM>(F, F3{pin[3 * q], pin[3 * q + 1], pin[3 * q + 2]}, dt, dirn, max_substeps, NAN);
        pout[3 * q] = r.x;
        pout[3 * q + 1] = r.y;
        pout[3 * q + 2] = r.z;
    }
}

// makeNoFluxProjection (:251-286) with projectAndApplyFriction (:30-44)
// over the listed faces: a blocked face takes the tangential part of the
// sampled velocity, reduced by Coulomb friction (coefficient 0.5,
// sdf_collider3.js:16).  The samples read the values of all components
// before any face is replaced, so the results wait in temp.
__global__ void __launch_bounds__(256) k_noflux(VelField F, Comps3 C, FaceLists L) {
    const int a = blockIdx.z;
    const CompDims &c = C.c[a];
    const unsigned n = L.count[a];
    const F3 o = comp_origin(F.g, a), oc = comp_origin(F.g, 3);
    for (unsigned q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        const unsigned f = (unsigned)L.list[a][q];
        int i, j, k;
        c.at(f, i, j, k);
        const F3 pt = index_pos(F.g, o, i, j, k);
        float res = C.d[a][f];
        if (face_blocked(F, L.cw[a], f, pt)) {
            const F3 vel = sample_vel(F, pt);
            const F3 gr = trilinear_gradient(F.phi, F.g, oc, pt);
            const float gl = sqrtf(gr.x * gr.x + gr.y * gr.y + gr.z * gr.z);
            res = 0.0f;
            if (gl > 0.0f) {
                const F3 nn{gr.x / gl, gr.y / gl, gr.z / gl};
                const float vn = vel.x * nn.x + vel.y * nn.y + vel.z * nn.z;
                F3 vt{vel.x - nn.x * vn, vel.y - nn.y * vn, vel.z - nn.z * vn};
                const float tl = sqrtf(vt.x * vt.x + vt.y * vt.y + vt.z * vt.z);
                if (tl > 0.0f) {
                    const float veln = fmaxf(-vn, 0.0f);
                    const float scale = fmaxf(1.0f - veln * 0.5f / tl, 0.0f);
                    vt = F3{vt.x * scale, vt.y * scale, vt.z * scale};
                }
                res = a == 0 ? vt.x : (a == 1 ? vt.y : vt.z);
            }
        }
        L.temp[a][q] = res;
    }
}
__global__ void __launch_bounds__(256) k_noflux_write(Comps3 C, FaceLists L) {
    const int a = blockIdx.z;
    const unsigned n = L.count[a];
    for (unsigned q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x)
        C.d[a][L.list[a][q]] = L.temp[a][q];
}

// blockedBoundary (:288-330): a collider cell's faces toward fluid cells
// take the collider velocity (0).  Four cells a thread; a cell outside the
// collider costs its share of one 16-byte load.
__global__ void __launch_bounds__(256) k_blocked(G3 g, CompDims c, const float *__restrict__ phi, float *u, float *v,
                                                 float *w) {
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const unsigned nq = (c.n + 3) / 4;
    for (unsigned q = blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += gridDim.x * blockDim.x) {
        const float4 p4 = __ldg(reinterpret_cast<const float4 *>(phi) + q);
        if (!(p4.x < 0.0f || p4.y < 0.0f || p4.z < 0.0f || p4.w < 0.0f)) continue;
        const float pv[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const unsigned f = 4 * q + m;
            if (f >= c.n || !(pv[m] < 0.0f)) continue;
            int i, j, k;
            c.at(f, i, j, k);
            auto solid = [&](int ii, int jj, int kk) { return phi[ii + nx * (jj + ny * kk)] < 0.0f; };
            if (i > 0 && !solid(i - 1, j, k)) u[i + (nx + 1) * (j + ny * k)] = 0.0f;
            if (i < nx - 1 && !solid(i + 1, j, k)) u[i + 1 + (nx + 1) * (j + ny * k)] = 0.0f;
            if (j > 0 && !solid(i, j - 1, k)) v[i + nx * (j + (ny + 1) * k)] = 0.0f;
            if (j < ny - 1 && !solid(i, j + 1, k)) v[i + nx * (j + 1 + (ny + 1) * k)] = 0.0f;
            if (k > 0 && !solid(i, j, k - 1)) w[i + nx * (j + ny * k)] = 0.0f;
            if (k < nz - 1 && !solid(i, j, k + 1)) w[i + nx * (j + ny * (k + 1))] = 0.0f;
        }
    }
}

// the clamp (clampComponent, |v| <= 100, non-finite -> 0) after the walls
// (zeroULeft .. zeroWFront)
__device__ __forceinline__ float clamp_vel(float val) {
    return (isnan(val) || isinf(val)) ? 0.0f : fminf(fmaxf(val, -100.0f), 100.0f);
}
__device__ __forceinline__ bool closed_face(const CompDims &c, int a, int closed, int i, int j, int k) {
    const int idx = a == 0 ? i : (a == 1 ? j : k), last = (a == 0 ? c.sx : (a == 1 ? c.sy : c.sz)) - 1;
    return (((closed >> (2 * a)) & 1) && idx == 0) || (((closed >> (2 * a + 1)) & 1) && idx == last);
}
// walls and clamp, four faces a thread (two quads' loads in flight); a face
// is written only when its bits change.  Most quads hold no wall face and no
// value to clamp: a test on the index along the component's axis and one on
// the magnitudes dismiss them, which keeps the pass near its read of the
// values (with the full test on each face it was bound by issue: 62 us for
// 256^3, cold).
__global__ void __launch_bounds__(256) k_walls_clamp(Comps3 C, int closed) {
    const int a = blockIdx.z;
    const CompDims &c = C.c[a];
    float *__restrict__ data = C.d[a];
    const unsigned nq = (c.n + 3) / 4, step = gridDim.x * blockDim.x;
    const unsigned plane = (unsigned)c.sx * (unsigned)c.sy;
    for (unsigned q0 = blockIdx.x * blockDim.x + threadIdx.x; q0 < nq; q0 += 2 * step) {
        const bool two = q0 + step < nq;
        const float4 v4[2] = {reinterpret_cast<const float4 *>(data)[q0],
                              two ? reinterpret_cast<const float4 *>(data)[q0 + step] : make_float4(0.f, 0.f, 0.f, 0.f)};
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const unsigned f0 = 4 * (q0 + p * step);
            const float vv[4] = {v4[p].x, v4[p].y, v4[p].z, v4[p].w};
            // no value to clamp: |v| <= 100 fails for a NaN too
            const bool plain = fabsf(vv[0]) <= 100.0f && fabsf(vv[1]) <= 100.0f && fabsf(vv[2]) <= 100.0f &&
                               fabsf(vv[3]) <= 100.0f;
            // whether f0 .. f0 + 3 can hold a face of the axis' end planes
            bool edge;
            const unsigned r = c.dx.div(f0);
            if (a == 0) {
                const unsigned i = f0 - r * (unsigned)c.sx;
                edge = i == 0 || i + 4 >= (unsigned)c.sx;
            } else if (a == 1) {
                const unsigned j = r - c.dy.div(r) * (unsigned)c.sy;
                edge = j == 0 || j + 5 >= (unsigned)c.sy;
            } else {
                edge = f0 < plane || f0 + 4 >= c.n - plane;
            }
            if (plain && !edge) continue;
            if (f0 >= c.n) break;
            int i, j, k;
            c.at(f0, i, j, k);
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const float w = clamp_vel(closed_face(c, a, closed, i, j, k) ? 0.0f : vv[m]);
                if (__float_as_uint(w) != __float_as_uint(vv[m]) && f0 + m < c.n) data[f0 + m] = w;
                if (++i == c.sx) {
                    i = 0;
                    if (++j == c.sy) j = 0, ++k;
                }
            }
        }
    }
}
// the same with inflows (buildInflowKernels) between the walls and the clamp
__global__ void __launch_bounds__(256, 6) k_walls_inflow_clamp(G3 g, Comps3 C, int closed, int n_in,
                                                               const float *const *__restrict__ in_phi,
                                                               const float *__restrict__ in_vel,
                                                               const int *__restrict__ in_mode) {
    const int a = blockIdx.z;
    const CompDims &c = C.c[a];
    float *__restrict__ data = C.d[a];
    const F3 o = comp_origin(g, a);
    const VelField F{g, nullptr, nullptr, nullptr, nullptr};
    for (unsigned f = blockIdx.x * blockDim.x + threadIdx.x; f < c.n; f += gridDim.x * blockDim.x) {
        int i, j, k;
        c.at(f, i, j, k);
        const float old = data[f];
        float val = closed_face(c, a, closed, i, j, k) ? 0.0f : old;
        const F3 pt = index_pos(g, o, i, j, k);
        for (int q = 0; q < n_in; ++q) {
            if (sample_phi(F, in_phi[q], pt) < 0.0f) {
                const float add = in_vel[3 * q + a];
                val = in_mode[q] ? val + add : add;
            }
        }
        val = clamp_vel(val);
        if (__float_as_uint(val) != __float_as_uint(old)) data[f] = val;
    }
}

// explicit viscosity: out = in + (dt nu) lap(in) inside the component's own
// axis range, Neumann past the array ends; the component's boundary planes
// copy through
__global__ void k_viscosity(G3 g, int a, const float *__restrict__ in, float *__restrict__ out, float c, float ihx,
                            float ihy, float ihz) {
    int s[3];
    comp_shape(g, a, s[0], s[1], s[2]);
    const long long n = (long long)s[0] * s[1] * s[2];
    const long long st[3] = {1, s[0], (long long)s[0] * s[1]};
    const float ih[3] = {ihx, ihy, ihz};
    for (long long f = blockIdx.x * (long long)blockDim.x + threadIdx.x; f < n; f += (long long)gridDim.x * blockDim.x) {
        int idx[3];
        unflatten(f, s[0], s[1], idx[0], idx[1], idx[2]);
        const float x = in[f];
        if (idx[a] == 0 || idx[a] == s[a] - 1) {
            out[f] = x;
            continue;
        }
        float lap = 0.0f;
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const float up = idx[b] + 1 < s[b] ? in[f + st[b]] : x;
            const float dn = idx[b] > 0 ? in[f - st[b]] : x;
            lap = lap + ((up - x) + (dn - x)) * ih[b];
        }
        out[f] = x + c * lap;
    }
}

int launch_blocks(long long n) { return (int)std::min<long long>((n + 255) / 256, 152LL * 16); }

int post(const char *what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return ff_set_error(FF_E_CUDA, "%s launch: %s", what, cudaGetErrorString(e));
    return FF_OK;
}

G3 geom_of(const int *res, const double *h, const double *o) {
    G3 g;
    g.nx = res[0];
    g.ny = res[1];
    g.nz = res[2];
    g.hx = (float)h[0];
    g.hy = (float)h[1];
    g.hz = (float)h[2];
    g.ox = o ? (float)o[0] : 0.0f;
    g.oy = o ? (float)o[1] : 0.0f;
    g.oz = o ? (float)o[2] : 0.0f;
    return g;
}

long long comp_count(const G3 &g, int a) {
    int sx, sy, sz;
    if (a == 3) return (long long)g.nx * g.ny * g.nz;
    comp_shape(g, a, sx, sy, sz);
    return (long long)sx * sy * sz;
}

bool field_is(ff_field f, long long count) { return f && f->dtype == FF_FLOAT && f->count == count; }

}  // namespace

// ----------------------------------------------------------------- advect --
struct ff_advect_s {
    ff_ctx ctx = nullptr;
    ff_advect_desc desc{};
    G3 g{};
    ff_field phi = nullptr;           // borrowed
    float *fwd[4] = {}, *bwd[4] = {};  // order-2 scratch per component (3 = scalar)
};

extern "C" int ff_advect3_create(ff_ctx ctx, const ff_advect_desc *d, ff_advect *out) {
    FF_CHECK(ctx && d && out, FF_E_ARG, "ff_advect3_create: NULL argument");
    FF_CHECK(d->resolution[0] > 0 && d->resolution[1] > 0 && d->resolution[2] > 0, FF_E_ARG,
             "createSemiLagrangianAdvectionSolver3: resolution must be positive");
    FF_CHECK(d->order == 1 || d->order == 2, FF_E_ARG, "createSemiLagrangianAdvectionSolver3: order must be 1 or 2");
    FF_CHECK(d->max_substeps > 0, FF_E_ARG, "createSemiLagrangianAdvectionSolver3: maxSubsteps must be positive");
    FF_TRY(check_grid32(d->resolution, "createSemiLagrangianAdvectionSolver3"));
    *out = nullptr;
    cudaSetDevice(ctx->device);
    ff_advect a = new ff_advect_s();
    a->ctx = ctx;
    a->desc = *d;
    a->g = geom_of(d->resolution, d->grid_spacing, d->origin);
    if (d->order == 2) {
        for (int c = 0; c < 4; ++c) {
            size_t bytes = (size_t)comp_count(a->g, c) * 4;
            int st = ff_dev_alloc((void **)&a->fwd[c], bytes, ctx->stream);
            if (st == FF_OK) st = ff_dev_alloc((void **)&a->bwd[c], bytes, ctx->stream);
            if (st != FF_OK) {
                ff_advect3_destroy(a);
                return st;
            }
        }
    }
    *out = a;
    return FF_OK;
}

extern "C" int ff_advect3_destroy(ff_advect a) {
    if (!a) return FF_OK;
    cudaStreamSynchronize(a->ctx->stream);
    for (int c = 0; c < 4; ++c) {
        ff_dev_free(a->fwd[c]);
        ff_dev_free(a->bwd[c]);
    }
    delete a;
    return FF_OK;
}

extern "C" int ff_advect3_set_dt(ff_advect a, double dt) {
    FF_CHECK(a, FF_E_ARG, "NULL advection solver");
    a->desc.dt = dt;
    return FF_OK;
}

extern "C" int ff_advect3_set_collider(ff_advect a, ff_field phi) {
    FF_CHECK(a, FF_E_ARG, "NULL advection solver");
    FF_CHECK(!phi || field_is(phi, comp_count(a->g, 3)), FF_E_ARG, "collider SDF must be a float cell field");
    a->phi = phi;
    return FF_OK;
}

// components a0 .. a0 + na - 1, one launch a stage
static int advect_components(ff_advect a, const VelField &F, int a0, int na, const float *const *src, float *const *out) {
    cudaStream_t s = a->ctx->stream;
    const float dt = (float)a->desc.dt;
    const int ms = a->desc.max_substeps, form = advect_form(F);
    long long n = 0;
    int planes = 0, blocks = 0;
    AdvectIO io{};
    for (int q = 0; q < na; ++q) {
        const int c = a0 + q;
        int sx = a->g.nx, sy = a->g.ny, sz = a->g.nz;
        if (c < 3) comp_shape(a->g, c, sx, sy, sz);
        n = std::max(n, (long long)sx * sy * sz);
        planes = std::max(planes, sz);
        blocks = std::max(blocks, TileMap(sx, sy).blocks());
        io.src[q] = src[q];
    }
    auto run = [&](auto stage, float *const *to) {
        constexpr int st = decltype(stage)::value;
        for (int q = 0; q < na; ++q) {
            io.fwd[q] = a->fwd[a0 + q];
            io.bwd[q] = a->bwd[a0 + q];
            io.out[q] = to[q];
        }
        if (form == FORM_PLAIN) {
            k_advect_plain<st><<<dim3((unsigned)launch_blocks(n), (unsigned)na), 256, 0, s>>>(F, a0, io, dt, ms);
            return;
        }
        const auto kernel = form == FORM_SHORT_P2 ? k_advect<st, FORM_SHORT_P2> : k_advect<st, FORM_SHORT>;
        for (int z0 = 0; z0 < planes; z0 += 65535)
            kernel<<<dim3((unsigned)blocks, (unsigned)na, (unsigned)std::min(65535, planes - z0)), 256, 0, s>>>(F, a0, io, dt,
                                                                                                              ms, z0);
    };
    if (a->desc.order == 1) {
        run(std::integral_constant<int, 0>(), out);
        return post("advect");
    }
    run(std::integral_constant<int, 1>(), a->fwd + a0);
    run(std::integral_constant<int, 2>(), a->bwd + a0);
    run(std::integral_constant<int, 3>(), out);
    return post("advect (MacCormack)");
}

static bool overlap(ff_field a, ff_field b) {
    const char *p = (const char *)a->d, *q = (const char *)b->d;
    return p < q + b->bytes && q < p + a->bytes;
}

extern "C" int ff_advect3_faces(ff_advect a, ff_field vu, ff_field vv, ff_field vw, ff_field iu, ff_field iv,
                                ff_field iw, ff_field ou, ff_field ov, ff_field ow) {
    FF_CHECK(a, FF_E_ARG, "NULL advection solver");
    ff_field vel[3] = {vu, vv, vw}, in[3] = {iu, iv, iw}, out[3] = {ou, ov, ow};
    for (int c = 0; c < 3; ++c)
        FF_CHECK(field_is(vel[c], comp_count(a->g, c)) && field_is(in[c], comp_count(a->g, c)) &&
                     field_is(out[c], comp_count(a->g, c)),
                 FF_E_ARG, "advectFaceCentered3: face field %d has the wrong shape or type", c);
    for (int c = 0; c < 3; ++c)
        FF_CHECK(out[c]->d != in[c]->d && out[c]->d != vel[c]->d, FF_E_ARG,
                 "advectFaceCentered3: output must not alias the input or the velocity");
    cudaSetDevice(a->ctx->device);
    const VelField F = trace_field({a->g, (const float *)vu->d, (const float *)vv->d, (const float *)vw->d,
                                    a->phi ? (const float *)a->phi->d : nullptr});
    const float *src[3] = {(const float *)iu->d, (const float *)iv->d, (const float *)iw->d};
    float *dst[3] = {(float *)ou->d, (float *)ov->d, (float *)ow->d};
    // fields that overlap across components: one after the other, as they are used
    bool apart = true;
    for (int c = 0; c < 3; ++c)
        for (int q = 0; q < 3; ++q)
            if (q != c)
                apart = apart && !overlap(out[c], in[q]) && !overlap(out[c], vel[q]) && !overlap(out[c], out[q]);
    if (apart) return advect_components(a, F, 0, 3, src, dst);
    for (int c = 0; c < 3; ++c) FF_TRY(advect_components(a, F, c, 1, src + c, dst + c));
    return FF_OK;
}

extern "C" int ff_advect3_scalar(ff_advect a, ff_field vu, ff_field vv, ff_field vw, ff_field s_in, ff_field s_out) {
    FF_CHECK(a, FF_E_ARG, "NULL advection solver");
    for (int c = 0; c < 3; ++c)
        FF_CHECK(field_is(c == 0 ? vu : (c == 1 ? vv : vw), comp_count(a->g, c)), FF_E_ARG,
                 "advectScalar3: velocity component %d has the wrong shape", c);
    FF_CHECK(field_is(s_in, comp_count(a->g, 3)) && field_is(s_out, comp_count(a->g, 3)) && s_in->d != s_out->d,
             FF_E_ARG, "advectScalar3: scalar fields must be distinct float cell fields");
    cudaSetDevice(a->ctx->device);
    const VelField F = trace_field({a->g, (const float *)vu->d, (const float *)vv->d, (const float *)vw->d,
                                    a->phi ? (const float *)a->phi->d : nullptr});
    const float *src = (const float *)s_in->d;
    float *dst = (float *)s_out->d;
    return advect_components(a, F, 3, 1, &src, &dst);
}

extern "C" int ff_advect3_trace(ff_advect a, ff_field vu, ff_field vv, ff_field vw, ff_field p_in, ff_field p_out,
                                int direction) {
    FF_CHECK(a && p_in && p_out, FF_E_ARG, "NULL argument");
    for (int c = 0; c < 3; ++c)
        FF_CHECK(field_is(c == 0 ? vu : (c == 1 ? vv : vw), comp_count(a->g, c)), FF_E_ARG,
                 "trace: velocity component %d has the wrong shape", c);
    FF_CHECK(p_in->dtype == FF_VEC3 && p_out->dtype == FF_VEC3 && p_in->count == p_out->count, FF_E_ARG,
             "trace: points must be vec3 fields of equal length");
    FF_CHECK(direction == 1 || direction == -1, FF_E_ARG, "trace: direction must be 1 or -1");
    cudaSetDevice(a->ctx->device);
    const VelField F = trace_field({a->g, (const float *)vu->d, (const float *)vv->d, (const float *)vw->d,
                                    a->phi ? (const float *)a->phi->d : nullptr});
    const long long n = p_in->count;
    if (n == 0) return FF_OK;
    const int form = point_form(F, n);
    const auto kernel = form == FORM_PLAIN ? k_trace<FORM_PLAIN> : form == FORM_SHORT ? k_trace<FORM_SHORT> : k_trace<FORM_SHORT_P2>;
    kernel<<<launch_blocks(n), 256, 0, a->ctx->stream>>>(F, n, (const float *)p_in->d, (float *)p_out->d,
                                                         (float)a->desc.dt, (float)direction, a->desc.max_substeps);
    return post("trace");
}

// --------------------------------------------------------------------- bc --
struct ff_bc_s {
    ff_ctx ctx = nullptr;
    G3 g{};
    int closed = 63;                       // DIRECTION_ALL_3D
    ff_field phi = nullptr, cw[3] = {};    // borrowed
    FaceLists lists{};                     // work arrays (cw filled in per call)
    int n_in = 0;
    const float **in_phi = nullptr;        // device array of n_in pointers
    float *in_vel = nullptr;
    int *in_mode = nullptr;
};

extern "C" int ff_bc3_create(ff_ctx ctx, const int *res, const double *h, const double *origin, ff_bc *out) {
    FF_CHECK(ctx && res && h && out, FF_E_ARG, "ff_bc3_create: NULL argument");
    FF_CHECK(res[0] > 0 && res[1] > 0 && res[2] > 0, FF_E_ARG, "createGridBlockedBoundaryConditionSolver3: bad resolution");
    FF_TRY(check_grid32(res, "createGridBlockedBoundaryConditionSolver3"));
    *out = nullptr;
    cudaSetDevice(ctx->device);
    ff_bc b = new ff_bc_s();
    b->ctx = ctx;
    b->g = geom_of(res, h, origin);
    int st = FF_OK;
    for (int a = 0; a < 3 && st == FF_OK; ++a) {
        const size_t n = (size_t)comp_count(b->g, a);
        st = ff_dev_alloc((void **)&b->lists.layer[a], n, ctx->stream);
        if (st == FF_OK) st = ff_dev_alloc((void **)&b->lists.list[a], n * 4, ctx->stream);
        if (st == FF_OK) st = ff_dev_alloc((void **)&b->lists.temp[a], n * 4, ctx->stream);
    }
    if (st == FF_OK) st = ff_dev_alloc((void **)&b->lists.count, 3 * sizeof(unsigned), ctx->stream);
    if (st != FF_OK) {
        ff_bc3_destroy(b);
        return st;
    }
    *out = b;
    return FF_OK;
}

extern "C" int ff_bc3_destroy(ff_bc b) {
    if (!b) return FF_OK;
    cudaStreamSynchronize(b->ctx->stream);
    for (int a = 0; a < 3; ++a) {
        ff_dev_free(b->lists.layer[a]);
        ff_dev_free(b->lists.list[a]);
        ff_dev_free(b->lists.temp[a]);
    }
    ff_dev_free(b->lists.count);
    ff_dev_free((void *)b->in_phi);
    ff_dev_free(b->in_vel);
    ff_dev_free(b->in_mode);
    delete b;
    return FF_OK;
}

extern "C" int ff_bc3_set_collider(ff_bc b, ff_field phi, ff_field wu, ff_field wv, ff_field ww) {
    FF_CHECK(b, FF_E_ARG, "NULL boundary solver");
    FF_CHECK(!phi || field_is(phi, comp_count(b->g, 3)), FF_E_ARG, "setCollider: SDF must be a float cell field");
    ff_field w[3] = {wu, wv, ww};
    FF_CHECK((!wu && !wv && !ww) || (wu && wv && ww), FF_E_ARG, "setCollider: give all three face weights or none");
    for (int a = 0; a < 3; ++a)
        FF_CHECK(!w[a] || field_is(w[a], comp_count(b->g, a)), FF_E_ARG, "setCollider: face weight %d shape", a);
    b->phi = phi;
    for (int a = 0; a < 3; ++a) b->cw[a] = phi ? w[a] : nullptr;
    return FF_OK;
}

extern "C" int ff_bc3_set_closed(ff_bc b, int flags) {
    FF_CHECK(b, FF_E_ARG, "NULL boundary solver");
    FF_CHECK(flags >= 0 && flags <= 63, FF_E_ARG, "closedDomainBoundaryFlag must be a DIRECTION_* mask");
    b->closed = flags;
    return FF_OK;
}

extern "C" int ff_bc3_set_inflows(ff_bc b, int n, const ff_field *phis, const double *velocities, const int *modes) {
    FF_CHECK(b && n >= 0 && (n == 0 || (phis && velocities && modes)), FF_E_ARG, "setInflows: bad arguments");
    FF_CHECK(n <= 64, FF_E_LIMIT, "setInflows: at most 64 inflows");
    std::vector<const float *> hp(n);
    std::vector<float> hv(3 * n);
    std::vector<int> hm(n);
    for (int q = 0; q < n; ++q) {
        FF_CHECK(field_is(phis[q], comp_count(b->g, 3)), FF_E_ARG, "setInflows: inflow %d SDF must be a float cell field", q);
        FF_CHECK(modes[q] == 0 || modes[q] == 1, FF_E_ARG, "setInflows: mode must be 0 (set) or 1 (add)");
        hp[q] = (const float *)phis[q]->d;
        for (int c = 0; c < 3; ++c) hv[3 * q + c] = (float)velocities[3 * q + c];
        hm[q] = modes[q];
    }
    cudaStream_t s = b->ctx->stream;
    FF_CUDA(cudaStreamSynchronize(s));
    ff_dev_free((void *)b->in_phi);
    ff_dev_free(b->in_vel);
    ff_dev_free(b->in_mode);
    b->in_phi = nullptr;
    b->in_vel = nullptr;
    b->in_mode = nullptr;
    b->n_in = 0;
    if (n == 0) return FF_OK;
    FF_TRY(ff_dev_alloc((void **)&b->in_phi, sizeof(float *) * n, s));
    FF_TRY(ff_dev_alloc((void **)&b->in_vel, sizeof(float) * 3 * n, s));
    FF_TRY(ff_dev_alloc((void **)&b->in_mode, sizeof(int) * n, s));
    FF_CUDA(cudaMemcpyAsync((void *)b->in_phi, hp.data(), sizeof(float *) * n, cudaMemcpyHostToDevice, s));
    FF_CUDA(cudaMemcpyAsync(b->in_vel, hv.data(), sizeof(float) * 3 * n, cudaMemcpyHostToDevice, s));
    FF_CUDA(cudaMemcpyAsync(b->in_mode, hm.data(), sizeof(int) * n, cudaMemcpyHostToDevice, s));
    FF_CUDA(cudaStreamSynchronize(s));
    b->n_in = n;
    return FF_OK;
}

// constrainVelocity(extrapolationDepth) (:427-477), in place on (u, v, w)
extern "C" int ff_bc3_constrain(ff_bc b, ff_field u, ff_field v, ff_field w, int depth) {
    FF_CHECK(b, FF_E_ARG, "NULL boundary solver");
    FF_CHECK(depth >= 0, FF_E_ARG, "constrainVelocity: depth must be >= 0");
    ff_field fs[3] = {u, v, w};
    for (int a = 0; a < 3; ++a)
        FF_CHECK(field_is(fs[a], comp_count(b->g, a)), FF_E_ARG, "constrainVelocity: velocity component %d shape", a);
    cudaSetDevice(b->ctx->device);
    cudaStream_t s = b->ctx->stream;
    Comps3 C;
    long long nmax = 0;
    for (int a = 0; a < 3; ++a) {
        C.c[a] = comp_dims(b->g, a);
        C.d[a] = (float *)fs[a]->d;
        nmax = std::max(nmax, comp_count(b->g, a));
    }
    const VelField F{b->g, C.d[0], C.d[1], C.d[2], b->phi ? (const float *)b->phi->d : nullptr};
    const dim3 faces(launch_blocks(nmax), 1, 3), quads(launch_blocks((nmax + 3) / 4), 1, 3);
    if (b->phi) {
        FaceLists L = b->lists;
        for (int a = 0; a < 3; ++a) L.cw[a] = b->cw[a] ? (const float *)b->cw[a]->d : nullptr;
        // the lists' lengths stay on the device: two blocks an SM and component
        const dim3 listed((unsigned)std::min<long long>((nmax + 255) / 256, 152LL * 2), 1, 3);
        FF_CUDA(cudaMemsetAsync(L.count, 0, 3 * sizeof(unsigned), s));
        if (L.cw[0]) k_mark<<<quads, 256, 0, s>>>(C, L);
        else k_mark_sdf<<<faces, 256, 0, s>>>(F, C, L);
        for (int it = 0, t = 1; it < depth; ++it, ++t) {
            if (t > LAYER_STEPS) {
                k_fold_list<<<listed, 256, 0, s>>>(L);
                t = 1;
            }
            k_extend_list<<<listed, 256, 0, s>>>(C, L, t);
        }
        k_noflux<<<listed, 256, 0, s>>>(F, C, L);
        k_noflux_write<<<listed, 256, 0, s>>>(C, L);
        k_blocked<<<launch_blocks((comp_count(b->g, 3) + 3) / 4), 256, 0, s>>>(b->g, comp_dims(b->g, 3), F.phi, C.d[0],
                                                                              C.d[1], C.d[2]);
    }
    if (b->n_in)
        k_walls_inflow_clamp<<<faces, 256, 0, s>>>(b->g, C, b->closed, b->n_in, b->in_phi, b->in_vel, b->in_mode);
    else
        k_walls_clamp<<<quads, 256, 0, s>>>(C, b->closed);
    return post("constrainVelocity");
}

// ------------------------------------------------------------ forces --
namespace {
__global__ void k_add_const(long long n, float *__restrict__ d, float fdt) {
    for (long long f = blockIdx.x * (long long)blockDim.x + threadIdx.x; f < n; f += (long long)gridDim.x * blockDim.x)
        d[f] = d[f] + fdt;
}
}  // namespace

// createExternalForceSolver3 (external_force_solver3.js:7-29) with a
// uniform force: u += f.x dt on every face of each component
extern "C" int ff_velocity3_add_force(ff_ctx ctx, const int *res, ff_field u, ff_field v, ff_field w, double fx,
                                      double fy, double fz, double dt) {
    FF_CHECK(ctx && res, FF_E_ARG, "ff_velocity3_add_force: NULL argument");
    const double unit[3] = {1.0, 1.0, 1.0};   // spacing does not enter
    const G3 g = geom_of(res, unit, nullptr);
    ff_field fs[3] = {u, v, w};
    const float fdt[3] = {(float)fx * (float)dt, (float)fy * (float)dt, (float)fz * (float)dt};
    cudaSetDevice(ctx->device);
    for (int a = 0; a < 3; ++a) {
        FF_CHECK(field_is(fs[a], comp_count(g, a)), FF_E_ARG, "add_force: component %d shape", a);
        k_add_const<<<launch_blocks(comp_count(g, a)), 256, 0, ctx->stream>>>(comp_count(g, a), (float *)fs[a]->d,
                                                                             fdt[a]);
    }
    return post("add_force");
}

// -------------------------------------------------------------- viscosity --
extern "C" int ff_viscosity3_apply(ff_ctx ctx, const int *res, const double *h, ff_field u, ff_field v, ff_field w,
                                   double nu, double dt, ff_field uo, ff_field vo, ff_field wo) {
    FF_CHECK(ctx && res && h, FF_E_ARG, "ff_viscosity3_apply: NULL argument");
    FF_TRY(check_grid32(res, "ff_viscosity3_apply"));
    const G3 g = geom_of(res, h, nullptr);
    ff_field in[3] = {u, v, w}, out[3] = {uo, vo, wo};
    for (int a = 0; a < 3; ++a)
        FF_CHECK(field_is(in[a], comp_count(g, a)) && field_is(out[a], comp_count(g, a)) && in[a]->d != out[a]->d,
                 FF_E_ARG, "viscosity: component %d must be distinct float face fields of the grid's shape", a);
    cudaSetDevice(ctx->device);
    const float ihx = 1.0f / ((float)h[0] * (float)h[0]), ihy = 1.0f / ((float)h[1] * (float)h[1]),
                ihz = 1.0f / ((float)h[2] * (float)h[2]);
    const float c = (float)dt * (float)nu;
    for (int a = 0; a < 3; ++a) {
        const long long n = comp_count(g, a);
        k_viscosity<<<launch_blocks(n), 256, 0, ctx->stream>>>(g, a, (const float *)in[a]->d, (float *)out[a]->d, c,
                                                               ihx, ihy, ihz);
    }
    return post("viscosity");
}

// ---------------------------------------------------------------- outflow --
// createGridOutflowSolver3 (src/grid/grid_outflow_solver3.js:79-210).  Each
// outflow is a cell-centred SDF on its own grid, inside where phi < 0
// (level_set_utils.js:5-9), sampled trilinearly (sdf_collider3.js:33-45).
namespace {

// extrapolate kernel of applyOutflowVelocityBC (:98-133) for one outflow and
// one component: faces inside the outflow relax toward the velocity one
// spacing upstream (pt + n h, n the unit SDF gradient) by the Courant number
// of the outward bulk speed, clamped to +-1e3; a zero gradient keeps the
// face.  Faces outside are not written (the copy kernel skips them too).
__global__ void k_outflow_relax(VelField F, int a, G3 pg, const float *__restrict__ phi, float dt,
                                float *__restrict__ dst) {
    int sx, sy, sz;
    comp_shape(F.g, a, sx, sy, sz);
    const long long n = (long long)sx * sy * sz;
    const F3 o = comp_origin(F.g, a), po = comp_origin(pg, 3);
    const float h = a == 0 ? F.g.hx : (a == 1 ? F.g.hy : F.g.hz);
    const float *cur_d = a == 0 ? F.u : (a == 1 ? F.v : F.w);
    for (long long f = blockIdx.x * (long long)blockDim.x + threadIdx.x; f < n; f += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        unflatten(f, sx, sy, i, j, k);
        const F3 pt = index_pos(F.g, o, i, j, k);
        if (!(trilinear(phi, pg.nx, pg.ny, pg.nz, pg, po, pt) < 0.0f)) continue;
        const float cur = cur_d[f];
        const F3 gr = trilinear_gradient(phi, pg, po, pt);
        const float gl = sqrtf(gr.x * gr.x + gr.y * gr.y + gr.z * gr.z);
        if (!(gl > 0.0f)) {
            dst[f] = cur;
            continue;
        }
        const F3 nn{gr.x / gl, gr.y / gl, gr.z / gl};
        const F3 up{pt.x + nn.x * h, pt.y + nn.y * h, pt.z + nn.z * h};
        const F3 bulk = sample_vel(F, pt);
        float dot = bulk.x * -nn.x;
        dot = dot + bulk.y * -nn.y;
        dot = dot + bulk.z * -nn.z;
        const float courant = fminf(fmaxf(fmaxf(0.0f, dot) * dt / h, 0.0f), 1.0f);
        const F3 uv = sample_vel(F, up);
        const float upc = a == 0 ? uv.x : (a == 1 ? uv.y : uv.z);
        const float relaxed = cur + (upc - cur) * courant;
        dst[f] = fminf(fmaxf(relaxed, -1.0e3f), 1.0e3f);
    }
}

// copy kernel (:137-150): faces inside the outflow take the relaxed value;
// also clearOutflowScalarField (:174-196) with src == nullptr (a = 3, the
// cells of a scalar grid, set to 0)
__global__ void k_outflow_copy(G3 g, int a, G3 pg, const float *__restrict__ phi, const float *__restrict__ src,
                               float *__restrict__ data) {
    int sx, sy, sz;
    if (a == 3) {
        sx = g.nx;
        sy = g.ny;
        sz = g.nz;
    } else {
        comp_shape(g, a, sx, sy, sz);
    }
    const long long n = (long long)sx * sy * sz;
    const F3 o = comp_origin(g, a), po = comp_origin(pg, 3);
    for (long long f = blockIdx.x * (long long)blockDim.x + threadIdx.x; f < n; f += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        unflatten(f, sx, sy, i, j, k);
        if (trilinear(phi, pg.nx, pg.ny, pg.nz, pg, po, index_pos(g, o, i, j, k)) < 0.0f)
            data[f] = src ? src[f] : 0.0f;
    }
}

// createOutflowPressureDirichlet3 (sdf_inflow_outflow3.js:44-64) at the cell
// centres of grid g (dataPosition, grid_data3.js:10-18): active where any
// outflow holds the centre; the target everywhere
__global__ void k_outflow_dirichlet(G3 g, int n_out, const float *const *__restrict__ phis,
                                    const G3 *__restrict__ pgs, float target, uint8_t *__restrict__ active,
                                    float *__restrict__ tgt) {
    const long long n = (long long)g.nx * g.ny * g.nz;
    const F3 o = comp_origin(g, 3);
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        unflatten(c, g.nx, g.ny, i, j, k);
        const F3 pt = index_pos(g, o, i, j, k);
        bool in = false;
        for (int q = 0; q < n_out; ++q) {
            const G3 pg = pgs[q];
            in |= trilinear(phis[q], pg.nx, pg.ny, pg.nz, pg, comp_origin(pg, 3), pt) < 0.0f;
        }
        active[c] = in ? 1 : 0;
        tgt[c] = target;
    }
}

}  // namespace

struct ff_outflow_s {
    ff_ctx ctx = nullptr;
    G3 g{};
    float dt = 0.0f;
    int apply = 1;
    std::vector<ff_field> phi;   // borrowed
    std::vector<G3> pg;
    float *dst[3] = {};
    const float **d_phi = nullptr;   // device copies for the Dirichlet kernel
    G3 *d_pg = nullptr;
};

extern "C" int ff_outflow3_destroy(ff_outflow o) {
    if (!o) return FF_OK;
    cudaStreamSynchronize(o->ctx->stream);
    for (int a = 0; a < 3; ++a) ff_dev_free(o->dst[a]);
    ff_dev_free((void *)o->d_phi);
    ff_dev_free(o->d_pg);
    delete o;
    return FF_OK;
}

extern "C" int ff_outflow3_create(ff_ctx ctx, const int *res, const double *h, const double *origin, int n,
                                  const ff_field *phis, const int *phi_res, const double *phi_h,
                                  const double *phi_origin, double dt, int apply_velocity_bc, ff_outflow *out) {
    FF_CHECK(ctx && res && h && out && n >= 0 && (n == 0 || (phis && phi_res && phi_h)), FF_E_ARG,
             "ff_outflow3_create: bad arguments");
    FF_CHECK(res[0] > 0 && res[1] > 0 && res[2] > 0, FF_E_ARG, "createGridOutflowSolver3: bad resolution");
    FF_CHECK(n <= 64, FF_E_LIMIT, "createGridOutflowSolver3: at most 64 outflows");
    FF_TRY(check_grid32(res, "createGridOutflowSolver3"));
    for (int q = 0; q < n; ++q) FF_TRY(check_grid32(phi_res + 3 * q, "createGridOutflowSolver3"));
    *out = nullptr;
    std::vector<G3> pg(n);
    for (int q = 0; q < n; ++q) {
        pg[q] = geom_of(phi_res + 3 * q, phi_h + 3 * q, phi_origin ? phi_origin + 3 * q : nullptr);
        FF_CHECK(pg[q].nx > 0 && pg[q].ny > 0 && pg[q].nz > 0 && field_is(phis[q], comp_count(pg[q], 3)), FF_E_ARG,
                 "createGridOutflowSolver3: outflow %d must be a float cell SDF of its grid's shape", q);
    }
    cudaSetDevice(ctx->device);
    ff_outflow o = new ff_outflow_s();
    o->ctx = ctx;
    o->g = geom_of(res, h, origin);
    o->dt = (float)dt;
    o->apply = apply_velocity_bc != 0;
    o->phi.assign(phis, phis + n);
    o->pg = pg;
    int st = FF_OK;
    for (int a = 0; a < 3 && st == FF_OK; ++a)
        st = ff_dev_alloc((void **)&o->dst[a], (size_t)comp_count(o->g, a) * 4, ctx->stream);
    if (st == FF_OK) st = ff_dev_alloc((void **)&o->d_phi, sizeof(float *) * std::max(1, n), ctx->stream);
    if (st == FF_OK) st = ff_dev_alloc((void **)&o->d_pg, sizeof(G3) * std::max(1, n), ctx->stream);
    if (st == FF_OK && n) {
        std::vector<const float *> hp(n);
        for (int q = 0; q < n; ++q) hp[q] = (const float *)phis[q]->d;
        if (cudaMemcpy(o->d_phi, hp.data(), sizeof(float *) * n, cudaMemcpyHostToDevice) != cudaSuccess ||
            cudaMemcpy(o->d_pg, pg.data(), sizeof(G3) * n, cudaMemcpyHostToDevice) != cudaSuccess)
            st = ff_set_error(FF_E_CUDA, "createGridOutflowSolver3: upload");
    }
    if (st != FF_OK) {
        ff_outflow3_destroy(o);
        return st;
    }
    *out = o;
    return FF_OK;
}

extern "C" int ff_outflow3_set_dt(ff_outflow o, double dt) {
    FF_CHECK(o, FF_E_ARG, "NULL outflow solver");
    o->dt = (float)dt;
    return FF_OK;
}

extern "C" int ff_outflow3_apply_velocity_bc(ff_outflow o, ff_field u, ff_field v, ff_field w) {
    FF_CHECK(o, FF_E_ARG, "NULL outflow solver");
    ff_field fs[3] = {u, v, w};
    for (int a = 0; a < 3; ++a)
        FF_CHECK(field_is(fs[a], comp_count(o->g, a)), FF_E_ARG, "applyOutflowVelocityBC: component %d shape", a);
    if (!o->apply) return FF_OK;
    cudaSetDevice(o->ctx->device);
    cudaStream_t s = o->ctx->stream;
    VelField F{o->g, (const float *)u->d, (const float *)v->d, (const float *)w->d, nullptr};
    for (size_t q = 0; q < o->phi.size(); ++q)
        for (int a = 0; a < 3; ++a) {
            const long long n = comp_count(o->g, a);
            const float *phi = (const float *)o->phi[q]->d;
            k_outflow_relax<<<launch_blocks(n), 256, 0, s>>>(F, a, o->pg[q], phi, o->dt, o->dst[a]);
            k_outflow_copy<<<launch_blocks(n), 256, 0, s>>>(o->g, a, o->pg[q], phi, o->dst[a], (float *)fs[a]->d);
        }
    return post("applyOutflowVelocityBC");
}

extern "C" int ff_outflow3_clear_scalar(ff_outflow o, ff_field scalar, const int *res, const double *h,
                                        const double *origin) {
    FF_CHECK(o && res && h, FF_E_ARG, "clearOutflowScalarField: NULL argument");
    const G3 sg = geom_of(res, h, origin);
    FF_CHECK(field_is(scalar, comp_count(sg, 3)), FF_E_ARG, "clearOutflowScalarField: float cell field expected");
    cudaSetDevice(o->ctx->device);
    const long long n = comp_count(sg, 3);
    for (size_t q = 0; q < o->phi.size(); ++q)
        k_outflow_copy<<<launch_blocks(n), 256, 0, o->ctx->stream>>>(sg, 3, o->pg[q], (const float *)o->phi[q]->d,
                                                                    nullptr, (float *)scalar->d);
    return post("clearOutflowScalarField");
}

extern "C" int ff_outflow3_dirichlet(ff_outflow o, const int *res, const double *h, const double *origin,
                                     double target, ff_field active, ff_field target_field) {
    FF_CHECK(o && res && h, FF_E_ARG, "outflow dirichlet: NULL argument");
    const G3 cg = geom_of(res, h, origin);
    const long long n = comp_count(cg, 3);
    FF_CHECK(active && active->dtype == FF_UINT8 && active->count == n && field_is(target_field, n), FF_E_ARG,
             "outflow dirichlet: active must be a uint8 and target a float cell field");
    cudaSetDevice(o->ctx->device);
    k_outflow_dirichlet<<<launch_blocks(n), 256, 0, o->ctx->stream>>>(cg, (int)o->phi.size(), o->d_phi, o->d_pg,
                                                                      (float)target, (uint8_t *)active->d,
                                                                      (float *)target_field->d);
    return post("outflow dirichlet");
}
