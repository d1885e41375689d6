// mpm_adjoint.cu -- the differentiable form of the substep: a batch of scenes
// of Tait water and fixed-corotated solid particles stepped on dense per-scene
// halo grids with a fixed dt per scene, the loss sum |x(T) - target|^2, and
// its adjoint by checkpoint and recompute (include/mpm_b200.h, mpma_*).
//
// The forward is the default path's arithmetic for these two models
// (prepareParticle, p2g, updateGrid + finishGridVelocity, g2p of
// src/lib/mpm/kernels/shaders.ts:808-963, :1072-1211, :1485-1777,
// :2114-2421): Tait stress -det * lambda * (det^-gamma - 1), fixed-corotated
// stress 2 mu (F - R) F^T + lambda J (J - 1), APIC transfer with the
// quadratic B-spline, liquid density-contrast acceleration, the deformation
// update in (I + h C)^k increments, liquid projection to sqrt(clamp(J)) R,
// wall cushion and friction, confinement.  Sums are scattered with vector
// atomics (their order is not fixed; the gradient does not need it to be).
//
// The adjoint differentiates that arithmetic exactly where it is smooth and
// keeps the forward's branch where it is not (subgradients): confinement and
// the wall factors act as masks, the liquid determinant clamp stops the
// gradient outside [0.5, 2], the increment count k and the stencil's base
// node are held.  The polar rotation of a 2x2 F with det F > 0 is the
// rotation by atan2(F10 - F01, F00 + F11), which is what both the forward and
// the adjoint use.
//
// A forward substep is two kernels: the grid update, and G2P with the P2G of
// the next substep (the particle's new state is in registers there).  Per
// backward segment of K substeps: the K substeps are recomputed from the
// segment's checkpoint, keeping each substep's input state and grid sums (the
// last segment's are kept by the forward pass), then each substep is reversed by
// four: the grid update again, the G2P adjoint (scatters the node-velocity
// adjoints), the grid adjoint, and the P2G adjoint (gathers them back to the
// particle and adds the parameter gradients).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/mpm_b200.h"
#include "mpm_device.cuh"
#include "mpm_launch.cuh"
#include "mpm_records.cuh"

namespace mpm {
int host_error(int code, const char *message);
void host_clear_error();
}  // namespace mpm

using namespace mpm;

namespace {

constexpr unsigned ADJ_THREADS = 256;


// Per-scene constants; tait, lambda_s and mu_s are the differentiated
// material parameters.
struct AdjScene {
    uint32_t n, p_base, node_base, node_w;
    uint32_t cells_x, cells_y, tile_base, tiles_x;  // 16x16-node tiles of the halo grid, row-major
    float dx, inv_dx, gs, dt;
    float gx, gy, domain_w, domain_h;
    float solid_mass, wall_friction, rho, gamma;
    float tait, lambda_s, mu_s, pad2;
};

struct AdjState {
    float2 *x, *v;
    float4 *C, *F;
};

struct AdjCtx {
    const AdjScene *scenes;
    const uint32_t *tag;       // per particle: scene << 1 | 1 for Tait water, 0 for a fixed-corotated solid
    const float *vol;          // per particle
    uint32_t n;
    uint32_t *status;
    AdjState in, out;
    float4 *sum_s, *sum_w;  // per node: solid (m, qx, qy, 0), water (m, qx, qy, V)
    float2 *gv_s;           // per node: solid velocity (k_adj_grid_fwd)
    float4 *gv_w;           // per node: water velocity (x, y), liquid mass, liquid volume
    // adjoints: of the substep's outputs (next) and inputs (cur)
    float2 *xb_next, *vb_next, *xb, *vb;
    float4 *Cb_next, *Fb_next, *Cb, *Fb;
    float2 *xg;            // the G2P part of the input position adjoint
    float4 *Fg;            // the G2P part of the input F adjoint
    float4 *ub_s;          // per node: solid velocity adjoint (x, y), then (Qx, Qy, M) adjoints, 0
    float4 *ub_w;          // per node: water velocity, liquid mass, liquid volume adjoints
    float4 *ub_s_prev, *ub_w_prev;  // those of the substep before, while the pass turns to it
    double *param_grad;    // per scene: tait, lambda_s, mu_s
    const float2 *target;  // per particle
    double *loss;          // per scene
    uint8_t *mark_out;     // per tile, solid and water: set when a position whose P2G is scattered reaches it, or NULL
};

constexpr int ADJ_TILE = 16;  // nodes per side of a tile of marks

constexpr uint32_t ADJ_ERR_STENCIL = 1u, ADJ_ERR_NONFINITE = 2u, ADJ_ERR_DETERMINANT = 4u;

__device__ __forceinline__ void adj_fail(const AdjCtx &c, uint32_t flag) { atomicOr(c.status, flag); }

// ------------------------------------------------------------ 2x2 helpers --

__device__ __forceinline__ float4 cofactor(float4 F) { return make_float4(F.w, -F.z, -F.y, F.x); }

// d(det)/dF for a row-major (F00, F01, F10, F11).
__device__ __forceinline__ float4 axpy4(float a, float4 x, float4 y)
{
    return make_float4(y.x + a * x.x, y.y + a * x.y, y.z + a * x.z, y.w + a * x.w);
}

// Rotation by phi = atan2(F10 - F01, F00 + F11), as (cos, sin); the polar
// rotation of F when det F > 0.
__device__ __forceinline__ float2 polar_angle(float4 F)
{
    const float a = F.x + F.w, b = F.z - F.y;
    const float r = sqrtf(a * a + b * b);
    return r > 0.0f ? make_float2(a / r, b / r) : make_float2(1.0f, 0.0f);
}

__device__ __forceinline__ float4 rotation(float2 cs) { return make_float4(cs.x, -cs.y, cs.y, cs.x); }

// Adds phi_bar * d(phi)/dF to Fb (phi = atan2(F10 - F01, F00 + F11)).
__device__ __forceinline__ float4 angle_adjoint(float4 F, float phi_bar, float4 Fb)
{
    const float a = F.x + F.w, b = F.z - F.y, r2 = a * a + b * b;
    if (!(r2 > 0.0f)) return Fb;
    const float da = -b / r2 * phi_bar, db = a / r2 * phi_bar;
    return make_float4(Fb.x + da, Fb.y - db, Fb.z + db, Fb.w + da);
}

// ------------------------------------------------------------- stencil ----

struct AdjStencil {
    int bx, by;
    float fx, fy;
    float wx[3], wy[3], dwx[3], dwy[3];  // weights and their derivatives in the fraction
};

__device__ __forceinline__ bool adj_stencil(const AdjScene &S, float2 x, AdjStencil &st)
{
    const float gx = __fmul_rn(x.x, S.inv_dx), gy = __fmul_rn(x.y, S.inv_dx);
    if (!finite_f(gx) || !finite_f(gy)) return false;
    st.bx = (int)floorf(__fsub_rn(gx, 0.5f));
    st.by = (int)floorf(__fsub_rn(gy, 0.5f));
    st.fx = __fsub_rn(gx, (float)st.bx);
    st.fy = __fsub_rn(gy, (float)st.by);
    if (st.bx < -1 || st.by < -1 || st.bx + 2 > (int)S.cells_x + 1 || st.by + 2 > (int)S.cells_y + 1) return false;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        st.wx[k] = quad_weight(st.fx, k);
        st.wy[k] = quad_weight(st.fy, k);
    }
    // d/df of 0.5 (1.5 - f)^2, 0.75 - (f - 1)^2, 0.5 (f - 0.5)^2
    st.dwx[0] = st.fx - 1.5f, st.dwx[1] = -2.0f * (st.fx - 1.0f), st.dwx[2] = st.fx - 0.5f;
    st.dwy[0] = st.fy - 1.5f, st.dwy[1] = -2.0f * (st.fy - 1.0f), st.dwy[2] = st.fy - 0.5f;
    return true;
}

__device__ __forceinline__ uint32_t adj_node(const AdjScene &S, int ix, int iy)
{
    return S.node_base + (uint32_t)(iy + 1) * S.node_w + (uint32_t)(ix + 1);
}

// ------------------------------------------------------------ materials ---

struct Prepared {
    float m, vliq, scale, det;
    float4 s, A;
};

// prepareParticle for the two differentiable models.
__device__ __forceinline__ bool adj_prepare(const AdjScene &S, bool liquid, float vol, float4 C, float4 F, Prepared &p)
{
    p.det = det2(F);
    if (!finite_f(p.det) || p.det <= 0.0f) return false;
    if (liquid) {
        const float pw = pow_wgsl(__fdiv_rn(1.0f, p.det), S.gamma);
        const float sigma = -p.det * (S.tait * (pw - 1.0f));
        p.s = make_float4(sigma, 0.f, 0.f, sigma);
        p.m = __fmul_rn(S.rho, vol);
        p.vliq = __fmul_rn(vol, p.det);
    } else {
        const float4 R = rotation(polar_angle(F));
        const float4 d = make_float4(F.x - R.x, F.y - R.y, F.z - R.z, F.w - R.w);
        const float shear = 2.0f * S.mu_s, volumetric = S.lambda_s * p.det * (p.det - 1.0f);
        p.s = make_float4(shear * (d.x * F.x + d.y * F.y) + volumetric, shear * (d.x * F.z + d.y * F.w),
                          shear * (d.z * F.x + d.w * F.y), shear * (d.z * F.z + d.w * F.w) + volumetric);
        p.m = S.solid_mass;
        p.vliq = 0.0f;
    }
    p.scale = -S.dt * vol * S.gs;
    p.A = make_float4(p.m * C.x + p.scale * p.s.x, p.m * C.y + p.scale * p.s.y, p.m * C.z + p.scale * p.s.z,
                      p.m * C.w + p.scale * p.s.w);
    return finite4(p.A);
}

// Stress adjoint: adds dL/dF to Fb and returns the parameter adjoints
// (tait, lambda_s, mu_s) for the stress adjoint sb.
__device__ __forceinline__ float3 stress_adjoint(const AdjScene &S, bool liquid, float4 F, float det, float4 sb,
                                                 float4 &Fb)
{
    if (liquid) {
        const float pw = pow_wgsl(__fdiv_rn(1.0f, det), S.gamma);
        const float sigma_b = sb.x + sb.w;
        // sigma = -tait (det^(1-gamma) - det)
        const float dsigma = -S.tait * ((1.0f - S.gamma) * pw - 1.0f);
        Fb = axpy4(sigma_b * dsigma, cofactor(F), Fb);
        return make_float3(sigma_b * -(det * pw - det), 0.f, 0.f);
    }
    const float2 cs = polar_angle(F);
    const float4 R = rotation(cs);
    const float4 D = make_float4(F.x - R.x, F.y - R.y, F.z - R.z, F.w - R.w);
    // mu: s : 2 (F - R) F^T
    const float4 DFt = make_float4(D.x * F.x + D.y * F.y, D.x * F.z + D.y * F.w, D.z * F.x + D.w * F.y,
                                   D.z * F.z + D.w * F.w);
    const float mu_b = 2.0f * (sb.x * DFt.x + sb.y * DFt.y + sb.z * DFt.z + sb.w * DFt.w);
    const float trace_b = sb.x + sb.w;
    const float lambda_b = trace_b * det * (det - 1.0f);
    Fb = axpy4(trace_b * S.lambda_s * (2.0f * det - 1.0f), cofactor(F), Fb);
    // 2 mu (F F^T - R F^T): (sb + sb^T) F - sb^T R for F, sb F for R
    const float m2 = 2.0f * S.mu_s;
    const float4 sym = make_float4(2.0f * sb.x, sb.y + sb.z, sb.z + sb.y, 2.0f * sb.w);
    const float4 symF = make_float4(sym.x * F.x + sym.y * F.z, sym.x * F.y + sym.y * F.w, sym.z * F.x + sym.w * F.z,
                                    sym.z * F.y + sym.w * F.w);
    const float4 sTR = make_float4(sb.x * R.x + sb.z * R.z, sb.x * R.y + sb.z * R.w, sb.y * R.x + sb.w * R.z,
                                   sb.y * R.y + sb.w * R.w);
    Fb = make_float4(Fb.x + m2 * (symF.x - sTR.x), Fb.y + m2 * (symF.y - sTR.y), Fb.z + m2 * (symF.z - sTR.z),
                     Fb.w + m2 * (symF.w - sTR.w));
    // R adjoint -m2 sb F, then through the angle: dR/dphi = (-sin, -cos, cos, -sin)
    const float4 sF = make_float4(sb.x * F.x + sb.y * F.y, sb.x * F.z + sb.y * F.w, sb.z * F.x + sb.w * F.y,
                                  sb.z * F.z + sb.w * F.w);
    const float4 Rb = make_float4(-m2 * sF.x, -m2 * sF.y, -m2 * sF.z, -m2 * sF.w);
    const float phi_b = Rb.x * -cs.y + Rb.y * -cs.x + Rb.z * cs.x + Rb.w * -cs.y;
    Fb = angle_adjoint(F, phi_b, Fb);
    return make_float3(0.f, lambda_b, mu_b);
}

// ------------------------------------------------------------ grid node ---

// The wall factors of updateGrid's applyWallCushion / applyWallTangentialFriction
// (shaders.ts:1438-1457) for a pre-wall velocity u at node (x, y).
__device__ __forceinline__ float cushion_factor(float u, int coord, int extent)
{
    const float cushion = fminf(WALL_CUSHION_CELLS, (float)extent / 4.0f);
    const float dist = u < 0.0f ? (float)coord : (float)(extent - coord);
    if (dist >= cushion) return 1.0f;
    return fminf(fmaxf(dist / cushion, 0.0f), 1.0f);
}

__device__ __forceinline__ float friction_factor(int coord, int extent, float friction)
{
    if (friction <= 0.0f) return 1.0f;
    const float dist = fmaxf(0.0f, fminf((float)coord, (float)(extent - coord)));
    const float cushion = fminf(WALL_CUSHION_CELLS, (float)extent / 4.0f);
    if (dist >= cushion) return 1.0f;
    return 1.0f - friction * (1.0f - fminf(fmaxf(dist / cushion, 0.0f), 1.0f));
}

// Node velocity from its sums (finishGridVelocity + walls); D receives the
// wall factors per axis.
__device__ __forceinline__ float2 node_velocity_adj(const AdjScene &S, float4 sum, int ix, int iy, float2 &D)
{
    D = make_float2(0.f, 0.f);
    if (!(sum.x > 0.0f)) return make_float2(0.f, 0.f);
    const float inv = __frcp_rn(sum.x);
    const float2 u0 = make_float2(sum.y * inv + S.dt * S.gx, sum.z * inv + S.dt * S.gy);
    const int cx = (int)S.cells_x, cy = (int)S.cells_y;
    D.x = cushion_factor(u0.x, ix, cx) * friction_factor(iy, cy, S.wall_friction);
    D.y = cushion_factor(u0.y, iy, cy) * friction_factor(ix, cx, S.wall_friction);
    return make_float2(u0.x * D.x, u0.y * D.y);
}

// --------------------------------------------------------------- G2P ------

// The forward G2P quantities of one particle that its adjoint reuses.
struct G2pFwd {
    float2 vp;       // interpolated velocity (after the liquid acceleration)
    float4 B;        // sum w u dp^T
    float pm, pv;    // interpolated liquid mass and volume
    float pdet;      // det of the input F
    float4 Cn;       // new C
    float4 trial;    // F before the projection
    uint32_t sub;    // deformation increments
    float2 xn;       // new position before confinement
};

__device__ __forceinline__ bool g2p_forward(const AdjCtx &c, const AdjScene &S, bool liquid, const AdjStencil &st,
                                            float2 x, float4 F0, G2pFwd &g)
{
    g.vp = make_float2(0.f, 0.f);
    g.B = make_float4(0.f, 0.f, 0.f, 0.f);
    g.pm = g.pv = 0.f;
#pragma unroll
    for (int oy = 0; oy < 3; ++oy) {
        const float dpy = ((float)oy - st.fy) * S.dx;
#pragma unroll
        for (int ox = 0; ox < 3; ++ox) {
            const float w = st.wx[ox] * st.wy[oy];
            const float dpx = ((float)ox - st.fx) * S.dx;
            const uint32_t n = adj_node(S, st.bx + ox, st.by + oy);
            float2 u;
            float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);  // liquid mass in x, liquid volume in w
            if (liquid) {
                const float4 gw = c.gv_w[n];
                u = make_float2(gw.x, gw.y);
                sum.x = gw.z;
                sum.w = gw.w;
            } else {
                u = c.gv_s[n];
            }
            g.vp.x += w * u.x;
            g.vp.y += w * u.y;
            g.B.x += w * u.x * dpx;
            g.B.y += w * u.x * dpy;
            g.B.z += w * u.y * dpx;
            g.B.w += w * u.y * dpy;
            if (liquid) {
                g.pm += w * sum.x;
                g.pv += w * sum.w;
            }
        }
    }
    g.pdet = det2(F0);
    if (liquid) {
        if (!(g.pm > 0.f) || !(g.pv > 0.f) || !(g.pdet > 0.f)) return false;
        const float pd = S.rho / g.pdet, ld = g.pm / g.pv;
        const float rd = (pd - ld) / pd;
        g.vp.x += S.dt * (rd * S.gx);
        g.vp.y += S.dt * (rd * S.gy);
    }
    g.Cn = make_float4(g.B.x * S.gs, g.B.y * S.gs, g.B.z * S.gs, g.B.w * S.gs);
    g.xn = make_float2(x.x + S.dt * g.vp.x, x.y + S.dt * g.vp.y);
    const float row = fmaxf(fabsf(g.Cn.x) + fabsf(g.Cn.y), fabsf(g.Cn.z) + fabsf(g.Cn.w));
    const float req = ceilf(S.dt * row * (1.0f / MAX_DEFORMATION_INCREMENT));
    if (!finite_f(req) || req > MAX_DEFORMATION_SUBSTEPS) return false;
    g.sub = max(1u, (uint32_t)req);
    g.trial = integrate_deformation(F0, g.Cn, S.dt, g.sub);
    float tdet = det2(g.trial);
    while (finite_f(tdet) && tdet <= 0.f && g.sub < 64u) {
        g.sub = min(g.sub * 2u, 64u);
        g.trial = integrate_deformation(F0, g.Cn, S.dt, g.sub);
        tdet = det2(g.trial);
    }
    return finite_f(tdet) && tdet > 0.f && finite2(g.vp) && finite4(g.Cn);
}

// projectLiquidDeformation (shaders.ts:474-488) as sqrt(clamp(det T)) R(T).
__device__ __forceinline__ float4 project_liquid(float4 T)
{
    const float2 cs = polar_angle(T);
    const float sc = sqrtf(fminf(fmaxf(det2(T), MIN_LIQUID_DETERMINANT), MAX_LIQUID_DETERMINANT));
    return make_float4(sc * cs.x, -sc * cs.y, sc * cs.y, sc * cs.x);
}

}  // namespace

// Marks the tiles that the stencil with base (bx, by) reaches (its corner
// nodes lie in at most four), a byte for solid particles and one for water.  Lanes
// of a warp storing to the same mark byte in one instruction make one memory
// transaction.
__device__ __forceinline__ void mark_tiles(uint8_t *mark, const AdjScene &S, bool liquid, int bx, int by)
{
    const uint32_t x0 = (uint32_t)(bx + 1) / ADJ_TILE, x1 = (uint32_t)(bx + 3) / ADJ_TILE;
    const uint32_t y0 = (uint32_t)(by + 1) / ADJ_TILE, y1 = (uint32_t)(by + 3) / ADJ_TILE;
    mark += 2u * S.tile_base + (liquid ? 1u : 0u);
    uint8_t *row0 = mark + 2u * y0 * S.tiles_x, *row1 = mark + 2u * y1 * S.tiles_x;
    row0[2u * x0] = 1u;
    if (x1 != x0) row0[2u * x1] = 1u;
    if (y1 != y0) {
        row1[2u * x0] = 1u;
        if (x1 != x0) row1[2u * x1] = 1u;
    }
}

// ------------------------------------------------------------- kernels ----

// The P2G of one particle: adds to the node sums and marks the tiles its
// stencil reaches (unless mark_out is NULL), or raises a status.
__device__ __forceinline__ void p2g_particle(const AdjCtx &c, const AdjScene &S, bool liquid, float2 x, float2 v, float4 C,
                                             float4 F, float vol)
{
    Prepared p;
    if (!adj_prepare(S, liquid, vol, C, F, p)) {
        adj_fail(c, ADJ_ERR_DETERMINANT);
        return;
    }
    AdjStencil st;
    if (!adj_stencil(S, x, st)) {
        adj_fail(c, ADJ_ERR_STENCIL);
        return;
    }
    if (c.mark_out) mark_tiles(c.mark_out, S, liquid, st.bx, st.by);
    float4 *sums = (liquid ? c.sum_w : c.sum_s) + adj_node(S, st.bx, st.by);
#pragma unroll
    for (int oy = 0; oy < 3; ++oy) {
        const float dpy = ((float)oy - st.fy) * S.dx;
#pragma unroll
        for (int ox = 0; ox < 3; ++ox) {
            const float w = st.wx[ox] * st.wy[oy];
            const float dpx = ((float)ox - st.fx) * S.dx;
            const float qx = p.m * v.x + p.A.x * dpx + p.A.y * dpy;
            const float qy = p.m * v.y + p.A.z * dpx + p.A.w * dpy;
            atomicAdd(sums + (uint32_t)oy * S.node_w + ox,
                      make_float4(w * p.m, w * qx, w * qy, liquid ? w * p.vliq : 0.f));
        }
    }
}

// P2G of the states in c.in (the first substep of a run; the others' comes
// with the G2P before them).
__global__ void __launch_bounds__(ADJ_THREADS) k_adj_p2g(AdjCtx c)
{
    follow();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const uint32_t tag = c.tag[i];
    p2g_particle(c, c.scenes[tag >> 1], (tag & 1u) != 0u, c.in.x[i], c.in.v[i], c.in.C[i], c.in.F[i], c.vol[i]);
}

// G2P of one substep, and with P2G the P2G of the next from the new state.
// Latency-bound (the gathered node velocities and the particle's own words from
// L2, issue active 40 % of cycles; the atomics use 22 % of L2's rate): 64 registers
// for 32 warps per SM, 56.6 us at 24 warps -> 52.3 us per million particles, where
// G2P and P2G as two kernels took 31 + 37 us and a launch more.
template <bool P2G>
__global__ void __launch_bounds__(ADJ_THREADS, 4) k_adj_g2p(AdjCtx c)
{
    follow();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const uint32_t tag = c.tag[i];
    const AdjScene &S = c.scenes[tag >> 1];
    const bool liquid = (tag & 1u) != 0u;
    const float2 x = c.in.x[i];
    const float4 F0 = c.in.F[i];
    const float vol = P2G ? c.vol[i] : 0.0f;
    AdjStencil st;
    G2pFwd g;
    if (!adj_stencil(S, x, st) || !g2p_forward(c, S, liquid, st, x, F0, g)) {
        adj_fail(c, ADJ_ERR_NONFINITE);
        return;
    }
    const float4 Fn = liquid ? project_liquid(g.trial) : g.trial;
    const float2 bx = confine_axis(g.xn.x, g.vp.x, S.domain_w);
    const float2 by = confine_axis(g.xn.y, g.vp.y, S.domain_h);
    const float2 xn = make_float2(bx.x, by.x), vn = make_float2(bx.y, by.y);
    c.out.x[i] = xn;
    c.out.v[i] = vn;
    c.out.C[i] = g.Cn;
    c.out.F[i] = Fn;
    if constexpr (P2G) p2g_particle(c, S, liquid, xn, vn, g.Cn, Fn, vol);
}

// The kernels over the grid take a tile of 16 x 16 nodes at a time, one node
// per thread, and leave what no stencil of the substep reaches (`mark`, set by
// the P2G, for solid and water) as it is: every node a substep adds to or reads
// lies in a marked tile, and the rest of the grid keeps stale values that no
// stencil reads.  The tiles are dealt to the CTAs one by one (marked ones lie
// together), a CTA reads the marks of its tiles together and then visits the
// marked ones: visit(scene, node, x, y, marks), marks 1 for solid and 2 for water,
// four times as much by the marks of the substep before.  No list of the marked
// tiles is built and no node cleared ahead of a substep: the grid update leaves the
// sums at zero.  64 scenes of 16,384 particles, 200 substeps forward and backward:
// 8 launches per substep forward and 7 backward -> 2 and 2 (and 2 to recompute a
// segment), 73.9 -> 48.9 ms; one scene of 1,024, 40 substeps: 2.08 -> 0.76 ms.
template <class Visit>
__device__ __forceinline__ void for_marked_nodes(const AdjCtx &c, const uint32_t *tile_scene, const uint8_t *mark,
                                                 const uint8_t *mark_prev, uint32_t n_tiles, const Visit &visit)
{
    __shared__ uint32_t s_tile[ADJ_THREADS], s_count;
    for (uint32_t first = blockIdx.x; first < n_tiles; first += gridDim.x * ADJ_THREADS) {
        __syncthreads();
        if (threadIdx.x == 0) s_count = 0u;
        __syncthreads();
        const uint64_t t = first + (uint64_t)threadIdx.x * gridDim.x;
        if (t < n_tiles) {
            // 1: solid, 0x100: water, four times as much for the substep before
            uint32_t both = reinterpret_cast<const uint16_t *>(mark)[t];
            if (mark_prev) both |= (uint32_t)reinterpret_cast<const uint16_t *>(mark_prev)[t] << 2;
            if (both != 0u) s_tile[atomicAdd(&s_count, 1u)] = (uint32_t)t << 4 | (both & 5u) | (both >> 7 & 10u);
        }
        __syncthreads();
        const uint32_t count = s_count;
        for (uint32_t k = 0; k < count; ++k) {
            const uint32_t entry = s_tile[k], tile = entry >> 4;
            const AdjScene &S = c.scenes[tile_scene[tile]];
            const uint32_t local = tile - S.tile_base;
            const uint32_t hx = (local % S.tiles_x) * ADJ_TILE + threadIdx.x % ADJ_TILE;
            const uint32_t hy = (local / S.tiles_x) * ADJ_TILE + threadIdx.x / ADJ_TILE;
            if (hx < S.node_w && hy < S.cells_y + 3u)
                visit(S, S.node_base + hy * S.node_w + hx, (int)hx - 1, (int)hy - 1, entry & 15u);
        }
    }
}

// The grid update (finishGridVelocity with the wall factors,
// node_velocity_adj) of one node: its velocity from its sums, for the G2P
// kernels; the water record also carries the node's liquid mass and volume.
__device__ __forceinline__ void grid_velocity(const AdjCtx &c, const AdjScene &S, uint32_t n, int ix, int iy, bool solid,
                                              bool water, float4 s, float4 w)
{
    float2 D;
    if (solid) c.gv_s[n] = node_velocity_adj(S, s, ix, iy, D);
    if (water) {
        const float2 u = node_velocity_adj(S, w, ix, iy, D);
        c.gv_w[n] = make_float4(u.x, u.y, w.x, w.w);
    }
}

// The grid update of the marked tiles' nodes.  ZERO: the sums are scratch; they
// are kept in tape_s / tape_w (unless NULL) and zeroed for the next P2G.  Else the
// sums are a kept substep's, and the node adjoints are zeroed for the G2P
// adjoint.
template <bool ZERO>
__global__ void __launch_bounds__(ADJ_THREADS) k_adj_grid_fwd(AdjCtx c, const uint32_t *tile_scene, const uint8_t *mark,
                                                              uint32_t n_tiles, float4 *tape_s, float4 *tape_w)
{
    follow();
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for_marked_nodes(c, tile_scene, mark, nullptr, n_tiles, [&](const AdjScene &S, uint32_t n, int ix, int iy, uint32_t marks) {
        const bool solid = (marks & 1u) != 0u, water = (marks & 2u) != 0u;
        float4 s, w;
        if (solid) s = c.sum_s[n];
        if (water) w = c.sum_w[n];
        grid_velocity(c, S, n, ix, iy, solid, water, s, w);
        if (solid) {
            if (ZERO && tape_s) tape_s[n] = s;
            (ZERO ? c.sum_s : c.ub_s)[n] = zero;
        }
        if (water) {
            if (ZERO && tape_w) tape_w[n] = w;
            (ZERO ? c.sum_w : c.ub_w)[n] = zero;
        }
    });
}

// The grid-update adjoint of one node and channel: the node velocity
// adjoints that the G2P adjoint scattered, b = (velocity x, y, liquid mass, liquid volume), to
// the adjoints of the node sums (u = D (q / m + dt g): momentum q, mass m; the
// liquid volume's passes through), once per node instead of once per particle
// reaching it.
__device__ __forceinline__ float4 grid_adjoint(const AdjScene &S, int ix, int iy, bool water, float4 sum, float4 b)
{
    float M_b = water ? b.z : 0.f, Qx_b = 0.f, Qy_b = 0.f;
    if (sum.x > 0.0f) {
        float2 D;
        node_velocity_adj(S, sum, ix, iy, D);
        const float inv = 1.0f / sum.x;
        const float udx = D.x * b.x, udy = D.y * b.y;
        Qx_b = udx * inv;
        Qy_b = udy * inv;
        M_b -= (udx * sum.y + udy * sum.z) * inv * inv;
    }
    return make_float4(Qx_b, Qy_b, M_b, water ? b.w : 0.f);
}

// The grid-update adjoint of the marked tiles' nodes, in place.  TURN: and the
// grid update of the substep before, whose sums and marks are given, with its node
// adjoints zeroed, as k_adj_grid_fwd<false> does it: one launch and one pass over
// the tiles fewer per substep.
template <bool TURN>
__global__ void __launch_bounds__(ADJ_THREADS) k_adj_grid_bwd(AdjCtx c, const uint32_t *tile_scene, const uint8_t *mark,
                                                              const uint8_t *mark_prev, uint32_t n_tiles,
                                                              const float4 *prev_s, const float4 *prev_w)
{
    follow();
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for_marked_nodes(c, tile_scene, mark, TURN ? mark_prev : nullptr, n_tiles,
                     [&](const AdjScene &S, uint32_t n, int ix, int iy, uint32_t marks) {
                         const bool solid = (marks & 1u) != 0u, water = (marks & 2u) != 0u;
                         const bool solid_prev = TURN && (marks & 4u) != 0u, water_prev = TURN && (marks & 8u) != 0u;
                         float4 s, w, us, uw, ps, pw;
                         if (solid) s = c.sum_s[n], us = c.ub_s[n];
                         if (water) w = c.sum_w[n], uw = c.ub_w[n];
                         if (solid_prev) ps = prev_s[n];
                         if (water_prev) pw = prev_w[n];
                         if (solid) c.ub_s[n] = grid_adjoint(S, ix, iy, false, s, us);
                         if (water) c.ub_w[n] = grid_adjoint(S, ix, iy, true, w, uw);
                         if (TURN) {
                             grid_velocity(c, S, n, ix, iy, solid_prev, water_prev, ps, pw);
                             if (solid_prev) c.ub_s_prev[n] = zero;
                             if (water_prev) c.ub_w_prev[n] = zero;
                         }
                     });
}

// Loss sum |x - target|^2 per scene (one atomic per warp whose particles
// share a scene) and its adjoint seeds.
__global__ void __launch_bounds__(ADJ_THREADS) k_adj_loss(AdjCtx c)
{
    follow();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < c.n;
    const uint32_t scene = valid ? c.tag[i] >> 1 : 0u;
    double term = 0.0;
    if (valid) {
        const float2 x = c.in.x[i], t = c.target[i];
        const float dx = x.x - t.x, dy = x.y - t.y;
        term = (double)dx * dx + (double)dy * dy;
        c.xb_next[i] = make_float2(2.0f * dx, 2.0f * dy);
        c.vb_next[i] = make_float2(0.f, 0.f);
        c.Cb_next[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        c.Fb_next[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const unsigned full = 0xffffffffu;
    const uint32_t lead = __shfl_sync(full, scene, 0);
    if (__all_sync(full, !valid || scene == lead)) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) term += __shfl_xor_sync(full, term, o);
        if ((threadIdx.x & 31u) == 0u) atomicAdd(&c.loss[lead], term);
    } else if (valid) {
        atomicAdd(&c.loss[scene], term);
    }
}

// A particle's adjoints of a state.
struct StateAdjoint {
    float2 x, v;
    float4 C, F;
};

// The G2P adjoint of one particle: from the adjoints of the substep's outputs
// to the node-velocity adjoints (added to ub_s / ub_w) and the G2P parts of
// the input position and F adjoints.
__device__ __forceinline__ void g2p_adjoint(const AdjCtx &c, uint32_t i, uint32_t tag, float2 x, float4 F0,
                                            const StateAdjoint &o, float4 *ub_s, float4 *ub_w)
{
    const AdjScene &S = c.scenes[tag >> 1];
    const bool liquid = (tag & 1u) != 0u;
    AdjStencil st;
    G2pFwd g;
    if (!adj_stencil(S, x, st) || !g2p_forward(c, S, liquid, st, x, F0, g)) {
        adj_fail(c, ADJ_ERR_NONFINITE);
        return;
    }
    const float2 xbo = o.x, vbo = o.v;
    const float4 Cbo = o.C, Fbo = o.F;
    // confinement: a clamped axis passes no gradient
    const float2 cxa = confine_axis(g.xn.x, g.vp.x, S.domain_w);
    const float2 cya = confine_axis(g.xn.y, g.vp.y, S.domain_h);
    const bool free_x = cxa.x == g.xn.x, free_y = cya.x == g.xn.y;
    float2 xb = make_float2(free_x ? xbo.x : 0.f, free_y ? xbo.y : 0.f);
    float2 vpb = make_float2(free_x ? vbo.x + S.dt * xbo.x : 0.f, free_y ? vbo.y + S.dt * xbo.y : 0.f);
    // projection
    float4 Tb = Fbo;
    if (liquid) {
        const float4 T = g.trial;
        const float2 cs = polar_angle(T);
        const float J = det2(T);
        const float Jc = fminf(fmaxf(J, MIN_LIQUID_DETERMINANT), MAX_LIQUID_DETERMINANT);
        const float sc = sqrtf(Jc);
        // F = sc (cos, -sin, sin, cos)
        const float sc_b = Fbo.x * cs.x - Fbo.y * cs.y + Fbo.z * cs.y + Fbo.w * cs.x;
        const float phi_b = sc * (Fbo.x * -cs.y + Fbo.y * -cs.x + Fbo.z * cs.x + Fbo.w * -cs.y);
        const float J_b = (J == Jc) ? sc_b * 0.5f / sc : 0.f;
        Tb = make_float4(0.f, 0.f, 0.f, 0.f);
        Tb = axpy4(J_b, cofactor(T), Tb);
        Tb = angle_adjoint(T, phi_b, Tb);
    }
    // deformation increments: T = U^k F0, U = I + h C'
    const float h = g.sub == 1u ? S.dt : __fdiv_rn(S.dt, (float)g.sub);
    const float4 U = make_float4(1.0f + h * g.Cn.x, h * g.Cn.y, h * g.Cn.z, 1.0f + h * g.Cn.w);
    float4 G = Tb, Ub = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int j = (int)g.sub - 1; j >= 0; --j) {
        float4 Fj = F0;  // U^j F0
        for (int q = 0; q < j; ++q)
            Fj = make_float4(U.x * Fj.x + U.y * Fj.z, U.x * Fj.y + U.y * Fj.w, U.z * Fj.x + U.w * Fj.z,
                             U.z * Fj.y + U.w * Fj.w);
        // Ub += G Fj^T; G = U^T G
        Ub = make_float4(Ub.x + G.x * Fj.x + G.y * Fj.y, Ub.y + G.x * Fj.z + G.y * Fj.w,
                         Ub.z + G.z * Fj.x + G.w * Fj.y, Ub.w + G.z * Fj.z + G.w * Fj.w);
        G = make_float4(U.x * G.x + U.z * G.z, U.x * G.y + U.z * G.w, U.y * G.x + U.w * G.z, U.y * G.y + U.w * G.w);
    }
    float4 Fg = G;
    const float4 Cnb = make_float4(Cbo.x + h * Ub.x, Cbo.y + h * Ub.y, Cbo.z + h * Ub.z, Cbo.w + h * Ub.w);
    const float4 Bb = make_float4(Cnb.x * S.gs, Cnb.y * S.gs, Cnb.z * S.gs, Cnb.w * S.gs);
    // liquid acceleration v += dt g (1 - ld pdet / rho), ld = pm / pv
    float pm_b = 0.f, pv_b = 0.f;
    if (liquid) {
        const float rd_b = S.dt * (S.gx * vpb.x + S.gy * vpb.y);
        const float ld = g.pm / g.pv;
        const float ld_b = -rd_b * g.pdet / S.rho;
        const float pdet_b = -rd_b * ld / S.rho;
        Fg = axpy4(pdet_b, cofactor(F0), Fg);
        pm_b = ld_b / g.pv;
        pv_b = -ld_b * g.pm / (g.pv * g.pv);
    }
    // interpolation: scatter the node adjoints; the position adjoint through
    // the weights and offsets
#pragma unroll
    for (int oy = 0; oy < 3; ++oy) {
        const float dpy = ((float)oy - st.fy) * S.dx;
#pragma unroll
        for (int ox = 0; ox < 3; ++ox) {
            const float w = st.wx[ox] * st.wy[oy];
            const float dpx = ((float)ox - st.fx) * S.dx;
            // the node velocity, liquid mass and volume once more
            const uint32_t n = adj_node(S, st.bx + ox, st.by + oy);
            const float4 gw = liquid ? c.gv_w[n] : make_float4(c.gv_s[n].x, c.gv_s[n].y, 0.f, 0.f);
            const float2 u = make_float2(gw.x, gw.y);
            // node velocity adjoint: w vpb + w Bb dp
            const float ubx = w * (vpb.x + Bb.x * dpx + Bb.y * dpy);
            const float uby = w * (vpb.y + Bb.z * dpx + Bb.w * dpy);
            if (liquid)
                atomicAdd(&ub_w[n], make_float4(ubx, uby, w * pm_b, w * pv_b));
            else
                atomicAdd(reinterpret_cast<float2 *>(&ub_s[n]), make_float2(ubx, uby));
            // d/dx of w: (dwx wy, wx dwy) / dx
            const float gwx = st.dwx[ox] * st.wy[oy] * S.inv_dx, gwy = st.wx[ox] * st.dwy[oy] * S.inv_dx;
            float sval = u.x * (vpb.x + Bb.x * dpx + Bb.y * dpy) + u.y * (vpb.y + Bb.z * dpx + Bb.w * dpy);
            if (liquid) sval += pm_b * gw.z + pv_b * gw.w;
            // dp = (k - f) dx: d/dx = -1 per axis
            xb.x += gwx * sval - w * (u.x * Bb.x + u.y * Bb.z);
            xb.y += gwy * sval - w * (u.x * Bb.y + u.y * Bb.w);
        }
    }
    c.xg[i] = xb;
    c.Fg[i] = Fg;
}

// The G2P adjoint of the last substep of a segment (the others' comes with
// the P2G adjoint of the substep after them).
__global__ void __launch_bounds__(ADJ_THREADS, 3) k_adj_g2p_bwd(AdjCtx c)
{
    follow();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const StateAdjoint o{c.xb_next[i], c.vb_next[i], c.Cb_next[i], c.Fb_next[i]};
    g2p_adjoint(c, i, c.tag[i], c.in.x[i], c.in.F[i], o, c.ub_s, c.ub_w);
}

// Sum of a value over the lanes of a warp whose particles all belong to one
// scene, else over the lanes of each scene separately through atomics.
__device__ __forceinline__ void add_param_grads(double *grad, uint32_t scene, float3 g, bool valid)
{
    const unsigned full = 0xffffffffu;
    const uint32_t lead = __shfl_sync(full, scene, 0);
    if (__all_sync(full, !valid || scene == lead)) {
        double a = valid ? g.x : 0.0, b = valid ? g.y : 0.0, d = valid ? g.z : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_xor_sync(full, a, o);
            b += __shfl_xor_sync(full, b, o);
            d += __shfl_xor_sync(full, d, o);
        }
        if ((threadIdx.x & 31u) == 0u) {
            if (a != 0.0) atomicAdd(grad + 3 * lead, a);
            if (b != 0.0) atomicAdd(grad + 3 * lead + 1, b);
            if (d != 0.0) atomicAdd(grad + 3 * lead + 2, d);
        }
    } else if (valid) {
        if (g.x != 0.f) atomicAdd(grad + 3 * scene, (double)g.x);
        if (g.y != 0.f) atomicAdd(grad + 3 * scene + 1, (double)g.y);
        if (g.z != 0.f) atomicAdd(grad + 3 * scene + 2, (double)g.z);
    }
}

// The P2G adjoint of one substep: each particle gathers, for its nine nodes,
// the adjoints of the node sums, then reverses its own P2G contribution and
// stress, adds the G2P parts, and has the adjoints of the substep's inputs and the
// parameter gradients.  TURN: those inputs are the outputs of the substep before,
// whose state is c.out and whose G2P adjoint follows at once; else they
// are written.  Bound by the latency of the gathers and by L1: the G2P
// adjoint reads its nodes' velocities a second time rather than keep them (shared
// memory for 36 KB a CTA took L1's room and a CTA per SM: per million particles
// 110.8 us, 96.8 without it, 91.8 with 64 registers for a fourth CTA; as two kernels
// 47 + 73).  Where the CTAs are at most two per SM, four cannot meet: the instance
// with room for all registers (1,024 particles: 7.6 -> 6.9 us, 65,536: 10.1 -> 9.6;
// above that line it loses, 98,304: 12.6 against 15.9).
template <bool TURN, int CTAS>
__global__ void __launch_bounds__(ADJ_THREADS, CTAS) k_adj_p2g_bwd(AdjCtx c)
{
    follow();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < c.n;
    const uint32_t tag = valid ? c.tag[i] : 0u, scene = tag >> 1;
    float3 pg = make_float3(0.f, 0.f, 0.f);
    StateAdjoint a{};
    bool ok = valid;
    if (valid) {
        const AdjScene &S = c.scenes[scene];
        const bool liquid = (tag & 1u) != 0u;
        const float2 x = c.in.x[i], v = c.in.v[i];
        const float4 C = c.in.C[i], F = c.in.F[i];
        const float vol = c.vol[i];
        Prepared p;
        AdjStencil st;
        ok = adj_prepare(S, liquid, vol, C, F, p) && adj_stencil(S, x, st);
        if (ok) {
            float2 xb = c.xg[i], vb = make_float2(0.f, 0.f);
            float4 Ab = make_float4(0.f, 0.f, 0.f, 0.f);
            float vliq_b = 0.f;
#pragma unroll
            for (int oy = 0; oy < 3; ++oy) {
                const float dpy = ((float)oy - st.fy) * S.dx;
#pragma unroll
                for (int ox = 0; ox < 3; ++ox) {
                    const float w = st.wx[ox] * st.wy[oy];
                    const float dpx = ((float)ox - st.fx) * S.dx;
                    const int ix = st.bx + ox, iy = st.by + oy;
                    const uint32_t n = adj_node(S, ix, iy);
                    // the node's sum adjoints (k_adj_grid_bwd): momentum, mass, liquid volume
                    const float4 g = liquid ? c.ub_w[n] : c.ub_s[n];
                    const float Qx_b = g.x, Qy_b = g.y, M_b = g.z, V_b = g.w;
                    // P2G adjoint of M += w m, Q += w (m v + A dp), V += w vliq
                    vb.x += w * p.m * Qx_b;
                    vb.y += w * p.m * Qy_b;
                    Ab.x += w * Qx_b * dpx;
                    Ab.y += w * Qx_b * dpy;
                    Ab.z += w * Qy_b * dpx;
                    Ab.w += w * Qy_b * dpy;
                    if (liquid) vliq_b += w * V_b;
                    const float qx = p.m * v.x + p.A.x * dpx + p.A.y * dpy;
                    const float qy = p.m * v.y + p.A.z * dpx + p.A.w * dpy;
                    const float sval = M_b * p.m + Qx_b * qx + Qy_b * qy + (liquid ? V_b * p.vliq : 0.f);
                    const float gwx = st.dwx[ox] * st.wy[oy] * S.inv_dx, gwy = st.wx[ox] * st.dwy[oy] * S.inv_dx;
                    xb.x += gwx * sval - w * (p.A.x * Qx_b + p.A.z * Qy_b);
                    xb.y += gwy * sval - w * (p.A.y * Qx_b + p.A.w * Qy_b);
                }
            }
            // A = m C + scale s
            const float4 Cb = make_float4(p.m * Ab.x, p.m * Ab.y, p.m * Ab.z, p.m * Ab.w);
            const float4 sb = make_float4(p.scale * Ab.x, p.scale * Ab.y, p.scale * Ab.z, p.scale * Ab.w);
            float4 Fb = c.Fg[i];
            if (liquid) Fb = axpy4(vliq_b * vol, cofactor(F), Fb);
            pg = stress_adjoint(S, liquid, F, p.det, sb, Fb);
            a = StateAdjoint{xb, vb, Cb, Fb};
            if (!finite2(xb) || !finite2(vb) || !finite4(Cb) || !finite4(Fb)) adj_fail(c, ADJ_ERR_NONFINITE);
        } else {
            adj_fail(c, ADJ_ERR_NONFINITE);
        }
    }
    add_param_grads(c.param_grad, scene, pg, ok);
    if (!ok) return;
    if constexpr (TURN) {
        g2p_adjoint(c, i, tag, c.out.x[i], c.out.F[i], a, c.ub_s_prev, c.ub_w_prev);
    } else {
        c.xb[i] = a.x;
        c.vb[i] = a.v;
        c.Cb[i] = a.C;
        c.Fb[i] = a.F;
    }
}

// ----------------------------------------------------------------- host ---

struct mpm_adjoint {
    int device = 0;
    cudaStream_t stream = nullptr;
    RecordStage *stage = nullptr;  // pinned staging of the device
    uint32_t n = 0, n_scenes = 0, n_nodes = 0;
    std::vector<AdjScene> scenes;
    AdjScene *d_scenes = nullptr;
    uint32_t *tag = nullptr;
    float *vol = nullptr;
    // the states of a run: init is state 0; checkpoint s (s > 0) state s * every;
    // the others alternate in ping.  tape[j] and tape_s / tape_w[j]: state and
    // sums of substep j of the segment tape_segment (-1: none yet).
    AdjState init{}, ping[2]{};
    std::vector<AdjState> checkpoints, tape;
    std::vector<float4 *> tape_s, tape_w;
    int tape_segment = -1;
    float4 *sum_s = nullptr, *sum_w = nullptr;  // zero between substeps
    uint8_t *mark = nullptr;                    // per substep (0 .. steps) and 16 x 16-node tile: solid, water
    size_t mark_count = 0;
    uint32_t *tile_scene = nullptr;             // per tile
    uint32_t n_tiles = 0, tile_ctas = 1;
    unsigned sms = 1;
    float2 *xb[2]{}, *vb[2]{}, *xg = nullptr;
    float4 *Cb[2]{}, *Fb[2]{}, *Fg = nullptr, *ub_w[2]{}, *ub_s[2]{};
    float2 *gv_s = nullptr;  // node velocities of the substep at hand
    float4 *gv_w = nullptr;
    // loss per scene, the status word (in 8 bytes), three parameter gradients per scene
    double *results = nullptr;
    float2 *target = nullptr, *final_x = nullptr;
    uint32_t steps = 0, every = 0;
    bool forward_done = false;
    cudaEvent_t ev[4]{};
    float forward_ms = 0.f, backward_ms = 0.f;

    double *loss() const { return results; }
    uint32_t *status() const { return reinterpret_cast<uint32_t *>(results + n_scenes); }
    double *param_grad() const { return results + n_scenes + 1; }
};

namespace {

template <typename T>
cudaError_t adj_alloc(T **ptr, size_t count)
{
    *ptr = nullptr;
    return cudaMalloc(reinterpret_cast<void **>(ptr), std::max<size_t>(count, 1) * sizeof(T));
}

cudaError_t alloc_state(AdjState &s, size_t n)
{
    cudaError_t e = adj_alloc(&s.x, n);
    if (e == cudaSuccess) e = adj_alloc(&s.v, n);
    if (e == cudaSuccess) e = adj_alloc(&s.C, n);
    if (e == cudaSuccess) e = adj_alloc(&s.F, n);
    return e;
}

void free_state(AdjState &s)
{
    for (void *p : {(void *)s.x, (void *)s.v, (void *)s.C, (void *)s.F})
        if (p) cudaFree(p);
    s = AdjState{};
}

void free_engine(mpm_adjoint *a)
{
    if (!a) return;
    cudaSetDevice(a->device);
    if (a->stream) cudaStreamSynchronize(a->stream);
    free_state(a->init);
    free_state(a->ping[0]);
    free_state(a->ping[1]);
    for (auto &s : a->checkpoints) free_state(s);
    for (auto &s : a->tape) free_state(s);
    for (float4 *p : a->tape_s) cudaFree(p);
    for (float4 *p : a->tape_w) cudaFree(p);
    void *ptrs[] = {a->mark,  a->tile_scene, a->d_scenes, a->tag,   a->vol,   a->sum_s, a->sum_w,
                    a->xb[0], a->xb[1],      a->vb[0],    a->vb[1], a->xg,    a->ub_s[0], a->ub_s[1], a->ub_w[0], a->ub_w[1], a->Cb[0], a->Cb[1],
                    a->Fb[0], a->Fb[1],      a->Fg,       a->gv_s,  a->gv_w,  a->results, a->target, a->final_x};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    for (cudaEvent_t e : a->ev)
        if (e) cudaEventDestroy(e);
    if (a->stream) cudaStreamDestroy(a->stream);
    if (a->stage) a->stage->release();
    delete a;
}

int err(int code, const char *fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    return host_error(code, buf);
}

#define ADJ_TRY(expr)                                                                                    \
    do {                                                                                                 \
        cudaError_t e__ = (expr);                                                                        \
        if (e__ != cudaSuccess) return err(MPM_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(e__)); \
    } while (0)

AdjCtx make_adj_ctx(mpm_adjoint *a, const AdjState &in, const AdjState &out, float4 *sum_s, float4 *sum_w, int adj)
{
    AdjCtx c{};
    c.scenes = a->d_scenes;
    c.tag = a->tag;
    c.vol = a->vol;
    c.n = a->n;
    c.status = a->status();
    c.in = in;
    c.out = out;
    c.sum_s = sum_s;
    c.sum_w = sum_w;
    c.xb_next = a->xb[adj];
    c.vb_next = a->vb[adj];
    c.Cb_next = a->Cb[adj];
    c.Fb_next = a->Fb[adj];
    c.xb = a->xb[1 - adj];
    c.vb = a->vb[1 - adj];
    c.Cb = a->Cb[1 - adj];
    c.Fb = a->Fb[1 - adj];
    c.xg = a->xg;
    c.Fg = a->Fg;
    c.ub_s = a->ub_s[0];
    c.ub_w = a->ub_w[0];
    c.gv_s = a->gv_s;
    c.gv_w = a->gv_w;
    c.param_grad = a->param_grad();
    c.target = a->target;
    c.loss = a->loss();
    return c;
}

unsigned blocks(uint32_t n) { return std::max(1u, (n + ADJ_THREADS - 1) / ADJ_THREADS); }

// Enqueues a kernel over the particles (one per thread) or over the tiles.
template <class... Args>
void over_particles(mpm_adjoint *a, void (*kernel)(Args...), Args... args)
{
    launch_following(a->stream, kernel, dim3(blocks(a->n)), dim3(ADJ_THREADS), 0, args...);
}

template <class... Args>
void over_tiles(mpm_adjoint *a, void (*kernel)(Args...), Args... args)
{
    launch_following(a->stream, kernel, dim3(std::min(a->n_tiles, a->tile_ctas)), dim3(ADJ_THREADS), 0, args...);
}

// The tile marks of substep k (of its input positions).
uint8_t *marks_of(mpm_adjoint *a, uint32_t k) { return a->mark + (size_t)k * a->n_tiles * 2u; }

const uint32_t *tile_scenes(const mpm_adjoint *a) { return a->tile_scene; }
const uint8_t *tile_marks(mpm_adjoint *a, uint32_t k) { return marks_of(a, k); }

// The input state of substep k of the forward pass, whose last segment runs on
// the tape (segment `last` from substep last * every).
const AdjState &state_of(mpm_adjoint *a, uint32_t k, uint32_t last)
{
    if (k == 0u) return a->init;
    if (k < a->steps && k % a->every == 0u) return a->checkpoints[k / a->every];
    if (k < a->steps && k / a->every == last) return a->tape[k % a->every];
    return a->ping[k & 1u];
}

// Substeps start .. start + len - 1 from state(start): the P2G of the first when
// `p2g_first`, then per substep the grid update and G2P with the next P2G.
// `tape` keeps the sums; the G2P of the last substep runs when `last_g2p`, with the
// P2G after it when `last_p2g`.  Every P2G marks the tiles of its positions
// (adding to the marks when a segment is recomputed: float atomics may move
// a position by its last bits).
template <class State>
cudaError_t run_substeps(mpm_adjoint *a, uint32_t start, uint32_t len, const State &state, bool tape, bool p2g_first,
                         bool last_g2p, bool last_p2g)
{
    if (p2g_first) {
        AdjCtx c = make_adj_ctx(a, state(start), state(start), a->sum_s, a->sum_w, 0);
        c.mark_out = marks_of(a, start);
        over_particles(a, k_adj_p2g, c);
    }
    for (uint32_t j = 0; j < len; ++j) {
        const uint32_t k = start + j;
        AdjCtx c = make_adj_ctx(a, state(k), state(k + 1u), a->sum_s, a->sum_w, 0);
        over_tiles(a, k_adj_grid_fwd<true>, c, tile_scenes(a), tile_marks(a, k), a->n_tiles,
                   tape ? a->tape_s[j] : nullptr, tape ? a->tape_w[j] : nullptr);
        if (j + 1u == len && !last_g2p) break;
        c.mark_out = marks_of(a, k + 1u);
        if (j + 1u < len || last_p2g)
            over_particles(a, k_adj_g2p<true>, c);
        else
            over_particles(a, k_adj_g2p<false>, c);
    }
    return cudaGetLastError();
}

int check_status(uint32_t st, const char *what)
{
    if (st != 0u)
        return err(MPM_ERR_STATE, "%s stopped: %s%s%s", what, (st & ADJ_ERR_STENCIL) ? "a particle left the grid; " : "",
                   (st & ADJ_ERR_DETERMINANT) ? "a deformation gradient lost its positive determinant; " : "",
                   (st & ADJ_ERR_NONFINITE) ? "a non-finite value appeared" : "");
    return MPM_OK;
}

}  // namespace

extern "C" {

int mpma_create(const mpm_config *configs, uint32_t scene_count, const uint32_t *particle_counts,
                const float *packed_particles, const float *gravity_xy, mpm_adjoint **out)
{
    host_clear_error();
    if (!configs || !particle_counts || !packed_particles || !gravity_xy || !out)
        return err(MPM_ERR_INVALID_ARGUMENT, "configs, particle_counts, packed_particles, gravity_xy and out must not be NULL");
    *out = nullptr;
    if (scene_count < 1) return err(MPM_ERR_INVALID_ARGUMENT, "a batch needs at least one scene");
    std::vector<AdjScene> scenes(scene_count);
    std::vector<uint32_t> tag;
    std::vector<float> vol;
    std::vector<float2> x, v;
    std::vector<float4> C, F;
    uint64_t total = 0, nodes = 0;
    std::vector<uint32_t> tile_scene;  // per tile
    {
        size_t all = 0;
        for (uint32_t k = 0; k < scene_count; ++k) all += particle_counts[k];
        for (auto *a : {&x, &v}) a->reserve(all);
        for (auto *a : {&C, &F}) a->reserve(all);
        vol.reserve(all);
        tag.reserve(all);
    }
    for (uint32_t k = 0; k < scene_count; ++k) {
        const mpm_config &cfg = configs[k];
        if (cfg.cells_x < 1 || cfg.cells_y < 1 || cfg.cells_x > 65536 || cfg.cells_y > 65536 || !(cfg.cell_size > 0.f))
            return err(MPM_ERR_INVALID_ARGUMENT, "scene %u: invalid grid", k);
        AdjScene &S = scenes[k];
        S.n = particle_counts[k];
        S.p_base = (uint32_t)total;
        S.node_base = (uint32_t)nodes;
        S.node_w = cfg.cells_x + 3;
        S.cells_x = cfg.cells_x;
        S.cells_y = cfg.cells_y;
        S.dx = cfg.cell_size;
        S.inv_dx = 1.0f / cfg.cell_size;
        S.gs = (float)(4.0 / ((double)cfg.cell_size * cfg.cell_size));
        S.gx = gravity_xy[2 * k];
        S.gy = gravity_xy[2 * k + 1];
        S.domain_w = (float)((double)cfg.cells_x * cfg.cell_size);
        S.domain_h = (float)((double)cfg.cells_y * cfg.cell_size);
        S.solid_mass = cfg.particle_mass;
        S.wall_friction = cfg.wall_friction;
        bool have_liquid = false, have_solid = false;
        for (uint32_t j = 0; j < S.n; ++j) {
            const float *w = packed_particles + (size_t)(total + j) * MPM_PARTICLE_WORDS;
            uint32_t model;
            std::memcpy(&model, &w[13], 4);
            const bool liq = model == MODEL_WATER;
            if (!liq && model != MODEL_FIXED_COROTATED)
                return err(MPM_ERR_INVALID_ARGUMENT,
                           "scene %u particle %u: the adjoint takes Tait water and fixed-corotated solids only", k, j);
            if (liq) {
                if (!(w[18] > 0.f) || !(w[14] > 0.f) || !(w[16] > 0.f))
                    return err(MPM_ERR_INVALID_ARGUMENT, "scene %u particle %u: water needs a Tait exponent", k, j);
                if (!have_liquid) {
                    S.tait = w[14], S.rho = w[16], S.gamma = w[18];
                    have_liquid = true;
                } else if (w[14] != S.tait || w[16] != S.rho || w[18] != S.gamma) {
                    return err(MPM_ERR_INVALID_ARGUMENT, "scene %u: every water particle must share its material", k);
                }
            } else {
                if (!have_solid) {
                    S.lambda_s = w[14], S.mu_s = w[15];
                    have_solid = true;
                } else if (w[14] != S.lambda_s || w[15] != S.mu_s) {
                    return err(MPM_ERR_INVALID_ARGUMENT, "scene %u: every solid particle must share its material", k);
                }
            }
            x.push_back(make_float2(w[0], w[1]));
            v.push_back(make_float2(w[2], w[3]));
            C.push_back(make_float4(w[4], w[5], w[6], w[7]));
            F.push_back(make_float4(w[8], w[9], w[10], w[11]));
            vol.push_back(w[17]);
            tag.push_back((k << 1) | (liq ? 1u : 0u));
        }
        total += S.n;
        nodes += (uint64_t)(cfg.cells_x + 3) * (cfg.cells_y + 3);
        S.tile_base = (uint32_t)tile_scene.size();
        S.tiles_x = (cfg.cells_x + 3 + ADJ_TILE - 1) / ADJ_TILE;
        tile_scene.insert(tile_scene.end(), (size_t)S.tiles_x * ((cfg.cells_y + 3 + ADJ_TILE - 1) / ADJ_TILE), k);
        // (this also keeps the tiles below 2^30)
        if (total > 0x7fffffffull || nodes > 0x7fffffffull)
            return err(MPM_ERR_INVALID_ARGUMENT, "the batch exceeds the GPU index range");
    }
    int device = configs[0].device, count = 0;
    ADJ_TRY(cudaGetDeviceCount(&count));
    if (device < 0 || device >= count) return err(MPM_ERR_INVALID_ARGUMENT, "device %d is not available", device);
    ADJ_TRY(cudaSetDevice(device));
    mpm_adjoint *a = new mpm_adjoint();
    a->device = device;
    a->stage = &RecordStage::of(device);
    a->stage->retain();
    a->n = (uint32_t)total;
    a->n_scenes = scene_count;
    a->n_nodes = (uint32_t)nodes;
    a->scenes = scenes;
    auto fail = [&](int code) {
        free_engine(a);
        return code;
    };
#define ADJ_ALLOC(ptr, cnt)                                                                             \
    do {                                                                                                \
        cudaError_t e__ = adj_alloc(&(ptr), (cnt));                                                     \
        if (e__ != cudaSuccess) return fail(err(MPM_ERR_CUDA, "cudaMalloc(%s) failed: %s", #ptr, cudaGetErrorString(e__))); \
    } while (0)
    if (cudaStreamCreateWithFlags(&a->stream, cudaStreamNonBlocking) != cudaSuccess)
        return fail(err(MPM_ERR_CUDA, "cudaStreamCreate failed"));
    for (cudaEvent_t &e : a->ev)
        if (cudaEventCreate(&e) != cudaSuccess) return fail(err(MPM_ERR_CUDA, "cudaEventCreate failed"));
    const size_t n = a->n;
    ADJ_ALLOC(a->d_scenes, scene_count);
    ADJ_ALLOC(a->tag, n);
    ADJ_ALLOC(a->vol, n);
    if (alloc_state(a->init, n) != cudaSuccess || alloc_state(a->ping[0], n) != cudaSuccess ||
        alloc_state(a->ping[1], n) != cudaSuccess)
        return fail(err(MPM_ERR_CUDA, "state allocation failed"));
    ADJ_ALLOC(a->sum_s, nodes);
    ADJ_ALLOC(a->sum_w, nodes);
    for (int b = 0; b < 2; ++b) {
        ADJ_ALLOC(a->xb[b], n);
        ADJ_ALLOC(a->vb[b], n);
        ADJ_ALLOC(a->Cb[b], n);
        ADJ_ALLOC(a->Fb[b], n);
    }
    ADJ_ALLOC(a->xg, n);
    ADJ_ALLOC(a->Fg, n);
    for (int b = 0; b < 2; ++b) {
        ADJ_ALLOC(a->ub_s[b], nodes);
        ADJ_ALLOC(a->ub_w[b], nodes);
    }
    ADJ_ALLOC(a->gv_s, nodes);
    ADJ_ALLOC(a->gv_w, nodes);
    ADJ_ALLOC(a->results, 4 * (size_t)scene_count + 1);
    ADJ_ALLOC(a->target, n);
    ADJ_ALLOC(a->final_x, n);
    a->n_tiles = (uint32_t)tile_scene.size();
    ADJ_ALLOC(a->tile_scene, tile_scene.size());
#undef ADJ_ALLOC
    int sms = 1;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
        return fail(err(MPM_ERR_CUDA, "device query failed"));
    a->sms = (unsigned)sms;
    a->tile_ctas = (uint32_t)sms * 8u;  // 2048 threads per SM
    bool ok = cudaMemcpy(a->d_scenes, scenes.data(), scene_count * sizeof(AdjScene), cudaMemcpyHostToDevice) == cudaSuccess;
    ok = ok && cudaMemcpy(a->tag, tag.data(), n * sizeof(uint32_t), cudaMemcpyHostToDevice) == cudaSuccess;
    ok = ok && cudaMemcpy(a->vol, vol.data(), n * sizeof(float), cudaMemcpyHostToDevice) == cudaSuccess;
    ok = ok && cudaMemcpy(a->init.x, x.data(), n * sizeof(float2), cudaMemcpyHostToDevice) == cudaSuccess;
    ok = ok && cudaMemcpy(a->init.v, v.data(), n * sizeof(float2), cudaMemcpyHostToDevice) == cudaSuccess;
    ok = ok && cudaMemcpy(a->init.C, C.data(), n * sizeof(float4), cudaMemcpyHostToDevice) == cudaSuccess;
    ok = ok && cudaMemcpy(a->init.F, F.data(), n * sizeof(float4), cudaMemcpyHostToDevice) == cudaSuccess;
    ok = ok && cudaMemset(a->results, 0, (4 * (size_t)scene_count + 1) * sizeof(double)) == cudaSuccess;
    ok = ok && cudaMemset(a->sum_s, 0, nodes * sizeof(float4)) == cudaSuccess;
    ok = ok && cudaMemset(a->sum_w, 0, nodes * sizeof(float4)) == cudaSuccess;
    ok = ok && cudaDeviceSynchronize() == cudaSuccess;  // before work of the engine's own stream
    ok = ok && cudaMemcpy(a->tile_scene, tile_scene.data(), tile_scene.size() * sizeof(uint32_t),
                          cudaMemcpyHostToDevice) == cudaSuccess;
    if (!ok) return fail(err(MPM_ERR_CUDA, "upload failed"));
    *out = a;
    return MPM_OK;
}

int mpma_set_parameters(mpm_adjoint *a, const float *parameters)
{
    host_clear_error();
    if (!a || !parameters) return err(MPM_ERR_INVALID_ARGUMENT, "engine and parameters must not be NULL");
    for (uint32_t k = 0; k < a->n_scenes; ++k) {
        const float *p = parameters + 3 * k;
        if (!std::isfinite(p[0]) || !std::isfinite(p[1]) || !std::isfinite(p[2]) || p[0] < 0.f)
            return err(MPM_ERR_INVALID_ARGUMENT, "scene %u: parameters must be finite", k);
        a->scenes[k].tait = p[0];
        a->scenes[k].lambda_s = p[1];
        a->scenes[k].mu_s = p[2];
    }
    ADJ_TRY(cudaSetDevice(a->device));
    ADJ_TRY(cudaMemcpy(a->d_scenes, a->scenes.data(), a->n_scenes * sizeof(AdjScene), cudaMemcpyHostToDevice));
    a->forward_done = false;
    return MPM_OK;
}

int mpma_get_parameters(mpm_adjoint *a, float *parameters)
{
    host_clear_error();
    if (!a || !parameters) return err(MPM_ERR_INVALID_ARGUMENT, "engine and parameters must not be NULL");
    for (uint32_t k = 0; k < a->n_scenes; ++k) {
        parameters[3 * k] = a->scenes[k].tait;
        parameters[3 * k + 1] = a->scenes[k].lambda_s;
        parameters[3 * k + 2] = a->scenes[k].mu_s;
    }
    return MPM_OK;
}

int mpma_set_velocities(mpm_adjoint *a, const float *velocities)
{
    host_clear_error();
    if (!a || !velocities) return err(MPM_ERR_INVALID_ARGUMENT, "engine and velocities must not be NULL");
    ADJ_TRY(cudaSetDevice(a->device));
    ADJ_TRY(a->stage->copy_in(a->stream, a->init.v, velocities, (size_t)a->n * sizeof(float2)));
    a->forward_done = false;
    return MPM_OK;
}

int mpma_forward(mpm_adjoint *a, uint32_t substeps, const float *dts, uint32_t checkpoint_every,
                 const float *targets, double *loss)
{
    host_clear_error();
    if (!a || !dts || !targets) return err(MPM_ERR_INVALID_ARGUMENT, "engine, dts and targets must not be NULL");
    if (substeps < 1) return err(MPM_ERR_INVALID_ARGUMENT, "substeps must be positive");
    if (checkpoint_every < 1 || checkpoint_every > 1024)
        return err(MPM_ERR_INVALID_ARGUMENT, "checkpoint_every must lie in [1, 1024]");
    for (uint32_t k = 0; k < a->n_scenes; ++k) {
        if (!(dts[k] > 0.f) || !std::isfinite(dts[k])) return err(MPM_ERR_INVALID_ARGUMENT, "scene %u: dt must be positive", k);
        a->scenes[k].dt = dts[k];
    }
    ADJ_TRY(cudaSetDevice(a->device));
    ADJ_TRY(cudaMemcpyAsync(a->d_scenes, a->scenes.data(), a->n_scenes * sizeof(AdjScene), cudaMemcpyHostToDevice, a->stream));
    ADJ_TRY(a->stage->copy_in(a->stream, a->target, targets, (size_t)a->n * sizeof(float2)));
    const uint32_t n_check = (substeps + checkpoint_every - 1) / checkpoint_every;
    if (a->checkpoints.size() != n_check || a->every != checkpoint_every) {
        a->tape_segment = -1;
        a->every = 0;
        for (auto &s : a->checkpoints) free_state(s);
        for (auto &s : a->tape) free_state(s);
        for (float4 *p : a->tape_s) cudaFree(p);
        for (float4 *p : a->tape_w) cudaFree(p);
        a->checkpoints.assign(n_check, AdjState{});
        a->tape.assign(checkpoint_every, AdjState{});
        a->tape_s.assign(checkpoint_every, nullptr);
        a->tape_w.assign(checkpoint_every, nullptr);
        // state 0 is the initial state, and substep 0 of a segment has its checkpoint
        for (uint32_t k = 1; k < n_check; ++k)
            if (alloc_state(a->checkpoints[k], a->n) != cudaSuccess) return err(MPM_ERR_CUDA, "checkpoint allocation failed");
        for (uint32_t j = 0; j < checkpoint_every; ++j) {
            if ((j > 0 && alloc_state(a->tape[j], a->n) != cudaSuccess) ||
                adj_alloc(&a->tape_s[j], a->n_nodes) != cudaSuccess || adj_alloc(&a->tape_w[j], a->n_nodes) != cudaSuccess)
                return err(MPM_ERR_CUDA, "recompute tape allocation failed");
        }
    }
    a->steps = substeps;
    a->every = checkpoint_every;
    const size_t marks = ((size_t)substeps + 1) * a->n_tiles * 2;
    if (a->mark_count < marks) {
        cudaFree(a->mark);
        a->mark = nullptr;
        a->mark_count = 0;
        if (adj_alloc(&a->mark, marks) != cudaSuccess) return err(MPM_ERR_CUDA, "tile mark allocation failed");
        a->mark_count = marks;
    }
    ADJ_TRY(cudaMemsetAsync(a->mark, 0, marks, a->stream));
    ADJ_TRY(cudaMemsetAsync(a->results, 0, (a->n_scenes + 1) * sizeof(double), a->stream));
    ADJ_TRY(cudaEventRecord(a->ev[0], a->stream));
    // the last segment (with checkpoint_every >= substeps the whole run) keeps
    // its states and sums, so the backward pass does not recompute it
    const uint32_t last = n_check - 1, last_start = last * checkpoint_every;
    const auto state = [&](uint32_t k) -> const AdjState & { return state_of(a, k, last); };
    if (last_start > 0) ADJ_TRY(run_substeps(a, 0, last_start, state, false, true, true, true));
    ADJ_TRY(run_substeps(a, last_start, substeps - last_start, state, true, last_start == 0, true, false));
    ADJ_TRY(cudaEventRecord(a->ev[1], a->stream));
    a->tape_segment = (int)last;
    const AdjState &final_state = state(substeps);
    over_particles(a, k_adj_loss, make_adj_ctx(a, final_state, final_state, a->sum_s, a->sum_w, 0));
    ADJ_TRY(cudaGetLastError());
    ADJ_TRY(cudaMemcpyAsync(a->final_x, final_state.x, (size_t)a->n * sizeof(float2), cudaMemcpyDeviceToDevice, a->stream));
    std::vector<double> got(a->n_scenes + 1);
    ADJ_TRY(cudaMemcpyAsync(got.data(), a->results, got.size() * sizeof(double), cudaMemcpyDeviceToHost, a->stream));
    ADJ_TRY(cudaStreamSynchronize(a->stream));
    uint32_t st;
    std::memcpy(&st, &got[a->n_scenes], sizeof st);
    const int rc = check_status(st, "the forward pass");
    if (rc != MPM_OK) return rc;
    ADJ_TRY(cudaEventElapsedTime(&a->forward_ms, a->ev[0], a->ev[1]));
    if (loss) std::memcpy(loss, got.data(), a->n_scenes * sizeof(double));
    a->forward_done = true;
    return MPM_OK;
}

int mpma_backward(mpm_adjoint *a, float *grad_velocities, double *grad_parameters)
{
    host_clear_error();
    if (!a) return err(MPM_ERR_INVALID_ARGUMENT, "engine must not be NULL");
    if (!a->forward_done) return err(MPM_ERR_STATE, "backward needs a completed forward pass of the same inputs");
    ADJ_TRY(cudaSetDevice(a->device));
    ADJ_TRY(cudaMemsetAsync(a->param_grad(), 0, 3 * a->n_scenes * sizeof(double), a->stream));
    ADJ_TRY(cudaEventRecord(a->ev[2], a->stream));
    int adj = 0;  // the adjoint of the current substep's outputs sits in buffer `adj` (seeded by the loss)
    const uint32_t K = a->every;
    for (int seg = (int)a->checkpoints.size() - 1; seg >= 0; --seg) {
        const uint32_t start = (uint32_t)seg * K, len = std::min(K, a->steps - start);
        // a substep's input state on the tape; the output of the last one is not kept
        const auto state = [&](uint32_t k) -> const AdjState & {
            if (k == start) return seg == 0 ? a->init : a->checkpoints[seg];
            return k < start + len ? a->tape[k - start] : a->ping[0];
        };
        if (a->tape_segment != seg) {
            a->tape_segment = -1;
            ADJ_TRY(run_substeps(a, start, len, state, true, true, false, false));
            a->tape_segment = seg;
        }
        // substep by substep from the segment's last; node adjoints of one
        // substep in one pair of buffers, of the one before it in the other
        int ub = 0;
        const auto substep = [&](uint32_t k) {
            const uint32_t j = k - start;
            AdjCtx c = make_adj_ctx(a, state(k), j > 0u ? state(k - 1u) : state(k), a->tape_s[j], a->tape_w[j], adj);
            c.ub_s = a->ub_s[ub], c.ub_w = a->ub_w[ub];
            c.ub_s_prev = a->ub_s[1 - ub], c.ub_w_prev = a->ub_w[1 - ub];
            return c;
        };
        const uint32_t last = start + len - 1u;
        over_tiles(a, k_adj_grid_fwd<false>, substep(last), tile_scenes(a), tile_marks(a, last), a->n_tiles, (float4 *)nullptr,
                   (float4 *)nullptr);
        over_particles(a, k_adj_g2p_bwd, substep(last));
        for (uint32_t k = last; k > start; --k) {
            over_tiles(a, k_adj_grid_bwd<true>, substep(k), tile_scenes(a), tile_marks(a, k), tile_marks(a, k - 1u), a->n_tiles,
                       (const float4 *)a->tape_s[k - 1u - start], (const float4 *)a->tape_w[k - 1u - start]);
            if (blocks(a->n) <= 2u * a->sms)
                over_particles(a, k_adj_p2g_bwd<true, 2>, substep(k));
            else
                over_particles(a, k_adj_p2g_bwd<true, 4>, substep(k));
            ub = 1 - ub;
        }
        over_tiles(a, k_adj_grid_bwd<false>, substep(start), tile_scenes(a), tile_marks(a, start), (const uint8_t *)nullptr,
                   a->n_tiles, (const float4 *)nullptr, (const float4 *)nullptr);
        over_particles(a, k_adj_p2g_bwd<false, 4>, substep(start));
        adj = 1 - adj;
        ADJ_TRY(cudaGetLastError());
    }
    ADJ_TRY(cudaEventRecord(a->ev[3], a->stream));
    std::vector<double> got(3 * (size_t)a->n_scenes + 1);
    ADJ_TRY(cudaMemcpyAsync(got.data(), a->results + a->n_scenes, got.size() * sizeof(double), cudaMemcpyDeviceToHost,
                            a->stream));
    ADJ_TRY(cudaStreamSynchronize(a->stream));
    uint32_t st;
    std::memcpy(&st, &got[0], sizeof st);
    const int rc = check_status(st, "the adjoint pass");
    if (rc != MPM_OK) return rc;
    ADJ_TRY(cudaEventElapsedTime(&a->backward_ms, a->ev[2], a->ev[3]));
    const size_t bytes = (size_t)a->n * sizeof(float2);
    if (grad_velocities) ADJ_TRY(a->stage->copy_out(a->stream, a->vb[adj], bytes, grad_velocities, bytes, nullptr));
    if (grad_parameters) std::memcpy(grad_parameters, got.data() + 1, 3 * a->n_scenes * sizeof(double));
    return MPM_OK;
}

int mpma_read_positions(mpm_adjoint *a, float *positions)
{
    host_clear_error();
    if (!a || !positions) return err(MPM_ERR_INVALID_ARGUMENT, "engine and positions must not be NULL");
    if (!a->forward_done) return err(MPM_ERR_STATE, "no forward pass has completed");
    ADJ_TRY(cudaSetDevice(a->device));
    const size_t bytes = (size_t)a->n * sizeof(float2);
    ADJ_TRY(a->stage->copy_out(a->stream, a->final_x, bytes, positions, bytes, nullptr));
    return MPM_OK;
}

int mpma_last_ms(mpm_adjoint *a, double *forward_ms, double *backward_ms)
{
    host_clear_error();
    if (!a) return err(MPM_ERR_INVALID_ARGUMENT, "engine must not be NULL");
    if (forward_ms) *forward_ms = a->forward_ms;
    if (backward_ms) *backward_ms = a->backward_ms;
    return MPM_OK;
}

void mpma_destroy(mpm_adjoint *a) { free_engine(a); }

}  // extern "C"
