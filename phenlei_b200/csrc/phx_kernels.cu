// sm_100a kernels of the NS per-iteration path (storage layout: see
// phx_internal.h).
//
// Per-cell sums are owner-computes gathers over the cell's faces in the
// reference's face order, so no atomics touch the state (the SA cell pass sums
// convection and diffusion side by side).  Metrics are formed and kept in FP64;
// the passes read face geometry derived from them in the working precision T,
// double (FP64 path) or float (mixed path).
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>

#include <algorithm>

#include "phx_internal.h"
#include "phx_device.cuh"
#include "phx_geometry.cuh"
#include "phx_physics.cuh"

namespace phx {

// ---------------------------------------------------------------------------
// Boundary: ghost-cell state per boundary face (NSSolverUnstruct::Boundary,
// NSSolverUnstruct.cpp:13404-13515): SymmetryBCRegion (:19413),
// ViscousAdiabaticWallBCRegion (:20988), FarfieldBCRegion (:21195).
// Computed in FP64 from the FP64 master state.  Interface ghosts keep the
// state the last halo exchange gave them (Boundary skips INTERFACE faces,
// :13474); their working record and laminar viscosity are formed from it.
// ---------------------------------------------------------------------------
template <class T>
__global__ void __launch_bounds__(kThreads) boundary_kernel(DevGrid g, NsConst c, double *q, Work<T> w,
                                                            bool writeVisl)
{
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= g.nBFace) return;
    const int nt = g.nTotal;
    const int le = g.lr[f].x, re = g.nCell + f;
    const double r = q[le], u = q[nt + le], v = q[2 * nt + le], wv = q[3 * nt + le], p = q[4 * nt + le];
    double fr[4];
    ld4(g.frec + (size_t)f * kF, fr);
    const double xn = fr[0], yn = fr[1], zn = fr[2];
    double o[5] = {r, u, v, wv, p};
    const int kind = g.bkind[f];
    if (kind == BK_INTERFACE) {
#pragma unroll
        for (int k = 0; k < 5; ++k) o[k] = q[k * nt + re];
    } else if (kind == BK_SYMMETRY) {
        const double vn = xn * u + yn * v + zn * wv;
        o[1] = u - 2.0 * xn * vn;
        o[2] = v - 2.0 * yn * vn;
        o[3] = wv - 2.0 * zn * vn;
    } else if (kind == BK_WALL) {
        o[1] = -u; o[2] = -v; o[3] = -wv;
    } else if (kind == BK_FARFIELD) {
        const double *pi = c.primInf;
        const double rO = pi[0], uO = pi[1], vO = pi[2], wO = pi[3], pO = pi[4];
        const double gl = c.gama;
        const double cO = sqrt(fabs(gl * pO / rO));
        const double vnO = xn * uO + yn * vO + zn * wO;
        const double vnI = xn * u + yn * v + zn * wv;
        const double cI = sqrt(fabs(gl * p / r));
        const double gm1 = gl - 1.0;
        const double velI = sqrt(u * u + v * v + wv * wv);
        if (velI > cI) {
            if (vnI < 0.0) { for (int k = 0; k < 5; ++k) o[k] = pi[k]; }
        } else {
            const double Rp = vnI + 2.0 * cI / gm1;
            const double Rm = vnO - 2.0 * cO / gm1;
            const double vnB = 0.5 * (Rp + Rm);
            const double cB = 0.25 * (Rp - Rm) * gm1;
            double s, vtx, vty, vtz;
            if (vnB >= 0.0) {
                s = p / pow(r, gl);
                vtx = u - xn * vnI; vty = v - yn * vnI; vtz = wv - zn * vnI;
            } else {
                s = pO / pow(rO, gl);
                vtx = uO - xn * vnO; vty = vO - yn * vnO; vtz = wO - zn * vnO;
            }
            const double rB = pow((cB * cB / (s * gl)), 1.0 / gm1);
            o[0] = rB;
            o[1] = vtx + xn * vnB;
            o[2] = vty + yn * vnB;
            o[3] = vtz + zn * vnB;
            o[4] = cB * cB * rB / gl;
        }
    }
    T t[5];
    for (int k = 0; k < 5; ++k) {
        q[k * nt + re] = o[k];
        t[k] = (T)o[k];
    }
    put_state<T>(w.qrec + (size_t)re * kQ, t, (T)c.gama);
    // laminar viscosity of the ghost for the SA step (NS ComputeViscousCoeff
    // covers the ghosts, NSSolverUnstruct.cpp:6733-6745)
    if (w.trec && writeVisl) w.trec[(size_t)re * kTr + 2] = sutherland(temperature(t, (T)c.coefState), (T)c.tsuth);
}

template <class T>
void launch_boundary(const DevGrid &g, const NsConst &c, double *q64, const Work<T> &w, cudaStream_t s)
{
    if (g.nBFace == 0) return;
    boundary_kernel<T><<<(g.nBFace + kThreads - 1) / kThreads, kThreads, 0, s>>>(g, c, q64, w, true);
}

template <class T>
void launch_boundary_post(const DevGrid &g, const NsConst &c, double *q64, const Work<T> &w, cudaStream_t s)
{
    if (g.nBFace == 0) return;
    boundary_kernel<T><<<(g.nBFace + kThreads - 1) / kThreads, kThreads, 0, s>>>(g, c, q64, w, false);
}

template <class T>
__global__ void __launch_bounds__(kThreads) sync_qrec_kernel(DevGrid g, NsConst c, const double *q, Work<T> w)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.nTotal) return;
    const int nt = g.nTotal;
    T t[5];
    for (int k = 0; k < 5; ++k) t[k] = (T)q[k * nt + i];
    put_state<T>(w.qrec + (size_t)i * kQ, t, (T)c.gama);
}

template <class T>
void launch_sync_qrec(const DevGrid &g, const NsConst &c, const double *q64, const Work<T> &w, cudaStream_t s)
{
    sync_qrec_kernel<T><<<(g.nTotal + kThreads - 1) / kThreads, kThreads, 0, s>>>(g, c, q64, w);
}

// ---------------------------------------------------------------------------
// Face geometry records of the full layout (phx_geometry.cuh).  Formed in the
// passes instead, the 1M-cell bump's gradient takes 139 us (118), its face and cell
// passes 300 (255) and its SA residual 241 (181), mixed: square roots, divisions and
// conversions in FP64 beside single-precision work.  In FP64 it comes to about the
// same (gradient 288 -> 250, face and cell passes 609 -> 628, SA residual 286 -> 319).
// ---------------------------------------------------------------------------
template <class T>
__global__ void __launch_bounds__(kThreads) face_geometry_kernel(DevGrid g, NsConst c, Work<T> w)
{
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= g.nFace) return;
    const int2 lr = ld(g.lr + f);
    T nr[4], r[5][4];
    form_normal<T>(g, c.gradient == 1, f, lr.x, lr.y, nr);
    st4(w.fnrm + (size_t)f * kNrm, nr);
    const int n = (c.viscous ? kGeo<true> : kGeo<false>) / 4;
    if (c.viscous) form_face<T, true>(g, f, lr.x, lr.y, r[0], r[1], r[2], r[3], r[4]);
    else form_face<T, false>(g, f, lr.x, lr.y, r[0], r[1], r[2], r[3], r[4]);
#pragma unroll
    for (int k = 0; k < 5; ++k)
        if (k < n) st4(w.fgeo + (size_t)f * n * 4 + k * 4, r[k]);
    if (w.fsa) {
        T sa[8];
        form_sa<T>(g, f, lr.x, lr.y, sa);
        st8(w.fsa + (size_t)f * kGeoSa, sa);
    }
}

template <class T>
void launch_face_geometry(const DevGrid &g, const NsConst &c, const Work<T> &w, cudaStream_t s)
{
    face_geometry_kernel<T><<<(g.nFace + kThreads - 1) / kThreads, kThreads, 0, s>>>(g, c, w);
}

// ---------------------------------------------------------------------------
// Gradient + limiter, fused per cell:
//  Green-Gauss cell gradient (UnstructGrid::CompGradientGGCell,
//  Geo_UnstructGrid.cpp:3220-3284) or least-squares gradient
//  (CompGradientLSQ, :3996-4085, weights of ComputeWeight :3761-3935) of the 5
//  primitives, and for viscous runs of the temperature (GetGradientField,
//  NSSolverUnstruct.cpp:18244-18330), accumulated in the reference's face
//  order; then the scalar Venkatakrishnan limiter from rho and p
//  (Limiter::VencatLimiter7, Limiter.cpp:1091-1200, neighbour min/max of
//  Limiter::MinMaxDiff :1202-1252 over interior faces), zeroed next to
//  far-field boundaries (SetLimitBoundary, Geo_UnstructGrid.cpp:10744-10775).
// ---------------------------------------------------------------------------
// GG-node node values (NSSolverUnstruct::ComputeNodeValue,
// NSSolverUnstruct.cpp:4734-5080, and ModifyNodeValue :5083-5116) of the
// current state: per node the 1/distance-weighted sum of its contributions in
// the reference's order (a boundary face gives 0.5 (owner + ghost), a cell its
// value) over the weight sum, 0 where the sum is not above SMALL.  The
// reference forms node values in PostSolve after the update and the boundary
// but without recomputing the temperature (Controller::PostSolve,
// Controller.cpp:5063-5205; SetBoundaryValueOfField :1467-1491), so the
// temperature node values its next gradient reads are those of the previous
// state: slot 6 takes slot 5 of the previous call (havePrev), or this state's
// after a state import, as at initialisation (NSSolver::InitDependentVariables,
// NSSolver.cpp:757-790).
template <class T>
__global__ void __launch_bounds__(kThreads) node_value_kernel(DevGrid g, NsConst c, Work<T> w, int havePrev)
{
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= g.nNode) return;
    const T coef = (T)c.coefState;
    T acc[6] = {0, 0, 0, 0, 0, 0};
    const int j1 = ld(g.node_off + n + 1);
    for (int j = ld(g.node_off + n); j < j1; ++j) {
        const int src = ld(g.node_src + j);
        const T wt = (T)ld(g.node_w + j);
        T v[6];
        if (src < 0) {
            const int fs = src & 0x7fffffff;
            const int le = ld(&g.lr[fs].x), re = g.nCell + fs;
            T ql[8], qg[8];
            ld8(w.qrec + (size_t)le * kQ, ql);
            ld8(w.qrec + (size_t)re * kQ, qg);
#pragma unroll
            for (int k = 0; k < 5; ++k) v[k] = T(0.5) * (ql[k] + qg[k]);
            v[5] = T(0.5) * (temperature(ql, coef) + temperature(qg, coef));
        } else {
            T qc[8];
            ld8(w.qrec + (size_t)src * kQ, qc);
#pragma unroll
            for (int k = 0; k < 5; ++k) v[k] = qc[k];
            v[5] = temperature(qc, coef);
        }
#pragma unroll
        for (int k = 0; k < 6; ++k) acc[k] += v[k] * wt;
    }
    const double ws = ld(g.node_wsum + n);
    T o[8];
#pragma unroll
    for (int k = 0; k < 6; ++k) o[k] = ws > kSmall ? acc[k] / (T)ws : T(0);
    T *r = w.nrec + (size_t)n * kN;
    o[6] = havePrev ? r[5] : o[5];
    o[7] = T(0);
    st8(r, o);
}

// Threads of a block in the passes with many registers: in double precision
// (142 here, 150 in the face pass) three blocks of 128 fit an SM, where one of 256
// did (1M-cell bump, FP64: 394 -> 289 us).
template <class T>
constexpr int kPassThreads = sizeof(T) == 4 ? 256 : 128;

// kGrad: 0 GG-cell, 1 least squares, 2 GG-node.  kCompact: geometry formed here, not stored.
template <class T, bool kTemp, int kGrad, bool kCompact>
__global__ void __launch_bounds__(kPassThreads<T>) gradient_limiter_kernel(DevGrid g, NsConst c, Work<T> w)
{
    constexpr bool kLsq = kGrad == 1;
    const int cell = blockIdx.x * blockDim.x + threadIdx.x;
    if (cell >= g.nCell) return;
    constexpr int NV = kTemp ? 6 : 5;   // variable 5: temperature
    T qc[8];
    ld8(w.qrec + (size_t)cell * kQ, qc);
    const T coef = (T)c.coefState;
    T vc[NV];
#pragma unroll
    for (int k = 0; k < 5; ++k) vc[k] = qc[k];
    if (kTemp) vc[NV - 1] = temperature(qc, coef);
    const T vol = (T)ld(g.xrec + (size_t)cell * kX + 3);
    T gx[NV], gy[NV], gz[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) gx[k] = gy[k] = gz[k] = T(0);
    T rmin = qc[0], rmax = qc[0], pmin = qc[4], pmax = qc[4];
    const int j0 = g.c2f_off[cell], j1 = g.c2f_off[cell + 1];
    for (int j = j0; j < j1; ++j) {
        const int2 e = ld(g.c2x + j);
        const bool isLeft = e.x >= 0;
        const int f = isLeft ? e.x : ~e.x;
        T qn[8], nr[4];
        ld8(w.qrec + (size_t)e.y * kQ, qn);
        if (kCompact) form_normal<T>(g, kLsq, f, isLeft ? cell : e.y, isLeft ? e.y : cell, nr);
        else ld4(w.fnrm + (size_t)f * kNrm, nr);
        T vn[NV];
#pragma unroll
        for (int k = 0; k < 5; ++k) vn[k] = qn[k];
        if (kTemp) vn[NV - 1] = temperature(qn, coef);
        if (kLsq) {
            // (q[re] - q[le]) (x[re] - x[le]) iwt in the face's own orientation,
            // added to both sides
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                const T dq = nr[3] * (isLeft ? vn[k] - vc[k] : vc[k] - vn[k]);
                gx[k] += dq * nr[0]; gy[k] += dq * nr[1]; gz[k] += dq * nr[2];
            }
        } else {
            const T nx = nr[0], ny = nr[1], nz = nr[2];
            T qf[NV];
#pragma unroll
            for (int k = 0; k < NV; ++k) qf[k] = T(0.5) * (isLeft ? (vc[k] + vn[k]) : (vn[k] + vc[k]));
            if (kGrad == 2 && (f >= g.nBFace || ld(g.btype + f) == PHX_BC_SYMMETRY)) {
                // UnstructGrid::CompGradientGGNode_NEW (Geo_UnstructGrid.cpp:4202-4309):
                // the average of the face's node values, in the face's node order
                T sn[NV];
#pragma unroll
                for (int k = 0; k < NV; ++k) sn[k] = T(0);
                const int a0 = ld(g.fn_off + f), a1 = ld(g.fn_off + f + 1);
                for (int a = a0; a < a1; ++a) {
                    T r[8];
                    ld8(w.nrec + (size_t)ld(g.fn_idx + a) * kN, r);
#pragma unroll
                    for (int k = 0; k < 5; ++k) sn[k] += r[k];
                    if (kTemp) sn[NV - 1] += r[6];
                }
                const T cnt = (T)(a1 - a0);
#pragma unroll
                for (int k = 0; k < NV; ++k) qf[k] = sn[k] / cnt;
            }
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                if (isLeft) { gx[k] += qf[k] * nx; gy[k] += qf[k] * ny; gz[k] += qf[k] * nz; }
                else { gx[k] -= qf[k] * nx; gy[k] -= qf[k] * ny; gz[k] -= qf[k] * nz; }
            }
        }
        if (f >= g.nBFace || ld(g.bkind + f) == BK_INTERFACE) {   // MinMaxDiff reads interface ghosts
            rmin = tmin(rmin, qn[0]); rmax = tmax(rmax, qn[0]);
            pmin = tmin(pmin, qn[4]); pmax = tmax(pmax, qn[4]);
        }
    }
    if (kLsq) {
        double m6[8];
        ld8(g.lsq + (size_t)cell * 8, m6);
        const T ixx = (T)m6[0], iyy = (T)m6[1], izz = (T)m6[2], ixy = (T)m6[3], ixz = (T)m6[4], iyz = (T)m6[5];
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const T tx = gx[k], ty = gy[k], tz = gz[k];
            gx[k] = ixx * tx + ixy * ty + ixz * tz;
            gy[k] = ixy * tx + iyy * ty + iyz * tz;
            gz[k] = ixz * tx + iyz * ty + izz * tz;
        }
    } else if (kGrad == 2) {
#pragma unroll
        for (int k = 0; k < NV; ++k) { gx[k] /= vol; gy[k] /= vol; gz[k] /= vol; }
    } else {
        const T ovol = T(1) / vol;
#pragma unroll
        for (int k = 0; k < NV; ++k) { gx[k] *= ovol; gy[k] *= ovol; gz[k] *= ovol; }
    }
    T gr[kG];
#pragma unroll
    for (int k = 0; k < 5; ++k) { gr[3 * k] = gx[k]; gr[3 * k + 1] = gy[k]; gr[3 * k + 2] = gz[k]; }
    gr[15] = T(0);
    T *go = w.grec + (size_t)cell * kG;
    st8(go, gr);
    st8(go + 8, gr + 8);
    if (kTemp) {
        gr[16] = gx[NV - 1]; gr[17] = gy[NV - 1]; gr[18] = gz[NV - 1]; gr[19] = T(0);
        st4(go + 16, gr + 16);
        // laminar viscosity of this NS step, read by the SA step after the update
        if (w.trec) w.trec[(size_t)cell * kTr + 2] = sutherland(vc[NV - 1], (T)c.tsuth);
    }
    T lim = T(1);
    if (c.limiter != PHX_LIMITER_NOLIM && c.firstOrder) {
        lim = T(0);
    } else if (c.limiter == PHX_LIMITER_BARTH) {
        // Limiter::BarthLimiter (Limiter.cpp:157-262) from rho and p: the face
        // extrapolation clipped to the neighbour min/max difference; a face whose
        // centre lies behind the cell's outward normal zeroes the limiter.  Each
        // candidate is >= 0, so visiting rho and p per face gives the reference's
        // two passes' minimum.
        const T dminr = rmin - qc[0], dmaxr = rmax - qc[0];
        const T dminp = pmin - qc[4], dmaxp = pmax - qc[4];
        const T small = (T)kSmall;
        for (int j = j0; j < j1; ++j) {
            const int e = ld(&g.c2x[j].x);
            const bool isLeft = e >= 0;
            const int f = isLeft ? e : ~e;
            T fn[4], dc[4];
            if (kCompact) {
                form_side<T>(g, f, cell, fn, dc);
            } else {
                const T *geo = w.fgeo + (size_t)f * kGeo<kTemp>;
                ld4(geo, fn);
                ld4(geo + (isLeft ? 4 : 8), dc);
            }
            const T dx = dc[0], dy = dc[1], dz = dc[2];
            const T ds = sqrt(dx * dx + dy * dy + dz * dz);
            const T nd = fn[0] * dx + fn[1] * dy + fn[2] * dz;
            const T dot = (isLeft ? nd : -nd) / (ds + small);
            if (dot < T(0)) { lim = T(0); continue; }
            T d = gx[0] * dx + gy[0] * dy + gz[0] * dz;
            if (d > dmaxr) lim = tmin(lim, dmaxr / (d + small));
            else if (d < dminr) lim = tmin(lim, dminr / (d + small));
            d = gx[4] * dx + gy[4] * dy + gz[4] * dz;
            if (d > dmaxp) lim = tmin(lim, dmaxp / (d + small));
            else if (d < dminp) lim = tmin(lim, dminp / (d + small));
        }
        if (g.farfield_adj[cell]) lim = T(0);
    } else if (c.limiter == PHX_LIMITER_VENCAT) {
        const T vp = (T)ld(g.volpow + cell);
        T er = (T)c.venkatK3 * qc[0]; er = er * qc[0]; er = er * vp;
        T ep = (T)c.venkatK3 * qc[4]; ep = ep * qc[4]; ep = ep * vp;
        const T dminr = rmin - qc[0], dmaxr = rmax - qc[0];
        const T dminp = pmin - qc[4], dmaxp = pmax - qc[4];
        const T small = (T)kSmall;
        for (int j = j0; j < j1; ++j) {
            const int e = ld(&g.c2x[j].x);
            T dc[4];
            if (kCompact) {
                T fn[4];
                form_side<T>(g, e >= 0 ? e : ~e, cell, fn, dc);
            } else ld4(w.fgeo + (size_t)(e >= 0 ? e : ~e) * kGeo<kTemp> + (e >= 0 ? 4 : 8), dc);
            const T dx = dc[0], dy = dc[1], dz = dc[2];
            T d = gx[0] * dx + gy[0] * dy + gz[0] * dz;
            if (d > small) lim = tmin(lim, venfun(dmaxr, d, er));
            else if (d < -small) lim = tmin(lim, venfun(dminr, d, er));
            d = gx[4] * dx + gy[4] * dy + gz[4] * dz;
            if (d > small) lim = tmin(lim, venfun(dmaxp, d, ep));
            else if (d < -small) lim = tmin(lim, venfun(dminp, d, ep));
        }
        if (g.farfield_adj[cell]) lim = T(0);
    }
    w.qrec[(size_t)cell * kQ + 7] = lim;
}

template <class T, bool kCompact>
static void launch_gradient(const DevGrid &g, const NsConst &c, const Work<T> &w, cudaStream_t s)
{
    constexpr int pt = kPassThreads<T>;
    const int blocks = (g.nCell + pt - 1) / pt;
    if (c.viscous) {
        if (c.gradient == 1) gradient_limiter_kernel<T, true, 1, kCompact><<<blocks, pt, 0, s>>>(g, c, w);
        else if (c.gradient == 2) gradient_limiter_kernel<T, true, 2, kCompact><<<blocks, pt, 0, s>>>(g, c, w);
        else gradient_limiter_kernel<T, true, 0, kCompact><<<blocks, pt, 0, s>>>(g, c, w);
    } else {
        if (c.gradient == 1) gradient_limiter_kernel<T, false, 1, kCompact><<<blocks, pt, 0, s>>>(g, c, w);
        else if (c.gradient == 2) gradient_limiter_kernel<T, false, 2, kCompact><<<blocks, pt, 0, s>>>(g, c, w);
        else gradient_limiter_kernel<T, false, 0, kCompact><<<blocks, pt, 0, s>>>(g, c, w);
    }
}

template <class T>
void launch_gradient_limiter(const DevGrid &g, const NsConst &c, const Work<T> &w, int nodePrev, cudaStream_t s)
{
    if (c.gradient == 2)
        node_value_kernel<T><<<(g.nNode + kThreads - 1) / kThreads, kThreads, 0, s>>>(g, c, w, nodePrev);
    if (g.compact) launch_gradient<T, true>(g, c, w, s);
    else launch_gradient<T, false>(g, c, w, s);
}

// ---------------------------------------------------------------------------
// Residual, pass 1 (one thread per face): MUSCL face states (GetQlQr /
// ReConstructFaceValue, NSSolverUnstruct.cpp:5507, :13991-14193), the wall /
// symmetry face fix (BoundaryQlQrFix, :13725-13951), the inviscid flux (Roe,
// with kScheme = 1 the other scheme uns_scheme_name selects, with kScheme = 2
// the rotated Van Leer scheme in an instantiation of its own) times the face area
// (InviscidFluxWrap, :14466-14488), the face term of the inviscid
// spectral radius (SpectrumRadiusInviscid, :5749-5850), and the dq-independent
// LU-SGS factors of both face uses (RoeAveragedVariables + GetRad +
// MXDQ_STD, :15097-15116, Jacobian.cpp:27-47).
// ---------------------------------------------------------------------------

// Roe-averaged spectral radius |vn| + c of a face (RoeAveragedVariables,
// Flux_Inviscid.cpp:15440-15465, and GetRad) from the cell records, whose slot 6
// is the total enthalpy: the same for both uses of the face.
template <class T>
__device__ __forceinline__ T roe_radius(const T *qL, const T *qR, T nx, T ny, T nz, T gm)
{
    const T t0 = sqrt(qR[0] / qL[0]), t1 = T(1) / (T(1) + t0);
    const T u = (qL[1] + qR[1] * t0) * t1, v = (qL[2] + qR[2] * t0) * t1, w = (qL[3] + qR[3] * t0) * t1;
    const T hm = (qL[6] + qR[6] * t0) * t1;
    return fabs(nx * u + ny * v + nz * w) + sqrt((gm - T(1)) * (hm - T(0.5) * (u * u + v * v + w * w)));
}

// The factors of a face use (kUse) for the sweeps: MXDQ_STD with ipn = -1
// (Jacobian.cpp:13-86).  Its eigenvalues l1 = (vn - rad) / 2, l2 = l1 + c / 2 and
// l3 = l1 - c / 2 make its coefficients (2 l1 - l2 - l3) / (2 c^2) and (l2 - l3) /
// (2 c) zero and one half, so the neighbour's term is
//   area (l1 dq - dc / 2 (1, u, h) + dh / 2 (0, n, vn)) - vspec dq
// with dc = vn dq0 - n . dq123 and dh of the neighbour's state (delta_flux).
template <class T>
__device__ __forceinline__ void sweep_use(const T *qn, T nx, T ny, T nz, T area, T rad, T vspec, T *v)
{
    const T vn = nx * qn[1] + ny * qn[2] + nz * qn[3], ha = T(0.5) * area;
    v[0] = ha * nx; v[1] = ha * ny; v[2] = ha * nz;
    v[3] = ha * (vn - rad) - vspec;
    v[4] = qn[1]; v[5] = qn[2]; v[6] = qn[3]; v[7] = qn[6];
}

// Where the sweeps' rows hold the factors of a face use (DevGrid::use), and a
// cell's right-hand side (slot = row * kSweepSlots + slot).
template <class T>
__device__ __forceinline__ T *use_at(const Work<T> &w, int at)
{
    const int i = at < 0 ? ~at : at;
    unsigned char *row = at < 0 ? w.rowb + (size_t)(i >> 5) * kRowNs<T, false> : w.rowf + (size_t)(i >> 5) * kRowNs<T, true>;
    return reinterpret_cast<T *>(row) + (i & 31) * kUse;
}
template <class T, bool kForward>
__device__ __forceinline__ T *lead_at(const Work<T> &w, int slot)
{
    unsigned char *row = (kForward ? w.rowf : w.rowb) + (size_t)(slot / kSweepSlots) * kRowNs<T, kForward>;
    return reinterpret_cast<T *>(row) + 32 * kUse + (slot % kSweepSlots) * (kForward ? kLeadF : kLeadB);
}

// One side of a face: the MUSCL state qo from the cell state qs and the cell's
// gradient (kept where its density or pressure is not positive), and for viscous
// runs, added to what the other side gave, the face gradient of u, v, w (weight
// wt) and the side's velocity and temperature at the foot of the normal line
// (offset x).  gp: the gradient record to use, null for none; recon: whether this
// side is reconstructed (boundary ghosts are used as they are; an interface ghost
// has the neighbouring zone's gradient, limiter and centre).
template <class T, bool kVisc>
__device__ __forceinline__ void face_side(const T *gp, bool recon, T lim, const T *d, const T *qs, T *qo, T wt, const T *x,
                                          T *F, T *foot, T &tfoot)
{
#pragma unroll
    for (int k = 0; k < 5; ++k) qo[k] = qs[k];
    if (kVisc) {
#pragma unroll
        for (int k = 0; k < 3; ++k) foot[k] = qs[k + 1];
    }
    if (!gp) return;
    T a[16];
    ld8(gp, a);
    ld8(gp + 8, a + 8);
    if (recon) {
        T tr[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) tr[k] = qs[k] + lim * (a[3 * k] * d[0] + a[3 * k + 1] * d[1] + a[3 * k + 2] * d[2]);
        if (tr[0] > T(0) && tr[4] > T(0)) {
#pragma unroll
            for (int k = 0; k < 5; ++k) qo[k] = tr[k];
        }
    }
    if (kVisc) {
        T b[4];
        ld4(gp + 16, b);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const T *gk = a + 3 * (k + 1);
            foot[k] += gk[0] * x[0] + gk[1] * x[1] + gk[2] * x[2];
#pragma unroll
            for (int m = 0; m < 3; ++m) F[3 * k + m] += wt * gk[m];
        }
        const T t0 = tfoot;
        tfoot += b[0] * x[0] + b[1] * x[1] + b[2] * x[2];
        if (tfoot < (T)kSmall) tfoot = t0;
    }
}

__device__ __forceinline__ void reset_reduce(Reduce *r)
{
    r->mindt_bits = 0x7FEFFFFFFFFFFFFFULL;  // largest finite double
    for (int k = 0; k < 5; ++k) r->resnorm[k] = 0.0;
    r->negcount = 0;
}

// Viscous flux times the area, F1..F4 (F0 is zero), and the face's viscous
// spectral-radius term, which is also the LU-SGS viscous factor of both face uses
// (SpectrumRadiusViscous method 2, NSSolverUnstruct.cpp:5930-5960;
// SolveLUSGSForward :15339-15357): GetVisFaceValue (:7126-7375, static adiabatic
// walls) and ComputeVisflux (:12977-13378, perfect gas).  The face gradient F of u,
// v, w has its normal part replaced by the normal derivative; what ComputeVisflux
// takes along two tangents is F less its normal part.
//
// The pass is bound by memory latency: three blocks per SM, of 256 threads on the
// mixed path and of 128 in double precision (at most 168 registers), and one side
// after the other, so that little is held at a time.  With the cell pass, on the
// 1M-cell bump: mixed 335 -> 255 us, FP64 918 -> 607 us against geometry formed
// in the pass, gradients read twice and 256 threads at 166 registers.
template <class T, bool kVisc, int kScheme, bool kCompact>
__global__ void __launch_bounds__(kPassThreads<T>, 3) face_flux_kernel(DevGrid g, NsConst c, Work<T> w, Reduce *red)
{
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f == 0) reset_reduce(red);   // for the cell pass and the update
    if (f >= g.nFace) return;
    const int2 lr = ld(g.lr + f);
    const int le = lr.x, re = lr.y;
    T gn[4], gl[4], gr[4], xl[4], xr[4];
    if (kCompact) {
        form_face<T, kVisc>(g, f, le, re, gn, gl, gr, xl, xr);
    } else {
        const T *geo = w.fgeo + (size_t)f * kGeo<kVisc>;
        ld4(geo, gn);
        ld4(geo + 4, gl);
        ld4(geo + 8, gr);
        if (kVisc) { ld4(geo + 12, xl); ld4(geo + 16, xr); }
    }
    T qL[8], qR[8];
    ld8(w.qrec + (size_t)le * kQ, qL);
    ld8(w.qrec + (size_t)re * kQ, qR);
    const T xn = gn[0], yn = gn[1], zn = gn[2], area = gn[3];
    const bool cellR = re < g.nCell || g.bkind[f] == BK_INTERFACE;
    T limL = qL[7], limR = qR[7];
    if (c.reconMethod == 1) { const T m = tmin(limL, limR); limL = limR = m; }
    const bool recon = !(kScheme != 0 && c.firstOrder);
    const T gm = (T)c.gama;
    T ql[5], qr[5], fl[8], fv[4], vspec = T(0);
    {
        T F[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, f1[3], f2[3];
        const T coef = (T)c.coefState;
        const T tl0 = kVisc ? temperature(qL, coef) : T(0), tr0 = kVisc ? temperature(qR, coef) : T(0);
        T tL = tl0, tR = tr0;
        face_side<T, kVisc>(w.grec + (size_t)le * kG, recon, limL, gl, qL, ql, gl[3], xl, F, f1, tL);
        // a boundary ghost has the owner's gradient (least squares, GG-node) or
        // none (GG-cell), as the reference's gradient routines leave them
        const T *gp = cellR ? w.grec + (size_t)re * kG : (kVisc && c.gradient != 0 ? w.grec + (size_t)le * kG : nullptr);
        face_side<T, kVisc>(gp, recon && cellR, limR, gr, qR, qr, cellR ? T(1) - gl[3] : T(0), xr, F, f2, tR);
        if (kVisc) {
            const T S = (T)c.tsuth, A = gr[3], B = xl[3], ds = xr[3];
            const T mul = T(0.5) * (sutherland(tl0, S) + sutherland(tr0, S));
            const T mut = w.trec ? T(0.5) * (w.trec[(size_t)le * kTr + 1] + w.trec[(size_t)re * kTr + 1]) : T(0);
            const T vis = mul + mut;
            vspec = T(2) * vis / (T(0.5) * (qL[0] + qR[0]) * ds * (T)c.reynolds + (T)kSmall) * (T(0.5) * area);
            // a wall's face velocity is zero whatever its ghost holds (GetVisFaceValue), where both
            // centres are projected; elsewhere ComputeVisflux takes the mean
            const bool rest = f < g.nBFace && g.bkind[f] == BK_WALL && (g.vflag[f] & 1);
            T fm[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                fm[k] = rest ? T(0) : T(0.5) * (qL[k + 1] + qR[k + 1]);
                const T dn = A * (f1[k] - fm[k]) + B * (f2[k] - fm[k]);
                const T dt = dn - (F[3 * k] * xn + F[3 * k + 1] * yn + F[3 * k + 2] * zn);
                F[3 * k] += xn * dt; F[3 * k + 1] += yn * dt; F[3 * k + 2] += zn * dt;
            }
            const T tM = T(0.5) * (tl0 + tr0);
            const T qn = (mul * (T)c.oPrl + mut * (T)c.oPrt) * (T)c.cp * (A * (tL - tM) + B * (tR - tM));
            const T div = T(2.0 / 3.0) * (F[0] + F[4] + F[8]);
            const T txx = vis * (T(2) * F[0] - div), tyy = vis * (T(2) * F[4] - div), tzz = vis * (T(2) * F[8] - div);
            const T txy = vis * (F[1] + F[3]), txz = vis * (F[2] + F[6]), tyz = vis * (F[5] + F[7]);
            const T v1 = xn * txx + yn * txy + zn * txz;
            const T v2 = xn * txy + yn * tyy + zn * tyz;
            const T v3 = xn * txz + yn * tyz + zn * tzz;
            const T v4 = fm[0] * v1 + fm[1] * v2 + fm[2] * v3 + qn;
            const T sc = -(T)c.oRe * area;
            fv[0] = sc * v1; fv[1] = sc * v2; fv[2] = sc * v3; fv[3] = sc * v4;
        }
    }
    if (f < g.nBFace) {
        const int bt = g.btype[f];
        if (bt == PHX_BC_SOLID_SURFACE || bt == PHX_BC_SYMMETRY) {
#pragma unroll
            for (int k = 0; k < 5; ++k) { const T a = T(0.5) * (qL[k] + qR[k]); ql[k] = a; qr[k] = a; }
            if (bt == PHX_BC_SYMMETRY) {
                const T vn = T(2) * (xn * ql[1] + yn * ql[2] + zn * ql[3]);
                qr[1] = ql[1] - vn * xn; qr[2] = ql[2] - vn * yn; qr[3] = ql[3] - vn * zn;
            } else if (g.bkind[f] == BK_WALL) {
                ql[1] = ql[2] = ql[3] = T(0);
                qr[1] = qr[2] = qr[3] = T(0);
            }
        }
    }
    if (kScheme == 0) roe_flux<T>(ql, qr, gm, gm, xn, yn, zn, (T)c.acoustic, (T)c.convective, fl);
    else if (kScheme == 2) vanleer_rotate_flux_fp64<T>(ql, qr, gm, gm, xn, yn, zn, fl);
    else other_flux<T>(c.scheme, ql, qr, gm, gm, xn, yn, zn, (T)c.ausmpwLim, fl);
#pragma unroll
    for (int k = 0; k < 5; ++k) fl[k] *= area;
    // inviscid spectral radius term from the face-mean state
    {
        const T vnl = xn * qL[1] + yn * qL[2] + zn * qL[3];
        const T vnr = xn * qR[1] + yn * qR[2] + zn * qR[3];
        const T gmm = T(0.5) * (gm + gm);
        const T pm = T(0.5) * (qL[4] + qR[4]);
        const T rm = T(0.5) * (qL[0] + qR[0]);
        const T vn = T(0.5) * (vnl + vnr);
        const T cm = sqrt(gmm * pm / rm);
        fl[5] = T(0.5) * area * (fabs(vn) + cm);
    }
    fl[6] = vspec;
    fl[7] = kVisc ? fv[0] : T(0);
    st8(w.flux + (size_t)f * kFlux, fl);
    if (kVisc) {
        const T r[4] = {fv[1], fv[2], fv[3], T(0)};
        st4(w.flux + (size_t)f * kFlux + 8, r);
    }
    // LU-SGS factors of the left cell's and the right cell's use
    const T rad = roe_radius<T>(qL, qR, xn, yn, zn, gm);
    T v[kUse];
    sweep_use<T>(qR, xn, yn, zn, area, rad, vspec, v);
    if (f < g.nBFace) {
        put_use(w.coef + (size_t)f * kUse, 0, v);
    } else if (!kCompact) {
        const int2 at = ld(g.use + f);
        put_use(use_at<T>(w, at.x), (at.x < 0 ? ~at.x : at.x) & 31, v);
        sweep_use<T>(qL, -xn, -yn, -zn, area, rad, vspec, v);
        put_use(use_at<T>(w, at.y), (at.y < 0 ? ~at.y : at.y) & 31, v);
    }
    if (kCompact) {
        w.frad[2 * (size_t)f] = rad;
        w.frad[2 * (size_t)f + 1] = vspec;
    }
}

// Residual, pass 2 (one thread per cell): res gathered from the face fluxes
// in the reference's face order with the sign LoadFlux applies
// (NSSolverUnstruct.cpp:6435-6495), the inviscid spectral radius, and the
// local time step (LocalTimeStep / LimitCFL, :5999-6118) with its device-wide
// minimum (Controller::ComputeMinTimeStep, Controller.cpp:706-752).
__device__ __forceinline__ void atomic_min_pos_double(unsigned long long *addr, double v)
{
    atomicMin(addr, (unsigned long long)__double_as_longlong(v));
}

template <class T, bool kVisc>
__global__ void __launch_bounds__(kThreads) cell_residual_kernel(DevGrid g, NsConst c, Work<T> w, Reduce *red, double cfl)
{
    const int cell = blockIdx.x * blockDim.x + threadIdx.x;
    double mydt = kLarge;
    if (cell < g.nCell) {
        // ViscousFlux is loaded after InviscidFlux (NSSolver::UpdateResiduals,
        // NSSolver.cpp:71-80): its sum, in the same face order, is added at the end
        T res[5] = {0, 0, 0, 0, 0}, rv[4] = {0, 0, 0, 0};
        T spec = T(0), vis = T(0);
        const int j1 = g.c2f_off[cell + 1];
        for (int j = g.c2f_off[cell]; j < j1; ++j) {
            const int e = ld(&g.c2x[j].x);
            const T *rec = w.flux + (size_t)(e >= 0 ? e : ~e) * kFlux, sg = e >= 0 ? T(-1) : T(1);
            T fl[8];
            ld8(rec, fl);
#pragma unroll
            for (int k = 0; k < 5; ++k) res[k] += sg * fl[k];
            spec += fl[5];
            if (kVisc) {
                T fv[4];
                ld4(rec + 8, fv);
                vis += fl[6];
                rv[0] += sg * fl[7];
#pragma unroll
                for (int k = 0; k < 3; ++k) rv[k + 1] += sg * fv[k];
            }
        }
        if (kVisc) {
#pragma unroll
            for (int k = 0; k < 4; ++k) res[k + 1] += rv[k];
        }
        T tot = spec;
        if (c.viscous) tot += vis;
        double cc = cfl;
        const double pc = (double)w.qrec[(size_t)cell * kQ + 4];
        const double plo = 0.001 * c.pTotal, phi = 0.02 * c.pTotal;
        if (pc < plo) cc = c.cflStart;
        else if (pc < phi) cc = (pc - phi) * (cfl - c.cflStart) / (phi - plo) + cfl;
        const double sk = ld(g.skew + cell);
        if (sk < 0.1) cc *= 0.1;
        else if (sk < 10.0) cc *= (1.0 - exp(0.0 - sk));
        const T vol = (T)ld(&g.xrec[(size_t)cell * kX + 3]);
        const T dt = (T)cc * vol / tot;
        w.dtraw[cell] = dt;
        mydt = (double)dt;
        // reciprocal of the LU-SGS diagonal for the unclamped time step, formed
        // as the sweep forms it (the sweep recomputes it where ktmax clamps dt)
        T dd = idiv(T(1), idiv(dt, vol));
        dd += spec;
        if (c.viscous) dd += vis;
        T out[8] = {res[0], res[1], res[2], res[3], res[4], idiv(T(1), dd), spec, vis};
        st8(w.crec + (size_t)cell * kC, out);
        out[6] = dt;
        out[7] = T(0);
        if (!g.compact) st8(lead_at<T, true>(w, ld(g.lead + cell)), out);
    }
    // block minimum, then one atomic per block, skipped when it cannot lower
    // the running minimum (positive doubles order like their bit patterns)
    for (int o = 16; o > 0; o >>= 1) mydt = fmin(mydt, __shfl_xor_sync(0xffffffffu, mydt, o));
    __shared__ double wmin[kThreads / 32];
    if ((threadIdx.x & 31) == 0) wmin[threadIdx.x >> 5] = mydt;
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = wmin[0];
        for (int i = 1; i < kThreads / 32; ++i) m = fmin(m, wmin[i]);
        const unsigned long long cur = *(volatile unsigned long long *)&red->mindt_bits;
        if (m < kLarge && (unsigned long long)__double_as_longlong(m) < cur) atomic_min_pos_double(&red->mindt_bits, m);
    }
}

template <class T, bool kCompact>
static void launch_face_flux(const DevGrid &g, const NsConst &c, const Work<T> &w, Reduce *red, cudaStream_t s)
{
    constexpr int ft = kPassThreads<T>;
    const int fb = (g.nFace + ft - 1) / ft;
    const int kind = c.scheme == PHX_SCHEME_ROE ? 0 : c.scheme == PHX_SCHEME_VANLEER_ROTATE ? 2 : 1;
    if (c.viscous) {
        if (kind == 0) face_flux_kernel<T, true, 0, kCompact><<<fb, ft, 0, s>>>(g, c, w, red);
        else if (kind == 2) face_flux_kernel<T, true, 2, kCompact><<<fb, ft, 0, s>>>(g, c, w, red);
        else face_flux_kernel<T, true, 1, kCompact><<<fb, ft, 0, s>>>(g, c, w, red);
    } else {
        if (kind == 0) face_flux_kernel<T, false, 0, kCompact><<<fb, ft, 0, s>>>(g, c, w, red);
        else if (kind == 2) face_flux_kernel<T, false, 2, kCompact><<<fb, ft, 0, s>>>(g, c, w, red);
        else face_flux_kernel<T, false, 1, kCompact><<<fb, ft, 0, s>>>(g, c, w, red);
    }
}

template <class T>
void launch_residual(const DevGrid &g, const NsConst &c, const Work<T> &w, Reduce *red, double cfl, cudaStream_t s)
{
    if (g.compact) launch_face_flux<T, true>(g, c, w, red, s);
    else launch_face_flux<T, false>(g, c, w, red, s);
    const int cb = (g.nCell + kThreads - 1) / kThreads;
    if (c.viscous) cell_residual_kernel<T, true><<<cb, kThreads, 0, s>>>(g, c, w, red, cfl);
    else cell_residual_kernel<T, false><<<cb, kThreads, 0, s>>>(g, c, w, red, cfl);
}

// ---------------------------------------------------------------------------
// LU-SGS (Controller::LUSGS, Controller.cpp:1878-1955) as a dataflow
// computation.  The forward sweep of the reference visits cells in
// increasing number and uses the just-updated dq of lower-numbered face
// neighbours; the backward sweep the reverse.  Here each sweep is one launch of
// one-warp blocks, each running its rows of the schedule (phx_schedule.cpp):
// eight cells a row, four lanes a cell, a lane per neighbour.  A neighbour's
// result is taken from the warp's shared memory where the schedule says that
// this warp computed it and still holds it, and otherwise polled in its
// write-once record (dqfwd, dqrec), filled with the sentinel before the sweep
// (sweep_reset_kernel): the data is its own completion flag, and a cell sees
// exactly the values the sequential sweep of the reference sees.  The records
// of the row after next are polled while this row's sum is formed, so a warp that
// runs behind the ones it reads from does not wait for L2 at all.  All warps
// are co-resident (cooperative launch) and their rows ascend in level, so the
// wait graph cannot cycle.  Every wait is bounded: a timeout sets
// Reduce::error and the kernel gives up.  The dq-independent MXDQ_STD factors
// were computed by the residual pass.
// ---------------------------------------------------------------------------

// Ghost-cell dq of a boundary face from the owner's forward dq dl
// (SetGhostDQLUSGS, NSSolverUnstruct.cpp:14767-14810; SetSymmBCGhostDQLUSGS
// :14812-14915 with the owner's state ql and the ghost's qg;
// SetWallBCGhostDQLUSGS :14917-15006; far field 0).
template <class T>
__device__ __forceinline__ void ghost_dq(int kind, T xn, T yn, T zn, const T *ql, const T *qg, T gm, const T *dl, T *o)
{
#pragma unroll
    for (int k = 0; k < 5; ++k) o[k] = T(0);
    if (kind == BK_SYMMETRY) {
        const T r = ql[0], u = ql[1], v = ql[2], ww = ql[3], pp = ql[4];
        const T em = idiv(idiv(pp, r), gm - T(1)) + T(0.5) * (u * u + v * v + ww * ww);
        T Q[5] = {r, r * u, r * v, r * ww, r * em};
        const T rm = qg[0], um = qg[1], vm = qg[2], wm = qg[3], pm = qg[4];
        const T pmg = idiv(pm, gm - T(1));
        const T rmu2 = rm * (um * um + vm * vm + wm * wm);
#pragma unroll
        for (int k = 0; k < 5; ++k) Q[k] += dl[k];
        o[0] = dl[0];
        T rvn = T(2) * (xn * dl[1] + yn * dl[2] + zn * dl[3]);
        o[1] = dl[1] - xn * rvn;
        o[2] = dl[2] - yn * rvn;
        o[3] = dl[3] - zn * rvn;
        rvn = T(2) * (xn * Q[1] + yn * Q[2] + zn * Q[3]);
        const T ru = Q[1] - xn * rvn, rv = Q[2] - yn * rvn, rw = Q[3] - zn * rvn;
        const T rq0 = idiv(T(1), Q[0]);
        const T pnew = Q[4] - T(0.5) * (Q[1] * Q[1] + Q[2] * Q[2] + Q[3] * Q[3]) * rq0;
        o[4] = pnew - pmg + T(0.5) * ((ru * ru + rv * rv + rw * rw) * rq0 - rmu2);
    } else if (kind == BK_WALL) {
        o[0] = dl[0]; o[1] = -dl[1]; o[2] = -dl[2]; o[3] = -dl[3]; o[4] = dl[4];
    }
}

// Delta flux of one neighbour (SolveLUSGSForward, NSSolverUnstruct.cpp:15118-15357)
// from the use's factors u (sweep_use) and the neighbour's dq; g1 = gamma - 1.
template <class T>
__device__ __forceinline__ void delta_flux(const T *u, T g1, const T *dq, T *df)
{
    const T vn = u[0] * u[4] + u[1] * u[5] + u[2] * u[6];
    const T ek = T(0.5) * g1 * (u[4] * u[4] + u[5] * u[5] + u[6] * u[6]);
    const T dc = vn * dq[0] - u[0] * dq[1] - u[1] * dq[2] - u[2] * dq[3];
    const T dh = ek * dq[0] - g1 * (u[4] * dq[1] + u[5] * dq[2] + u[6] * dq[3] - dq[4]);
    df[0] = u[3] * dq[0] - dc;
    df[1] = u[3] * dq[1] - u[4] * dc + u[0] * dh;
    df[2] = u[3] * dq[2] - u[5] * dc + u[1] * dh;
    df[3] = u[3] * dq[3] - u[6] * dc + u[2] * dh;
    df[4] = u[3] * dq[4] - u[7] * dc + vn * dh;
}

// Boundary part of the backward sweep: per cell with boundary faces the sum of
// their ghosts' delta fluxes, in the cell's face order (the reference numbers
// boundary faces first, so the backward sum starts with them).  An interface
// ghost holds the neighbouring zone's forward dq, set by the halo exchange
// between the sweeps (SetGhostDQLUSGS leaves it to CommunicationDQ,
// Controller.cpp:1917-1924).  Everything here is known once the forward sweep
// has ended; inside the sweep it sat on the critical path of the wall and
// symmetry cells.
template <class T>
__global__ void __launch_bounds__(kThreads) sweep_ghost_kernel(DevGrid g, NsConst c, Work<T> w)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.nGhostCell) return;
    const int2 gc = ld(g.ghost_cell + i);
    const int cell = gc.x;
    const T gm = (T)c.gama;
    T ql[8], dl[8], sum[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    ld8(w.qrec + (size_t)cell * kQ, ql);
    ld8(w.dqfwd + (size_t)ld(g.lead + cell) * kD, dl);
    const int j1 = ld(g.c2f_off + cell + 1);
    for (int j = ld(g.c2f_off + cell); j < j1; ++j) {
        const int f = ld(&g.c2x[j].x);   // a boundary face's only cell is its left cell
        if (f < 0 || f >= g.nBFace) break;
        const int kind = ld(g.bkind + f), ghost = g.nCell + f;
        double fr[4];
        ld4(g.frec + (size_t)f * kF, fr);
        T qg[8], u[kUse], dq[8], df[5];
        ld8(w.qrec + (size_t)ghost * kQ, qg);
        get_use(w.coef + (size_t)f * kUse, 0, u);
        if (kind == BK_INTERFACE) ld8(w.dqghost + (size_t)f * kD, dq);
        else ghost_dq<T>(kind, (T)fr[0], (T)fr[1], (T)fr[2], ql, qg, gm, dl, dq);
        delta_flux<T>(u, gm - T(1), dq, df);
#pragma unroll
        for (int m = 0; m < 5; ++m) sum[m] += df[m];
    }
    st8(g.compact ? w.gsum + (size_t)i * kLeadF : lead_at<T, false>(w, gc.y) + 8, sum);
}

// One sweep: a warp per block, so that the few warps of a small mesh spread over
// the SMs.  What bounds it is the chain of dependent rows, about the sum of the
// mesh's extents, times the time from a result to the next row's, and that is
// the warp's instructions for a row one after the other (0.36 us forward, 0.29
// us backward in single precision, 0.8 us where the records of a row are polled
// when the row begins): whatever does not depend on dq is formed by the face and
// cell passes or by the schedule, and a row arrives by one copy.
// Both sweeps, mixed, against levels dealt out over all SMs with every result
// through L2: 8k hexahedra 170 -> 106 us, the 200k plate 515 -> 256 us, 1M
// tetrahedra 960 -> 590 us, the 1M-cell bump with prisms 978 -> 537 us.
// Shared memory in front of the stages: the warp's results and a zero, barriers.
template <class T>
constexpr int kSweepHead = (kSweepZero + 1) * 8 * (int)sizeof(T) + (sizeof(T) == 4 ? 96 : 64);
static_assert(kSweepHead<float> % 128 == 0 && kSweepHead<double> % 128 == 0, "aligned stages");

// Compact layout: the rows hold the schedule alone.  A lane forms its factors from
// the neighbour's state, the metrics and the face's two spectral terms, as the face
// pass does for full rows; right-hand sides lie by cell.  A row
// names the uses and cells of the warp's row after next, so that these loads are on
// their way for two rows (16M-cell bump, mixed, both NS sweeps: 5.6 ms, 7.8 when they
// begin with their row, 3.1 with full rows).
template <class T>
struct UseIn {
    int2 e;          // face (sign bit: the normal points into the cell), neighbour (-1: none)
    double n[4];
    T q[4], hm, rad, vspec;
};
template <class T>
__device__ __forceinline__ void fetch_use(const DevGrid &g, const Work<T> &w, int2 e, UseIn<T> &s)
{
    s.e = e;
    if (e.y < 0) return;
    const int f = e.x & 0x7fffffff;
    const T *q = w.qrec + (size_t)e.y * kQ;
    ld4(g.frec + (size_t)f * kF, s.n);
    ld4(q, s.q);
    s.hm = ld(q + 6);
    s.rad = ld(w.frad + 2 * (size_t)f);
    s.vspec = ld(w.frad + 2 * (size_t)f + 1);
}
template <class T>
__device__ __forceinline__ void form_use(const UseIn<T> &s, T *u)
{
    if (s.e.y < 0) {
#pragma unroll
        for (int k = 0; k < kUse; ++k) u[k] = T(0);
        return;
    }
    const T sg = s.e.x < 0 ? T(-1) : T(1);
    const T qn[8] = {s.q[0], s.q[1], s.q[2], s.q[3], T(0), T(0), s.hm, T(0)};
    sweep_use<T>(qn, sg * (T)s.n[0], sg * (T)s.n[1], sg * (T)s.n[2], (T)s.n[3], s.rad, s.vspec, u);
}
// Right-hand side of a cell (lane 0 of its slot; -1: none): residual (5), reciprocal diagonal, forward: time step.
template <class T, bool kForward>
__device__ __forceinline__ void fetch_lead(const Work<T> &w, int cell, T *q)
{
    if (cell < 0) return;
    ld8((kForward ? w.crec : w.lead) + (size_t)cell * kC, q);
    if (kForward) q[6] = ld(w.dtraw + cell);
}

// kCompact: registers for as many warps an SM as the schedule may be made for (sweep_max_warps)
template <class T, bool kForward, bool kCompact>
__global__ void __launch_bounds__(32, kCompact ? (sizeof(T) == 4 ? 16 : 12) : 0)
    lusgs_kernel(DevGrid g, NsConst c, Work<T> w, Reduce *red, int stages)
{
    constexpr int kLead = kForward ? kLeadF : kLeadB, kRow = kCompact ? kRowCompact : kRowNs<T, kForward>;
    using Pipe = RowPipe<kRow>;
    constexpr int kLeadOff = 32 * kUse * (int)sizeof(T), kRowOff = kRow - kSweepRow * 4;
    extern __shared__ __align__(128) unsigned char sm[];
    T *loc = reinterpret_cast<T *>(sm);
    const SweepDev &sw = kForward ? g.fwd : g.bwd;
    const int t = threadIdx.x, slot = t / kSweepLanes, lane = t % kSweepLanes;
    const int row0 = ld(sw.row_off + blockIdx.x), nrow = ld(sw.row_off + blockIdx.x + 1) - row0;
    if (nrow <= 0) return;
    if (t < 8) loc[kSweepZero * 8 + t] = T(0);
    const double mindt = __longlong_as_double((long long)red->mindt_bits);
    const T clamp = c.ktmax > 0 ? (T)(c.ktmax * mindt) : (T)kLarge;
    const T g1 = (T)c.gama - T(1);
    const int viscous = c.viscous, held = kForward && c.holdCell >= 0 ? c.holdCell : -2;
    T *out = kForward ? w.dqfwd : w.dqrec;
    T *mine = out + ((size_t)row0 * kSweepSlots + slot) * kD;   // record of this slot in the current row
    Pipe pipe;
    pipe.start(sm + kSweepHead<T>, reinterpret_cast<uint64_t *>(loc + (kSweepZero + 1) * 8), kForward ? w.rowf : w.rowb,
               row0, nrow, stages, t);
    // the entry of this lane in a row, and a first look at the record it polls
    auto entry = [&](const int *p, int &en, T *v) {
        en = p[t];
        if (en >= 0) poll5_load(out + (size_t)en * kD, v);
    };
    T va[5], vb[5], rhs[5];
    UseIn<T> ua, ub;
    T qa[8], qb[8];
    int ea, eb;
    if (kCompact) {
        const int2 *fu = sw.first_use + blockIdx.x * 64;
        const int *fc = sw.first_cell + blockIdx.x * 16;
        fetch_use<T>(g, w, fu[t], ua);
        fetch_use<T>(g, w, fu[32 + t], ub);
        fetch_lead<T, kForward>(w, lane == 0 ? fc[slot] : -1, qa);
        fetch_lead<T, kForward>(w, lane == 0 ? fc[8 + slot] : -1, qb);
    }
    entry(sw.first + blockIdx.x * 64, ea, va);
    entry(sw.first + blockIdx.x * 64 + 32, eb, vb);
    bool ok = true;
    auto step = [&](int i, int &en, T *v, UseIn<T> &in, T *qin) -> bool {
        const unsigned char *row = pipe.at(pipe.slot) + i * kRow;
        const int4 info = reinterpret_cast<const int4 *>(row + kRowOff + 128)[slot];
        const T *lead = reinterpret_cast<const T *>(row + kLeadOff) + slot * kLead;
        T u[kUse], q[8], b[5] = {0, 0, 0, 0, 0};
        if (kCompact) {
            form_use<T>(in, u);
            fetch_use<T>(g, w, reinterpret_cast<const int2 *>(row)[t], in);
#pragma unroll
            for (int m = 0; m < 8; ++m) q[m] = qin[m];
            fetch_lead<T, kForward>(w, lane == 0 ? reinterpret_cast<const int *>(row + 256)[slot] : -1, qin);
            if (!kForward && lane == 0 && info.w > 0) {
                const T *gs = w.gsum + (size_t)(info.w - 1) * kLeadF;
                ld4(gs, b);
                b[4] = ld(gs + 4);
            }
        } else {
            get_use(reinterpret_cast<const T *>(row) + t * kUse, t, u);
        }
        if (en < 0) {
            const T *a = loc + ~en * 8;
            T o[4];
            get4(a, o);
#pragma unroll
            for (int m = 0; m < 4; ++m) v[m] = o[m];
            v[4] = a[4];
        }
        // fault injection (phx_fault_hold_cell): the held cell waits on
        // nothing that is ever set, so its wait runs out
        const bool hold = kForward && lane == 0 && info.x == held;
        bool ready = (en < 0 || poll5_done(v)) && !hold;
        if (!__all_sync(0xffffffffu, ready)) {
            long long spins = 0;
            do {
                ++spins;
                if (spins > c.spinLimit) {
                    if (t == 0) atomicExch(&red->error, PHX_ERR_TIMEOUT);
                    return false;
                }
                if ((spins & 1023) == 0 && __any_sync(0xffffffffu, ((volatile int *)&red->error)[0] != 0)) return false;
                if (!ready && en >= 0) ready = poll5(out + (size_t)en * kD, v) && !hold;
            } while (!__all_sync(0xffffffffu, ready));
        }
        T df[5];
        delta_flux<T>(u, g1, v, df);
        // the row after next, while this row's sum is formed
        entry(reinterpret_cast<const int *>(row + kRowOff), en, v);
        // sum in the cell's face order, on the cell's first lane; the backward
        // sum starts with the boundary faces
        T sum[5];
        if (kForward) {
#pragma unroll
            for (int m = 0; m < 5; ++m) sum[m] = df[m];
        } else {
            if (!kCompact) {
                get4(lead + (kForward ? 0 : 8), b);
                b[4] = lead[kForward ? 0 : 12];
            }
#pragma unroll
            for (int m = 0; m < 5; ++m) sum[m] = b[m] + df[m];
        }
        if ((info.y & kSweepMulti) && (info.y & kSweepCarry)) {
#pragma unroll
            for (int m = 0; m < 5; ++m) sum[m] = rhs[m] + df[m];
        }
#pragma unroll
        for (int j = 1; j < kSweepLanes; ++j) {
#pragma unroll
            for (int m = 0; m < 5; ++m) sum[m] += __shfl_down_sync(0xffffffffu, df[m], j);
        }
        if (info.y & kSweepMulti) {
#pragma unroll
            for (int m = 0; m < 5; ++m) rhs[m] = sum[m];
        }
        __syncwarp();   // the row's reads of loc
        if (lane == 0 && info.x >= 0) {
            // reciprocal of the diagonal (NSSolverUnstruct.cpp:15867-15935),
            // 1 / (dt' / vol) + spectral radii, dt' = min(dt, ktmax min dt)
            // (ReduceMaxTimeStep, :5717-5745): formed by the residual pass for
            // the raw dt, by the forward sweep where the clamp applies
            T o[5];
            if (!kCompact) get8(lead, q);
            if (kForward && q[6] > clamp) {
                const T *cr = w.crec + (size_t)info.x * kC;
                T d = idiv(T(1), idiv(clamp, (T)ld(g.xrec + (size_t)info.x * kX + 3)));
                d += ld(cr + 6);
                if (viscous) d += ld(cr + 7);
                q[5] = idiv(T(1), d);
            }
            // dq = (res - Ux - L dq) / D, Ux = 0 for a single sweep
            // (LUSGSInitialization, Controller.cpp:1765-1777)
#pragma unroll
            for (int m = 0; m < 5; ++m) { q[m] -= sum[m]; o[m] = q[m] * q[5]; }
            T *own = loc + (info.y & 255) * 8;
            st4(own, o);
            own[4] = o[4];
            publish5(mine, o);
            if (kForward) st8(kCompact ? w.lead + (size_t)info.x * kLeadF : lead_at<T, false>(w, info.z), q);
        }
        mine += kSweepSlots * kD;
        __syncwarp();
        return true;
    };
    int k = 0;
    while (ok && k < pipe.nstage) {
        ok = pipe.wait() && step(0, ea, va, ua, qa) && (2 * k + 1 >= nrow || step(1, eb, vb, ub, qb));
        if (!ok) break;
        pipe.advance(t);
        ++k;
    }
    if (!ok) {
        if (t == 0 && ((volatile int *)&red->error)[0] == 0) atomicExch(&red->error, PHX_ERR_TIMEOUT);
        __syncwarp();
        pipe.drain(k);
    }
}

// Fills the sweeps' polled records (forward dq, final dq) with the sentinel.
template <class T>
__global__ void __launch_bounds__(kThreads) sweep_reset_kernel(int rowsF, int rowsB, T *f, T *b)
{
    constexpr int kQuads = kSweepSlots * kD / 4;
    const T s = sweep_sentinel<T>(), v[4] = {s, s, s, s};
    const long long nf = (long long)rowsF * kQuads, nb = (long long)rowsB * kQuads, n = max(nf, nb);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        if (i < nf) st4(f + i * 4, v);
        if (i < nb) st4(b + i * 4, v);
    }
}

// Shared memory of a sweep's warp with the given number of stages.
template <class T, bool kForward, bool kCompact>
static int sweep_smem(int stages)
{
    return kSweepHead<T> + stages * RowPipe<kCompact ? kRowCompact : kRowNs<T, kForward>>::kStage;
}

// Warps of the sweeps that are resident together with two stages each: the
// schedule is made for at most this many.  PHX_LUSGS_MAX_BLOCKS caps them
// (tuning; tests of many rows per warp).
template <class T>
int sweep_max_warps(int numSMs)
{
    int n = 16;
    auto resident = [&](auto kernel, int most, int two) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        int k = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, kernel, 32, two);
        n = std::min(n, k);
    };
    resident(lusgs_kernel<T, true, false>, sweep_smem<T, true, false>(4), sweep_smem<T, true, false>(2));
    resident(lusgs_kernel<T, false, false>, sweep_smem<T, false, false>(4), sweep_smem<T, false, false>(2));
    resident(lusgs_kernel<T, true, true>, sweep_smem<T, true, true>(4), sweep_smem<T, true, true>(2));
    resident(lusgs_kernel<T, false, true>, sweep_smem<T, false, true>(4), sweep_smem<T, false, true>(2));
    n = std::max(1, n) * numSMs;
    if (const char *cap = getenv("PHX_LUSGS_MAX_BLOCKS")) {
        const int v = atoi(cap);
        if (v > 0 && n > v) n = v;
    }
    return n;
}
template int sweep_max_warps<double>(int);
template int sweep_max_warps<float>(int);

template <class T, bool kForward, bool kCompact>
static cudaError_t launch_sweep(const DevGrid &g, const NsConst &c, const Work<T> &w, Reduce *red, int numSMs, cudaStream_t s)
{
    const int warps = (kForward ? g.fwd : g.bwd).nWarps;
    // more stages where the warps leave shared memory to spare (224 KB of an SM,
    // 1 KB of each block the system's)
    int stages = 2;
    const int perSM = (warps + numSMs - 1) / numSMs;
    while (stages < 4 && perSM * (sweep_smem<T, kForward, kCompact>(stages + 1) + 1024) <= 224 * 1024) ++stages;
    DevGrid gg = g;
    NsConst cc = c;
    Work<T> ww = w;
    Reduce *rr = red;
    void *args[] = {&gg, &cc, &ww, &rr, &stages};
    return cudaLaunchCooperativeKernel((void *)lusgs_kernel<T, kForward, kCompact>, dim3(warps), dim3(32), args,
                                       sweep_smem<T, kForward, kCompact>(stages), s);
}

template <class T>
int launch_lusgs(const DevGrid &g, const NsConst &c, const Work<T> &w, Reduce *red, int numSMs, cudaStream_t s,
                 int sweeps)
{
    cudaError_t e = cudaSuccess;
    if (sweeps & kSweepForward) {
        const long long n = (long long)std::max(g.fwd.nRows, g.bwd.nRows) * kSweepSlots * kD / 4;
        const int rb = (int)std::min<long long>((n + kThreads - 1) / kThreads, (long long)numSMs * 16);
        sweep_reset_kernel<T><<<rb, kThreads, 0, s>>>(g.fwd.nRows, g.bwd.nRows, w.dqfwd, w.dqrec);
        e = g.compact ? launch_sweep<T, true, true>(g, c, w, red, numSMs, s)
                      : launch_sweep<T, true, false>(g, c, w, red, numSMs, s);
    }
    if (e == cudaSuccess && (sweeps & kSweepBackward)) {
        if (g.nGhostCell > 0)
            sweep_ghost_kernel<T><<<(g.nGhostCell + kThreads - 1) / kThreads, kThreads, 0, s>>>(g, c, w);
        e = g.compact ? launch_sweep<T, false, true>(g, c, w, red, numSMs, s)
                      : launch_sweep<T, false, false>(g, c, w, red, numSMs, s);
    }
    return e == cudaSuccess ? 0 : (int)e;
}

// ---------------------------------------------------------------------------
// Update (NSSolverUnstruct::UpdateFlowField, NSSolverUnstruct.cpp:14587-14765):
// Q_cons (FP64, from the FP64 master primitive state) += dq, back to
// primitive.  Cells whose density or pressure drop below 1e-6 of the free
// stream are listed for the ordered SolutionFix pass.  Also reduces the
// residual monitor sum res_m^2 in FP64 (Residual.cpp:534-600).  q_old is read
// and q_new written (ghosts copied), so the repair pass can see the
// pre-update state of neighbours that come later in the reference's order,
// as the in-place sequential loop of the reference does.
// ---------------------------------------------------------------------------
// Cells the ordered repair pass takes per iteration; more than that means the
// run has diverged: the pass sets PHX_ERR_NUMERIC and leaves the state alone.
static constexpr int kMaxNeg = 4096;

template <class T>
__global__ void __launch_bounds__(kThreads) update_kernel(DevGrid g, NsConst c, Work<T> w, const double *qo,
                                                          double *qn, Reduce *red, int *neglist)
{
    const int nt = g.nTotal, nc = g.nCell;
    const int n = nc > g.nBFace ? nc : g.nBFace;
    const double gm = c.gama;
    double rs[5] = {0, 0, 0, 0, 0};
    for (int cell = blockIdx.x * blockDim.x + threadIdx.x; cell < n; cell += gridDim.x * blockDim.x) {
        if (cell < nc) {
            const double r = qo[cell], u = qo[nt + cell], v = qo[2 * nt + cell], ww = qo[3 * nt + cell],
                         p = qo[4 * nt + cell];
            const double em = (p / r) / (gm - 1.0) + 0.5 * (u * u + v * v + ww * ww);
            double Q[5] = {r, r * u, r * v, r * ww, r * em};
            T dq[8];
            ld8(w.dqrec + (size_t)ld(g.last + cell) * kD, dq);
#pragma unroll
            for (int k = 0; k < 5; ++k) Q[k] += (double)dq[k];
            double prim[5];
            if (Q[0] <= 0.0) {
                prim[0] = Q[0]; prim[1] = u; prim[2] = v; prim[3] = ww; prim[4] = p;
            } else {
                const double od = 1.0 / Q[0];
                const double um = Q[1] * od, vm = Q[2] * od, wm = Q[3] * od;
                const double ie = Q[4] - 0.5 * Q[0] * (um * um + vm * vm + wm * wm);
                prim[0] = Q[0]; prim[1] = um; prim[2] = vm; prim[3] = wm; prim[4] = (gm - 1.0) * ie;
            }
            if (prim[0] < 1.0e-6 * c.primInf[0] || prim[4] < 1.0e-6 * c.primInf[4]) {
                const int slot = atomicAdd(&red->negcount, 1);
                if (slot < kMaxNeg) neglist[slot] = cell;
            }
            T t[5];
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                qn[k * nt + cell] = prim[k];
                t[k] = (T)prim[k];
            }
            put_state<T>(w.qrec + (size_t)cell * kQ, t, (T)gm);
            T cr[8];
            ld8(w.crec + (size_t)cell * kC, cr);
#pragma unroll
            for (int k = 0; k < 5; ++k) rs[k] += (double)cr[k] * (double)cr[k];
        }
        if (cell < g.nBFace) {
            const int gc = nc + cell;
#pragma unroll
            for (int k = 0; k < 5; ++k) qn[k * nt + gc] = qo[k * nt + gc];
        }
    }
    // residual monitor sums: warp shuffle, then one FP64 atomic per block and variable
    __shared__ double part[kThreads / 32][5];
    const int wid = threadIdx.x >> 5, ln = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        double v = rs[k];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (ln == 0) part[wid][k] = v;
    }
    __syncthreads();
    if (threadIdx.x < 5) {
        double v = 0.0;
        for (int i = 0; i < kThreads / 32; ++i) v += part[i][threadIdx.x];
        if (v != 0.0) atomicAdd(&red->resnorm[threadIdx.x], v);
    }
}

template <class T>
void launch_update(const DevGrid &g, const NsConst &c, const Work<T> &w, const double *q64, double *q64_new,
                   Reduce *red, int *neglist, int numSMs, cudaStream_t s)
{
    const int n = g.nCell > g.nBFace ? g.nCell : g.nBFace;
    int blocks = (n + kThreads - 1) / kThreads;
    if (blocks > numSMs * 8) blocks = numSMs * 8;
    update_kernel<T><<<blocks, kThreads, 0, s>>>(g, c, w, q64, q64_new, red, neglist);
}

// SolutionFix (NSSolverUnstruct.cpp:14509-14585) for the listed cells, in the
// reference's cell order: neighbour averages of rho,u,v,w,p (|rho|, |p|),
// neighbours earlier in the reference's order taken after their update,
// later ones before.  One block: the list (at most kMaxNeg cells; empty in
// healthy runs) is sorted by reference number with a bitonic sort in shared
// memory, then one thread repairs the cells in that order.
static constexpr int kFixThreads = 1024;

template <class T>
__global__ void __launch_bounds__(kFixThreads) solution_fix_kernel(DevGrid g, NsConst c, Work<T> w, const double *qo,
                                                                   double *qn, Reduce *red, int *neglist, double *hist)
{
    __shared__ int key[kMaxNeg], val[kMaxNeg];
    if (hist && threadIdx.x == 0) {
        // the residual monitor of the step
        const double v = sqrt(red->resnorm[0] / (double)g.nCell);
        if ((!(v == v) || v > 1.0e300) && red->error == 0) red->error = PHX_ERR_NUMERIC;
        *hist = v;
    }
    const int n = red->negcount;
    if (n <= 0) return;
    if (n > kMaxNeg) {
        if (threadIdx.x == 0) red->error = PHX_ERR_NUMERIC;
        return;
    }
    int m = 1;
    while (m < n) m <<= 1;
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const int v = i < n ? neglist[i] : -1;
        key[i] = i < n ? g.orig[v] : 0x7fffffff;
        val[i] = v;
    }
    __syncthreads();
    for (int k = 2; k <= m; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = threadIdx.x; i < m; i += blockDim.x) {
                const int l = i ^ j;
                if (l > i) {
                    const bool up = (i & k) == 0;
                    if ((key[i] > key[l]) == up) {
                        const int tk = key[i]; key[i] = key[l]; key[l] = tk;
                        const int tv = val[i]; val[i] = val[l]; val[l] = tv;
                    }
                }
            }
            __syncthreads();
        }
    }
    if (threadIdx.x != 0) return;
    const int nt = g.nTotal;
    const double rlim = 1.0e-6 * c.primInf[0], plim = 1.0e-6 * c.primInf[4];
    for (int i = 0; i < n; ++i) {
        const int cell = val[i];
        const int oc = key[i];
        double acc[5] = {0, 0, 0, 0, 0}, wsum = 0.0;
        for (int j = g.c2f_off[cell]; j < g.c2f_off[cell + 1]; ++j) {
            const int nb = g.c2x[j].y;
            const double *src = (g.orig[nb] < oc) ? qn : qo;
            if (src[nb] < rlim || src[4 * nt + nb] < plim) continue;
            wsum += 1.0;
            for (int k = 0; k < 5; ++k) {
                double fv = src[k * nt + nb];
                if (k == 0 || k == 4) fv = fabs(fv);
                acc[k] += fv;
            }
        }
        double prim[5];
        if (wsum > 0.0) { const double o = 1.0 / wsum; for (int k = 0; k < 5; ++k) prim[k] = acc[k] * o; }
        else for (int k = 0; k < 5; ++k) prim[k] = c.primInf[k];
        T t[5];
        for (int k = 0; k < 5; ++k) { qn[k * nt + cell] = prim[k]; t[k] = (T)prim[k]; }
        put_state<T>(w.qrec + (size_t)cell * kQ, t, (T)c.gama);
    }
}

template <class T>
void launch_solution_fix(const DevGrid &g, const NsConst &c, const Work<T> &w, const double *q64, double *q64_new,
                         Reduce *red, int *neglist, double *hist, cudaStream_t s)
{
    solution_fix_kernel<T><<<1, kFixThreads, 0, s>>>(g, c, w, q64, q64_new, red, neglist, hist);
}

// ---------------------------------------------------------------------------
// Layout conversion between the reference order (API) and storage order.
// ---------------------------------------------------------------------------
template <class T>
__global__ void export_kernel(DevGrid g, const T *rec, int stride, int first, int count, int step, int n, double *out,
                              int outLen, const int *at)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int o = g.orig[i], r = at ? at[i] : i;
    for (int k = 0; k < count; ++k) out[(size_t)k * outLen + o] = (double)rec[(size_t)r * stride + first + k * step];
}

template <class T>
void launch_export(const DevGrid &g, const T *rec, int stride, int first, int count, int step, int n, double *out,
                   int outLen, cudaStream_t s, const int *at)
{
    export_kernel<T><<<(n + kThreads - 1) / kThreads, kThreads, 0, s>>>(g, rec, stride, first, count, step, n, out,
                                                                       outLen, at);
}

__global__ void import_q_kernel(DevGrid g, const double *in, double *q)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.nTotal) return;
    const int o = g.orig[i], nt = g.nTotal;
    for (int k = 0; k < 5; ++k) q[(size_t)k * nt + i] = in[(size_t)k * nt + o];
}

__global__ void export_q_kernel(DevGrid g, const double *q, double *out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.nTotal) return;
    const int o = g.orig[i], nt = g.nTotal;
    for (int k = 0; k < 5; ++k) out[(size_t)k * nt + o] = q[(size_t)k * nt + i];
}

void launch_import_q(const DevGrid &g, const double *in, double *q64, cudaStream_t s)
{
    import_q_kernel<<<(g.nTotal + kThreads - 1) / kThreads, kThreads, 0, s>>>(g, in, q64);
}

void launch_export_q(const DevGrid &g, const double *q64, double *out, cudaStream_t s)
{
    export_q_kernel<<<(g.nTotal + kThreads - 1) / kThreads, kThreads, 0, s>>>(g, q64, out);
}

// Residual monitor of the current residual record: out[m] += sum_c res_m^2
// (FP64; block sums, one atomic per block and equation; out zeroed first).
template <class T>
__global__ void __launch_bounds__(kThreads) resnorm_kernel(DevGrid g, Work<T> w, double *out)
{
    double s[5] = {0, 0, 0, 0, 0};
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < g.nCell; c += gridDim.x * blockDim.x) {
        T cr[8];
        ld8(w.crec + (size_t)c * kC, cr);
#pragma unroll
        for (int k = 0; k < 5; ++k) s[k] += (double)cr[k] * (double)cr[k];
    }
    __shared__ double part[kThreads / 32][5];
    const int wid = threadIdx.x >> 5, ln = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        double v = s[k];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (ln == 0) part[wid][k] = v;
    }
    __syncthreads();
    if (threadIdx.x < 5) {
        double v = 0.0;
        for (int i = 0; i < kThreads / 32; ++i) v += part[i][threadIdx.x];
        if (v != 0.0) atomicAdd(out + threadIdx.x, v);
    }
}

template <class T>
void launch_resnorm(const DevGrid &g, const Work<T> &w, double *out, int numSMs, cudaStream_t s)
{
    cudaMemsetAsync(out, 0, sizeof(double) * 5, s);
    int blocks = (g.nCell + kThreads - 1) / kThreads;
    if (blocks > numSMs * 8) blocks = numSMs * 8;
    resnorm_kernel<T><<<blocks, kThreads, 0, s>>>(g, w, out);
}
template void launch_resnorm<double>(const DevGrid &, const Work<double> &, double *, int, cudaStream_t);
template void launch_resnorm<float>(const DevGrid &, const Work<float> &, double *, int, cudaStream_t);

// Explicit instantiations for the FP64 and mixed paths.
#define PHX_INSTANTIATE(T)                                                                                         \
    template void launch_face_geometry<T>(const DevGrid &, const NsConst &, const Work<T> &, cudaStream_t);        \
    template void launch_boundary<T>(const DevGrid &, const NsConst &, double *, const Work<T> &, cudaStream_t);   \
    template void launch_gradient_limiter<T>(const DevGrid &, const NsConst &, const Work<T> &, int, cudaStream_t); \
    template void launch_residual<T>(const DevGrid &, const NsConst &, const Work<T> &, Reduce *, double,           \
                                     cudaStream_t);                                                                 \
    template int launch_lusgs<T>(const DevGrid &, const NsConst &, const Work<T> &, Reduce *, int, cudaStream_t,   \
                                 int);                                                                             \
    template void launch_boundary_post<T>(const DevGrid &, const NsConst &, double *, const Work<T> &,           \
                                          cudaStream_t);                                                            \
    template void launch_update<T>(const DevGrid &, const NsConst &, const Work<T> &, const double *, double *,     \
                                   Reduce *, int *, int, cudaStream_t);                                             \
    template void launch_solution_fix<T>(const DevGrid &, const NsConst &, const Work<T> &, const double *,         \
                                         double *, Reduce *, int *, double *, cudaStream_t);                        \
    template void launch_sync_qrec<T>(const DevGrid &, const NsConst &, const double *, const Work<T> &,            \
                                      cudaStream_t);                                                                \
    template void launch_export<T>(const DevGrid &, const T *, int, int, int, int, int, double *, int, cudaStream_t, \
                                   const int *);
PHX_INSTANTIATE(double)
PHX_INSTANTIATE(float)

}  // namespace phx
