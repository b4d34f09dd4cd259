// Face geometry of the passes in the working precision (records: kNrm, kGeo,
// kGeoSa), formed in FP64 from the metrics: FaceWeight (Geo_UnstructGrid.cpp:
// 2420-2478) and the geometric part of ComputeVisflux (NSSolverUnstruct.cpp:
// 13147-13236).  Interface faces are interior faces (FaceWeight,
// Geo_UnstructGrid.cpp:2475).  Kept by face_geometry_kernel or formed in the passes.
#pragma once
#include "phx_device.cuh"

namespace phx {

// Unit normal times area, or, least squares, the vector from the left to the
// right centre and the weight.
template <class T>
__device__ __forceinline__ void form_normal(const DevGrid &g, bool lsq, int f, int le, int re, T *nr)
{
    double fr[8];
    ld8(g.frec + (size_t)f * kF, fr);
    if (lsq) {
        double xl[4], xr[4];
        ld4(g.xrec + (size_t)le * kX, xl);
        ld4(g.xrec + (size_t)re * kX, xr);
#pragma unroll
        for (int k = 0; k < 3; ++k) nr[k] = (T)(xr[k] - xl[k]);
    } else {
#pragma unroll
        for (int k = 0; k < 3; ++k) nr[k] = (T)(fr[k] * fr[3]);
    }
    nr[3] = (T)fr[7];
}

// The limiters' part: unit normal and area, face centre less the cell's.
template <class T>
__device__ __forceinline__ void form_side(const DevGrid &g, int f, int cell, T *fn, T *dc)
{
    double fr[8], xc[4];
    ld8(g.frec + (size_t)f * kF, fr);
    ld4(g.xrec + (size_t)cell * kX, xc);
#pragma unroll
    for (int k = 0; k < 4; ++k) fn[k] = (T)fr[k];
#pragma unroll
    for (int k = 0; k < 3; ++k) dc[k] = (T)(fr[4 + k] - xc[k]);
}

// The face pass's record, in its five (inviscid: three) quarters.
template <class T, bool kVisc>
__device__ __forceinline__ void form_face(const DevGrid &g, int f, int le, int re, T *gn, T *gl, T *gr, T *xol, T *xor_)
{
    double fr[8], xl[4], xr[4], dl[3], dr[3];
    ld8(g.frec + (size_t)f * kF, fr);
    ld4(g.xrec + (size_t)le * kX, xl);
    ld4(g.xrec + (size_t)re * kX, xr);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        dl[k] = fr[4 + k] - xl[k];
        dr[k] = fr[4 + k] - xr[k];
        gn[k] = (T)fr[k];
        gl[k] = (T)dl[k];
        gr[k] = (T)dr[k];
    }
    gn[3] = (T)fr[3];
    gl[3] = T(1);
    gr[3] = T(0);
    if (!kVisc) return;
    const bool bnd = f < g.nBFace && g.bkind[f] != BK_INTERFACE;
    const double d1 = sqrt(dl[0] * dl[0] + dl[1] * dl[1] + dl[2] * dl[2]);
    const double d2 = sqrt(dr[0] * dr[0] + dr[1] * dr[1] + dr[2] * dr[2]);
    if (!bnd) gl[3] = (T)(d2 / (d1 + d2 + kSmall));
    const double dL = -(fr[0] * dl[0] + fr[1] * dl[1] + fr[2] * dl[2]);
    const double dR = -(fr[0] * dr[0] + fr[1] * dr[1] + fr[2] * dr[2]);
    const int vf = g.vflag[f];
    double A = 0.0, B = 0.0;
    if (vf & 2) {
        const double wl = bnd ? 1.0 : dL * dL / (dL * dL + dR * dR);
        A = wl / dL;
        B = (1.0 - wl) / dR;
    }
    gr[3] = (T)A;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        xol[k] = vf & 1 ? (T)(fr[k] * dL + dl[k]) : T(0);
        xor_[k] = vf & 1 ? (T)(fr[k] * dR + dr[k]) : T(0);
    }
    xol[3] = (T)B;
    xor_[3] = (T)fabs(fr[0] * (xr[0] - xl[0]) + fr[1] * (xr[1] - xl[1]) + fr[2] * (xr[2] - xl[2]));
}

// The SA face pass's record: the normal derivative of TurbSolverUnstr::
// ComputeVisflux (TurbSolverUnstr.cpp:4438-4674) is the weighted differences to
// the mean of both sides, or across the whole distance on boundary faces other
// than symmetry.
template <class T>
__device__ __forceinline__ void form_sa(const DevGrid &g, int f, int le, int re, T *o)
{
    double fr[8], xl[4], xr[4];
    ld8(g.frec + (size_t)f * kF, fr);
    ld4(g.xrec + (size_t)le * kX, xl);
    ld4(g.xrec + (size_t)re * kX, xr);
    double C = 0.0;
    if (g.vflag[f] & 4) {
        const double dL = -(fr[0] * (fr[4] - xl[0]) + fr[1] * (fr[5] - xl[1]) + fr[2] * (fr[6] - xl[2]));
        const double dR = -(fr[0] * (fr[4] - xr[0]) + fr[1] * (fr[5] - xr[1]) + fr[2] * (fr[6] - xr[2]));
        const double wl = dL * dL / (dL * dL + dR * dR);
        C = 0.5 * ((1.0 - wl) / dR - wl / dL);
        if (f < g.nBFace && g.bkind[f] != BK_INTERFACE && g.btype[f] != PHX_BC_SYMMETRY)
            C = 1.0 / ((xr[0] - xl[0]) * fr[0] + (xr[1] - xl[1]) * fr[1] + (xr[2] - xl[2]) * fr[2]);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) o[k] = (T)fr[k];
    o[4] = (T)C;
    o[5] = (T)(1.0 / (0.5 * (xl[3] + xr[3])));
    o[6] = o[7] = T(0);
}

}  // namespace phx
