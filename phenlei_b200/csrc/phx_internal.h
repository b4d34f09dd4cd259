// Internal definitions of the phx library: the device-side grid, the
// working arrays of one precision, and the kernel launchers.
//
// Storage layout.  The API speaks the reference's layout (original cell and
// face numbers, structure-of-arrays).  On the device, cells are stored in a
// space-filling-curve (Morton) order of their centroids and faces grouped by
// their storage owner, so that face neighbours lie close in memory; gathered
// per-cell and per-face data are array-of-structs records read with vector
// loads.  The reference's numbering is kept wherever it decides an order:
// every cell's face list is sorted by the reference face number (the order
// LoadFlux and the Green-Gauss loop accumulate in), and the LU-SGS
// schedules come from the reference cell numbers.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <vector>

#include "../../include/phx.h"

namespace phx {

constexpr double kSmall = 1.0e-40;  // API/Common/include/Precision.h:27 (SMALL, TINY)
constexpr double kLarge = 1.0e40;   // Precision.h:26 (LARGE)

// Boundary handling classes, resolved once from (bcType, viscousType) the way
// NSSolverUnstruct::Boundary dispatches (NSSolverUnstruct.cpp:13469-13512).
enum BcKind : int32_t {
    BK_SYMMETRY = 0,   // SymmetryBCRegion (also inviscid solid walls)
    BK_WALL = 1,       // ViscousAdiabaticWallBCRegion
    BK_FARFIELD = 2,   // FarfieldBCRegion
    BK_EXTRAP = 3,     // OutflowBCRegion / extrapolation
    BK_INTERFACE = 4,  // a face cut by a partition (PHENGLEI::INTERFACE): the ghost is the neighbouring part's
                       // cell, filled by halo exchanges; every pass but the boundary treats the face as interior
};

// Record strides (elements).
constexpr int kQ = 8;      // qrec: rho u v w p | c2 hm | limiter
constexpr int kG = 20;     // grec: (d/dx, d/dy, d/dz) of var k at 3k..3k+2 | pad | temperature gradient 16..18 | pad
constexpr int kC = 8;      // crec: res0..4 | 1 / LU-SGS diagonal (unclamped dt) | inviscid | viscous spectral radius
constexpr int kD = 8;      // dqrec / dflux: 5 values | pad
constexpr int kF = 8;      // frec (FP64): nx ny nz area xfc yfc zfc | least-squares face weight
constexpr int kX = 4;      // xrec (FP64): xcc ycc zcc vol
constexpr int kFlux = 12;  // face flux record: inviscid F0..4 (times area) | inviscid and viscous spectral parts |
                           // viscous F1..4 (times area; F0 is zero) | pad
// Face geometry in the working precision, formed in FP64 from the metrics
// (phx_geometry.cuh).  fnrm: unit normal times area (least squares: vector
// from the left to the right centre, weight).  fgeo: unit normal, area | face
// centre less left centre, left weight of the face gradient | less right centre,
// A | for viscous runs: left offset, B | right offset, centre distance along the
// normal.  A and B are the weights of the left and right difference to the face
// value in the normal derivative, the offsets lead from a centre to its foot on
// the normal line (zero where a face has no such term).
constexpr int kNrm = 4;
template <bool kVisc>
constexpr int kGeo = kVisc ? 20 : 12;
constexpr int kN = 8;      // nrec (GG-node): q node values (5), temperature node values of this
                           // iteration's state, those the gradient uses (the previous state's), pad
// LU-SGS factors of a face use, as the sweeps read them (sweep_use): unit normal
// from the cell to the neighbour times half the area, diagonal factor | the
// neighbour's u v w, total enthalpy.  Whole 32-byte sectors: with 48-byte records
// the passes that write them took 6 % longer.
constexpr int kUse = 8;
constexpr int kLeadF = 8;  // forward right-hand side of a cell: residual (5) | reciprocal diagonal | time step | pad
constexpr int kLeadB = 16; // backward: residual less the forward sums (5), reciprocal diagonal, pad | boundary part (5), pad
constexpr int kLeadT = 2;  // SA sweeps: right-hand side | reciprocal spectral radius
constexpr int kSweepLanes = 4;   // LU-SGS lanes (neighbour entries) per slot of a schedule row
constexpr int kSweepSlots = 8;   // slots (cells) of a row: one warp
constexpr int kMaxCellFaces = 8; // faces of a cell
constexpr int kSweepLocal = 8;   // rows whose results a warp's shared memory holds
constexpr int kSweepFirst = 8, kSweepLast = 16;   // flags of the host schedule: first, last row of a cell
// A schedule row on the device (kSweepRow words): per lane the entry of the row
// after next of its warp, the place of the neighbour's record (>= 0: it is
// polled) or ~ the shared-memory slot of its result (kSweepZero: none, reads
// zeros); then per slot {storage cell (-1: idle, or not the cell's last row),
// shared-memory slot of the result | kSweepMulti (the row holds a cell of several
// rows) | kSweepCarry (not the cell's first), forward: slot of the cell's last
// backward row; backward, in the first row of a cell with boundary faces: its place
// in ghost_cell + 1}.
constexpr int kSweepRow = 64, kSweepZero = kSweepLocal * kSweepSlots;
constexpr int kSweepMulti = 256, kSweepCarry = 512;
// Bytes of a row as the sweeps copy it: factors of the lanes' face uses, right-
// hand sides of the cells, schedule row; NS (both sweeps) and SA.
template <class T, bool kForward>
constexpr int kRowNs = (32 * kUse + kSweepSlots * (kForward ? kLeadF : kLeadB)) * (int)sizeof(T) + kSweepRow * 4;
// Compact layout: of the warp's row after next, the lanes' uses {face, neighbour} and the slots' cells (-1: none, or
// not the cell's last row); schedule row.
constexpr int kRowCompact = 32 * 8 + kSweepSlots * 4 + kSweepRow * 4;
template <class T>
constexpr int kRowSa = (32 + kSweepSlots * kLeadT) * (int)sizeof(T) + kSweepRow * 4;
constexpr long long kDefaultSpinLimit = 20000000LL;   // polls per dependency wait (~1-2 s)
// Spalart-Allmaras records
constexpr int kTr = 4;     // trec: nu~ | eddy viscosity | laminar viscosity of the NS step | pad
constexpr int kTg = 4;     // tgrad: d nu~ / dx, dy, dz | pad
constexpr int kTc = 4;     // tcrec: res_turb | spec_turb | its reciprocal | pad (compact: backward right-hand side)
constexpr int kTf = 4;     // tface: convection and first diffusion flux | second diffusion flux (times the side's own
                           // diffusivity) | spectral terms of the left and of the right cell
// SA face geometry (working precision, formed in FP64): unit normal, area |
// factor of the difference right less left in the normal derivative | one over
// the mean volume | pad.
constexpr int kGeoSa = 8;

// Schedule of one LU-SGS sweep (phx_schedule.cpp): warp w runs rows
// [row_off[w], row_off[w + 1]).
struct SweepDev {
    int nWarps, nRows;
    const int *row_off;
    const int *first;    // [nWarps][2][32] entries of the warp's first two rows
    const int2 *first_use;    // compact layout: [nWarps][2][32] their uses
    const int *first_cell;    // compact layout: [nWarps][2][8] and cells
};

// Read-only device grid (FP64 metrics, connectivity, schedules), storage order.
struct DevGrid {
    // 0, full layout: the face geometry is stored, and the LU-SGS rows hold all that the
    // sweeps need, written by the passes.  1, compact layout (large meshes): the passes
    // form the geometry, the rows hold the schedule alone and the sweeps gather their
    // factors; the same values.
    int compact;
    int nCell, nBFace, nFace, nTotal;
    const int2 *lr;              // [nFace] left, right (boundary face f: right = nCell + f)
    const double *frec;          // [nFace][kF]
    const double *xrec;          // [nTotal][kX]
    const double *skew;          // [nCell]
    const double *volpow;        // [nCell] pow(pow(vol, 1/3), 3) as VencatLimiter7 forms it
    const double *walldist;      // [nCell]
    const double *lsq;           // [nCell][8] inverse least-squares matrix ixx iyy izz ixy ixz iyz | pad (lsq only)
    // [nFace] viscous-flux geometry switches of ComputeVisflux: bit 0 = both
    // centre angles above skewnessAngle (project the cell values onto the
    // normal line), bit 1 = both angles positive and |dL|, |dR| > TINY (form
    // the normal derivative), bit 2 = both angles above turbSkewnessAngle and
    // |dL|, |dR| > TINY (the SA diffusion's normal derivative); pure geometry,
    // decided on the host
    const uint8_t *vflag;
    const int *c2f_off;          // faces of each cell, ordered by the reference face number:
    const int2 *c2x;             // {face, ~ it where the cell is the right cell; cell or ghost behind it}
    const int *orig;             // [nTotal] reference number of each cell (ghost: nCell + reference face)
    const int32_t *bkind;        // [nBFace] BcKind
    const int32_t *btype;        // [nBFace] bcType
    const uint8_t *farfield_adj; // [nCell] 1 if the cell touches a limiter-zeroing boundary
    SweepDev fwd, bwd;           // LU-SGS schedules
    const int2 *use;             // [nFace] (full layout) lane (row * 32 + lane) of the left and of the right cell's use of the face;
                                 // >= 0 in the forward sweep, ~ it in the backward sweep (interior faces)
    const int *lead;             // [nCell] slot (row * kSweepSlots + slot) of the cell's last forward row
    const int *last;             // [nCell] and of its last backward row
    int nGhostCell;              // cells with boundary faces: {storage cell, slot of its first backward row}
    const int2 *ghost_cell;
    // GG-node (gradientName 2): per storage node, its contributions {storage
    // cell, or storage boundary face with the sign bit set} with 1/distance
    // weights in the reference's order and their sum; per storage face, its
    // storage nodes in the face's node order
    int nNode;
    const int *node_off, *node_src;
    const double *node_w, *node_wsum;
    const int *fn_off, *fn_idx;
    // GG-node of the SA variable: per storage node, the {owner, other side}
    // pairs whose values it averages, in the reference's order
    const int *tn_off;
    const int2 *tn_pairs;
    double avgVol;
};

// Scalars of the NS path (derived from phx_params as the reference's
// Param_NSSolverUnstruct and PerfectGas do).
struct NsConst {
    double gama, coefState, pTotal;
    double primInf[5];
    double acoustic, convective;   // Roe entropy-fix coefficients
    int scheme;                    // PHX_SCHEME_* in use (Van Leer during the flow initialisation)
    int firstOrder;                // flow initialisation: no reconstruction, zero limiter
    double ausmpwLim;              // AusmpwPlusLimiter
    double venkatK3;               // K^3 / (avgVol^(1/3))^3, as VencatLimiter7 forms it
    int viscous;                   // viscousType
    int limiter;                   // 0 none, 1 vencat
    int reconMethod;
    double cflStart, cflEnd;
    int cflVaryStep;
    double ktmax;
    int nSweeps;
    double lusgsTol;
    double reynolds;
    int gradient;                  // 0 Green-Gauss cell, 1 least squares
    // viscous terms (Param_NSSolverUnstruct / PerfectGas): 1/Re, 1/Pr, 1/Pr_t,
    // cp = 1 / ((gamma - 1) M^2), Sutherland constant over the reference
    // temperature, skewness switch of the viscous flux (degrees)
    double oRe, oPrl, oPrt, cp, tsuth, skewAngle;
    // Spalart-Allmaras (viscousType 3): free-stream nu~ and eddy viscosity of
    // far-field inflow ghosts, turbCFLScale
    double nutInf, vistInf, turbCflScale;
    int saSource;                  // 0 exact source, 1 learned source (exact for nu~ <= 0), 2 learned inside its
                                   // training hull, exact outside
    long long spinLimit;           // polls per device-side dependency wait before PHX_ERR_TIMEOUT
    int holdCell;                  // fault injection: storage cell whose forward LU-SGS result never comes (the
                                   // wait on it runs out); -1 off
};

// Working arrays of one precision T (double: FP64 path, float: mixed path).
template <class T>
struct Work {
    T *qrec;        // [nTotal][kQ] working state, c2 = |gamma p / rho|, total enthalpy, limiter
    // full layout | compact layout
    union {
        T *fnrm;    // [nFace][kNrm] face geometry
        T *frad;    // [nFace][2] Roe spectral radius, viscous spectral term
    };
    union {
        T *fgeo;    // [nFace][kGeo] face geometry
        T *lead;    // [nCell][kLeadF] right-hand side of the backward sweep
    };
    union {
        T *fsa;     // [nFace][kGeoSa] SA face geometry (SA runs; else null)
        T *gsum;    // [nGhostCell][kLeadF] boundary part of the backward right-hand side
    };
    T *grec;        // [nTotal][kG] primitive gradients (ghost rows: interface ghosts only, from the halo exchange)
    T *flux;        // [nFace][kFlux] face flux times area and inviscid spectral radius term (in the scratch)
    T *coef;        // [nBFace][kUse] LU-SGS factors of the boundary faces' uses
    unsigned char *rowf, *rowb;   // [rows][kRowNs] (compact: [kRowCompact]) rows of the forward and the backward sweep
    T *crec;        // [nCell][kC] residual, diagonal, spectral radii
    T *dtraw;       // [nCell] CFL * vol / spectral radius, before the ktmax clamp
    // LU-SGS dq, write-once per sweep, by the slot of the cell's last row (a
    // row's eight records are written together, and mostly read together)
    T *dqrec;       // [backward rows][kSweepSlots][kD] backward sweep
    T *dqfwd;       // [forward rows][kSweepSlots][kD] forward sweep
    T *dqghost;     // [nBFace][kD] forward dq behind interface faces, from the halo exchange between the sweeps
    T *trec;        // [nTotal][kTr] SA variable, eddy and laminar viscosity (SA runs; else null)
    T *nrec;        // [nNode][kN] GG-node node values (GG-node runs; else null)
};

// Spalart-Allmaras working arrays (one precision T; the FP64 master nu~ is qt64).
template <class T>
struct TurbWork {
    double *qt64;   // [nTotal] master nu~
    T *tgrad;       // [nCell][kTg] gradient of nu~
    T *tcrec;       // [nCell][kTc] residual, spectral radius, its reciprocal, pad
    T *tface;       // [nFace][kTf] face terms (in the scratch)
    unsigned char *trowf, *trowb;   // [rows][kRowSa] LU-SGS rows (compact: the NS sweeps' rows)
    T *tmat;        // [nFace][2] compact layout: LU-SGS matrix of the left and the right cell's use
    T *tdq;         // [backward rows][kSweepSlots] LU-SGS dq (write-once per sweep, by slot as the NS records)
    T *tdqf;        // [forward rows][kSweepSlots] forward-sweep dq
    T *tsrc;        // [nCell] source computed by the learned-source kernel (sa_source != 0)
    T *qtnode;      // [nNode] GG-node node values of nu~ for the next SA gradient (GG-node runs; else null)
};

struct Reduce {
    unsigned long long mindt_bits;  // min over cells of dtraw (positive doubles order as integers)
    double resnorm[5];
    int negcount;
    int error;                      // PHX_ERR_TIMEOUT / PHX_ERR_NUMERIC
};

// Kernel launchers (phx_kernels.cu).
// The stored face geometry from the FP64 metrics.
template <class T>
void launch_face_geometry(const DevGrid &g, const NsConst &c, const Work<T> &w, cudaStream_t s);
template <class T>
void launch_boundary(const DevGrid &g, const NsConst &c, double *q64, const Work<T> &w, cudaStream_t s);
template <class T>
void launch_gradient_limiter(const DevGrid &g, const NsConst &c, const Work<T> &w, int nodePrev, cudaStream_t s);
template <class T>
void launch_residual(const DevGrid &g, const NsConst &c, const Work<T> &w, Reduce *red, double cfl, cudaStream_t s);
// Resident warps of the sweeps (NS; SA's kernels hold at least as many).
template <class T>
int sweep_max_warps(int numSMs);
template <class T>
int sa_sweep_max_warps(int numSMs);
// LU-SGS sweeps: bit 0 of `sweeps` runs the forward sweep (after resetting
// the sweep records), bit 1 the backward sweep; 3 runs both in one launch.
constexpr int kSweepForward = 1, kSweepBackward = 2, kSweepBoth = 3;
template <class T>
int launch_lusgs(const DevGrid &g, const NsConst &c, const Work<T> &w, Reduce *red, int numSMs, cudaStream_t s,
                 int sweeps = kSweepBoth);
template <class T>
void launch_update(const DevGrid &g, const NsConst &c, const Work<T> &w, const double *q64, double *q64_new,
                   Reduce *red, int *neglist, int numSMs, cudaStream_t s);
// The ordered repair pass; with hist, also the step's residual monitor into it.
template <class T>
void launch_solution_fix(const DevGrid &g, const NsConst &c, const Work<T> &w, const double *q64, double *q64_new,
                         Reduce *red, int *neglist, double *hist, cudaStream_t s);
// Refreshes qrec (state, c2, hm) of all cells and ghosts from the FP64 master state.
template <class T>
void launch_sync_qrec(const DevGrid &g, const NsConst &c, const double *q64, const Work<T> &w, cudaStream_t s);
// Export of record fields into reference-order SoA: out[k * outLen +
// orig[i]] = rec[i * stride + first + k * step] for k < count, i < n.
// `at` (if given): where record i lies.
template <class T>
void launch_export(const DevGrid &g, const T *rec, int stride, int first, int count, int step, int n, double *out,
                   int outLen, cudaStream_t s, const int *at = nullptr);
// q64[k][i] = in[k][orig[i]] and the inverse.
void launch_import_q(const DevGrid &g, const double *in, double *q64, cudaStream_t s);
void launch_export_q(const DevGrid &g, const double *q64, double *out, cudaStream_t s);
// out[m] = sum over cells of res_m^2 (FP64 device reduction of the residual record).
template <class T>
void launch_resnorm(const DevGrid &g, const Work<T> &w, double *out, int numSMs, cudaStream_t s);
// NS boundary after the update (Controller::PostSolve): ghost states only,
// the laminar viscosity of the ghosts keeps its value of the NS step.
template <class T>
void launch_boundary_post(const DevGrid &g, const NsConst &c, double *q64, const Work<T> &w, cudaStream_t s);
// Spalart-Allmaras step (phx_sa.cu).
template <class T>
void launch_sa_boundary(const DevGrid &g, const NsConst &c, const double *q64, const Work<T> &w,
                        const TurbWork<T> &t, cudaStream_t s);
struct MlpDev;
template <class T>
void launch_sa_residual(const DevGrid &g, const NsConst &c, const double *q64, const Work<T> &w,
                        const TurbWork<T> &t, Reduce *red, const MlpDev *mlp, unsigned long long *nmlp, int numSMs,
                        cudaStream_t s);
// Learned SA source (phx_mlp.cu): source of every cell into t.tsrc; training-sample capture.
template <class T>
void launch_mlp_source(const DevGrid &g, const NsConst &c, const Work<T> &w, const TurbWork<T> &t,
                       const MlpDev &mlp, Reduce *red, unsigned long long *nmlp, int numSMs, cudaStream_t s);
template <class T>
void launch_mlp_capture(const DevGrid &g, const NsConst &c, const Work<T> &w, const TurbWork<T> &t, float *feat,
                        float *targ, int *cells, float *scales, long long cap, unsigned long long *count,
                        cudaStream_t s);
template <class T>
void launch_turb_node_values(const DevGrid &g, const Work<T> &w, const TurbWork<T> &t, cudaStream_t s);
template <class T>
int launch_sa_lusgs(const DevGrid &g, const NsConst &c, const Work<T> &w, const TurbWork<T> &t, Reduce *red,
                    int numSMs, cudaStream_t s, int sweeps = kSweepBoth);
template <class T>
void launch_sa_update(const DevGrid &g, const NsConst &c, const Work<T> &w, const TurbWork<T> &t, cudaStream_t s);
// Wall force sums (16 doubles, the last zero) of the current state.
template <class T>
void launch_forces(const DevGrid &g, const NsConst &c, const Work<T> &w, const double *q64, double *out,
                   cudaStream_t s);
// qt64[i] = in[orig[i]] and the working copy in trec, cells and ghosts.
template <class T>
void launch_import_turb(const DevGrid &g, const double *in, const TurbWork<T> &t, const Work<T> &w, cudaStream_t s);
// trec slot 1 (eddy viscosity) of cells and ghosts from in[orig[i]].
template <class T>
void launch_import_vist(const DevGrid &g, const double *in, const Work<T> &w, cudaStream_t s);
// Halo exchange of a partitioned grid (phx_halo.cu): pack gathers rows of
// the cells `send` (storage indices) into buf, unpack scatters rows of buf
// into the ghosts `recv` (storage indices); `field` is a PHX_HALO_* code and
// a row holds halo_row_bytes<T>(field) bytes.
template <class T>
size_t halo_row_bytes(int field);
template <class T>
void launch_halo_pack(const DevGrid &g, int field, const double *q64, const Work<T> &w, const TurbWork<T> &t,
                      const int *send, int n, unsigned char *buf, cudaStream_t s);
template <class T>
void launch_halo_unpack(const DevGrid &g, const NsConst &c, int field, double *q64, const Work<T> &w,
                        const TurbWork<T> &t, const int *recv, int n, const unsigned char *buf, cudaStream_t s);

}  // namespace phx
