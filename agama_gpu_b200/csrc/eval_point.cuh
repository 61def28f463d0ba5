// eval_point.cuh -- one point of a leaf, and the write of a point's result: shared by the
// evaluation kernels (eval.cu, split.cu).
#pragma once
#include "agb_dev.cuh"
#include "multipole.cuh"
#include "cylspline.cuh"
#include "analytic.cuh"

// internal mode of agb_eval_vjp_force: the VJP plus the force of the same leaves
// (written to the `hess` pointer as [N,3]) from the same per-point sums
#define AGB_MODE_VJPF 5

__host__ __device__ constexpr int stage_rec(int mode)
{
    return mode == AGB_MODE_HESS ? 10 : mode == AGB_MODE_GRAD ? 4 : mode == AGB_MODE_VJP ? 3
         : mode == AGB_MODE_VJPF ? 6 : 1;
}
#define AGB_STAGE_MAX_REC 10

// AN: the tree holds analytic leaves only (no expansion code compiled in: a
// small register footprint and more resident blocks for the Hessian modes)
template <int MODE, typename R, bool EXACT, bool AN = false>
__device__ __forceinline__ void eval_component(const DevComp& c, double x, double y, double z,
                                               PointOut& o)
{
    switch (c.kind) {
    case AGB_KIND_MULTIPOLE:     if (!AN) multipole_point<MODE, R>(c, x, y, z, o); break;
    case AGB_KIND_CYLSPLINE:     if (!AN) cylspline_point<MODE, EXACT, R>(c, x, y, z, o); break;
    case AGB_KIND_NFW:           nfw_point<MODE>(c.p, x, y, z, o); break;
    case AGB_KIND_PLUMMER:       plummer_point<MODE>(c.p, x, y, z, o); break;
    case AGB_KIND_HERNQUIST:     hernquist_point<MODE>(c.p, x, y, z, o); break;
    case AGB_KIND_DEHNEN:        dehnen_point<MODE>(c.p, x, y, z, o); break;
    case AGB_KIND_ISOCHRONE:     isochrone_point<MODE>(c.p, x, y, z, o); break;
    case AGB_KIND_MIYAMOTONAGAI: mn_point<MODE>(c.p, x, y, z, o); break;
    case AGB_KIND_LOGHALO:       loghalo_point<MODE>(c.p, x, y, z, o); break;
    case AGB_KIND_DISKANSATZ:    diskansatz_point<MODE>(c.p, x, y, z, o); break;
    case AGB_KIND_UNIFORMACC:    uniform_point<MODE>(c.p, x, y, z, o); break;
    default: break;
    }
}

// one point's result: the VJP contraction or the outputs, into the sorted-order record of
// position pos or the arrays' row i
template <int MODE>
__device__ __forceinline__ void eval_write(const EvalArgs& a, long long pos, long long i,
                                           double phi, double g0, double g1, double g2,
                                           const double h[6], double rho)
{
    constexpr bool VJP = MODE == AGB_MODE_VJP || MODE == AGB_MODE_VJPF;
    if (VJP) {
        // L(Phi, F): dL/dx = gPhi grad(Phi) + (dF/dx)^T gF = gPhi grad(Phi) - H gF
        const double gp = a.gphi ? a.gphi[i] : 0.0;
        double f0 = 0.0, f1 = 0.0, f2 = 0.0;
        if (a.gforce) { f0 = a.gforce[3 * i]; f1 = a.gforce[3 * i + 1]; f2 = a.gforce[3 * i + 2]; }
        const double v0 = gp * g0 - (h[0] * f0 + h[3] * f1 + h[5] * f2);
        const double v1 = gp * g1 - (h[3] * f0 + h[1] * f1 + h[4] * f2);
        const double v2 = gp * g2 - (h[5] * f0 + h[4] * f1 + h[2] * f2);
        if (MODE == AGB_MODE_VJPF) {
            if (a.stage) {
                double* o = a.stage + 6 * pos;
                o[0] = v0; o[1] = v1; o[2] = v2; o[3] = -g0; o[4] = -g1; o[5] = -g2;
            } else {
                a.grad[3 * i] = v0; a.grad[3 * i + 1] = v1; a.grad[3 * i + 2] = v2;
                a.hess[3 * i] = -g0; a.hess[3 * i + 1] = -g1; a.hess[3 * i + 2] = -g2;
            }
            return;
        }
        double* o = a.stage ? a.stage + 3 * pos : a.grad + 3 * i;
        o[0] = v0; o[1] = v1; o[2] = v2;
        return;
    }
    const double sg = (a.out_flags & AGB_OUT_NEGATE) ? -1.0 : 1.0;
    if (MODE == AGB_MODE_DENS) {
        if (a.stage) a.stage[pos] = rho;
        else a.rho[i] = rho;
        return;
    }
    if (a.stage) {
        // sorted order: consecutive threads write consecutive records
        constexpr int REC = stage_rec(MODE);
        double* o = a.stage + REC * pos;
        o[0] = phi;
        if (MODE != AGB_MODE_POT) { o[1] = sg * g0; o[2] = sg * g1; o[3] = sg * g2; }
        if (MODE == AGB_MODE_HESS) {
            #pragma unroll
            for (int q = 0; q < 6; ++q) o[4 + q] = sg * h[q];
        }
        return;
    }
    if (a.phi) a.phi[i] = phi;
    if (MODE != AGB_MODE_POT && a.grad) {
        a.grad[3 * i] = sg * g0; a.grad[3 * i + 1] = sg * g1; a.grad[3 * i + 2] = sg * g2;
    }
    if (MODE == AGB_MODE_HESS) {
        #pragma unroll
        for (int q = 0; q < 6; ++q) a.hess[6 * i + q] = sg * h[q];
    }
}
