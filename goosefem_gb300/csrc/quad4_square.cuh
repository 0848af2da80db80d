// The FP64 closed forms that the explicit step's kernels share: the element forces of a uniform
// square Quad4 element and the velocity estimates of a lumped-mass class.
#pragma once

#include "common.cuh"

namespace gfgpu {

struct VerletCoef {
    double dt, h, c, eta; // h = 0.5 dt, c = 0.5 dt^2
};

// Per-class coefficients of the three velocity estimates in closed form. With be = m^-1 eta,
// h = dt/2 and mR = m^-1 (fext - f), the sequence v1 = v + dt a, a1 = mR - be v1, w = v + h a,
// v2 = w + h a1, a2 = mR - be v2, v' = w + h a2, a' = mR - be v' is
//   v' = c1 v + c2 a + c3 mR,  c1 = (1 - h be) + h^2 be^2,  c2 = h (1 - h be) + h^2 be^2 dt,
//   c3 = h (1 - h be),  a' = mR - be v'
// (10 FP64 instructions per free dof instead of 14).
struct MassClassTab {
    int n;
    double mi[GFGPU_MASS_CLASSES], be[GFGPU_MASS_CLASSES], c1[GFGPU_MASS_CLASSES],
        c2[GFGPU_MASS_CLASSES], c3[GFGPU_MASS_CLASSES];
};

// The table in shared memory (written by the block's first threads; the caller synchronises).
struct MassClassShared {
    double t[5][GFGPU_MASS_CLASSES];
    __device__ __forceinline__ void load(const MassClassTab& tab)
    {
        const int c = threadIdx.x;
        if (c < GFGPU_MASS_CLASSES) {
            t[0][c] = tab.mi[c];
            t[1][c] = tab.be[c];
            t[2][c] = tab.c1[c];
            t[3][c] = tab.c2[c];
            t[4][c] = tab.c3[c];
        }
    }
    // velocity and acceleration of one component of class c under the internal force f
    __device__ __forceinline__ void update(int c, double f, bool has_fext, double fx, double vn, double an,
                                           double h, double& vv, double& aa) const
    {
        if (c < GFGPU_MASS_CLASSES) {
            const double mi = t[0][c];
            const double mR = has_fext ? mi * (fx - f) : -mi * f;
            vv = fma(t[4][c], mR, fma(t[3][c], an, t[2][c] * vn));
            aa = fma(-t[1][c], vv, mR);
        }
        else {
            // prescribed: the solve leaves a untouched; v follows the estimates
            aa = an;
            vv = fma(h, an + an, vn);
        }
    }
};

// Forces of a square element from its nodal displacements and coefficients {L, M}, {N, kH}
// (k_quad4_square_coef): 34 FP64 instructions.
__device__ __forceinline__ void quad4_square_forces(double2 u0, double2 u1, double2 u2, double2 u3, double2 c01,
                                                    double2 c23, double2 (&f)[4])
{
    const double L = c01.x, M = c01.y, N = c23.x, kH = c23.y;
    const double px = u2.x - u0.x, qx = u1.x - u3.x;
    const double py = u2.y - u0.y, qy = u1.y - u3.y;
    const double A1x = px + qx, A2x = px - qx, A3x = (u0.x + u2.x) - (u1.x + u3.x);
    const double A1y = py + qy, A2y = py - qy, A3y = (u0.y + u2.y) - (u1.y + u3.y);
    const double Lt = L * (A1x + A2y);
    const double P0 = fma(M, A1x, Lt), Q1 = fma(M, A2y, Lt);
    const double P1 = N * (A1y + A2x); // = Q0
    const double H0 = kH * A3x, H1 = kH * A3y;
    const double Sx = P0 + P1, Dx = P0 - P1, Sy = P1 + Q1, Dy = P1 - Q1;
    f[0] = make_double2(H0 - Sx, H1 - Sy);
    f[1] = make_double2(Dx - H0, Dy - H1);
    f[2] = make_double2(Sx + H0, Sy + H1);
    f[3] = make_double2(-(Dx + H0), -(Dy + H1));
}

} // namespace gfgpu
