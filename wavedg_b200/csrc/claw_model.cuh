// Flux models and face geometry of the conservation-law path, shared by the fused collocation
// kernel (claw_line.cu) and the exact-quadrature Euler kernels (claw.cu).
//
//   ClawEuler    the compressible Euler system of examples/cl2d.cpp:67-126 (gamma 1.4) with its
//                local Lax-Friedrichs flux; exterior boundary state = interior state.
//   ClawLinear   f = A_0 u, g = A_1 u (Advection<true>), upwind flux
//                fh = 1/2 (n.A)(a + b) + 1/2 |n.A| (a - b), |n.A| per element side from a table
//                formed at set-up; exterior boundary state 0 (AdvectionHomogeneousBC<true>).
//
// flux: r = a f(q) + b g(q), a contravariant component with the vector (a, b).
// face: r += 2 w fh(n, qL, qR), exactly antisymmetric (n, qL, qR) -> (-n, qR, qL): the products of
// the two states are rounded before they are added.
#pragma once

#include <cuda_runtime.h>

#include "launch.hpp"

namespace wdg
{
    struct ClawEuler
    {
        static constexpr bool LINEAR = false;
        static constexpr double gamma = 1.4;
        // velocities and pressure over density with one reciprocal
        __device__ __forceinline__ static void primitive(const double *q, double &ir, double &u, double &v, double &p)
        {
            ir = 1.0 / q[0];
            u = q[1] * ir;
            v = q[2] * ir;
            p = (gamma - 1.0) * (q[3] - 0.5 * q[0] * (u * u + v * v));
        }
        // the state carried along (a, b) and the pressure acting along it
        __device__ __forceinline__ static void carry(double a, double b, double u, double v, double p, const double *q,
                                                     double *f)
        {
            const double s = a * u + b * v;
            f[0] = q[0] * s;
            f[1] = q[1] * s + a * p;
            f[2] = q[2] * s + b * p;
            f[3] = (q[3] + p) * s;
        }
        template <int NV>
        __device__ __forceinline__ static void flux(const double *, double a, double b, const double *q, double *f)
        {
            double ir, u, v, p;
            primitive(q, ir, u, v, p);
            carry(a, b, u, v, p, q, f);
        }
        template <int NV>
        __device__ __forceinline__ static void exterior(const double *q, double *x)
        {
#pragma unroll
            for (int d = 0; d < NV; ++d)
                x[d] = q[d];
        }
        template <int NV>
        __device__ __forceinline__ static void face(const double *, const double *, double nx, double ny, double w,
                                                    const double *qL, const double *qR, double *r)
        {
            double iL, uL, vL, pL, iR, uR, vR, pR;
            primitive(qL, iL, uL, vL, pL);
            primitive(qR, iR, uR, vR, pR);
            const double c = fmax(sqrt(uL * uL + vL * vL) + sqrt(gamma * pL * iL),
                                  sqrt(uR * uR + vR * vR) + sqrt(gamma * pR * iR));
            const double nL = nx * uL + ny * vL, nR = nx * uR + ny * vR, ps = pL + pR;
            const double s0 = __dadd_rn(__dmul_rn(qL[0], nL), __dmul_rn(qR[0], nR));
            const double s1 = __dadd_rn(__dmul_rn(qL[1], nL), __dmul_rn(qR[1], nR)) + nx * ps;
            const double s2 = __dadd_rn(__dmul_rn(qL[2], nL), __dmul_rn(qR[2], nR)) + ny * ps;
            const double s3 = __dadd_rn(__dmul_rn(qL[3] + pL, nL), __dmul_rn(qR[3] + pR, nR));
            r[0] += w * (s0 + c * (qL[0] - qR[0]));
            r[1] += w * (s1 + c * (qL[1] - qR[1]));
            r[2] += w * (s2 + c * (qL[2] - qR[2]));
            r[3] += w * (s3 + c * (qL[3] - qR[3]));
        }
    };

    struct ClawLinear
    {
        static constexpr bool LINEAR = true;
        // A_0, A_1 as A(d, c, k) = A[d + nv (c + nv k)]
        template <int NV>
        __device__ __forceinline__ static void flux(const double *A, double a, double b, const double *q, double *f)
        {
#pragma unroll
            for (int d = 0; d < NV; ++d)
            {
                double s0 = 0.0, s1 = 0.0;
#pragma unroll
                for (int c = 0; c < NV; ++c)
                {
                    s0 += A[d + NV * c] * q[c];
                    s1 += A[d + NV * c + NV * NV] * q[c];
                }
                f[d] = a * s0 + b * s1;
            }
        }
        template <int NV>
        __device__ __forceinline__ static void exterior(const double *, double *x)
        {
#pragma unroll
            for (int d = 0; d < NV; ++d)
                x[d] = 0.0;
        }
        // absA: |n.A| of the side
        template <int NV>
        __device__ __forceinline__ static void face(const double *A, const double *absA, double nx, double ny, double w,
                                                    const double *qL, const double *qR, double *r)
        {
#pragma unroll
            for (int d = 0; d < NV; ++d)
            {
                double c = 0.0, u = 0.0;
#pragma unroll
                for (int k = 0; k < NV; ++k)
                {
                    const double nA = nx * A[d + NV * k] + ny * A[d + NV * k + NV * NV];
                    c += nA * (qL[k] + qR[k]);
                    u += absA[d + NV * k] * (qL[k] - qR[k]);
                }
                r[d] += w * (c + u);
            }
        }
    };

    // outward unit normal and measure (length / 2) of side s of an element with corners c
    // (StraightEdge, wavedg/Edge.hpp:107-122); side s runs from corner p0 to p1: 0: 0 -> 1,
    // 1: 1 -> 2, 2: 3 -> 2, 3: 0 -> 3 (sides 2 and 3 against the counter-clockwise order)
    __device__ __forceinline__ void claw_side(const double *c, int s, double &nx, double &ny, double &meas)
    {
        const int p0 = (s == 0 || s == 3) ? 0 : (s == 1 ? 1 : 3), p1 = (s == 0) ? 1 : (s == 3 ? 3 : 2);
        const double dx = c[2 * p1] - c[2 * p0], dy = c[2 * p1 + 1] - c[2 * p0 + 1];
        const double len = sqrt(dx * dx + dy * dy), sgn = (s >= 2) ? -1.0 : 1.0;
        nx = sgn * dy / len;
        ny = -sgn * dx / len;
        meas = 0.5 * len;
    }
} // namespace wdg
