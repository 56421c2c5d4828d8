// Exterior states of the wave system's boundary codes, shared by the collocation and the
// exact-quadrature kernels.  Code 0 is the absorbing state wavedg/WaveEquation.hpp:77-84
// intends (the reference evaluates p_e before u_e), 1 reflecting (:64-69), 2 Dirichlet p = 0.
#pragma once

namespace wdg
{
    // a b + c, a b + c d and a b - c d: in FP64 fused as written (the second product rounded), so that
    // every kernel rounds alike; in FP32 left to the compiler's contraction
    __device__ __forceinline__ double mad(double a, double b, double c) { return fma(a, b, c); }
    __device__ __forceinline__ float mad(float a, float b, float c) { return a * b + c; }
    __device__ __forceinline__ double mul2_add(double a, double b, double c, double d) { return fma(a, b, c * d); }
    __device__ __forceinline__ float mul2_add(float a, float b, float c, float d) { return a * b + c * d; }
    __device__ __forceinline__ double mul2_sub(double a, double b, double c, double d) { return fma(a, b, -(c * d)); }
    __device__ __forceinline__ float mul2_sub(float a, float b, float c, float d) { return a * b - c * d; }

    // exterior state of a boundary node: 0 absorbing, 1 reflecting, 2 Dirichlet p = 0
    template <typename Real>
    __device__ __forceinline__ void exterior(int code, Real nx, Real ny, const Real q[3], Real x[3])
    {
        if (code == 1)
        {
            x[0] = q[0];
            const Real s = Real(2) * nx * ny;
            x[1] = mul2_sub(mul2_sub(ny, ny, nx, nx), q[1], s, q[2]);
            x[2] = mul2_add(-s, q[1], mul2_sub(nx, nx, ny, ny), q[2]);
        }
        else if (code == 0)
        {
            const Real out = mad(ny, q[2], mad(nx, q[1], q[0]));
            const Real tan = mul2_sub(ny, q[1], nx, q[2]);
            x[1] = mul2_add(ny, tan, Real(0.5) * nx, out);
            x[2] = mul2_add(-nx, tan, Real(0.5) * ny, out);
            x[0] = mul2_add(nx, x[1], ny, x[2]);
        }
        else
        {
            x[0] = -q[0];
            x[1] = q[1];
            x[2] = q[2];
        }
    }

} // namespace wdg
