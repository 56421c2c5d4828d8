// The wave system's stage on grid lines, shared by the kernels that take a lane per line
// (stage_ws.cuh: streaming chunks; stage_res.cu: elements resident for many stages): the basis
// tables, the sides' geometry and upwind flux, and the volume sums of a column and of a row.
// The two kernels step bit-identically: everything that rounds is formed here, in FP64 with the fused
// multiply-adds written out, so that no compiler's choice of which product to fuse comes between.
// (FP32 stepping keeps the contraction its results have always had.)
// (Each translation unit that includes this has its own copy of the tables to fill.)
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <vector>

#include "common.hpp"
#include "launch.hpp"
#include "wave_bc.cuh"

namespace wdg
{
    // ------------------------------------------------------------------ tables
    struct BasisTab
    {
        double x[kMaxN], w[kMaxN], D[kMaxN * kMaxN];     // GLL nodes, weights, D[l + n j] = phi_j'(x_l)
        double gx[kMaxN], gw[kMaxN], B[kMaxN * kMaxN];   // n-point Gauss-Legendre and B[q + n j] = phi_j(gx_q)
        float xf[kMaxN], wf[kMaxN], Df[kMaxN * kMaxN];
    };
    static __constant__ BasisTab c_tab[kMaxN + 1];

    static int upload_basis_tab(int device)
    {
        static std::mutex mu;
        static uint64_t done = 0;
        std::lock_guard<std::mutex> lock(mu);
        if (device < 0 || device >= 64)
            return fail(WDG_ERR_ARG, "device ordinal out of range");
        if (done & (1ull << device))
            return WDG_OK;
        std::vector<BasisTab> tab(kMaxN + 1);
        for (int n = kMinN; n <= kMaxN; ++n)
        {
            BasisTab &T = tab[n];
            gauss_lobatto(n, T.x, T.w);
            deriv_matrix(n, T.x, T.D);
            gauss_legendre(n, T.gx, T.gw);
            interp_matrix(n, T.x, n, T.gx, T.B);
            for (int k = 0; k < n; ++k)
            {
                T.xf[k] = (float)T.x[k];
                T.wf[k] = (float)T.w[k];
            }
            for (int k = 0; k < n * n; ++k)
                T.Df[k] = (float)T.D[k];
        }
        WDG_CUDA(cudaMemcpyToSymbol(c_tab, tab.data(), sizeof(BasisTab) * (kMaxN + 1)));
        done |= (1ull << device);
        return WDG_OK;
    }

    template <typename Real>
    struct Tab;
    template <>
    struct Tab<double>
    {
        static __device__ __forceinline__ double x(int n, int i) { return c_tab[n].x[i]; }
        static __device__ __forceinline__ double w(int n, int i) { return c_tab[n].w[i]; }
        static __device__ __forceinline__ double D(int n, int k) { return c_tab[n].D[k]; }
    };
    template <>
    struct Tab<float>
    {
        static __device__ __forceinline__ float x(int n, int i) { return c_tab[n].xf[i]; }
        static __device__ __forceinline__ float w(int n, int i) { return c_tab[n].wf[i]; }
        static __device__ __forceinline__ float D(int n, int k) { return c_tab[n].Df[k]; }
    };

    // The column sums' strides (row j of an element, element): columns are written at 3 i, rows read at
    // j * row, both with as few wavefronts as the 16 double-wide banks of a half-warp allow
    struct SumStride
    {
        int row, el;
    };
    __host__ __device__ constexpr int sum_waves(int n, int a, int e)
    {
        int waves = 0;
        for (int h = 0; h < 2; ++h)
        {
            int cnt[16] = {}, most = 0;
            for (int i = 16 * h; i < 16 * h + 16 && i < 32 / n * n; ++i)
                if (++cnt[(i / n * e + i % n * a) & 15] > most)
                    most = cnt[(i / n * e + i % n * a) & 15];
            waves += most;
        }
        return waves;
    }
    __host__ __device__ constexpr SumStride sum_strides(int n)
    {
        SumStride b{3 * n, 3 * n * n};
        int cost = 1 << 30;
        for (int row = 3 * n; row < 3 * n + 8; ++row)
            for (int el = row * n; el < row * n + 6; ++el)
            {
                const int c = 32 * (sum_waves(n, 3, el) + sum_waves(n, row, el)) + (el - 3 * n * n) / 2;
                if (c < cost)
                {
                    cost = c;
                    b.row = row;
                    b.el = el;
                }
            }
        return b;
    }
    // the same where the host has n at run time: a table made by the compiler, for the search takes a host
    // core 10 us
    inline SumStride sum_strides_at(int n)
    {
        struct Table
        {
            SumStride s[kMaxN + 1];
        };
        static constexpr Table t = []
        {
            Table m{};
            for (int k = kMinN; k <= kMaxN; ++k)
                m.s[k] = sum_strides(k);
            return m;
        }();
        return t.s[n];
    }

    template <int N>
    __device__ __forceinline__ int partner_stride(uint32_t byte)
    {
        const uint32_t c = byte & 3u;
        return (c == 0) ? 3 : (c == 1) ? -3 : (c == 2) ? 3 * N : -3 * N;
    }

    // a metric term of the bilinear map, linear in x: ((1 - x) a + (1 + x) b) / 4
    template <typename Real>
    __device__ __forceinline__ Real metric(Real x, Real a, Real b)
    {
        return Real(0.25) * mul2_add(Real(1) - x, a, Real(1) + x, b);
    }
    // the low-storage update (wavedg/ode.hpp:66-93) of one value: the register d, the state q
    template <typename Real>
    __device__ __forceinline__ Real rk_register(bool has_du, Real a, Real d, Real dt, Real r)
    {
        return has_du ? mul2_add(a, d, dt, r) : dt * r;
    }
    template <typename Real>
    __device__ __forceinline__ Real rk_state(Real q, Real b, Real d) { return mad(b, d, q); }

    // upwind numerical flux through a face with outward normal n, weight
    // h = w_k * meas / 2:  r -= h [C (q + x) + |C| (q - x)],  |C| = C^2
    template <typename Real>
    __device__ __forceinline__ void upwind(Real nx, Real ny, Real h, const Real q[3], const Real x[3], Real r[3])
    {
        const Real sp = q[0] + x[0], su = q[1] + x[1], sv = q[2] + x[2];
        const Real jp = q[0] - x[0], ju = q[1] - x[1], jv = q[2] - x[2];
        const Real nj = mul2_add(nx, ju, ny, jv);
        r[0] = mad(-h, mul2_add(nx, su, ny, sv) + jp, r[0]);
        r[1] = mad(-h, mul2_add(nx, sp, nx, nj), r[1]);
        r[2] = mad(-h, mul2_add(ny, sp, ny, nj), r[2]);
    }

    // Outward unit normal and half measure (length / 4) of side SIDE of an element with corners
    // (c01, c23, c45, c67) (StraightEdge, wavedg/Edge.hpp:107-122)
    template <typename Real, int SIDE>
    __device__ __forceinline__ void line_side(const double2 c01, const double2 c23, const double2 c45, const double2 c67,
                                              Real &nx, Real &ny, Real &hm)
    {
        // side SIDE runs from corner p0 to p1: 0: 0->1, 1: 1->2, 2: 3->2, 3: 0->3
        const double2 a0 = (SIDE == 0 || SIDE == 3) ? c01 : (SIDE == 1) ? c23 : c67;
        const double2 a1 = (SIDE == 0) ? c23 : (SIDE == 3) ? c67 : c45;
        if constexpr (sizeof(Real) == 4)
        {
            // FP32 stepping: the side's length and normal in FP32 from FP64 corner differences
            const float dx = (float)(a1.x - a0.x), dy = (float)(a1.y - a0.y);
            const float s2 = mul2_add(dx, dx, dy, dy), rs = rsqrtf(s2);
            const float sgn = (SIDE >= 2) ? -1.f : 1.f;
            nx = sgn * dy * rs;
            ny = -sgn * dx * rs;
            hm = 0.25f * s2 * rs;
        }
        else
        {
            const double dx = a1.x - a0.x, dy = a1.y - a0.y;
            const double s2 = mul2_add(dx, dx, dy, dy), rs = rsqrt(s2);
            const double sgn = (SIDE >= 2) ? -1.0 : 1.0;
            nx = (Real)(sgn * dy * rs);
            ny = (Real)(-sgn * dx * rs);
            hm = (Real)(0.25 * s2 * rs);
        }
    }
    // Upwind flux of one face node (own trace `own`, weight w_k times the side's half measure),
    // subtracted into r: the closed form of EdgeFlux (source/EdgeFlux.cpp:7-139), with the neighbour's
    // trace x or, on a boundary side (bit 7 of its byte), the exterior state of WaveBC
    template <typename Real>
    __device__ __forceinline__ void line_face(uint32_t byte, Real nx, Real ny, Real h, const Real *own, const Real *nbr,
                                              Real &r0, Real &r1, Real &r2)
    {
        const Real q[3] = {own[0], own[1], own[2]};
        Real x[3];
        if (byte & 0x80u)
            exterior<Real>((int)((byte >> 3) & 3u), nx, ny, q, x);
        else
        {
            x[0] = nbr[0];
            x[1] = nbr[1];
            x[2] = nbr[2];
        }
        Real r[3] = {r0, r1, r2};
        upwind<Real>(nx, ny, h, q, x, r);
        r0 = r[0];
        r1 = r[1];
        r2 = r[2];
    }

    // Column i of an element (values ue, node-major, 3 per node), weight wi: contravariant eta-fluxes of
    // the wave system (source/Div.cpp:5-53): G = W (-y_xi u + x_xi v, -y_xi p, x_xi p); along a column
    // x_eta, y_eta are constant and x_xi, y_xi vary linearly with eta.  Adds sum_l D(l, j) G(i, l)
    // (div_2d_c, source/Div.cpp:131-179) to the sums.
    template <int N, typename Real>
    __device__ __forceinline__ void line_column(const double2 c01, const double2 c23, const double2 c45, const double2 c67,
                                                const Real *ue, int i, Real wi, Real (&sp)[N], Real (&su)[N], Real (&sv)[N])
    {
        const Real dx0 = Real(c23.x - c01.x), dx1 = Real(c45.x - c67.x);
        const Real dy0 = Real(c23.y - c01.y), dy1 = Real(c45.y - c67.y);
#pragma unroll
        for (int l = 0; l < N; ++l)
        {
            const Real el = Tab<Real>::x(N, l);
            const Real Xxi = metric(el, dx0, dx1), Yxi = metric(el, dy0, dy1);
            const Real W = wi * Tab<Real>::w(N, l);
            const Real *nd = ue + 3 * (i + N * l);
            const Real p = nd[0], u = nd[1], v = nd[2];
            const Real WYx = W * Yxi, WXx = W * Xxi;
            const Real Gp = mul2_sub(WXx, v, WYx, u), Gu = -WYx * p, Gv = WXx * p;
#pragma unroll
            for (int j = 0; j < N; ++j)
            {
                const Real d = Tab<Real>::D(N, l + N * j);
                sp[j] = mad(d, Gp, sp[j]);
                su[j] = mad(d, Gu, su[j]);
                sv[j] = mad(d, Gv, sv[j]);
            }
        }
    }

    // Row j at eta = x_j, weight wj, of values q0, q1, q2: F = W (y_eta u - x_eta v, y_eta p, -x_eta p); along
    // a row x_xi, y_xi are constant and x_eta, y_eta vary linearly with xi.  VOL: adds sum_l D(l, i) F(l, j)
    // to the sums; MASS: forms the inverse mass 1 / (w_i w_j det J) (MassMatrix<true>,
    // source/MassMatrix.cpp:6-28) of the row's nodes.
    template <int N, typename Real, bool MASS>
    __device__ __forceinline__ void line_row(const double2 c01, const double2 c23, const double2 c45, const double2 c67,
                                             Real eta, Real wj, bool vol, const Real (&q0)[N], const Real (&q1)[N],
                                             const Real (&q2)[N], Real (&ap)[N], Real (&au)[N], Real (&av)[N], Real (&mv)[N])
    {
        const Real Xxi = metric(eta, Real(c23.x - c01.x), Real(c45.x - c67.x));
        const Real Yxi = metric(eta, Real(c23.y - c01.y), Real(c45.y - c67.y));
        const Real ex0 = Real(c67.x - c01.x), ex1 = Real(c45.x - c23.x);
        const Real ey0 = Real(c67.y - c01.y), ey1 = Real(c45.y - c23.y);
#pragma unroll
        for (int l = 0; l < N; ++l)
        {
            const Real xl = Tab<Real>::x(N, l);
            const Real Xeta = metric(xl, ex0, ex1), Yeta = metric(xl, ey0, ey1);
            const Real W = Tab<Real>::w(N, l) * wj;
            if constexpr (MASS)
            {
                if constexpr (sizeof(Real) == 4)
                    mv[l] = __frcp_rn(W * mul2_sub(Xxi, Yeta, Yxi, Xeta));
                else
                    mv[l] = Real(1) / (W * mul2_sub(Xxi, Yeta, Yxi, Xeta));
            }
            if (vol)
            {
                const Real WYe = W * Yeta, WXe = W * Xeta;
                const Real Fp = mul2_sub(WYe, q1[l], WXe, q2[l]), Fu = WYe * q0[l], Fv = -WXe * q0[l];
#pragma unroll
                for (int i = 0; i < N; ++i)
                {
                    const Real d = Tab<Real>::D(N, l + N * i);
                    ap[i] = mad(d, Fp, ap[i]);
                    au[i] = mad(d, Fu, au[i]);
                    av[i] = mad(d, Fv, av[i]);
                }
            }
        }
    }
} // namespace wdg
