// Right-hand sides and time-stepping stages with exact quadrature, one fused launch, lanes on
// grid lines (included by exactq.cu, claw.cu and vadvect.cu, each with its own model):
//
//   wave system        Div<false>, EdgeFlux<false>, MassMatrix<false>
//   Euler system       DivF2D<false>, EdgeFluxF2D<false>, MassMatrix<false>
//   scalar advection   Div<false>, EdgeFlux<false> with a varying coefficient, MassMatrix<false>
//
// The mass matrix.  det J of a bilinear quad has degree one in each direction, so the n-point
// Gauss-Legendre rule integrates phi_i phi_j det J exactly and the matrix that the (n + 1)-point
// rule of MassMatrix<false> (source/MassMatrix.cpp:84-227) gives is
//     M = (B x B)^T diag(w_k w_l det J(g_k, g_l)) (B x B),
// B the n x n interpolation from the basis nodes to the Gauss points g.  So
//     M^{-1} r = (T x T) diag(1 / (w w det J)) r^,   T = B^{-1},   r^ = (T x T)^T r,
// and r^ needs no extra work: it is r with the Lagrange basis psi on the Gauss points as test
// functions, i.e. the projections below use psi and psi' in place of phi and phi'.  No dense
// n^2 x n^2 inverse is stored or read.
//
// A warp owns EW = 32 / Q elements (Q volume points per direction).
//   1  lane = (element, node row [, half of the variables]): the row to the Q points along xi
//   2  lane = (element, column of points): the column to the Q points along eta, at each point the
//      contravariant fluxes F, G, contracted at once along eta with psi (F) and psi' (G): no flux
//      is stored at a point
//   3  lane = (element, row of Gauss points): the xi contraction with psi' and psi, the sides'
//      projected fluxes, 1 / (w w det J), T along xi
//   4  lane = (element, node column): T along eta and the RHS or stage update
// and between 1 and 2 the sides: both traces at the face points (lane per point), the numerical
// flux, and its projection on psi along the side (lane per side and variable).  The contraction
// matrices have the same indices in every lane of a warp, so they are constant-bank operands.
//
// What bounds it: the latency of the phases' chains at 12 resident warps per SM, then the shared-
// memory pipe (49 to 54 % busy) and FP64 issue; the state and the tables of the measured sizes stay in
// L2.  128 x 128, N = 5, per launch: wave system 91 -> 27 us, Euler 382 -> 62 us, scalar advection on
// Gauss-Legendre points 127 -> 18 us against a warp per element with generic loops and a dense
// inverse mass matrix (3400, 7950 and 3300 warp instructions per element; now 490, 1620, 490).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "common.hpp"
#include "launch.hpp"

namespace wdg
{
    void lagrange_deriv_at(int n, const double *x, int nq, const double *xq, double *D);

    constexpr int kXWarps = 4;

    // One degree's matrices: rows are points, columns basis functions (phi: the basis the state is
    // expanded in, psi: the Lagrange basis on the n Gauss points)
    template <int N, int Q, int QF>
    struct XTab
    {
        double P[Q][N], Pt[Q][N], Dt[Q][N]; // phi, psi, psi' at the volume points
        double Pf[QF][N], Pft[QF][N];       // phi, psi at the face points (psi times the weights where
                                            // the model's flux does not hold them)
        double R[N][N];                     // Pft^T Pf: a side's trace to its projection
        double T[N][N];                     // psi at the basis nodes
        double xq[Q], wq[Q];
        double xg[N], wg[N], sm[N], sp[N];  // Gauss points and weights, psi(-1), psi(+1)
        double e[N];                        // phi(-1) (Gauss-Legendre bases' traces)
    };

    template <class M>
    struct XTabs
    {
        template <int N>
        using One = XTab<N, M::q(N), M::qf(N)>;
        One<2> t2;
        One<3> t3;
        One<4> t4;
        One<5> t5;
        One<6> t6;
        One<7> t7;
        One<8> t8;
        One<9> t9;
    };
    template <int N, class Tabs>
    __host__ __device__ __forceinline__ auto &xtab(Tabs &t)
    {
        if constexpr (N == 2) return t.t2;
        else if constexpr (N == 3) return t.t3;
        else if constexpr (N == 4) return t.t4;
        else if constexpr (N == 5) return t.t5;
        else if constexpr (N == 6) return t.t6;
        else if constexpr (N == 7) return t.t7;
        else if constexpr (N == 8) return t.t8;
        else return t.t9;
    }

    template <int N, int Q, int QF>
    inline void xtab_fill(XTab<N, Q, QF> &t, bool legendre, bool weighted)
    {
        double x[N], w[N], xf[QF], wf[QF];
        if (legendre)
            gauss_legendre(N, x, w);
        else
            gauss_lobatto(N, x, w);
        gauss_legendre(N, t.xg, t.wg);
        gauss_legendre(Q, t.xq, t.wq);
        gauss_legendre(QF, xf, wf);
        std::vector<double> B((size_t)(Q > QF ? Q : QF) * N);
        auto put = [&](int rows, double *dst) // column-major (rows x N) -> row-major
        {
            for (int r = 0; r < rows; ++r)
                for (int c = 0; c < N; ++c)
                    dst[r * N + c] = B[r + (size_t)rows * c];
        };
        interp_matrix(N, x, Q, t.xq, B.data());
        put(Q, &t.P[0][0]);
        interp_matrix(N, t.xg, Q, t.xq, B.data());
        put(Q, &t.Pt[0][0]);
        lagrange_deriv_at(N, t.xg, Q, t.xq, B.data());
        put(Q, &t.Dt[0][0]);
        interp_matrix(N, x, QF, xf, B.data());
        put(QF, &t.Pf[0][0]);
        interp_matrix(N, t.xg, QF, xf, B.data());
        put(QF, &t.Pft[0][0]);
        for (int q = 0; q < QF && weighted; ++q)
            for (int m = 0; m < N; ++m)
                t.Pft[q][m] *= wf[q];
        for (int m = 0; m < N; ++m)
            for (int k = 0; k < N; ++k)
            {
                t.R[m][k] = 0.0;
                for (int q = 0; q < QF; ++q)
                    t.R[m][k] += t.Pft[q][m] * t.Pf[q][k];
            }
        interp_matrix(N, t.xg, N, x, B.data());
        put(N, &t.T[0][0]);
        const double ends[2] = {-1.0, 1.0};
        interp_matrix(N, t.xg, 1, ends, t.sm);
        interp_matrix(N, t.xg, 1, ends + 1, t.sp);
        interp_matrix(N, x, 1, ends, t.e);
    }
    template <class M>
    inline void xtabs_fill(XTabs<M> &t, bool legendre)
    {
        xtab_fill(t.t2, legendre, M::WEIGHTED);
        xtab_fill(t.t3, legendre, M::WEIGHTED);
        xtab_fill(t.t4, legendre, M::WEIGHTED);
        xtab_fill(t.t5, legendre, M::WEIGHTED);
        xtab_fill(t.t6, legendre, M::WEIGHTED);
        xtab_fill(t.t7, legendre, M::WEIGHTED);
        xtab_fill(t.t8, legendre, M::WEIGHTED);
        xtab_fill(t.t9, legendre, M::WEIGHTED);
    }

    // Every det J at the n x n Gauss points positive: exactly when M is positive definite (M is
    // congruent to the diagonal above), which the Cholesky factorisation of the reference's
    // MassMatrix<false> needs
    inline int exact_mass_check(const wdg_mesh &mesh, int n)
    {
        std::vector<double> g(n), w(n);
        gauss_legendre(n, g.data(), w.data());
        for (int el = 0; el < mesh.nel; ++el)
            for (int l = 0; l < n; ++l)
                for (int k = 0; k < n; ++k)
                {
                    double J[4];
                    quad_jacobian(&mesh.corners[8 * (size_t)el], g[k], g[l], J);
                    if (!(J[0] * J[3] - J[2] * J[1] > 0.0))
                        return fail(WDG_ERR_ARG, "an element mass matrix is not positive definite");
                }
        return WDG_OK;
    }

    // r <- M^{-1} r of one element by one warp, n and the variable count at run time (the table-driven
    // advection kernel): T (row-major n x n) holds psi_m(x_k), c the corners, tmp holds nv n^2 values
    __device__ inline void x_mass_inv(int n, int nv, const double *T, const double *xg, const double *wg, const double *c,
                                      double *r, double *tmp, int lane)
    {
        const int m = nv * n * n;
        if (n <= 3)
        {
            // both directions at once: at most nine terms, and two passes fewer
            for (int o = lane; o < m; o += 32)
            {
                const int d = o % nv, i = (o / nv) % n, j = o / (nv * n);
                double s = 0.0, J[4];
                for (int l = 0; l < n; ++l)
                    for (int k = 0; k < n; ++k)
                        s += __ldg(T + i + n * k) * __ldg(T + j + n * l) * r[d + nv * (k + n * l)];
                quad_jacobian(c, __ldg(xg + i), __ldg(xg + j), J);
                tmp[o] = s / (__ldg(wg + i) * __ldg(wg + j) * (J[0] * J[3] - J[2] * J[1]));
            }
            __syncwarp();
            for (int o = lane; o < m; o += 32)
            {
                const int d = o % nv, i = (o / nv) % n, j = o / (nv * n);
                double s = 0.0;
                for (int l = 0; l < n; ++l)
                    for (int k = 0; k < n; ++k)
                        s += __ldg(T + n * i + k) * __ldg(T + n * j + l) * tmp[d + nv * (k + n * l)];
                r[o] = s;
            }
            __syncwarp();
            return;
        }
        // (T x T)^T r at the Gauss points
        for (int o = lane; o < m; o += 32)
        {
            const int d = o % nv, i = (o / nv) % n, l = o / (nv * n);
            double s = 0.0;
            for (int k = 0; k < n; ++k)
                s += __ldg(T + i + n * k) * r[d + nv * (k + n * l)];
            tmp[o] = s;
        }
        __syncwarp();
        for (int o = lane; o < m; o += 32)
        {
            const int d = o % nv, i = (o / nv) % n, j = o / (nv * n);
            double s = 0.0, J[4];
            for (int k = 0; k < n; ++k)
                s += __ldg(T + j + n * k) * tmp[d + nv * (i + n * k)];
            quad_jacobian(c, __ldg(xg + i), __ldg(xg + j), J);
            r[o] = s / (__ldg(wg + i) * __ldg(wg + j) * (J[0] * J[3] - J[2] * J[1]));
        }
        __syncwarp();
        for (int o = lane; o < m; o += 32)
        {
            const int d = o % nv, i = (o / nv) % n, l = o / (nv * n);
            double s = 0.0;
            for (int k = 0; k < n; ++k)
                s += __ldg(T + n * i + k) * r[d + nv * (k + n * l)];
            tmp[o] = s;
        }
        __syncwarp();
        for (int o = lane; o < m; o += 32)
        {
            const int d = o % nv, i = (o / nv) % n, j = o / (nv * n);
            double s = 0.0;
            for (int k = 0; k < n; ++k)
                s += __ldg(T + n * j + k) * tmp[d + nv * (i + n * k)];
            r[o] = s;
        }
        __syncwarp();
    }

    // A device copy of what x_mass reads for a basis with nodes x
    struct MassTables
    {
        double *T = nullptr, *xg = nullptr, *wg = nullptr;
    };
    int mass_tables(int n, const double *x, MassTables &t);
    void mass_tables_free(MassTables &t);

    // The operators M and M^{-1} on arrays of nv interleaved variables, for a basis with nodes x: the
    // matrices go with each launch
    struct MassOp
    {
        int n = 0;
        double T[kMaxN * kMaxN], B[kMaxN * kMaxN], xg[kMaxN], wg[kMaxN]; // psi_m(x_k), phi_k(g_m) (row-major), the Gauss rule
    };
    MassOp mass_op(int n, const double *x);
    // y <- M x or M^{-1} x (x and y may be the same array)
    int mass_launch(const MassOp &t, int nel, int nv, bool inverse, const double *corners, const double *x, double *y,
                    cudaStream_t s);

    struct XArgs
    {
        ClawArgs c;           // state, output, stage coefficients, geometry, partner table, error word
        const double *F;      // wave system: forcing load vector (nullable) times fs
        double fs;
        double *acc;          // wave system: FP64 filter of the last RK4 stage (nullable) += acc_c u'
        double acc_c;
        const double *op, *G; // advection: volume and face tables
        const int *nb;        // Gauss-Legendre bases: the sides' neighbours
    };

    // Shared-memory strides.  A warp's 64-bit accesses go out in halves of 16 lanes, conflict-free when
    // the 16 addresses differ modulo 16.  Lanes are (element, column i) at i * sp and (element, row l,
    // part) at l * nv + part, elements e (mod 16) apart; of all strides the pair with the fewest
    // wavefronts is taken (odd variable counts: none above two per access), then su, the stride of the
    // nodal rows, likewise.
    struct XStride
    {
        int sp, su, e;
    };
    constexpr int x_waves(int lanes, int q, int parts, int n, int a, int b, int e)
    {
        int waves = 0;
        for (int h = 0; h < 2; ++h)
        {
            int cnt[16] = {}, most = 0;
            for (int i = 16 * h; i < 16 * h + 16 && i < lanes; ++i)
            {
                const int el = i / q, ln = i % q;
                if (ln >= n * parts)
                    continue;
                const int at = (el * e + (ln % n) * a + (ln / n) * b) & 15;
                if (++cnt[at] > most)
                    most = cnt[at];
            }
            waves += most;
        }
        return waves;
    }
    constexpr XStride x_strides(int n, int nv, int q, int parts)
    {
        XStride best{n * nv, n * nv, 0};
        int cost = 1 << 30;
        const int lanes = (32 / q) * q;
        for (int sp = n * nv; sp < n * nv + 16; ++sp)
            for (int e = 0; e < 16; ++e)
            {
                const int c = 64 * (3 * x_waves(lanes, q, 1, q, sp, 0, e) + 4 * x_waves(lanes, q, parts, n, nv, 1, e)) +
                              sp - n * nv;
                if (c < cost)
                {
                    cost = c;
                    best.sp = sp;
                    best.e = e;
                }
            }
        cost = 1 << 30;
        for (int su = n * nv; su < n * nv + 16; ++su)
        {
            const int c = 64 * x_waves(lanes, q, parts, n, su, 1, best.e) + su;
            if (c < cost)
            {
                cost = c;
                best.su = su;
            }
        }
        return best;
    }

    template <int N, class M>
    struct XShape
    {
        static constexpr int NV = M::NV, Q = M::q(N), QF = M::qf(N), NN = N * N, ND = NV * NN;
        static constexpr int EW = 32 / Q;          // elements per warp
        static constexpr bool COLLOC = Q == N;     // the volume points are the Gauss points: psi = identity
        // row lanes per row: two, with every other variable each, where the lanes are there
        static constexpr int PARTS = (Q >= 2 * N && NV % 2 == 0) ? 2 : 1;
        static constexpr int VP = NV / PARTS;
        static constexpr XStride ST = x_strides(N, NV, Q, PARTS);
        static constexpr int SP = ST.sp, SU = ST.su; // doubles per column of points, per nodal row
        static constexpr int H1 = Q * SP;
        // both traces at the face points, the flux over the first
        static constexpr int TQ = 4 * QF * NV;
        static constexpr int H2 = (H1 > 2 * TQ || M::LINEAR) ? H1 : 2 * TQ;
        static constexpr int TN = 4 * N * NV; // a trace array
        // per element: nodal values | two half-contracted arrays (the first also the interpolated
        // columns, the second the face points) | neighbour traces, later the projected side fluxes | own
        // traces (Gauss-Legendre bases) | side normals and measures | corners
        static constexpr int oH = N * SU, oH2 = oH + H1, oT = oH2 + H2, oT0 = oT + TN, oS = oT0 + (M::LEG ? TN : 0),
                             oC = oS + 12;
        static constexpr int ES = oC + 8 + ((ST.e - (oC + 8)) & 15);
        static constexpr size_t smem = sizeof(double) * (size_t)(kXWarps * EW * ES);
        // columns of points kept in registers while the accumulators leave room for them
        static constexpr bool REG = COLLOC || 3 * N * NV <= 64;
        static_assert(smem <= 227 * 1024, "a CTA's elements fit shared memory");
        static constexpr int MINB = N <= 5 ? 3 : 2;
        // shared-memory place of value v (of ND) of an element's nodal data
        __device__ static __forceinline__ int node(int v) { return (v / (N * NV)) * SU + v % (N * NV); }
    };

    // outward unit normal and measure (length / 2) of side s (StraightEdge, wavedg/Edge.hpp:107-122)
    __device__ __forceinline__ void x_side(const double *c, int s, double &nx, double &ny, double &meas)
    {
        const int p0 = (s == 0 || s == 3) ? 0 : (s == 1 ? 1 : 3), p1 = (s == 0) ? 1 : (s == 3 ? 3 : 2);
        const double dx = c[2 * p1] - c[2 * p0], dy = c[2 * p1 + 1] - c[2 * p0 + 1];
        const double len = sqrt(dx * dx + dy * dy), sgn = (s >= 2) ? -1.0 : 1.0;
        nx = sgn * dy / len;
        ny = -sgn * dx / len;
        meas = 0.5 * len;
    }
    // face-node k of side s in the staged rows: base + k * stride (source/FaceProlongator.cpp:508-514)
    template <int N, class S>
    __device__ __forceinline__ int x_face_base(int s)
    {
        return s == 1 ? S::NV * (N - 1) : s == 2 ? S::SU * (N - 1) : 0;
    }
    template <class S>
    __device__ __forceinline__ int x_face_stride(int s) { return (s & 1) ? S::SU : S::NV; }
    // LegendreFaceProlongator's node map (source/FaceProlongator.cpp:716-737): the node at distance m
    // from side s at position i along it, rows `su` apart
    template <int N>
    __device__ __forceinline__ int x_line(int s, int i, int m, int su)
    {
        const int x = (s == 0 || s == 2) ? i : (s == 1 ? N - 1 - m : m);
        const int y = (s == 1 || s == 3) ? i : (s == 2 ? N - 1 - m : m);
        return x + su * y;
    }
    // asynchronous 8-byte copies to shared memory, in groups
    __device__ __forceinline__ void x_copy8(double *dst, const double *src)
    {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                     : "memory");
    }
    __device__ __forceinline__ void x_copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
    template <int LEFT>
    __device__ __forceinline__ void x_copy_wait()
    {
        asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
    }

    // what a stage reads beside its input: the RK4 register or SSPRK3's first state (null: nothing)
    __device__ __forceinline__ const double *x_prev(const ClawArgs &a)
    {
        return (a.mode == CLAW_RK4) ? (a.rk_a == 0.0 ? nullptr : a.du) : (a.mode == CLAW_SSP1 || a.mode == CLAW_SSP2) ? a.base
                                                                                                                 : nullptr;
    }
    // the RHS or one stage of ode::RungeKutta4 / ode::SSPRK3 (wavedg/ode.hpp:66-93, 145-186) of one
    // value: g its place, q the staged state, p x_prev's value, y the RHS; the new state where there is one
    __device__ __forceinline__ double x_stage(const ClawArgs &a, size_t g, double q, double p, double y)
    {
        double v;
        switch (a.mode)
        {
        case CLAW_RHS:
            v = y;
            break;
        case CLAW_RK4:
        {
            const double kd = (a.rk_a == 0.0) ? a.dt * y : a.rk_a * p + a.dt * y;
            a.du[g] = kd;
            v = q + a.rk_b * kd;
            break;
        }
        case CLAW_SSP0:
            v = q + a.dt * y;
            break;
        case CLAW_SSP1:
            v = 0.25 * (q + 3.0 * p + a.dt * y);
            break;
        default: // CLAW_SSP2
            v = (p + 2.0 * q + 2.0 * a.dt * y) / 3.0;
            break;
        }
        a.out[g] = v;
        return v;
    }

    template <int N, class M>
    __global__ void __launch_bounds__(32 * kXWarps, XShape<N, M>::MINB) xline_kernel(const XArgs A)
    {
        using S = XShape<N, M>;
        constexpr int NV = S::NV, Q = S::Q, QF = S::QF, NN = S::NN, ND = S::ND, EW = S::EW, SP = S::SP, SU = S::SU;
        constexpr int VP = S::VP, PT = S::PARTS;
        extern __shared__ double xsm[];
        const ClawArgs &a = A.c;
        const auto &tab = M::template table<N>();
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        double *base = xsm + (size_t)warp * EW * S::ES;
        const long long limit = (long long)a.nel * NN; // nodes a neighbour index may name
        const int le = lane / Q, ln = lane - le * Q;   // element of the warp, line
        double *E = base + le * S::ES;                 // this lane's element
        const int ngroups = (a.nel + EW - 1) / EW;
        for (int g = blockIdx.x * kXWarps + warp; g < ngroups; g += gridDim.x * kXWarps)
        {
            const int e0 = g * EW, ne = min(EW, a.nel - e0);
            const bool on = le < ne;
            // row lanes: row l, variables part, part + PT, ...
            const bool row = on && ln < N * PT;
            const int l = ln % N, part = ln / N;
            // ---- nodal values and corners by asynchronous copies; meanwhile the side codes and partner
            // offsets of this lane's face nodes, all in flight together, then (second copy group) the
            // traces T(s, k, d) of the sides' neighbours
            for (int o = lane; o < ne * ND; o += 32)
                x_copy8(base + (o / ND) * S::ES + S::node(o % ND), a.x + (size_t)e0 * ND + o);
            for (int o = lane; o < ne * 8; o += 32)
                x_copy8(base + (o >> 3) * S::ES + S::oC + (o & 7), a.corners + 8 * (size_t)e0 + o);
            x_copy_commit();
            constexpr int IT = (EW * 4 * N + 31) / 32; // face nodes per lane
            uint32_t byte[IT];
            int off[IT];
#pragma unroll
            for (int t = 0; t < IT; ++t)
            {
                const int o = lane + 32 * t, el = e0 + o / (4 * N), s = (o / N) & 3;
                byte[t] = 0x100u; // past the group
                off[t] = -1;
                if (o < ne * 4 * N)
                {
                    byte[t] = (__ldg(a.fcode + el) >> (8 * s)) & 0xffu;
                    off[t] = M::LEG ? __ldg(A.nb + 4 * (size_t)el + s)
                                    : __ldg(reinterpret_cast<const int *>(a.fbase + el) + s);
                }
            }
#pragma unroll
            for (int t = 0; t < IT; ++t)
            {
                const int o = lane + 32 * t, s = (o / N) & 3, k = o % N;
                if (byte[t] & 0x180u)
                    continue; // a boundary side, or past the group
                double *t1 = base + (o / (4 * N)) * S::ES + S::oT + NV * (s * N + k);
                if constexpr (M::LEG)
                {
                    // sum_k phi_k(-1) u(node at distance k from the side) (source/FaceProlongator.cpp:806-834);
                    // one variable
                    const int nel = off[t] >> 3, ns = (off[t] >> 1) & 3, kk = (off[t] & 1) ? N - 1 - k : k;
                    double w = 0.0;
                    if (off[t] < 0 || nel >= a.nel)
                        atomicOr(a.err, 2u);
                    else
#pragma unroll
                        for (int m = 0; m < N; ++m)
                            w += __ldg(a.x + (size_t)NN * nel + x_line<N>(ns, kk, m, N)) * tab.e[m];
                    t1[0] = w;
                }
                else
                {
                    const uint32_t sc = byte[t] & 3u;
                    const int stride = (sc == 0) ? 1 : (sc == 1) ? -1 : (sc == 2) ? N : -N; // in nodes
                    const long long pn = (long long)(off[t] / 3) + (long long)k * stride;
                    if (off[t] < 0 || pn < 0 || pn >= limit)
                    {
                        atomicOr(a.err, 2u);
                        byte[t] |= 0x200u; // the own trace below
                    }
                    else
#pragma unroll
                        for (int d = 0; d < NV; ++d)
                            x_copy8(t1 + d, a.x + (size_t)NV * pn + d);
                }
            }
            x_copy_commit();
            x_copy_wait<1>();
            __syncwarp();
            for (int o = lane; o < ne * 4; o += 32)
            {
                double *Eo = base + (o >> 2) * S::ES;
                double nx, ny, meas;
                x_side(Eo + S::oC, o & 3, nx, ny, meas);
                double *sn = Eo + S::oS + 3 * (o & 3);
                sn[0] = nx;
                sn[1] = ny;
                sn[2] = meas;
            }
            // ---- 1: rows to the points along xi; H[i][l][d], column-of-points major
            if (row)
            {
                double v[N][VP];
#pragma unroll
                for (int k = 0; k < N; ++k)
#pragma unroll
                    for (int d = 0; d < VP; ++d)
                        v[k][d] = E[SU * l + NV * k + part + PT * d];
#pragma unroll
                for (int i = 0; i < Q; ++i)
                {
                    double s[VP];
#pragma unroll
                    for (int d = 0; d < VP; ++d)
                        s[d] = 0.0;
#pragma unroll
                    for (int k = 0; k < N; ++k)
#pragma unroll
                        for (int d = 0; d < VP; ++d)
                            s[d] += tab.P[i][k] * v[k][d];
#pragma unroll
                    for (int d = 0; d < VP; ++d)
                        E[S::oH + i * SP + l * NV + part + PT * d] = s[d];
                }
            }
            if constexpr (M::FORCE)
            {
                static_assert(S::COLLOC && PT == 1, "the forcing's columns wait where phase 2 puts its own");
                if (A.F && row)
                {
                    // the forcing's load vector against psi along xi
                    const double *Fe = A.F + (size_t)(e0 + le) * ND + NV * N * l;
                    double f[N][NV];
#pragma unroll
                    for (int k = 0; k < N; ++k)
#pragma unroll
                        for (int d = 0; d < NV; ++d)
                            f[k][d] = __ldg(Fe + NV * k + d);
#pragma unroll
                    for (int i = 0; i < N; ++i)
#pragma unroll
                        for (int d = 0; d < NV; ++d)
                        {
                            double s = 0.0;
#pragma unroll
                            for (int k = 0; k < N; ++k)
                                s += tab.T[k][i] * f[k][d];
                            E[S::oH2 + i * SP + l * NV + d] = A.fs * s;
                        }
                }
            }
            x_copy_wait<0>();
            __syncwarp();
            // ---- sides.  Exterior states (and the own traces of Gauss-Legendre bases)
#pragma unroll
            for (int t = 0; t < IT; ++t)
            {
                const int o = lane + 32 * t, s = (o / N) & 3, k = o % N;
                double *Eo = base + (o / (4 * N)) * S::ES, *t1 = Eo + S::oT + NV * (s * N + k);
                if (byte[t] & 0x100u)
                    continue;
                if constexpr (M::LEG)
                {
                    double v = 0.0;
#pragma unroll
                    for (int m = 0; m < N; ++m)
                        v += Eo[x_line<N>(s, k, m, SU)] * tab.e[m];
                    Eo[S::oT0 + s * N + k] = v;
                    if (byte[t] & 0x80u)
                        t1[0] = 0.0;
                }
                else
                {
                    const double *own = Eo + x_face_base<N, S>(s) + k * x_face_stride<S>(s);
                    if (byte[t] & 0x80u)
                        M::exterior((int)((byte[t] >> 3) & 3u), Eo + S::oS + 3 * s, own, t1);
                    else if (byte[t] & 0x200u)
#pragma unroll
                        for (int d = 0; d < NV; ++d)
                            t1[d] = own[d];
                    if constexpr (M::LINEAR)
                        M::combine(Eo + S::oS + 3 * s, own, t1);
                }
            }
            __syncwarp();
            if constexpr (M::LINEAR)
            {
                // the flux is linear with coefficients constant along the side: it is the nodal
                // combinations' two scalars through R
#pragma unroll
                for (int o = lane; o < ((EW * 8 + 31) & ~31); o += 32)
                {
                    const bool act = o < ne * 8;
                    const int s = (o >> 1) & 3, which = o & 1;
                    double *Eo = base + (act ? o >> 3 : 0) * S::ES, *t1 = Eo + S::oT + NV * s * N;
                    double v[N], m[N];
#pragma unroll
                    for (int k = 0; k < N; ++k)
                    {
                        v[k] = t1[NV * k + which];
                        m[k] = 0.0;
                    }
                    __syncwarp(); // both of the side's lanes have read it
#pragma unroll
                    for (int k = 0; k < N; ++k)
#pragma unroll
                        for (int j = 0; j < N; ++j)
                            m[j] += tab.R[j][k] * v[k];
                    if (act)
#pragma unroll
                        for (int k = 0; k < N; ++k)
                            M::spread(Eo + S::oS + 3 * s, which, m[k], t1 + NV * k);
                }
            }
            else
            {
                // both traces to the face points, lane per (element, side, variable); in the face array
                // point p = s QF + q of variable d is at d 4 QF + p
                for (int o = lane; o < ne * 4 * NV; o += 32)
                {
                    const int s = (o / NV) & 3, d = o % NV;
                    double *Eo = base + (o / (4 * NV)) * S::ES, *qp = Eo + S::oH2 + d * 4 * QF + s * QF;
                    const double *own = M::LEG ? Eo + S::oT0 + s * N : Eo + x_face_base<N, S>(s) + d;
                    const int os = M::LEG ? 1 : x_face_stride<S>(s);
                    const double *nb = Eo + S::oT + NV * s * N + d;
                    double v[N], w[N];
#pragma unroll
                    for (int k = 0; k < N; ++k)
                    {
                        v[k] = own[k * os];
                        w[k] = nb[NV * k];
                    }
#pragma unroll
                    for (int q = 0; q < QF; ++q)
                    {
                        double x = 0.0, y = 0.0;
#pragma unroll
                        for (int k = 0; k < N; ++k)
                        {
                            x += tab.Pf[q][k] * v[k];
                            y += tab.Pf[q][k] * w[k];
                        }
                        qp[q] = x;
                        qp[S::TQ + q] = y;
                    }
                }
                __syncwarp();
                // the numerical flux: what the element adds
                for (int o = lane; o < ne * 4 * QF; o += 32)
                {
                    const int eo = o / (4 * QF), pt = o % (4 * QF), s = pt / QF;
                    double *Eo = base + eo * S::ES, *qp = Eo + S::oH2 + pt;
                    double qL[NV], qR[NV], uf[NV];
#pragma unroll
                    for (int d = 0; d < NV; ++d)
                    {
                        qL[d] = qp[d * 4 * QF];
                        qR[d] = qp[S::TQ + d * 4 * QF];
                    }
                    M::template face<N>(A, e0 + eo, s, pt - s * QF, Eo + S::oS + 3 * s, qL, qR, uf);
#pragma unroll
                    for (int d = 0; d < NV; ++d)
                        qp[d * 4 * QF] = uf[d];
                }
                __syncwarp();
                // against psi along the side
                for (int o = lane; o < ne * 4 * NV; o += 32)
                {
                    const int s = (o / NV) & 3, d = o % NV;
                    double *Eo = base + (o / (4 * NV)) * S::ES;
                    const double *uf = Eo + S::oH2 + d * 4 * QF + s * QF;
                    double m[N];
#pragma unroll
                    for (int k = 0; k < N; ++k)
                        m[k] = 0.0;
#pragma unroll
                    for (int q = 0; q < QF; ++q)
                    {
                        const double f = uf[q];
#pragma unroll
                        for (int k = 0; k < N; ++k)
                            m[k] += tab.Pft[q][k] * f;
                    }
#pragma unroll
                    for (int k = 0; k < N; ++k)
                        Eo[S::oT + NV * (s * N + k) + d] = m[k];
                }
            }
            __syncwarp();
            // ---- 2: column i of points
            if (on)
            {
                const int i = ln;
                double *H = E + S::oH + i * SP, *H2 = E + S::oH2 + i * SP;
                const double *c = E + S::oC;
                const double xi = tab.xq[i], wi = tab.wq[i];
                const double Xe = 0.25 * ((1.0 - xi) * (c[6] - c[0]) + (1.0 + xi) * (c[4] - c[2]));
                const double Ye = 0.25 * ((1.0 - xi) * (c[7] - c[1]) + (1.0 + xi) * (c[5] - c[3]));
                const double dx0 = c[2] - c[0], dx1 = c[4] - c[6], dy0 = c[3] - c[1], dy1 = c[5] - c[7];
                double v[S::REG ? N : 1][NV], fa[S::COLLOC ? 1 : N][NV], ga[N][NV];
                if constexpr (S::REG)
                {
#pragma unroll
                    for (int j = 0; j < N; ++j)
#pragma unroll
                        for (int d = 0; d < NV; ++d)
                            v[j][d] = H[j * NV + d];
                }
#pragma unroll
                for (int j = 0; j < N; ++j)
#pragma unroll
                    for (int d = 0; d < NV; ++d)
                    {
                        ga[j][d] = 0.0;
                        if constexpr (!S::COLLOC)
                            fa[j][d] = 0.0;
                    }
                if constexpr (M::FORCE)
                    if (A.F)
                    {
                        // + the forcing's column against psi along eta
                        for (int k = 0; k < N; ++k)
#pragma unroll
                            for (int d = 0; d < NV; ++d)
                            {
                                const double f = H2[k * NV + d];
#pragma unroll
                                for (int j = 0; j < N; ++j)
                                    ga[j][d] += tab.T[k][j] * f;
                            }
                    }
                // a collocated column's F goes straight to its row slot, over the interpolated column
                // it no longer needs once that is in registers (REG holds for every collocated shape)
                static_assert(!S::COLLOC || S::REG, "collocated columns live in registers");
                auto point = [&](int j)
                {
                    double U[NV], F[NV], G[NV];
#pragma unroll
                    for (int d = 0; d < NV; ++d)
                        U[d] = 0.0;
#pragma unroll
                    for (int m = 0; m < N; ++m)
#pragma unroll
                        for (int d = 0; d < NV; ++d)
                            U[d] += tab.P[j][m] * (S::REG ? v[S::REG ? m : 0][d] : H[m * NV + d]);
                    const double eta = tab.xq[j], W = wi * tab.wq[j];
                    const double Xx = 0.25 * ((1.0 - eta) * dx0 + (1.0 + eta) * dx1);
                    const double Yx = 0.25 * ((1.0 - eta) * dy0 + (1.0 + eta) * dy1);
                    M::template point<Q>(A, e0 + le, i, j, W * Xx, W * Yx, W * Xe, W * Ye, U, F, G);
#pragma unroll
                    for (int m = 0; m < N; ++m)
#pragma unroll
                        for (int d = 0; d < NV; ++d)
                        {
                            ga[m][d] += tab.Dt[j][m] * G[d];
                            if constexpr (!S::COLLOC)
                                fa[m][d] += tab.Pt[j][m] * F[d];
                        }
                    if constexpr (S::COLLOC)
#pragma unroll
                        for (int d = 0; d < NV; ++d)
                            H[j * NV + d] = F[d];
                };
                if constexpr (Q <= 7)
                {
#pragma unroll
                    for (int j = 0; j < Q; ++j)
                        point(j);
                }
                else
                {
#pragma unroll 1
                    for (int j = 0; j < Q; ++j)
                        point(j);
                }
#pragma unroll
                for (int j = 0; j < N; ++j)
#pragma unroll
                    for (int d = 0; d < NV; ++d)
                    {
                        H2[j * NV + d] = ga[j][d];
                        if constexpr (!S::COLLOC)
                            H[j * NV + d] = fa[j][d];
                    }
            }
            __syncwarp();
            // ---- 3: row l of Gauss points.  What the stage reads beside its input is asked for first
            double r[N][VP], p[N][VP];
            const size_t ge = (size_t)(e0 + le) * ND;
            const double *prev = x_prev(a);
#pragma unroll
            for (int k = 0; k < N; ++k)
#pragma unroll
                for (int d = 0; d < VP; ++d)
                    p[k][d] = (row && prev) ? prev[ge + NV * (M::LEG ? l * N + k : k * N + l) + part + PT * d] : 0.0;
            if (row)
            {
                const double *H = E + S::oH + l * NV + part, *H2 = E + S::oH2 + l * NV + part, *Sf = E + S::oT + part;
                const double *c = E + S::oC;
#pragma unroll
                for (int k = 0; k < N; ++k)
#pragma unroll
                    for (int d = 0; d < VP; ++d)
                        r[k][d] = S::COLLOC ? H2[k * SP + PT * d] : 0.0;
#pragma unroll
                for (int i = 0; i < Q; ++i)
#pragma unroll
                    for (int d = 0; d < VP; ++d)
                    {
                        const double f = H[i * SP + PT * d], gg = S::COLLOC ? 0.0 : H2[i * SP + PT * d];
#pragma unroll
                        for (int k = 0; k < N; ++k)
                        {
                            r[k][d] += tab.Dt[i][k] * f;
                            if constexpr (!S::COLLOC)
                                r[k][d] += tab.Pt[i][k] * gg;
                        }
                    }
                const double el = tab.xg[l], wl = tab.wg[l], sml = tab.sm[l], spl = tab.sp[l];
                const double Xx = 0.25 * ((1.0 - el) * (c[2] - c[0]) + (1.0 + el) * (c[4] - c[6]));
                const double Yx = 0.25 * ((1.0 - el) * (c[3] - c[1]) + (1.0 + el) * (c[5] - c[7]));
                double s1[VP], s3[VP];
#pragma unroll
                for (int d = 0; d < VP; ++d)
                {
                    s1[d] = Sf[NV * (N + l) + PT * d];
                    s3[d] = Sf[NV * (3 * N + l) + PT * d];
                }
#pragma unroll
                for (int k = 0; k < N; ++k)
                {
                    const double xi = tab.xg[k];
                    const double Xe = 0.25 * ((1.0 - xi) * (c[6] - c[0]) + (1.0 + xi) * (c[4] - c[2]));
                    const double Ye = 0.25 * ((1.0 - xi) * (c[7] - c[1]) + (1.0 + xi) * (c[5] - c[3]));
                    const double mi = 1.0 / (wl * tab.wg[k] * (Xx * Ye - Yx * Xe));
#pragma unroll
                    for (int d = 0; d < VP; ++d)
                        r[k][d] = mi * (r[k][d] + sml * Sf[NV * k + PT * d] + spl * Sf[NV * (2 * N + k) + PT * d] +
                                        tab.sm[k] * s3[d] + tab.sp[k] * s1[d]);
                }
            }
            // ---- 4: to the basis nodes (Gauss-Legendre bases are there), output
            auto finish = [&](int i, int j, const double *pv, const double *y)
            {
                const size_t gn = ge + NV * (j * N + i) + part;
                const double *u = E + SU * j + NV * i + part;
#pragma unroll
                for (int d = 0; d < VP; ++d)
                {
                    const double v = x_stage(a, gn + PT * d, u[PT * d], pv[d], y[d]);
                    if constexpr (M::FORCE) // the WaveHoltz filter of a step's last stage
                        if (A.acc)
                            A.acc[gn + PT * d] += A.acc_c * v;
                }
            };
            if constexpr (M::LEG)
            {
                if (row)
#pragma unroll
                    for (int k = 0; k < N; ++k)
                        finish(k, l, p[k], r[k]);
            }
            else
            {
                __syncwarp(); // every row has read H
                if (row)
                {
#pragma unroll
                    for (int k = 0; k < N; ++k)
#pragma unroll
                        for (int d = 0; d < VP; ++d)
                        {
                            double s = 0.0;
#pragma unroll
                            for (int m = 0; m < N; ++m)
                                s += tab.T[k][m] * r[m][d];
                            E[S::oH + k * SP + l * NV + part + PT * d] = s;
                        }
                }
                __syncwarp();
                if (row)
                {
                    // lane = node column l
                    double v[N][VP];
#pragma unroll
                    for (int m = 0; m < N; ++m)
#pragma unroll
                        for (int d = 0; d < VP; ++d)
                            v[m][d] = E[S::oH + l * SP + m * NV + part + PT * d];
#pragma unroll
                    for (int j = 0; j < N; ++j)
                    {
                        double y[VP];
#pragma unroll
                        for (int d = 0; d < VP; ++d)
                        {
                            y[d] = 0.0;
#pragma unroll
                            for (int m = 0; m < N; ++m)
                                y[d] += tab.T[j][m] * v[m][d];
                        }
                        finish(l, j, p[j], y);
                    }
                }
            }
            __syncwarp(); // the staging is reused by the next group
        }
    }

    // shared memory above 48 KB is opted in when a handle is created, before any capture
    template <int N, class M>
    cudaError_t xline_prepare_n()
    {
        return cudaFuncSetAttribute(xline_kernel<N, M>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)XShape<N, M>::smem);
    }
    template <int N, class M>
    cudaError_t xline_launch_n(const XArgs &A, cudaStream_t s)
    {
        using S = XShape<N, M>;
        const int ngroups = (A.c.nel + S::EW - 1) / S::EW;
        // one group per warp: the block scheduler evens out the last wave
        const int blocks = std::max(1, (ngroups + kXWarps - 1) / kXWarps);
        xline_kernel<N, M><<<blocks, 32 * kXWarps, S::smem, s>>>(A);
        return cudaGetLastError();
    }
#define WDG_XLINE_CASES(CALL)          \
    switch (n)                         \
    {                                  \
    case 2: return CALL(2);            \
    case 3: return CALL(3);            \
    case 4: return CALL(4);            \
    case 5: return CALL(5);            \
    case 6: return CALL(6);            \
    case 7: return CALL(7);            \
    case 8: return CALL(8);            \
    case 9: return CALL(9);            \
    default: return cudaErrorInvalidValue; \
    }
    template <class M>
    cudaError_t xline_prepare(int n)
    {
#define WDG_X(NV_) xline_prepare_n<NV_, M>()
        WDG_XLINE_CASES(WDG_X)
#undef WDG_X
    }
    template <class M>
    cudaError_t xline_launch(int n, const XArgs &A, cudaStream_t s)
    {
#define WDG_X(NV_) xline_launch_n<NV_, M>(A, s)
        WDG_XLINE_CASES(WDG_X)
#undef WDG_X
    }
} // namespace wdg
