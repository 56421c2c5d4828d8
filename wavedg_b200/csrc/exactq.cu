// C-ABI: the wave system with exact quadrature (approx_quad = false).
//
//   WaveEquation(mesh, basis, false)  source/WaveEquation.cpp:5-30
//     Div<false>       source/Div.cpp:312-361 (op_2d_cc), div_2d_q :469-588
//     EdgeFlux<false>  source/EdgeFlux.cpp:496-535, flux_action_2d_q :548-622
//   WaveBC(mesh, bc, basis, false)    source/WaveEquation.cpp:70-105, 190-215
//   MassMatrix<false>(mesh, basis)    source/MassMatrix.cpp:84-230; chol, solve_chol,
//                                     mult_chol in source/linalg.cpp:5-100
//
// Quadrature rules are the reference's defaults for bilinear elements (Gauss-Legendre):
// Div 1 + ((n-2) + (n-1) + 1) / 2 points per direction, EdgeFlux and MassMatrix
// 1 + (2 (n-1) + 2) / 2.  Face prolongation, the exterior states of the boundary codes and
// the argument staging are the collocation handle's (an internal wdg_wave, FP64).
//
// FP64 only.  The accuracy path for callers that set approx_quad = false.  The RHS and every
// RK4 stage (WaveHoltz periods included) are one fused launch (xline_kernel of
// exact_line.cuh: volume term, the four sides through the partner table, forcing, the inverse mass
// matrix as two one-dimensional contractions around a diagonal, the stage update); the operator
// entry points (Div, EdgeFlux, the mass matrix and its inverse) keep component kernels in the
// reference layouts: one CTA per element for the volume term, one thread per edge for the face
// term, a lane per grid line for the mass matrix.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "exact_line.cuh"
#include "wave_bc.cuh"
#include "wave_impl.hpp"

using namespace wdg;

struct wdg_waveq
{
    wdg_wave *w = nullptr;
    int n = 0, nqd = 0, nqf = 0, nqm = 0;
    double *d_xd = nullptr, *d_wd = nullptr, *d_Pd = nullptr, *d_Dd = nullptr; // Div rule, P(i,k), D(i,k)
    double *d_wf = nullptr, *d_Pf = nullptr;                                   // face rule, P(i,k)
    double *d_nI = nullptr, *d_nB = nullptr; // per edge (n_x, n_y, |E| / 2)
    MassOp mass;
    double *d_uf = nullptr, *d_uB = nullptr; // face traces
};

namespace wdg
{
    // D(i, j) = phi_j'(xq_i) for the Lagrange basis on the nodes x, by the barycentric
    // derivative formula: at a node the diagonal form, elsewhere the quotient form
    // (lagrange_basis_deriv, source/lagrange_interpolation.cpp:33-50, 96-139)
    void lagrange_deriv_at(int n, const double *x, int nq, const double *xq, double *D)
    {
        std::vector<double> lw(n), B((size_t)nq * n);
        for (int i = 0; i < n; ++i)
        {
            double p = 1.0;
            for (int j = 0; j < n; ++j)
                if (j != i)
                    p *= x[i] - x[j];
            lw[i] = 1.0 / p;
        }
        const auto mm = std::minmax_element(lw.begin(), lw.end());
        const double diff = *mm.second - *mm.first;
        for (double &v : lw)
            v /= diff;
        interp_matrix(n, x, nq, xq, B.data());
        const double eps = 2.220446049250313e-16;
        for (int j = 0; j < n; ++j)
            for (int i = 0; i < nq; ++i)
            {
                const double x0 = xq[i], p = B[i + (size_t)nq * j];
                int at = -1;
                for (int k = 0; k < n; ++k)
                    if (x0 == x[k] || std::abs(x0 - x[k]) <= eps)
                        at = k;
                double A = 0.0, S = 0.0;
                if (at >= 0)
                {
                    S = -lw[at];
                    for (int k = 0; k < n; ++k)
                        if (k != at)
                            A += lw[k] * (p - (k == j ? 1.0 : 0.0)) / (x0 - x[k]);
                }
                else
                    for (int k = 0; k < n; ++k)
                    {
                        const double t = lw[k] / (x0 - x[k]);
                        A += t * (p - (k == j ? 1.0 : 0.0)) / (x0 - x[k]);
                        S += t;
                    }
                D[i + (size_t)nq * j] = A / S;
            }
    }

    template <int N>
    struct MassArgs
    {
        double A[N][N], xg[N], wg[N]; // psi_m(x_k) at [k][m] (inverse), phi_k(g_m) at [m][k] (action)
        const double *corners, *x;
        double *y;
        int nel, nv, ew, rs;
    };
    // M = (B x B)^T D (B x B) and its inverse (T x T) D^{-1} (T x T)^T.  A warp owns ew whole elements, a lane
    // a grid line of one of them, one variable after the other, in place: rows, columns (to the Gauss points,
    // D, and back: the column is this lane's alone), rows.  The staged rows are rs (odd) doubles apart, so
    // that neither pass has two lanes on a bank; the matrices are constant-bank operands.  Bound by memory: 16 bytes a value.
    // 128 x 128, inverse, one and three variables: n = 2: 18 and 18 -> 4.5 and 5.5 us, n = 5: 21 and 49 -> 6.5
    // and 10 us against a warp per element with generic loops (dense inverses: 6.2 and 6.2, 22 and 42 us).
    template <int N, bool INV>
    __global__ void __launch_bounds__(128) mass_kernel(const __grid_constant__ MassArgs<N> a)
    {
        extern __shared__ double sx[];
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nv = a.nv, rs = a.rs, m = nv * N;
        const int e0 = (blockIdx.x * (int)(blockDim.x >> 5) + warp) * a.ew, ne = min(a.ew, a.nel - e0);
        if (ne <= 0)
            return;
        double *E = sx + (size_t)warp * a.ew * N * rs;
        const size_t first = (size_t)e0 * N * m;
        for (int o = lane; o < ne * N * m; o += 32)
            E[(o / m) * rs + o % m] = a.x[first + o];
        const int le = lane / N, ln = lane - le * N;
        const bool on = le < ne;
        double *R = E + (le * N + ln) * rs, *C = E + le * N * rs + ln * nv;
        double w[N];
        if (on)
        {
            double c[8], J[4];
#pragma unroll
            for (int k = 0; k < 8; ++k)
                c[k] = __ldg(a.corners + 8 * (size_t)(e0 + le) + k);
#pragma unroll
            for (int j = 0; j < N; ++j)
            {
                quad_jacobian(c, a.xg[ln], a.xg[j], J);
                w[j] = a.wg[ln] * a.wg[j] * (J[0] * J[3] - J[2] * J[1]);
                if (INV)
                    w[j] = 1.0 / w[j];
            }
        }
        // v -> to the points along a line (`to`), or back
        auto line = [&](double (&v)[N], bool to)
        {
            double s[N];
#pragma unroll
            for (int i = 0; i < N; ++i)
            {
                s[i] = 0.0;
#pragma unroll
                for (int k = 0; k < N; ++k)
                    s[i] += (to != INV ? a.A[i][k] : a.A[k][i]) * v[k];
            }
#pragma unroll
            for (int i = 0; i < N; ++i)
                v[i] = s[i];
        };
        __syncwarp();
        if (on)
            for (int d = 0; d < nv; ++d)
            {
                double v[N];
#pragma unroll
                for (int k = 0; k < N; ++k)
                    v[k] = R[k * nv + d];
                line(v, true);
#pragma unroll
                for (int k = 0; k < N; ++k)
                    R[k * nv + d] = v[k];
            }
        __syncwarp();
        if (on)
            for (int d = 0; d < nv; ++d)
            {
                double v[N];
#pragma unroll
                for (int k = 0; k < N; ++k)
                    v[k] = C[k * rs + d];
                line(v, true);
#pragma unroll
                for (int k = 0; k < N; ++k)
                    v[k] *= w[k];
                line(v, false);
#pragma unroll
                for (int k = 0; k < N; ++k)
                    C[k * rs + d] = v[k];
            }
        __syncwarp();
        if (on)
            for (int d = 0; d < nv; ++d)
            {
                double v[N];
#pragma unroll
                for (int k = 0; k < N; ++k)
                    v[k] = R[k * nv + d];
                line(v, false);
#pragma unroll
                for (int k = 0; k < N; ++k)
                    R[k * nv + d] = v[k];
            }
        __syncwarp();
        for (int o = lane; o < ne * N * m; o += 32)
            a.y[first + o] = E[(o / m) * rs + o % m];
    }

    template <int N>
    int mass_launch_n(const MassOp &t, int nel, int nv, bool inverse, const double *corners, const double *x, double *y,
                      cudaStream_t s)
    {
        MassArgs<N> a;
        for (int i = 0; i < N; ++i)
        {
            for (int k = 0; k < N; ++k)
                a.A[i][k] = inverse ? t.T[i * N + k] : t.B[i * N + k];
            a.xg[i] = t.xg[i];
            a.wg[i] = t.wg[i];
        }
        a.corners = corners;
        a.x = x;
        a.y = y;
        a.nel = nel;
        a.nv = nv;
        a.rs = (nv * N) | 1;
        // 48 KB: one element at least (callers bound nv), then a lane per line, then warps
        const size_t element = sizeof(double) * N * a.rs, room = 48 * 1024;
        a.ew = (int)std::max<size_t>(1, std::min<size_t>(32 / N, room / element));
        const int wpb = (int)std::max<size_t>(1, std::min<size_t>(4, room / (element * a.ew)));
        const unsigned blocks = (unsigned)(((nel + a.ew - 1) / a.ew + wpb - 1) / wpb);
        const size_t smem = element * a.ew * wpb;
        if (inverse)
            mass_kernel<N, true><<<blocks, 32 * wpb, smem, s>>>(a);
        else
            mass_kernel<N, false><<<blocks, 32 * wpb, smem, s>>>(a);
        WDG_CUDA(cudaGetLastError());
        return WDG_OK;
    }
    int mass_launch(const MassOp &t, int nel, int nv, bool inverse, const double *corners, const double *x, double *y,
                    cudaStream_t s)
    {
        switch (t.n)
        {
        case 2: return mass_launch_n<2>(t, nel, nv, inverse, corners, x, y, s);
        case 3: return mass_launch_n<3>(t, nel, nv, inverse, corners, x, y, s);
        case 4: return mass_launch_n<4>(t, nel, nv, inverse, corners, x, y, s);
        case 5: return mass_launch_n<5>(t, nel, nv, inverse, corners, x, y, s);
        case 6: return mass_launch_n<6>(t, nel, nv, inverse, corners, x, y, s);
        case 7: return mass_launch_n<7>(t, nel, nv, inverse, corners, x, y, s);
        case 8: return mass_launch_n<8>(t, nel, nv, inverse, corners, x, y, s);
        case 9: return mass_launch_n<9>(t, nel, nv, inverse, corners, x, y, s);
        default: return fail(WDG_ERR_UNSUPPORTED, "mass matrix: n_colloc must be 2..9");
        }
    }

    MassOp mass_op(int n, const double *x)
    {
        MassOp t;
        std::vector<double> C((size_t)n * n);
        t.n = n;
        gauss_legendre(n, t.xg, t.wg);
        auto rows = [&](double *R) // column-major -> row-major
        {
            for (int r = 0; r < n; ++r)
                for (int c = 0; c < n; ++c)
                    R[r * n + c] = C[r + (size_t)n * c];
        };
        interp_matrix(n, t.xg, n, x, C.data());
        rows(t.T);
        interp_matrix(n, x, n, t.xg, C.data());
        rows(t.B);
        return t;
    }

    int mass_tables(int n, const double *x, MassTables &t)
    {
        const MassOp m = mass_op(n, x);
        auto put = [](double **d, const double *v, size_t count) -> int
        {
            WDG_TRY(device_alloc(d, count));
            WDG_CUDA(cudaMemcpy(*d, v, sizeof(double) * count, cudaMemcpyHostToDevice));
            return WDG_OK;
        };
        WDG_TRY(put(&t.T, m.T, (size_t)n * n));
        WDG_TRY(put(&t.xg, m.xg, (size_t)n));
        return put(&t.wg, m.wg, (size_t)n);
    }
    void mass_tables_free(MassTables &t)
    {
        for (double *p : {t.T, t.xg, t.wg})
            if (p)
                cudaFree(p);
        t = MassTables{};
    }
} // namespace wdg

namespace
{
    constexpr int kMaxQ = 16;

    int qdiv(int n) { return 1 + ((n - 2) + (n - 1) + 1) / 2; }
    int qface(int n) { return 1 + (2 * (n - 1) + 2) / 2; }

    // QuadElement::jacobian (source/Element.cpp:21-27): J = (x_xi, y_xi, x_eta, y_eta)
    __host__ __device__ inline void jac(const double *c, double xi, double eta, double J[4])
    {
        J[0] = 0.25 * ((1.0 - eta) * (c[2] - c[0]) + (1.0 + eta) * (c[4] - c[6]));
        J[1] = 0.25 * ((1.0 - eta) * (c[3] - c[1]) + (1.0 + eta) * (c[5] - c[7]));
        J[2] = 0.25 * ((1.0 - xi) * (c[6] - c[0]) + (1.0 + xi) * (c[4] - c[2]));
        J[3] = 0.25 * ((1.0 - xi) * (c[7] - c[1]) + (1.0 + xi) * (c[5] - c[3]));
    }

    // ---------------------------------------------------------------- Div<false>
    // One CTA per element, shared memory per element: u, P u (one direction), U at the points,
    // the two contravariant fluxes, and the two half-contracted sums.  Accumulates into du.
    __global__ void qdiv_kernel(int n, int q, int nel, const double *__restrict__ corners,
                                const double *__restrict__ xd, const double *__restrict__ wd,
                                const double *__restrict__ Pd, const double *__restrict__ Dd,
                                const double *__restrict__ u, double *du)
    {
        extern __shared__ double sm[];
        const int nn = n * n, qq = q * q;
        double *su = sm;                 // (3, n, n)
        double *Pu = su + 3 * nn;        // (n, 3, q)
        double *Uq = Pu + 3 * n * q;     // (3, q, q)
        double *Fq = Uq + 3 * qq;        // (2, 3, q, q)
        double *Df = Fq + 6 * qq;        // (q, 3, n)
        double *Pg = Df + 3 * q * n;     // (q, 3, n)
        const int t = threadIdx.x, T = blockDim.x;
        for (int el = blockIdx.x; el < nel; el += gridDim.x)
        {
            const double *ue = u + (size_t)3 * nn * el;
            for (int k = t; k < 3 * nn; k += T)
                su[k] = ue[k];
            __syncthreads();
            // Pu(l, d, i) = sum_k P(i, k) u(d, k, l)
            for (int o = t; o < 3 * n * q; o += T)
            {
                const int l = o % n, d = (o / n) % 3, i = o / (3 * n);
                double s = 0.0;
                for (int k = 0; k < n; ++k)
                    s += Pd[i + q * k] * su[d + 3 * (k + n * l)];
                Pu[o] = s;
            }
            __syncthreads();
            // U(d, i, j) = sum_l P(j, l) Pu(l, d, i)
            for (int o = t; o < 3 * qq; o += T)
            {
                const int d = o % 3, i = (o / 3) % q, j = o / (3 * q);
                double s = 0.0;
                for (int l = 0; l < n; ++l)
                    s += Pd[j + q * l] * Pu[l + n * (d + 3 * i)];
                Uq[o] = s;
            }
            __syncthreads();
            // contravariant fluxes of the wave system at the points (op_2d_cc with the wave
            // table: F = W (y_eta u - x_eta v, y_eta p, -x_eta p), G = W (-y_xi u + x_xi v, -y_xi p, x_xi p))
            const double *ce = corners + 8 * (size_t)el;
            for (int o = t; o < qq; o += T)
            {
                const int i = o % q, j = o / q;
                double J[4];
                jac(ce, xd[i], xd[j], J);
                const double W = wd[i] * wd[j];
                const double Xxi = J[0] * W, Yxi = J[1] * W, Xeta = J[2] * W, Yeta = J[3] * W;
                const double *U = Uq + 3 * o;
                double *F = Fq + 6 * o;
                F[0] = Yeta * U[1] - Xeta * U[2];
                F[1] = -Yxi * U[1] + Xxi * U[2];
                F[2] = Yeta * U[0];
                F[3] = -Yxi * U[0];
                F[4] = -Xeta * U[0];
                F[5] = Xxi * U[0];
            }
            __syncthreads();
            // Df(j, d, k) = sum_i D(i, k) F(d, i, j);  Pg(j, d, k) = sum_i P(i, k) G(d, i, j)
            for (int o = t; o < 3 * q * n; o += T)
            {
                const int j = o % q, d = (o / q) % 3, k = o / (3 * q);
                double df = 0.0, pg = 0.0;
                for (int i = 0; i < q; ++i)
                {
                    df += Dd[i + q * k] * Fq[2 * d + 6 * (i + q * j)];
                    pg += Pd[i + q * k] * Fq[2 * d + 1 + 6 * (i + q * j)];
                }
                Df[o] = df;
                Pg[o] = pg;
            }
            __syncthreads();
            // du(d, k, l) += sum_j P(j, l) Df(j, d, k) + D(j, l) Pg(j, d, k)
            double *de = du + (size_t)3 * nn * el;
            for (int o = t; o < 3 * nn; o += T)
            {
                const int d = o % 3, k = (o / 3) % n, l = o / (3 * n);
                double s = 0.0;
                for (int j = 0; j < q; ++j)
                    s += Pd[j + q * l] * Df[j + q * (d + 3 * k)] + Dd[j + q * l] * Pg[j + q * (d + 3 * k)];
                de[o] += s;
            }
            __syncthreads();
        }
    }

    // ---------------------------------------------------------------- EdgeFlux<false>
    // One thread per edge: both sides' traces to the face points, upwind flux there (a = -1,
    // b = -1/2 of the wave system, in closed form: side 0 contributes -1/2 v (v . U0),
    // v = (1, n_x, n_y); side 1 +1/2 w (w . U1), w = (1, -n_x, -n_y)), weighted by
    // w_q |E| / 2, then back to the nodes; side 1 gets the negative.  fb may equal ub.
    __global__ void qflux_kernel(int n, int q, int ne, const double *__restrict__ nrm, const double *__restrict__ wf,
                                 const double *__restrict__ Pf, const double *ub, double *fb)
    {
        const int e = blockIdx.x * blockDim.x + threadIdx.x;
        if (e >= ne)
            return;
        const double nx = nrm[3 * e], ny = nrm[3 * e + 1], meas = nrm[3 * e + 2];
        double uf[kMaxQ][3];
        for (int i = 0; i < q; ++i)
        {
            double U0[3], U1[3];
            for (int d = 0; d < 3; ++d)
            {
                double a = 0.0, b = 0.0;
                for (int j = 0; j < n; ++j)
                {
                    a += ub[j + n * (d + 3 * (0 + 2 * (size_t)e))] * Pf[i + q * j];
                    b += ub[j + n * (d + 3 * (1 + 2 * (size_t)e))] * Pf[i + q * j];
                }
                U0[d] = a;
                U1[d] = b;
            }
            const double w = wf[i] * meas;
            const double s0 = -0.5 * w * (U0[0] + nx * U0[1] + ny * U0[2]);
            const double s1 = 0.5 * w * (U1[0] - nx * U1[1] - ny * U1[2]);
            uf[i][0] = s0 + s1;
            uf[i][1] = nx * (s0 - s1);
            uf[i][2] = ny * (s0 - s1);
        }
        for (int d = 0; d < 3; ++d)
            for (int i = 0; i < n; ++i)
            {
                double f = 0.0;
                for (int j = 0; j < q; ++j)
                    f += uf[j][d] * Pf[j + q * i];
                fb[i + n * (d + 3 * (0 + 2 * (size_t)e))] = f;
                fb[i + n * (d + 3 * (1 + 2 * (size_t)e))] = -f;
            }
    }

    // ---------------------------------------------------------------- fused RHS / RK4 stage
    // The model of exact_line.cuh: what rhs_dev's operators add up to, with the boundary codes'
    // exterior states at the nodes, the closed-form upwind flux with the element's own outward
    // normal (so the two elements of an edge add exactly opposite terms), the forcing s F, and the
    // WaveHoltz filter on the last stage.
    struct WaveX
    {
        static constexpr int NV = 3;
        static constexpr bool LEG = false, FORCE = true, LINEAR = true, WEIGHTED = true;
        __host__ __device__ static constexpr int q(int n) { return n; }
        __host__ __device__ static constexpr int qf(int n) { return n + 1; }
        template <int N>
        __device__ static const XTab<N, N, N + 1> &table();
        __device__ static void exterior(int code, const double *sn, const double *own, double *x)
        {
            const double o[3] = {own[0], own[1], own[2]};
            wdg::exterior<double>(code, sn[0], sn[1], o, x);
        }
        template <int Q>
        __device__ static void point(const XArgs &, int, int, int, double Xx, double Yx, double Xe, double Ye,
                                     const double *U, double *F, double *G)
        {
            F[0] = Ye * U[1] - Xe * U[2];
            G[0] = -Yx * U[1] + Xx * U[2];
            F[1] = Ye * U[0];
            G[1] = -Yx * U[0];
            F[2] = -Xe * U[0];
            G[2] = Xx * U[0];
        }
        // The upwind flux of side 0 is -1/2 v (v . U0), v = (1, n_x, n_y), of side 1 +1/2 w (w . U1),
        // w = (1, -n_x, -n_y) (as qflux_kernel): with s0, s1 those scalars at a face node, t becomes
        // (s0 + s1, s0 - s1), which spread turns into the side's three projected fluxes
        __device__ static void combine(const double *sn, const double *o, double *t)
        {
            const double h = 0.5 * sn[2];
            const double s0 = -h * (o[0] + sn[0] * o[1] + sn[1] * o[2]), s1 = h * (t[0] - sn[0] * t[1] - sn[1] * t[2]);
            t[0] = s0 + s1;
            t[1] = s0 - s1;
        }
        __device__ static void spread(const double *sn, int which, double v, double *t)
        {
            if (which == 0)
                t[0] = v;
            else
            {
                t[1] = sn[0] * v;
                t[2] = sn[1] * v;
            }
        }
    };
    __constant__ XTabs<WaveX> c_wave_x;
    template <int N>
    __device__ const XTab<N, N, N + 1> &WaveX::table() { return xtab<N>(c_wave_x); }

    size_t face_count(const wdg_waveq *h, int type)
    {
        return (size_t)h->n * 3 * 2 * (type == 0 ? h->w->nI : h->w->nB);
    }

    int exact_launch(wdg_waveq *h, const XArgs &a)
    {
        WDG_CUDA(xline_launch<WaveX>(h->n, a, h->w->stream));
        return WDG_OK;
    }

    // nsteps of ode::RungeKutta4 on device array u (not a rotation buffer), one fused launch per
    // stage: the rotation u -> B -> C -> B -> C -> u of the wave handle's buffers; with F, the
    // forcing F s(t) at the stage times; with acc, acc += c_filter[step] u after each step
    int exact_rk4(wdg_waveq *h, double *u, double dt, double t, int nsteps, const double *F, double omega,
                   double *acc, const double *c_filter)
    {
        wdg_wave *w = h->w;
        WDG_TRY(ensure_states(w));
        double *B = static_cast<double *>(w->d_state[1]), *Cb = static_cast<double *>(w->d_state[2]);
        XArgs a{};
        a.c = claw_args(w, u, nullptr);
        a.c.du = static_cast<double *>(w->d_du);
        a.c.mode = CLAW_RK4;
        a.c.dt = dt;
        a.F = F;
        for (int step = 0; step < nsteps; ++step)
        {
            const double *src = u;
            for (int st = 0; st < 5; ++st)
            {
                double *dst = (st == 4) ? u : ((st % 2 == 0) ? B : Cb);
                a.c.x = src;
                a.c.out = dst;
                a.c.rk_a = rk4a[st];
                a.c.rk_b = rk4b[st];
                a.fs = F ? -std::sin(omega * (t + rk4c[st] * dt)) / omega : 0.0;
                a.acc = (st == 4) ? acc : nullptr;
                a.acc_c = (st == 4 && acc) ? c_filter[step] : 0.0;
                WDG_TRY(exact_launch(h, a));
                src = dst;
            }
            t += dt;
        }
        return WDG_OK;
    }

    // ---------------------------------------------------------------- device-side operators
    int div_dev(wdg_waveq *h, const double *u, double *du)
    {
        wdg_wave *w = h->w;
        const int n = h->n, q = h->nqd;
        const size_t smem = sizeof(double) * (3 * n * n + 3 * n * q + 3 * q * q + 6 * q * q + 6 * q * n);
        qdiv_kernel<<<(unsigned)std::min(w->nel, 148 * 16), 64, smem, w->stream>>>(n, q, w->nel, w->d_corners, h->d_xd,
                                                                                   h->d_wd, h->d_Pd, h->d_Dd, u, du);
        WDG_CUDA(cudaGetLastError());
        return WDG_OK;
    }
    int flux_dev(wdg_waveq *h, int type, const double *ub, double *fb)
    {
        wdg_wave *w = h->w;
        const int ne = (type == 0) ? w->nI : w->nB;
        if (ne == 0)
            return WDG_OK;
        qflux_kernel<<<(unsigned)((ne + 127) / 128), 128, 0, w->stream>>>(h->n, h->nqf, ne, type == 0 ? h->d_nI : h->d_nB,
                                                                          h->d_wf, h->d_Pf, ub, fb);
        WDG_CUDA(cudaGetLastError());
        return WDG_OK;
    }
    int mass_dev(wdg_waveq *h, int nv, const double *x, double *y, bool inverse)
    {
        return mass_launch(h->mass, h->w->nel, nv, inverse, h->w->d_corners, x, y, h->w->stream);
    }
    // du += Div u + Prol_I^T Flux_I Prol_I u
    int wave_dev(wdg_waveq *h, const double *u, double *du)
    {
        wdg_wave *w = h->w;
        WDG_TRY(div_dev(h, u, du));
        if (w->nI)
        {
            WDG_CUDA(launch_prolong(w->geo, 0, u, h->d_uf, w->stream));
            WDG_TRY(flux_dev(h, 0, h->d_uf, h->d_uf));
            WDG_CUDA(launch_prolong_t(w->geo, 0, h->d_uf, du, w->stream));
        }
        return WDG_OK;
    }
    // du += Prol_B^T Flux_B (exterior states) Prol_B u
    int bc_dev(wdg_waveq *h, const double *u, double *du)
    {
        wdg_wave *w = h->w;
        if (!w->nB)
            return WDG_OK;
        WDG_CUDA(launch_prolong(w->geo, 1, u, h->d_uB, w->stream));
        WDG_CUDA(launch_apply_bc(w->geo, h->d_uB, w->stream));
        WDG_TRY(flux_dev(h, 1, h->d_uB, h->d_uB));
        WDG_CUDA(launch_prolong_t(w->geo, 1, h->d_uB, du, w->stream));
        return WDG_OK;
    }
    // dudt = M^{-1} (A u + B u + s F), one fused launch
    int rhs_dev(wdg_waveq *h, const double *u, double *dudt, const double *F, double s)
    {
        XArgs a{};
        a.c = claw_args(h->w, u, dudt);
        a.c.mode = CLAW_RHS;
        a.F = F;
        a.fs = s;
        return exact_launch(h, a);
    }

    typedef int (*Unary)(wdg_waveq *, const double *, double *);
    int accumulate_entry(wdg_waveq *h, const double *u, double *du, Unary f)
    {
        if (!h)
            return fail(WDG_ERR_ARG, "null exact-quadrature discretisation");
        if (u == du)
            return fail(WDG_ERR_ARG, "input and output arrays must differ");
        DeviceScope g(h->w->device);
        HostArg a[2];
        WDG_TRY(bind_arg(h->w, 0, u, h->w->ndof, true, false, a[0]));
        WDG_TRY(bind_arg(h->w, 1, du, h->w->ndof, true, true, a[1]));
        WDG_TRY(f(h, a[0].dev, a[1].dev));
        return finish_args(h->w, a, 2);
    }
} // namespace

namespace wdg
{
    // RK buffers and the resident state exist before a period is captured into a graph
    int waveq_prepare(wdg_waveq *h)
    {
        DeviceScope g(h->w->device);
        return ensure_states(h->w);
    }

    // One WaveHoltz period on the exact-quadrature operators, the sequence rk4_run runs on the
    // collocation kernels: nt RK4 steps of u' = M^{-1}(A u + B u + F s(t)), s(t) =
    // -sin(omega t) / omega at the stage times (F may be NULL), then acc += c_filter[step] u
    // after each step (source/WaveHoltz.cpp:55-121).  On the handle's current stream.
    int waveq_period(wdg_waveq *h, double *u, double dt, int nt, const double *F, double omega, double *acc,
                     const double *c_filter)
    {
        return exact_rk4(h, u, dt, 0.0, nt, F, omega, acc, c_filter);
    }

    // P = M^{-1}(A + B) W on the exact operators (WaveHoltz::postprocess's RHS)
    int waveq_rhs_device(wdg_waveq *h, const double *u, double *dudt) { return rhs_dev(h, u, dudt, nullptr, 0.0); }
} // namespace wdg

extern "C"
{
    int wdg_waveq_create(const wdg_mesh *mesh, int n_colloc, const int *bc, int device, wdg_waveq **out)
    {
        if (!mesh || !out)
            return fail(WDG_ERR_ARG, "wdg_waveq_create: null argument");
        *out = nullptr;
        if (n_colloc < 2 || n_colloc > 9)
            return fail(WDG_ERR_UNSUPPORTED, "wdg_waveq_create: n_colloc must be 2..9");
        wdg_wave *w = nullptr;
        WDG_TRY(wdg_wave_create(mesh, n_colloc, bc, WDG_FP64, device, &w));
        wdg_waveq *h = new wdg_waveq;
        h->w = w;
        h->n = n_colloc;
        h->nqd = qdiv(n_colloc);
        h->nqf = qface(n_colloc);
        h->nqm = qface(n_colloc);
        DeviceScope g(w->device);
        {
            // the fused kernel's matrices (once per device) and its shared memory, before any period
            // is captured into a graph
            static std::mutex mu;
            static uint64_t set = 0;
            std::lock_guard<std::mutex> lock(mu);
            cudaError_t e = cudaSuccess;
            if (!(set & (1ull << (w->device & 63))))
            {
                std::vector<XTabs<WaveX>> t(1);
                xtabs_fill(t[0], false);
                e = cudaMemcpyToSymbol(c_wave_x, t.data(), sizeof(XTabs<WaveX>));
                if (e == cudaSuccess)
                    set |= 1ull << (w->device & 63);
            }
            if (e == cudaSuccess)
                e = xline_prepare<WaveX>(n_colloc);
            if (e != cudaSuccess)
            {
                wdg_wave_destroy(w);
                delete h;
                return cuda_fail(e, "wdg_waveq_create: fused kernel");
            }
        }
        const int n = n_colloc, c = n * n;
        std::vector<double> x(n), wg(n);
        gauss_lobatto(n, x.data(), wg.data());
        // Div rule and its interpolation / derivative matrices
        std::vector<double> xd(h->nqd), wd(h->nqd), Pd((size_t)h->nqd * n), Dd((size_t)h->nqd * n);
        gauss_legendre(h->nqd, xd.data(), wd.data());
        interp_matrix(n, x.data(), h->nqd, xd.data(), Pd.data());
        lagrange_deriv_at(n, x.data(), h->nqd, xd.data(), Dd.data());
        // face rule
        std::vector<double> xf(h->nqf), wf(h->nqf), Pf((size_t)h->nqf * n);
        gauss_legendre(h->nqf, xf.data(), wf.data());
        interp_matrix(n, x.data(), h->nqf, xf.data(), Pf.data());
        // per edge: outward normal of elements[0] and |E| / 2 (StraightEdge, wavedg/Edge.hpp:107-122)
        auto normals = [&](const std::vector<EdgeRec> &list)
        {
            std::vector<double> nr(3 * list.size());
            for (size_t e = 0; e < list.size(); ++e)
            {
                const double *cr = &mesh->corners[8 * (size_t)list[e].el0];
                const int s = list[e].s0;
                const double dx = cr[2 * kSideTo[s]] - cr[2 * kSideFrom[s]];
                const double dy = cr[2 * kSideTo[s] + 1] - cr[2 * kSideFrom[s] + 1];
                const double len = std::sqrt(dx * dx + dy * dy), sgn = (s >= 2) ? -1.0 : 1.0;
                nr[3 * e] = sgn * dy / len;
                nr[3 * e + 1] = -sgn * dx / len;
                nr[3 * e + 2] = 0.5 * len;
            }
            return nr;
        };
        const std::vector<double> nI = normals(mesh->interior), nB = normals(mesh->boundary);
        int st = exact_mass_check(*mesh, n);
        auto chk = [&](int r)
        {
            if (st == WDG_OK)
                st = r;
        };
        chk(device_alloc(&h->d_xd, xd.size()));
        chk(device_alloc(&h->d_wd, wd.size()));
        chk(device_alloc(&h->d_Pd, Pd.size()));
        chk(device_alloc(&h->d_Dd, Dd.size()));
        chk(device_alloc(&h->d_wf, wf.size()));
        chk(device_alloc(&h->d_Pf, Pf.size()));
        chk(device_alloc(&h->d_nI, nI.size()));
        chk(device_alloc(&h->d_nB, nB.size()));
        chk(device_alloc(&h->d_uf, face_count(h, 0)));
        chk(device_alloc(&h->d_uB, face_count(h, 1)));
        if (st == WDG_OK)
        {
            chk(device_put(h->d_xd, xd));
            chk(device_put(h->d_wd, wd));
            chk(device_put(h->d_Pd, Pd));
            chk(device_put(h->d_Dd, Dd));
            chk(device_put(h->d_wf, wf));
            chk(device_put(h->d_Pf, Pf));
            chk(device_put(h->d_nI, nI));
            chk(device_put(h->d_nB, nB));
            h->mass = mass_op(n, x.data());
        }
        if (st == WDG_OK)
        {
            const int smax = (int)(sizeof(double) * (3 * c + 3 * n * h->nqd + 9 * h->nqd * h->nqd + 6 * h->nqd * n));
            if (smax > 48 * 1024)
            {
                const cudaError_t e = cudaFuncSetAttribute(qdiv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smax);
                if (e != cudaSuccess)
                    st = cuda_fail(e, "wdg_waveq_create: shared memory attribute");
            }
        }
        if (st != WDG_OK)
        {
            wdg_waveq_destroy(h);
            return st;
        }
        *out = h;
        return WDG_OK;
    }

    void wdg_waveq_destroy(wdg_waveq *h)
    {
        if (!h)
            return;
        {
            DeviceScope g(h->w ? h->w->device : 0);
            for (double *p : {h->d_xd, h->d_wd, h->d_Pd, h->d_Dd, h->d_wf, h->d_Pf, h->d_nI, h->d_nB, h->d_uf, h->d_uB})
                if (p)
                    cudaFree(p);
        }
        if (h->w)
            wdg_wave_destroy(h->w);
        delete h;
    }

    int wdg_waveq_rules(const wdg_waveq *h, int *n_div, int *n_face, int *n_mass)
    {
        if (!h)
            return fail(WDG_ERR_ARG, "null exact-quadrature discretisation");
        if (n_div)
            *n_div = h->nqd;
        if (n_face)
            *n_face = h->nqf;
        if (n_mass)
            *n_mass = h->nqm;
        return WDG_OK;
    }

    int wdg_waveq_wave(const wdg_waveq *h, wdg_wave **wave)
    {
        if (!h || !wave)
            return fail(WDG_ERR_ARG, "wdg_waveq_wave: null argument");
        *wave = h->w;
        return WDG_OK;
    }

    int wdg_waveq_div_action(wdg_waveq *h, const double *u, double *du) { return accumulate_entry(h, u, du, div_dev); }
    int wdg_waveq_wave_action(wdg_waveq *h, const double *u, double *du) { return accumulate_entry(h, u, du, wave_dev); }
    int wdg_waveq_wavebc_action(wdg_waveq *h, const double *u, double *du) { return accumulate_entry(h, u, du, bc_dev); }

    int wdg_waveq_edge_flux(wdg_waveq *h, int type, const double *ub, double *fb)
    {
        if (!h || (type != 0 && type != 1) || !ub || !fb)
            return fail(WDG_ERR_ARG, "wdg_waveq_edge_flux: bad arguments");
        DeviceScope g(h->w->device);
        const size_t cnt = face_count(h, type);
        HostArg a[2];
        if (ub == fb)
        {
            WDG_TRY(bind_arg(h->w, 0, ub, cnt, true, true, a[0]));
            WDG_TRY(flux_dev(h, type, a[0].dev, a[0].dev));
            return finish_args(h->w, a, 1);
        }
        WDG_TRY(bind_arg(h->w, 0, ub, cnt, true, false, a[0]));
        WDG_TRY(bind_arg(h->w, 1, fb, cnt, false, true, a[1]));
        WDG_TRY(flux_dev(h, type, a[0].dev, a[1].dev));
        return finish_args(h->w, a, 2);
    }

    int wdg_waveq_mass_inv(wdg_waveq *h, int n_var, double *x)
    {
        if (!h || n_var < 1 || n_var > 16)
            return fail(WDG_ERR_ARG, "wdg_waveq_mass_inv: bad arguments");
        DeviceScope g(h->w->device);
        HostArg a;
        WDG_TRY(bind_arg(h->w, 0, x, (size_t)n_var * h->n * h->n * h->w->nel, true, true, a));
        WDG_TRY(mass_dev(h, n_var, a.dev, a.dev, true));
        return finish_args(h->w, &a, 1);
    }

    int wdg_waveq_mass_action(wdg_waveq *h, int n_var, const double *x, double *y)
    {
        if (!h || n_var < 1 || n_var > 16 || !x || !y)
            return fail(WDG_ERR_ARG, "wdg_waveq_mass_action: bad arguments");
        DeviceScope g(h->w->device);
        const size_t cnt = (size_t)n_var * h->n * h->n * h->w->nel;
        HostArg a[2];
        WDG_TRY(bind_arg(h->w, 0, x, cnt, true, false, a[0]));
        WDG_TRY(bind_arg(h->w, 1, y, cnt, false, true, a[1]));
        WDG_TRY(mass_dev(h, n_var, a[0].dev, a[1].dev, false));
        return finish_args(h->w, a, 2);
    }

    int wdg_waveq_rhs(wdg_waveq *h, const double *u, double *dudt, const double *F, double s)
    {
        if (!h || !u || !dudt)
            return fail(WDG_ERR_ARG, "wdg_waveq_rhs: bad arguments");
        if (u == dudt)
            return fail(WDG_ERR_ARG, "input and output arrays must differ");
        DeviceScope g(h->w->device);
        HostArg a[3];
        int na = 2;
        WDG_TRY(bind_arg(h->w, 0, u, h->w->ndof, true, false, a[0]));
        WDG_TRY(bind_arg(h->w, 1, dudt, h->w->ndof, false, true, a[1]));
        if (F)
        {
            WDG_TRY(bind_arg(h->w, 2, F, h->w->ndof, true, false, a[2]));
            na = 3;
        }
        WDG_TRY(rhs_dev(h, a[0].dev, a[1].dev, F ? a[2].dev : nullptr, s));
        return finish_args(h->w, a, na);
    }

    int wdg_waveq_rk4_steps(wdg_waveq *h, double *u, double dt, double *t, int nsteps)
    {
        if (!h || !u || !t || nsteps < 0)
            return fail(WDG_ERR_ARG, "wdg_waveq_rk4_steps: bad arguments");
        DeviceScope g(h->w->device);
        wdg_wave *w = h->w;
        HostArg a;
        WDG_TRY(bind_arg(w, 0, u, w->ndof, true, true, a));
        WDG_TRY(exact_rk4(h, a.dev, dt, *t, nsteps, nullptr, 0.0, nullptr, nullptr));
        for (int s = 0; s < nsteps; ++s)
            *t += dt; // ode::RungeKutta4::step advances t once per step
        return finish_args(w, &a, 1);
    }
}
