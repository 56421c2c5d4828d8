// Fused kernel of the conservation-law path: u_t + div F(u) = 0 with nodal DG on GLL nodes,
// approximate quadrature, one launch per RHS evaluation or time-stepping stage.
//
//   volume   per node the contravariant fluxes of F(u) and the D contraction (DivF2D<true>::action,
//            wavedg/DivF.hpp:203-260; Div<true> for a linear flux);
//   faces    per face node the numerical flux with the element's own outward normal, subtracted
//            times w_k |E| / 2 (EdgeFluxF2D<true>::action, wavedg/EdgeFluxF.hpp:138-180, with the sign
//            flip and transpose prolongation of examples/cl2d.cpp:175-219); the neighbour's trace is
//            read from the stage's input through the partner table of the fused wave kernels;
//   mass     M^{-1} = 1 / (w_i w_j det J) (MassMatrix<true>);
//   output   the RHS, or one stage of ode::RungeKutta4 or ode::SSPRK3 (wavedg/ode.hpp:66-93,
//            145-186) applied in the same pass.
// Each face contribution uses the element's own normal and the numerical flux's antisymmetry,
// which holds exactly in floating point for both models, so the two elements of an edge add exactly
// opposite terms, as the reference's edge loop does.
//
// A CTA is one warp, persistent over groups of EW = 32 / N whole elements, a lane per grid line with
// all variables:
//   column pass  lane (element, column i): eta-fluxes node by node, contracted at once with D
//                (constant-bank operands), the two face nodes of sides 0 and 2, the sums to shared memory
//   row pass     lane (element, row j): xi-fluxes likewise, sides 3 and 1, + the column sums, M^{-1},
//                the update in place
// State and register come and go by cp.async.bulk, one copy per element (padded element strides keep
// the passes off each other's banks), where an element is a whole number of 16-byte units and the arrays are
// aligned, else by 8-byte copies and plain stores (one and three variables at odd n); the neighbour traces of the next group are gathered with
// cp.async as soon as the current group is done with its own, their table entries loaded a group
// ahead.  A warp never waits for another one.
//
// What bounds it: the FP64 chains of a line at ten resident warps per SM (the staging of six elements
// is 19 KB for the Euler system at N = 5; shared-memory pipe 49 % busy, one instruction issued every
// 4 to 5 cycles and scheduler).  256 x 256, N = 5: Euler SSPRK3 stage 241 -> 73 us, linear n_var 2
// RK4 stage 123 -> 44 us against a warp per element with a lane per node, which spent 1800 warp
// instructions per Euler element on index arithmetic and per-node metrics (now 456).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <vector>

#include "claw_model.cuh"
#include "common.hpp"
#include "launch.hpp"
#include "ptx.cuh"
#include "wave_impl.hpp"

namespace wdg
{
    namespace
    {
        struct LineTab
        {
            double D[kMaxN + 1][kMaxN * kMaxN], x[kMaxN + 1][kMaxN], w[kMaxN + 1][kMaxN]; // D[n][l n + j] = phi_j'(x_l)
        };
        __constant__ LineTab c_line;

        int upload_line_tables(int device)
        {
            DeviceScope scope(device);
            static std::mutex mu;
            static uint64_t done = 0;
            std::lock_guard<std::mutex> lock(mu);
            if (done & (1ull << (device & 63)))
                return WDG_OK;
            std::vector<LineTab> t(1);
            for (int n = kMinN; n <= kMaxN; ++n)
            {
                std::vector<double> D((size_t)n * n);
                gauss_lobatto(n, t[0].x[n], t[0].w[n]);
                deriv_matrix(n, t[0].x[n], D.data()); // D[l + n j]
                for (int l = 0; l < n; ++l)
                    for (int j = 0; j < n; ++j)
                        t[0].D[n][l * n + j] = D[l + n * j];
            }
            WDG_CUDA(cudaMemcpyToSymbol(c_line, t.data(), sizeof(LineTab)));
            done |= 1ull << (device & 63);
            return WDG_OK;
        }

        // wavefronts of a warp's access of `width` doubles a lane, lane (element, line) at line * a +
        // element * e: 32 / (2 width) lanes go out together, conflict-free on different 8 width-byte banks
        constexpr int l_waves(int n, int ew, int a, int e, int width)
        {
            int waves = 0;
            const int per = 16 / width;
            for (int h = 0; h < 32 / per; ++h)
            {
                int cnt[16] = {}, most = 0;
                for (int i = per * h; i < per * (h + 1) && i < n * ew; ++i)
                {
                    const int at = ((i / n) * e + (i % n) * a) / width % per;
                    if (++cnt[at] > most)
                        most = cnt[at];
                }
                waves += most;
            }
            return waves;
        }
        struct LineStride
        {
            int eu, s1, eh;
        };
        constexpr LineStride l_strides(int n, int nv, int ew)
        {
            const int w = nv % 2 == 0 ? 2 : 1, nd = nv * n * n;
            LineStride b{nd + (nd & 1), n, 0};
            int cost = 1 << 30;
            for (int eu = nd + (nd & 1); eu < nd + 18; eu += 2)
            {
                const int c = 8 * (l_waves(n, ew, nv, eu, w) + l_waves(n, ew, nv * n, eu, w)) + (eu - nd);
                if (c < cost)
                {
                    cost = c;
                    b.eu = eu;
                }
            }
            cost = 1 << 30;
            for (int s1 = n; s1 < n + 6; ++s1)
                for (int pad = 0; pad < 16; ++pad)
                {
                    const int eh = nv * n * s1 + pad;
                    const int c = 16 * (l_waves(n, ew, s1, eh, 1) + l_waves(n, ew, 1, eh, 1)) + (eh - nd) / 4;
                    if (c < cost)
                    {
                        cost = c;
                        b.s1 = s1;
                        b.eh = eh;
                    }
                }
            return b;
        }

        template <int N, int NV, class M>
        struct LineShape
        {
            static constexpr int NN = N * N, ND = NV * NN;
            static constexpr int AB = M::LINEAR ? 4 * NV * NV : 0; // |n.A| of the four sides
            // elements per warp: a lane per line, less where the staging of many variables would leave
            // fewer than five warps on an SM
            static constexpr int fit = (44 * 1024 / 8) / (3 * ND + 4 * N * NV + AB + 24);
            static constexpr int EW = 32 / N < fit ? 32 / N : (fit < 1 ? 1 : fit);
            static constexpr LineStride ST = l_strides(N, NV, EW);
            static constexpr int EU = ST.eu, S1 = ST.s1, EH = ST.eh, ET = 4 * N * NV;
            // doubles: state | register | neighbour traces | |n.A| | corners | column sums | mbarrier
            static constexpr int oK = EW * EU, oT = 2 * EW * EU, oA = oT + EW * ET, oC = oA + EW * AB, oH = oC + EW * 8,
                                 oB = (oH + EW * EH + 1) & ~1, total = oB + 2;
            static constexpr size_t smem = sizeof(double) * (size_t)total;
            static_assert(smem <= 227 * 1024, "a warp's elements fit shared memory");
            static constexpr int FIT = (int)(227 * 1024 / (smem + 1024));
            // the warps that the registers a line's sums and state want leave room for; an SM's quarters hold
            // them, so that 13 warps get those of 16 (128 a thread) and 9 those of 12 (168), and some shapes spill
            // (n = 5, n_var 2: 100 bytes; n = 2, n_var 7: 700)
            static constexpr int REGS = 65536 / 32 / (4 * N * NV + 110 < 255 ? 4 * N * NV + 110 : 255);
            static constexpr int MINB = FIT < 1 ? 1 : FIT > REGS ? REGS : FIT;
            static constexpr bool BULK = ND % 2 == 0; // whole 16-byte units per element
            // node loops stay rolled where a line's sums are many: unrolled, their hoisted loads spill
            static constexpr int UNROLL = N * NV > 15 ? 1 : N;
        };

        // constant coefficients go with the launch, so that they are constant-bank operands
        template <int NV, class M>
        struct LineArgs
        {
            ClawArgs c;
            double A[M::LINEAR ? 2 * NV * NV : 1];
        };

        // NV consecutive values, in 16-byte pieces where they are aligned
        template <int NV>
        __device__ __forceinline__ void l_get(const double *p, double *q)
        {
            if constexpr (NV % 2 == 0)
            {
#pragma unroll
                for (int d = 0; d < NV; d += 2)
                {
                    const double2 v = *reinterpret_cast<const double2 *>(p + d);
                    q[d] = v.x;
                    q[d + 1] = v.y;
                }
            }
            else
#pragma unroll
                for (int d = 0; d < NV; ++d)
                    q[d] = p[d];
        }
        template <int NV>
        __device__ __forceinline__ void l_put(double *p, const double *q)
        {
            if constexpr (NV % 2 == 0)
            {
#pragma unroll
                for (int d = 0; d < NV; d += 2)
                    *reinterpret_cast<double2 *>(p + d) = make_double2(q[d], q[d + 1]);
            }
            else
#pragma unroll
                for (int d = 0; d < NV; ++d)
                    p[d] = q[d];
        }

        // what the element adds at one face node: own state q, side s, weight w_k |E| / 2 with the normal
        // from the side's corners
        template <int NV, class M, int SIDE>
        __device__ __forceinline__ void l_face(uint32_t codes, const double *c, double wk, const double *coef,
                                               const double *absA, const double *q, const double *t, double *r)
        {
            // side s runs from corner p0 to p1: 0: 0 -> 1, 1: 1 -> 2, 2: 3 -> 2, 3: 0 -> 3
            constexpr int p0 = (SIDE == 0 || SIDE == 3) ? 0 : (SIDE == 1 ? 1 : 3), p1 = (SIDE == 0) ? 1 : (SIDE == 3 ? 3 : 2);
            const double dx = c[2 * p1] - c[2 * p0], dy = c[2 * p1 + 1] - c[2 * p0 + 1];
            const double s2 = dx * dx + dy * dy, rs = rsqrt(s2), sgn = (SIDE >= 2) ? -1.0 : 1.0;
            const double nx = sgn * dy * rs, ny = -sgn * dx * rs;
            double x[NV];
            if (codes & (0x80u << (8 * SIDE)))
                M::template exterior<NV>(q, x);
            else
                l_get<NV>(t, x);
            M::template face<NV>(coef, absA, nx, ny, -0.25 * wk * (s2 * rs), q, x, r);
        }

        template <int N, int NV, class M>
        __global__ void __launch_bounds__(32, LineShape<N, NV, M>::MINB) claw_line_kernel(const __grid_constant__ LineArgs<NV, M> args)
        {
            const ClawArgs &a = args.c;
            const double *coef = args.A;
            using S = LineShape<N, NV, M>;
            constexpr int NN = S::NN, ND = S::ND, EW = S::EW, EU = S::EU, S1 = S::S1;
            extern __shared__ __align__(128) double lsm[];
            const int lane = threadIdx.x, G = gridDim.x;
            double *U = lsm, *K = lsm + S::oK, *T = lsm + S::oT, *AB = lsm + S::oA, *C = lsm + S::oC, *H = lsm + S::oH;
            uint64_t *full = reinterpret_cast<uint64_t *>(lsm + S::oB);
            const double *D = c_line.D[N], *xn = c_line.x[N], *wn = c_line.w[N];
            const int le = lane / N, ln = lane - le * N;
            const int ngroups = (a.nel + EW - 1) / EW;
            // what the pass reads beside its input and writes beside its output (null: nothing)
            const double *prev = (a.mode == CLAW_RK4)                            ? (a.rk_a == 0.0 ? nullptr : a.du)
                                 : (a.mode == CLAW_SSP1 || a.mode == CLAW_SSP2) ? a.base
                                 : (a.mode == CLAW_DIV)                         ? a.out
                                                                                : nullptr;
            double *reg = (a.mode == CLAW_RK4) ? a.du : nullptr;
            const bool bulk = S::BULK && a.aligned;
            if (lane == 0)
            {
                mbar_init(full, 1);
                fence_mbar_init();
            }
            __syncwarp();

            constexpr int IT = (EW * 4 * N + 31) / 32; // face nodes per lane
            uint32_t byte[IT];
            int off[IT];
            // side codes and partner offsets of this lane's face nodes of group g (the volume term alone wants none)
            auto tables = [&](int g)
            {
#pragma unroll
                for (int t = 0; t < IT; ++t)
                {
                    const int o = lane + 32 * t, el = g * EW + o / (4 * N), s = (o / N) & 3;
                    byte[t] = 0x80u;
                    off[t] = -1;
                    if ((M::LINEAR || a.mode != CLAW_DIV) && g < ngroups && o < EW * 4 * N && el < a.nel)
                    {
                        byte[t] = (__ldg(a.fcode + el) >> (8 * s)) & 0xffu;
                        off[t] = __ldg(reinterpret_cast<const int *>(a.fbase + el) + s);
                    }
                }
            };
            // the neighbour traces T(s, k, d); an index outside the state is reported and not read
            auto gather = [&]()
            {
#pragma unroll
                for (int t = 0; t < IT; ++t)
                {
                    const int o = lane + 32 * t, k = o % N;
                    if (byte[t] & 0x80u)
                        continue;
                    const uint32_t sc = byte[t] & 3u;
                    const int stride = (sc == 0) ? 1 : (sc == 1) ? -1 : (sc == 2) ? N : -N; // in nodes
                    const long long pn = (long long)(off[t] / 3) + (long long)k * stride;
                    double *dst = T + (size_t)NV * o;
                    if (off[t] < 0 || pn < 0 || pn >= (long long)a.nel * NN)
                    {
                        atomicOr(a.err, 2u);
#pragma unroll
                        for (int d = 0; d < NV; ++d)
                            dst[d] = 1.0;
                    }
                    else if (NV % 2 == 0 && a.aligned)
#pragma unroll
                        for (int d = 0; d + 1 < NV; d += 2)
                            cp_async<16>(dst + d, a.x + (size_t)NV * pn + d);
                    else
#pragma unroll
                        for (int d = 0; d < NV; ++d)
                            cp_async<8>(dst + d, a.x + (size_t)NV * pn + d);
                }
            };
            // state, register, corners and |n.A| of group g
            auto load = [&](int g)
            {
                const int e0 = g * EW, ne = min(EW, a.nel - e0);
                if (bulk)
                {
                    if (lane == 0)
                        mbar_expect_tx(full, (uint32_t)(ne * (8 * (ND * (prev ? 2 : 1) + S::AB) + 64)));
                    __syncwarp();
                    if (lane < ne)
                    {
                        const size_t e = (size_t)(e0 + lane);
                        bulk_g2s(U + lane * EU, a.x + e * ND, 8 * ND, full);
                        if (prev)
                            bulk_g2s(K + lane * EU, prev + e * ND, 8 * ND, full);
                        bulk_g2s(C + lane * 8, a.corners + 8 * e, 64, full);
                        if constexpr (M::LINEAR)
                            bulk_g2s(AB + lane * S::AB, a.absA + e * S::AB, 8 * S::AB, full);
                    }
                }
                else
                {
                    for (int o = lane; o < ne * ND; o += 32)
                    {
                        const int at = (o / ND) * EU + o % ND;
                        cp_async<8>(U + at, a.x + (size_t)e0 * ND + o);
                        if (prev)
                            cp_async<8>(K + at, prev + (size_t)e0 * ND + o);
                    }
                    for (int o = lane; o < ne * 8; o += 32)
                        cp_async<8>(C + o, a.corners + 8 * (size_t)e0 + o);
                    if constexpr (M::LINEAR)
                        for (int o = lane; o < ne * S::AB; o += 32)
                            cp_async<8>(AB + o, a.absA + (size_t)e0 * S::AB + o);
                }
            };

            int g = blockIdx.x;
            if (g >= ngroups)
                return;
            tables(g);
            load(g);
            gather();
            cp_async_commit();
            bool ok = true;
            for (int m = 0; g < ngroups; ++m, g += G)
            {
                const int e0 = g * EW, ne = min(EW, a.nel - e0);
                const bool on = le < ne && lane < EW * N;
                const uint32_t codes = on ? __ldg(a.fcode + e0 + le) : 0u;
                tables(g + G);
                if (bulk && !__all_sync(0xffffffffu, mbar_wait(full, m & 1)))
                {
                    ok = false;
                    break;
                }
                cp_async_wait<0>();
                __syncwarp();
                double c[8];
                if (on)
                {
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        c[k] = C[8 * le + k];
                }
                const double *Te = T + (on ? le * S::ET : 0), *Ae = AB + (on ? le * S::AB : 0);
                double *Ue = U + (on ? le * EU : 0), *Ke = K + (on ? le * EU : 0), *He = H + (on ? le * S::EH : 0);
                const double xl = on ? xn[ln] : 0.0, wl = on ? wn[ln] : 0.0;
                if (on)
                {
                    // ---- column i = ln
                    double s[N][NV];
#pragma unroll
                    for (int j = 0; j < N; ++j)
#pragma unroll
                        for (int d = 0; d < NV; ++d)
                            s[j][d] = 0.0;
#pragma unroll S::UNROLL
                    for (int l = 0; l < N; ++l)
                    {
                        double q[NV], f[NV];
                        l_get<NV>(Ue + NV * (ln + N * l), q);
                        const double W = wl * wn[l];
                        const double Xx = 0.25 * ((1.0 - xn[l]) * (c[2] - c[0]) + (1.0 + xn[l]) * (c[4] - c[6]));
                        const double Yx = 0.25 * ((1.0 - xn[l]) * (c[3] - c[1]) + (1.0 + xn[l]) * (c[5] - c[7]));
                        M::template flux<NV>(coef, -(W * Yx), W * Xx, q, f);
#pragma unroll
                        for (int j = 0; j < N; ++j)
#pragma unroll
                            for (int d = 0; d < NV; ++d)
                                s[j][d] += D[l * N + j] * f[d];
                        if (a.mode != CLAW_DIV)
                        {
                            if (l == 0)
                                l_face<NV, M, 0>(codes, c, wl, coef, Ae, q, Te + NV * ln, s[0]);
                            if (l == N - 1)
                                l_face<NV, M, 2>(codes, c, wl, coef, Ae + 2 * NV * NV, q, Te + NV * (2 * N + ln),
                                                 s[N - 1]);
                        }
                    }
#pragma unroll
                    for (int j = 0; j < N; ++j)
#pragma unroll
                        for (int d = 0; d < NV; ++d)
                            He[(d * N + ln) * S1 + j] = s[j][d];
                }
                __syncwarp();
                if (on)
                {
                    // ---- row j = ln: along a row x_xi, y_xi are constant
                    const double Xx = 0.25 * ((1.0 - xl) * (c[2] - c[0]) + (1.0 + xl) * (c[4] - c[6]));
                    const double Yx = 0.25 * ((1.0 - xl) * (c[3] - c[1]) + (1.0 + xl) * (c[5] - c[7]));
                    double r[N][NV];
#pragma unroll
                    for (int i = 0; i < N; ++i)
#pragma unroll
                        for (int d = 0; d < NV; ++d)
                            r[i][d] = He[(d * N + i) * S1 + ln];
#pragma unroll S::UNROLL
                    for (int l = 0; l < N; ++l)
                    {
                        double q[NV], f[NV];
                        l_get<NV>(Ue + NV * (l + N * ln), q);
                        const double W = wl * wn[l];
                        const double Xe = 0.25 * ((1.0 - xn[l]) * (c[6] - c[0]) + (1.0 + xn[l]) * (c[4] - c[2]));
                        const double Ye = 0.25 * ((1.0 - xn[l]) * (c[7] - c[1]) + (1.0 + xn[l]) * (c[5] - c[3]));
                        M::template flux<NV>(coef, W * Ye, -(W * Xe), q, f);
#pragma unroll
                        for (int i = 0; i < N; ++i)
#pragma unroll
                            for (int d = 0; d < NV; ++d)
                                r[i][d] += D[l * N + i] * f[d];
                        if (a.mode != CLAW_DIV)
                        {
                            if (l == 0)
                                l_face<NV, M, 3>(codes, c, wl, coef, Ae + 3 * NV * NV, q, Te + NV * (3 * N + ln), r[0]);
                            if (l == N - 1)
                                l_face<NV, M, 1>(codes, c, wl, coef, Ae + NV * NV, q, Te + NV * (N + ln), r[N - 1]);
                        }
                    }
                    // ---- M^{-1} and the update, in place: the row is this lane's alone
#pragma unroll
                    for (int i = 0; i < N; ++i)
                    {
                        double *un = Ue + NV * (i + N * ln), *kn = Ke + NV * (i + N * ln);
                        double q[NV], p[NV], y[NV];
                        // MassMatrix<true>: w_i w_j det J
                        const double Xe = 0.25 * ((1.0 - xn[i]) * (c[6] - c[0]) + (1.0 + xn[i]) * (c[4] - c[2]));
                        const double Ye = 0.25 * ((1.0 - xn[i]) * (c[7] - c[1]) + (1.0 + xn[i]) * (c[5] - c[3]));
                        const double mi = (a.mode == CLAW_DIV) ? 1.0 : 1.0 / (wl * wn[i] * (Xx * Ye - Yx * Xe));
#pragma unroll
                        for (int d = 0; d < NV; ++d)
                            y[d] = r[i][d] * mi;
                        if (a.mode == CLAW_RK4)
                        {
                            l_get<NV>(un, q);
                            if (prev)
                                l_get<NV>(kn, p);
#pragma unroll
                            for (int d = 0; d < NV; ++d)
                            {
                                y[d] = prev ? a.rk_a * p[d] + a.dt * y[d] : a.dt * y[d];
                                q[d] += a.rk_b * y[d];
                            }
                            l_put<NV>(kn, y);
                            l_put<NV>(un, q);
                            continue;
                        }
                        if (a.mode != CLAW_RHS)
                        {
                            l_get<NV>(un, q);
                            if (prev)
                                l_get<NV>(kn, p);
#pragma unroll
                            for (int d = 0; d < NV; ++d)
                                y[d] = (a.mode == CLAW_SSP0)   ? q[d] + a.dt * y[d]
                                       : (a.mode == CLAW_SSP1) ? 0.25 * (q[d] + 3.0 * p[d] + a.dt * y[d])
                                       : (a.mode == CLAW_SSP2) ? (p[d] + 2.0 * q[d] + 2.0 * a.dt * y[d]) / 3.0
                                                               : p[d] + y[d]; // CLAW_DIV
                        }
                        l_put<NV>(un, y);
                    }
                }
                // ---- out, and the next group in
                if (bulk)
                {
                    fence_async_smem();
                    __syncwarp();
                    if (lane < ne)
                    {
                        const size_t e = (size_t)(e0 + lane);
                        bulk_s2g(a.out + e * ND, U + lane * EU, 8 * ND);
                        if (reg)
                            bulk_s2g(reg + e * ND, K + lane * EU, 8 * ND);
                        bulk_commit();
                    }
                }
                else
                {
                    __syncwarp();
                    for (int o = lane; o < ne * ND; o += 32)
                    {
                        const int at = (o / ND) * EU + o % ND;
                        a.out[(size_t)e0 * ND + o] = U[at];
                        if (reg)
                            reg[(size_t)e0 * ND + o] = K[at];
                    }
                }
                if (g + G < ngroups)
                {
                    gather();
                    bulk_wait_read(); // this lane's stores have read the staging
                    __syncwarp();
                    load(g + G);
                    cp_async_commit();
                }
            }
            if (!ok && lane == 0)
                atomicOr(a.err, 1u);
            cp_async_wait<0>();
            bulk_wait_all();
        }

        // EdgeFluxF2D<true>::action for the Euler system on face traces (n, 4, 2, edges): thread per
        // (face node, edge); fB = +- w_i |E| / 2 fh(n, side 0, side 1), n the outward normal of the
        // edge's first element (in place allowed: a thread reads its node's traces before writing)
        __global__ void euler_face_flux_kernel(int n, int ne, const int *__restrict__ edges,
                                               const double *__restrict__ corners, const double *ub, double *fb)
        {
            const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
            if (q >= (long long)n * ne)
                return;
            const int i = (int)(q % n), e = (int)(q / n);
            const int el = edges[5 * (size_t)e], s = edges[5 * (size_t)e + 1];
            double c[8];
            for (int k = 0; k < 8; ++k)
                c[k] = corners[8 * (size_t)el + k];
            double nx, ny, meas, qL[4], qR[4], fh[4] = {0.0, 0.0, 0.0, 0.0};
            claw_side(c, s, nx, ny, meas);
            for (int d = 0; d < 4; ++d)
            {
                qL[d] = ub[i + n * (d + 4 * (0 + 2 * (size_t)e))];
                qR[d] = ub[i + n * (d + 4 * (1 + 2 * (size_t)e))];
            }
            ClawEuler::face<4>(nullptr, nullptr, nx, ny, 0.5 * c_line.w[n][i] * meas, qL, qR, fh);
            for (int d = 0; d < 4; ++d)
            {
                fb[i + n * (d + 4 * (0 + 2 * (size_t)e))] = fh[d];
                fb[i + n * (d + 4 * (1 + 2 * (size_t)e))] = -fh[d];
            }
        }

        template <int N, int NV, class M>
        cudaError_t launch_nv(const ClawArgs &a, cudaStream_t s)
        {
            using S = LineShape<N, NV, M>;
            // resident CTAs of this kernel on each device, found once (and its shared memory opted in)
            static std::atomic<int> resident[64];
            int dev = 0;
            cudaGetDevice(&dev);
            int grid = resident[dev & 63].load(std::memory_order_relaxed);
            if (grid == 0)
            {
                int per_sm = 0, sms = 0;
                cudaError_t e = cudaFuncSetAttribute(claw_line_kernel<N, NV, M>,
                                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::smem);
                if (e == cudaSuccess)
                    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, claw_line_kernel<N, NV, M>, 32, S::smem);
                if (e == cudaSuccess)
                    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
                if (e != cudaSuccess)
                    return e;
                grid = std::max(1, per_sm) * sms;
                resident[dev & 63].store(grid, std::memory_order_relaxed);
            }
            const int ngroups = (a.nel + S::EW - 1) / S::EW;
            LineArgs<NV, M> args;
            args.c = a;
            for (int k = 0; k < (M::LINEAR ? 2 * NV * NV : 0); ++k)
                args.A[k] = a.A[k];
            claw_line_kernel<N, NV, M><<<std::max(1, std::min(grid, ngroups)), 32, S::smem, s>>>(args);
            return cudaGetLastError();
        }

        template <int N>
        cudaError_t launch_n(int model, int nv, const ClawArgs &a, cudaStream_t s)
        {
            if (model == 0)
                return nv == 4 ? launch_nv<N, 4, ClawEuler>(a, s) : cudaErrorInvalidValue;
            switch (nv)
            {
            case 1: return launch_nv<N, 1, ClawLinear>(a, s);
            case 2: return launch_nv<N, 2, ClawLinear>(a, s);
            case 3: return launch_nv<N, 3, ClawLinear>(a, s);
            case 4: return launch_nv<N, 4, ClawLinear>(a, s);
            case 5: return launch_nv<N, 5, ClawLinear>(a, s);
            case 6: return launch_nv<N, 6, ClawLinear>(a, s);
            case 7: return launch_nv<N, 7, ClawLinear>(a, s);
            case 8: return launch_nv<N, 8, ClawLinear>(a, s);
            default: return cudaErrorInvalidValue;
            }
        }
    } // namespace

    int claw_prepare(int device) { return upload_line_tables(device); }

    cudaError_t launch_claw(int model, int n, int nv, const ClawArgs &args, cudaStream_t s)
    {
        ClawArgs a = args;
        // bulk and 16-byte copies: every array the pass touches by them on a 16-byte boundary (the
        // handle's own are)
        a.aligned = (((uintptr_t)a.x | (uintptr_t)a.out | (uintptr_t)a.du | (uintptr_t)a.base) & 15u) == 0;
        switch (n)
        {
        case 2: return launch_n<2>(model, nv, a, s);
        case 3: return launch_n<3>(model, nv, a, s);
        case 4: return launch_n<4>(model, nv, a, s);
        case 5: return launch_n<5>(model, nv, a, s);
        case 6: return launch_n<6>(model, nv, a, s);
        case 7: return launch_n<7>(model, nv, a, s);
        case 8: return launch_n<8>(model, nv, a, s);
        case 9: return launch_n<9>(model, nv, a, s);
        default: return cudaErrorInvalidValue;
        }
    }
    cudaError_t launch_euler_face_flux(int n, int ne, const int *edges, const double *corners, const double *ub,
                                       double *fb, cudaStream_t s)
    {
        if (ne == 0)
            return cudaSuccess;
        const long long tot = (long long)n * ne;
        euler_face_flux_kernel<<<(unsigned)((tot + 127) / 128), 128, 0, s>>>(n, ne, edges, corners, ub, fb);
        return cudaGetLastError();
    }
} // namespace wdg
