// Resident RK4: many stages of the wave system in one launch, the elements staying on chip.
//
// A mesh whose state, RK register and per-element tables fit the shared memory of the chip needs HBM
// for nothing but its first load and last store.  One cooperative launch (one CTA per SM) runs all
// stages of nsteps steps; every warp owns whole groups of EW = 32 / N elements for the launch and
// steps them with the line passes of wave_line.cuh, bit for bit what the streaming kernel
// (stage_ws.cuh) computes.  Between stages only the sides' traces travel, through two buffers in L2
// (element, side, node, field padded to four), so that a face node is one access and a side is
// contiguous.
//
// Synchronisation is between neighbouring groups only.  A group's flag counts the traces it has
// published (released after them); before its face terms a group waits until its neighbours' flags
// show theirs.  Stage s reads buffer s & 1 and publishes its result to the other one: a group that has
// seen its neighbours' traces of stage s knows that they are done reading its own of stage s - 1,
// which it overwrites next (the neighbour relation is symmetric).  The column sums of the
// volume term are formed before the wait, so the flag's way through L2 is mostly hidden.  Flags
// only grow: every launch counts on from the handle's last value.  Every wait is bounded by the
// handle's limit; a warp whose wait runs out records it and leaves, and the others follow.
//
// What is formed once per launch instead of once per stage: the sides' normals and measures and the
// inverse mass at the nodes.
//
// What bounds it: the latency of a group's chain (column sums, flags, traces, row sums, update) with
// ten warps per SM, and the shared-memory pipe behind it (about 480 wavefronts per group and stage);
// with one group per warp, the chain alone.  Per stage, FP64: 128 x 128, N = 5: 17.4 -> 7.7 us (forced
// and unforced periods of WaveHoltz together), 32 x 32, N = 4: 8.2 -> 2.7 us against stage launches.
// Tried, when the first stood at 9.1 us: flags released late, after the next group's column sums (9.5 us); traces read in the state's
// layout (12.2 us), staged through shared memory (11.0 us), in 16-byte pieces (10.4 us).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "ptx.cuh"
#include "wave_impl.hpp"
#include "wave_line.cuh"

namespace wdg
{
    namespace
    {
        constexpr int kResMaxWarps = 12; // 170 registers a thread
        constexpr int kFlagStride = 4;   // flags 32 bytes apart: one sector each

        template <typename Real>
        struct ResArgs
        {
            Real *A;    // state, in and out
            Real *T[2]; // trace buffers (element, side, node, 4)
            const double *corners;
            const int4 *fbase;
            const uint32_t *fcode;
            unsigned long long *flags, base;
            unsigned *err;
            int nel, ngroups, nsteps;
            Real a[5], b[5], dt;
            const Real *F;         // forcing (nullable) times fscale[5 step + stage]
            const double *fscale;
            double *acc;           // FP64 filter (nullable): += cfilter[step] u after each step
            const double *cfilter;
            unsigned long long wait_ns;
            int test_skip; // test hook: the group whose warp leaves before the first stage (-1: none)
        };

        // one group's shared memory (bytes)
        struct ResLayout
        {
            int u, k, m, s, c, t, w, code, bytes;
        };
        template <typename Real>
        __host__ __device__ constexpr ResLayout res_layout(int n)
        {
            ResLayout L{};
            const int ew = 32 / n, nn = n * n, r = (int)sizeof(Real);
            L.c = 0;                       // corners (8 doubles per element)
            L.u = L.c + ew * 64;           // state
            L.k = L.u + ew * 3 * nn * r;   // RK register
            L.m = L.k + ew * 3 * nn * r;   // inverse mass
            L.s = L.m + ew * nn * r;       // sides: n_x, n_y, length / 4 (13 apart: different banks)
            L.t = (L.s + ew * 13 * r + 15) & ~15;       // per side: where the neighbour's trace begins (-1: nowhere)
            L.w = L.t + ew * 16;           // the neighbours' groups
            L.code = L.w + ew * 16;        // side codes (bits 0, 6: the neighbour's trace runs backwards, is missing)
            L.bytes = (L.code + ew * 4 + 15) & ~15;
            return L;
        }
        // FP32 stepping adds the forcing where the streaming kernel does, to the row's finished sums, so that
        // batches of either kind give the same bits; its values then need a place of their own.  FP64 adds it
        // to the column's sums and lets it share the scratch: that place would cost a warp or two.
        template <typename Real>
        constexpr bool kLateForcing = sizeof(Real) == 4;
        __host__ __device__ constexpr int res_forcing(int n, int real)
        {
            return real == 4 ? ((32 / n) * 3 * n * n * real + 15) & ~15 : 0;
        }
        // a warp's scratch: the forcing (FP64), then the column sums of a group
        __host__ __device__ constexpr int res_scratch(int n, SumStride sums, int real)
        {
            return ((32 / n) * sums.el * real + 15) & ~15;
        }

        __device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long *p)
        {
            unsigned long long v;
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
            return v;
        }
        __device__ __forceinline__ void st_release(unsigned long long *p, unsigned long long v)
        {
            asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
        }
        // until the flag reaches `want`; false when the limit runs out or another warp's did
        __device__ __forceinline__ bool res_wait(const unsigned long long *flag, unsigned long long want, unsigned *err,
                                                 uint64_t limit_ns)
        {
            if (ld_acquire(flag) >= want)
                return true;
            const uint64_t t0 = globaltimer_ns();
            for (;;)
            {
                for (int q = 0; q < 32; ++q)
                    if (ld_acquire(flag) >= want)
                        return true;
                if (globaltimer_ns() - t0 > limit_ns || (*(volatile unsigned *)err & 1u))
                    return false;
            }
        }

        template <int N, typename Real>
        __global__ void __launch_bounds__(32 * kResMaxWarps, 1) res_kernel(const ResArgs<Real> a)
        {
            constexpr int NN = N * N, ND = 3 * NN, EW = 32 / N;
            constexpr ResLayout L = res_layout<Real>(N);
            extern __shared__ __align__(128) unsigned char rsm[];
            const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, W = blockDim.x >> 5;
            const int g_lo = (int)((long long)blockIdx.x * a.ngroups / gridDim.x);
            const int ng = (int)((long long)(blockIdx.x + 1) * a.ngroups / gridDim.x) - g_lo; // this CTA's groups
            const int most = (a.ngroups + gridDim.x - 1) / gridDim.x;
            unsigned char *groups = rsm;
            constexpr SumStride RS = sum_strides(N);
            constexpr int kScratch = res_scratch(N, RS, sizeof(Real));
            constexpr bool LATE = kLateForcing<Real>;
            const int scratch = kScratch + (a.F ? res_forcing(N, sizeof(Real)) : 0);
            Real *Rc = reinterpret_cast<Real *>(groups + (size_t)most * L.bytes + (size_t)warp * scratch);
            Real *Fc = LATE ? Rc + kScratch / (int)sizeof(Real) : Rc; // the group's forcing
            const int le = lane / N, ln = lane - le * N;
            const bool lane_on = lane < EW * N;
            const Real xm = lane_on ? Tab<Real>::x(N, ln) : Real(0), wm = lane_on ? Tab<Real>::w(N, ln) : Real(0);
            const uint64_t wlim = wait_limit(a.wait_ns);

            // ---- this warp's groups: state, corners, tables; side geometry and inverse mass
            for (int sl = warp; sl < ng; sl += W)
            {
                unsigned char *gb = groups + (size_t)sl * L.bytes;
                const int e0 = (g_lo + sl) * EW, ne = min(EW, a.nel - e0);
                Real *U = reinterpret_cast<Real *>(gb + L.u);
                double *C = reinterpret_cast<double *>(gb + L.c);
                for (int o = lane; o < ne * ND; o += 32)
                    cp_async<sizeof(Real)>(U + o, a.A + (size_t)e0 * ND + o);
                for (int o = lane; o < ne * 8; o += 32)
                    cp_async<8>(C + o, a.corners + 8 * (size_t)e0 + o);
                cp_async_commit();
                int *Tn = reinterpret_cast<int *>(gb + L.t), *Wn = reinterpret_cast<int *>(gb + L.w);
                uint32_t *code = reinterpret_cast<uint32_t *>(gb + L.code);
                for (int o = lane; o < ne; o += 32)
                {
                    uint32_t cd = __ldg(a.fcode + e0 + o);
                    const int4 fb = __ldg(a.fbase + e0 + o);
#pragma unroll
                    for (int s = 0; s < 4; ++s)
                    {
                        const int off = (s == 0) ? fb.x : (s == 1) ? fb.y : (s == 2) ? fb.z : fb.w;
                        const uint32_t byte = (cd >> (8 * s)) & 0xffu;
                        int own = -1, at = -1;
                        if (!(byte & 0x80u))
                        {
                            // an index outside the state is reported and its side left out
                            const int end = off + (N - 1) * partner_stride<N>(byte);
                            if (off < 0 || end < 0 || off + 3 > a.nel * ND || end + 3 > a.nel * ND)
                            {
                                atomicOr(a.err, 2u);
                                cd |= 0x40u << (8 * s);
                            }
                            else
                            {
                                // the neighbour's side from where its face-node facing node 0 lies and
                                // the walk along it
                                const int nd = off / 3 % NN, sc = byte & 3u;
                                const int ns = sc < 2 ? (nd / N == 0 ? 0 : 2) : (nd % N == 0 ? 3 : 1);
                                own = off / ND / EW;
                                at = (off / ND * 4 + ns) * N;
                                cd = (cd & ~(3u << (8 * s))) | ((uint32_t)(sc & 1) << (8 * s));
                            }
                        }
                        Tn[4 * o + s] = at;
                        Wn[4 * o + s] = own;
                    }
                    code[o] = cd;
                }
            }
            cp_async_wait<0>();
            __syncwarp();
            for (int sl = warp; sl < ng; sl += W)
            {
                unsigned char *gb = groups + (size_t)sl * L.bytes;
                const int ne = min(EW, a.nel - (g_lo + sl) * EW);
                if (!lane_on || le >= ne)
                    continue;
                const double2 *c2 = reinterpret_cast<const double2 *>(gb + L.c) + 4 * le;
                const double2 c01 = c2[0], c23 = c2[1], c45 = c2[2], c67 = c2[3];
                Real *Sg = reinterpret_cast<Real *>(gb + L.s) + 13 * le, *Mi = reinterpret_cast<Real *>(gb + L.m) + NN * le;
                if (ln == 0)
                {
                    line_side<Real, 0>(c01, c23, c45, c67, Sg[0], Sg[1], Sg[2]);
                    line_side<Real, 1>(c01, c23, c45, c67, Sg[3], Sg[4], Sg[5]);
                }
                if (ln == 1)
                {
                    line_side<Real, 2>(c01, c23, c45, c67, Sg[6], Sg[7], Sg[8]);
                    line_side<Real, 3>(c01, c23, c45, c67, Sg[9], Sg[10], Sg[11]);
                }
                Real z[N] = {}, mv[N];
                line_row<N, Real, true>(c01, c23, c45, c67, xm, wm, false, z, z, z, z, z, z, mv);
#pragma unroll
                for (int i = 0; i < N; ++i)
                    Mi[N * ln + i] = mv[i];
            }
            __syncwarp();

            // one face node's values to or from a trace buffer (L2 only on the way in: other SMs write it)
            auto put = [](Real *t, Real p, Real u, Real v)
            {
                if constexpr (sizeof(Real) == 8)
                {
                    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(t), "d"(p), "d"(u), "d"(v), "d"(0.0)
                                 : "memory");
                }
                else
                    *reinterpret_cast<float4 *>(t) = make_float4(p, u, v, 0.f);
            };
            auto get = [](const Real *t, Real (&x)[3])
            {
                if constexpr (sizeof(Real) == 8)
                {
                    double pad;
                    asm volatile("ld.global.cg.v4.f64 {%0, %1, %2, %3}, [%4];"
                                 : "=d"(x[0]), "=d"(x[1]), "=d"(x[2]), "=d"(pad)
                                 : "l"(t)
                                 : "memory");
                }
                else
                {
                    const float4 a0 = __ldcg(reinterpret_cast<const float4 *>(t));
                    x[0] = a0.x;
                    x[1] = a0.y;
                    x[2] = a0.z;
                }
            };
            // row j of element el (values q, a node apart 3): its face nodes' place in trace buffer T
            auto publish_row = [&](Real *T, int el, int j, auto q)
            {
                Real *t = T + (size_t)el * (16 * N);
                put(t + (3 * N + j) * 4, q(0, 0), q(0, 1), q(0, 2));
                put(t + (N + j) * 4, q(N - 1, 0), q(N - 1, 1), q(N - 1, 2));
                if (j == 0 || j == N - 1)
#pragma unroll
                    for (int i = 0; i < N; ++i)
                        put(t + ((j == 0 ? 0 : 2 * N) + i) * 4, q(i, 0), q(i, 1), q(i, 2));
            };
            for (int sl = warp; sl < ng; sl += W)
            {
                unsigned char *gb = groups + (size_t)sl * L.bytes;
                const int g = g_lo + sl, ne = min(EW, a.nel - g * EW);
                if (lane_on && le < ne)
                {
                    const Real *row = reinterpret_cast<const Real *>(gb + L.u) + le * ND + 3 * N * ln;
                    publish_row(a.T[0], g * EW + le, ln, [&](int i, int d) { return row[3 * i + d]; });
                }
                __syncwarp();
                if (lane == 0)
                    st_release(a.flags + (size_t)kFlagStride * g, a.base + 1);
            }

            // test hook: no flag of this warp's groups goes on, so their neighbours' waits run out
            if (a.test_skip >= g_lo && a.test_skip < g_lo + ng && (a.test_skip - g_lo) % W == warp)
                return;

            // ---- the stages
            const int nst = 5 * a.nsteps;
            bool ok = true;
            for (int stg = 0, st = 0, step = 0; stg < nst && ok; ++stg)
            {
                const Real *src = a.T[stg & 1];
                Real *dst = a.T[(stg + 1) & 1];
                const bool last = stg == nst - 1, has_du = st > 0;
                const Real fs = a.F ? (Real)__ldg(a.fscale + stg) : Real(0);
                for (int sl = warp; sl < ng; sl += W)
                {
                    unsigned char *gb = groups + (size_t)sl * L.bytes;
                    const int g = g_lo + sl, e0 = g * EW, ne = min(EW, a.nel - e0);
                    const bool act = lane_on && le < ne;
                    const int ae = act ? le : 0;
                    Real *Ue = reinterpret_cast<Real *>(gb + L.u) + ae * ND, *Ke = reinterpret_cast<Real *>(gb + L.k) + ae * ND;
                    const Real *Sg = reinterpret_cast<const Real *>(gb + L.s) + 13 * ae;
                    const Real *Mi = reinterpret_cast<const Real *>(gb + L.m) + NN * ae;
                    const uint32_t codes = reinterpret_cast<const uint32_t *>(gb + L.code)[ae];
                    const double2 *c2 = reinterpret_cast<const double2 *>(gb + L.c) + 4 * ae;
                    const double2 c01 = c2[0], c23 = c2[1], c45 = c2[2], c67 = c2[3];
                    Real *rc = Rc + ae * RS.el;
                    if (a.F)
                    {
                        for (int o = lane; o < ne * ND; o += 32)
                            cp_async<sizeof(Real)>(Fc + o, a.F + (size_t)e0 * ND + o);
                        cp_async_commit();
                    }
                    // column pass, volume (and forcing): needs nothing from the neighbours
                    Real sp[N], su[N], sv[N];
#pragma unroll
                    for (int j = 0; j < N; ++j)
                        sp[j] = su[j] = sv[j] = 0;
                    Real own0[3] = {}, own2[3] = {}; // the column's face nodes
                    if (act)
                    {
                        line_column<N, Real>(c01, c23, c45, c67, Ue, ln, wm, sp, su, sv);
#pragma unroll
                        for (int d = 0; d < 3; ++d)
                        {
                            own0[d] = Ue[3 * ln + d];
                            own2[d] = Ue[3 * (ln + N * (N - 1)) + d];
                        }
                    }
                    if (!LATE && a.F)
                    {
                        cp_async_wait<0>();
                        __syncwarp();
                        if (act)
                        {
#pragma unroll
                            for (int j = 0; j < N; ++j)
                            {
                                const Real *o = Fc + ae * ND + 3 * (ln + N * j);
                                sp[j] += fs * o[0];
                                su[j] += fs * o[1];
                                sv[j] += fs * o[2];
                            }
                        }
                        __syncwarp(); // the column sums take the forcing's place
                    }
                    bool seen = true;
                    const int *Wn = reinterpret_cast<const int *>(gb + L.w), *Tn = reinterpret_cast<const int *>(gb + L.t);
                    for (int o = lane; o < 4 * ne; o += 32)
                        if (Wn[o] >= 0)
                            seen = seen && res_wait(a.flags + (size_t)kFlagStride * Wn[o], a.base + stg + 1, a.err, wlim);
                    if (!__all_sync(0xffffffffu, seen))
                    {
                        ok = false;
                        break;
                    }
                    __syncwarp(); // a side's traces are read by other lanes than the one that acquired its flag
                    // this line's four face nodes in the neighbours' traces, all in flight together
                    Real x[4][3];
#pragma unroll
                    for (int s = 0; s < 4; ++s)
                    {
                        const int at = act ? Tn[4 * ae + s] : -1, k = ((codes >> (8 * s)) & 1u) ? N - 1 - ln : ln;
                        if (at >= 0)
                            get(src + 4 * (size_t)(at + k), x[s]);
                        else
                            x[s][0] = x[s][1] = x[s][2] = 0;
                    }
                    auto face = [&](int s, const Real *own, Real &r0, Real &r1, Real &r2)
                    {
                        const uint32_t byte = (codes >> (8 * s)) & 0xffu;
                        if (!(byte & 0x40u))
                            line_face<Real>(byte, Sg[3 * s], Sg[3 * s + 1], wm * Sg[3 * s + 2], own, x[s], r0, r1, r2);
                    };
                    if (act)
                    {
                        const int i = ln;
                        face(0, own0, sp[0], su[0], sv[0]);
                        face(2, own2, sp[N - 1], su[N - 1], sv[N - 1]);
#pragma unroll
                        for (int j = 0; j < N; ++j)
                        {
                            Real *o = rc + RS.row * j + 3 * i;
                            o[0] = sp[j];
                            o[1] = su[j];
                            o[2] = sv[j];
                        }
                    }
                    if (LATE)
                        cp_async_wait<0>();
                    __syncwarp();
                    if (act)
                    {
                        const int j = ln;
                        Real *row = Ue + 3 * N * j, *drow = Ke + 3 * N * j;
                        Real q0[N], q1[N], q2[N], ap[N], au[N], av[N], none[N];
#pragma unroll
                        for (int l = 0; l < N; ++l)
                        {
                            q0[l] = row[3 * l];
                            q1[l] = row[3 * l + 1];
                            q2[l] = row[3 * l + 2];
                            ap[l] = au[l] = av[l] = 0;
                        }
                        line_row<N, Real, false>(c01, c23, c45, c67, xm, wm, true, q0, q1, q2, ap, au, av, none);
                        const Real own3[3] = {q0[0], q1[0], q2[0]}, own1[3] = {q0[N - 1], q1[N - 1], q2[N - 1]};
                        face(3, own3, ap[0], au[0], av[0]);
                        face(1, own1, ap[N - 1], au[N - 1], av[N - 1]);
#pragma unroll
                        for (int i = 0; i < N; ++i)
                        {
                            const Real *cr = rc + RS.row * j + 3 * i;
                            const Real mv = Mi[N * j + i];
                            Real r0 = ap[i] + cr[0], r1 = au[i] + cr[1], r2 = av[i] + cr[2];
                            if (LATE && a.F)
                            {
                                const Real *f = Fc + ae * ND + 3 * (i + N * j);
                                r0 += fs * f[0];
                                r1 += fs * f[1];
                                r2 += fs * f[2];
                            }
                            r0 *= mv;
                            r1 *= mv;
                            r2 *= mv;
                            Real *dn = drow + 3 * i;
                            const Real d0 = rk_register(has_du, a.a[st], dn[0], a.dt, r0);
                            const Real d1 = rk_register(has_du, a.a[st], dn[1], a.dt, r1);
                            const Real d2 = rk_register(has_du, a.a[st], dn[2], a.dt, r2);
                            const Real u0 = rk_state(q0[i], a.b[st], d0), u1 = rk_state(q1[i], a.b[st], d1), u2 = rk_state(q2[i], a.b[st], d2);
                            dn[0] = d0;
                            dn[1] = d1;
                            dn[2] = d2;
                            row[3 * i] = q0[i] = u0;
                            row[3 * i + 1] = q1[i] = u1;
                            row[3 * i + 2] = q2[i] = u2;
                        }
                        if (!last)
                            publish_row(dst, e0 + le, j, [&](int i, int d) { return d == 0 ? q0[i] : d == 1 ? q1[i] : q2[i]; });
                    }
                    __syncwarp(); // the group's traces are written; the scratch is free
                    if (!last && lane == 0)
                        st_release(a.flags + (size_t)kFlagStride * g, a.base + stg + 2);
                    if (a.acc && st == 4)
                    {
                        // this warp alone writes these; a reduction leaves the addition to L2
                        const Real *U = reinterpret_cast<const Real *>(gb + L.u);
                        const double cf = __ldg(a.cfilter + step);
                        for (int o = lane; o < ne * ND; o += 32)
                            atomicAdd(a.acc + (size_t)e0 * ND + o, cf * (double)U[o]);
                    }
                }
                if (++st == 5)
                {
                    st = 0;
                    ++step;
                }
            }
            if (!ok)
            {
                if (lane == 0)
                    atomicOr(a.err, 1u);
                cp_async_wait<0>();
                return;
            }
            // ---- the state back
            for (int sl = warp; sl < ng; sl += W)
            {
                const int e0 = (g_lo + sl) * EW, ne = min(EW, a.nel - e0);
                const Real *U = reinterpret_cast<const Real *>(groups + (size_t)sl * L.bytes + L.u);
                for (int o = lane; o < ne * ND; o += 32)
                    a.A[(size_t)e0 * ND + o] = U[o];
            }
        }

        template <int N, typename Real>
        cudaError_t launch_n(const ResArgs<Real> &a, const ResPlan &p, cudaStream_t s)
        {
            static std::atomic<uint64_t> set{0}; // devices whose shared memory limit is raised
            int dev = 0;
            cudaGetDevice(&dev);
            const uint64_t bit = 1ull << (dev & 63);
            if (!(set.load(std::memory_order_relaxed) & bit))
            {
                const cudaError_t e = cudaFuncSetAttribute(res_kernel<N, Real>,
                                                           cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
                if (e != cudaSuccess)
                    return e;
                set.fetch_or(bit, std::memory_order_relaxed);
            }
            void *args[] = {const_cast<ResArgs<Real> *>(&a)};
            return cudaLaunchCooperativeKernel((const void *)res_kernel<N, Real>, dim3(p.ctas), dim3(32 * p.warps), args,
                                               p.smem, s);
        }
    } // namespace

    int upload_res_tables(int device) { return upload_basis_tab(device); }

    ResPlan res_plan(int n, bool fp32, int nel, int sms, int max_ctas, bool forced)
    {
        ResPlan p;
        p.ngroups = (nel + 32 / n - 1) / (32 / n);
        p.ctas = std::min(sms, p.ngroups);
        if (max_ctas > 0)
            p.ctas = std::min(p.ctas, max_ctas);
        if (p.ctas < 1)
            return p;
        const int most = (p.ngroups + p.ctas - 1) / p.ctas;
        const size_t gb = (size_t)(fp32 ? res_layout<float>(n).bytes : res_layout<double>(n).bytes);
        const size_t sc = (size_t)res_scratch(n, sum_strides_at(n), fp32 ? 4 : 8) + (forced ? res_forcing(n, fp32 ? 4 : 8) : 0);
        // as few rounds of groups per warp as twelve warps allow, the warps evened out over them; fewer
        // warps where their scratch is what does not fit
        for (int rounds = (most + kResMaxWarps - 1) / kResMaxWarps; rounds <= most && rounds <= 4 * kResMaxWarps; ++rounds)
        {
            p.warps = (most + rounds - 1) / rounds;
            p.smem = most * gb + p.warps * sc;
            p.fits = p.smem <= 227 * 1024;
            if (p.fits || most * gb + sc > 227 * 1024)
                break;
        }
        // with fewer than six warps an SM of many groups loses more to latency than the streaming kernel to L2
        if (p.warps < std::min(most, 6))
            p.fits = false;
        return p;
    }

    template <typename Real>
    int res_rk4(wdg_wave *w, const ResPlan &p, Real *A, double dt, int nsteps, const RKExtras &x, bool &ran, cudaStream_t stream)
    {
        ran = false;
        if ((x.F && !x.d_fscale) || (x.acc && !x.d_cfilter))
            return fail(WDG_ERR_ARG, "resident steps: forcing or filter without its table");
        ResArgs<Real> a{};
        a.A = A;
        a.T[0] = static_cast<Real *>(w->d_trace[0]);
        a.T[1] = static_cast<Real *>(w->d_trace[1]);
        a.corners = w->d_corners;
        a.fbase = w->d_fbase;
        a.fcode = w->d_fcode;
        a.flags = w->d_flags;
        a.err = w->d_err;
        a.nel = w->nel;
        a.ngroups = p.ngroups;
        for (int k = 0; k < 5; ++k)
        {
            a.a[k] = (Real)rk4a[k];
            a.b[k] = (Real)rk4b[k];
        }
        a.dt = (Real)dt;
        a.F = static_cast<const Real *>(x.F);
        a.acc = x.acc;
        a.wait_ns = w->wait_ns;
        a.test_skip = w->test_skip - 1;
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        WDG_CUDA(cudaStreamIsCapturing(stream, &cap));
        constexpr int kSteps = 4096; // per launch
        for (int s0 = 0; s0 < nsteps; s0 += kSteps)
        {
            a.nsteps = std::min(kSteps, nsteps - s0);
            a.fscale = x.d_fscale ? x.d_fscale + 5 * s0 : nullptr;
            a.cfilter = x.d_cfilter ? x.d_cfilter + s0 : nullptr;
            // A replayed graph repeats this launch with the same base, so its flags start below it again;
            // launches outside a graph count on from a base no replay has reached, the first from zero
            const bool captured = cap == cudaStreamCaptureStatusActive;
            if (captured || !w->flags_set)
                WDG_CUDA(cudaMemsetAsync(w->d_flags, 0, sizeof(unsigned long long) * kFlagStride * p.ngroups, stream));
            a.base = w->flag_base;
            cudaError_t e = cudaErrorInvalidValue;
            switch (w->n)
            {
            case 2: e = launch_n<2, Real>(a, p, stream); break;
            case 3: e = launch_n<3, Real>(a, p, stream); break;
            case 4: e = launch_n<4, Real>(a, p, stream); break;
            case 5: e = launch_n<5, Real>(a, p, stream); break;
            case 6: e = launch_n<6, Real>(a, p, stream); break;
            case 7: e = launch_n<7, Real>(a, p, stream); break;
            case 8: e = launch_n<8, Real>(a, p, stream); break;
            case 9: e = launch_n<9, Real>(a, p, stream); break;
            default: break;
            }
            if (e == cudaErrorCooperativeLaunchTooLarge && s0 == 0)
            {
                cudaGetLastError(); // fewer SMs than the plan counted on: the streaming kernel runs
                return WDG_OK;
            }
            if (e != cudaSuccess)
                return cuda_fail(e, "resident stage kernel launch");
            w->flag_base += 5ull * a.nsteps + 1;
            w->flags_set = w->flags_set || !captured;
            w->test_skip = 0; // this launch only
            a.test_skip = -1;
            ran = true;
        }
        return WDG_OK;
    }
    template int res_rk4<double>(wdg_wave *, const ResPlan &, double *, double, int, const RKExtras &, bool &, cudaStream_t);
    template int res_rk4<float>(wdg_wave *, const ResPlan &, float *, double, int, const RKExtras &, bool &, cudaStream_t);

    size_t res_flag_count(int n, int nel) { return (size_t)kFlagStride * ((nel + 32 / n - 1) / (32 / n)); }
} // namespace wdg
