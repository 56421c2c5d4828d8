// RK stage of meshes too large to stay resident: one warp per CTA, every warp on its own (included by
// kernels.cu after stage_ws.cuh, whose consumer code it runs, so the two step bit-identically).
//
// A warp is persistent over groups of EW = floor(32 / n) whole elements.  It loads a group's state,
// register and corners with cp.async.bulk, runs the column and the row pass in place and stores both
// back with cp.async.bulk.  The next group's pieces are asked into L2 before the current one is
// computed, its table entries are read then too, and its neighbour traces are gathered (cp.async) as soon
// as the passes are done with the current ones.  Warps share nothing, so their copies and their
// arithmetic overlap each other's; a producer warp, a ring and a CTA's barriers cost registers and shared
// memory that hold more consumers here (FP64, n = 5: 12 warps per SM against 8 + 2 producers).
//
// The gather takes a side by the neighbouring lanes of a part of the warp, since the L1 serves a line
// at a time: 3 n values lie in 1 to n lines.  Below n = 4 a lane takes its side value by value (the
// shuffles that hand out the sides cost more than the lines: 600 x 600, n = 3, FP32: 51.6 against 58.5 us).
// An FP32 group need not be a whole number of 16-byte units: it is loaded with the few bytes around it,
// and stored in its whole units by bulk copies, the values beside them one by one.
//
// What bounds it: per element the shared-memory pipe (90 wavefronts at n = 5, three quarters busy), the passes' dependent
// FP64 chains with three warps per scheduler, and in FP32 the issue slots; HBM follows (512 x 512, n = 5:
// 90 us a stage in FP64 and 46 in FP32 at the copy rate).  us a stage, against the warp-specialised kernel as
// it was: FP64: 600 x 600, n = 3: 102 -> 81; 512 x 512, n = 4: 141 -> 96, n = 5: 139 -> 113; 400 x 400,
// n = 6: 141 -> 105, n = 7: 228 -> 160; 350 x 350, n = 8: 338 -> 184; 300 x 300, n = 9: 323 -> 174.  FP32:
// 60 -> 52, 81 -> 55, 84 -> 78, 71 -> 66, 92 -> 88, 151 -> 84, 103 -> 99.  Forced periods of WaveHoltz,
// 300 x 300, n = 5: 1105 -> 869 ms.  Tried: neighbours of the same group read where they lie instead of gathered
// (n = 5 -1 %, n = 6 +20 %), side metrics by one lane a side (+6 %), more warps at fewer registers (n = 5: 154 us,
// spills), groups of two rounds (FP32 n = 5: 90 us).
namespace wdg
{
    // A group is a warp-round: EW = floor(32 / n) whole elements, a lane per grid line.
    // shared memory:  state | register | neighbour traces (4 n, 3) | corners | side codes |
    //                 column sums | mbarrier
    // State and register start as far from a 16-byte boundary as they do in memory.
    template <int N, typename Real>
    struct LineGroup
    {
        static constexpr int ND = 3 * N * N, G = 32 / N, real = sizeof(Real);
        static constexpr int size = G * ND * real;                    // a group's state
        static constexpr int ub = (size + (size % 16 ? 30 : 0)) & ~15; // its place: up to 12 bytes before, up to 15 after
        static constexpr int hb = 2 * ub, cb = hb + ((G * 12 * N * real + 15) & ~15), kb = cb + 64 * G;
        static constexpr int sb = (kb + 4 * G + 15) & ~15;
        static constexpr int bb = sb + ((G * stream_sums(N).el * real + 15) & ~15);
        static constexpr int bytes = bb + 16;
        static constexpr int fit = (227 * 1024) / (bytes + 1024);
        static constexpr int regs = real == 4 ? (N <= 8 ? 16 : 12) : N <= 6 ? 12 : 8; // warps the registers leave room for
        static constexpr int MINB = fit < regs ? fit : regs;
        static constexpr int PT = (4 * G + 31) / 32; // (element, side) pairs per lane
    };

    // EXTRA: launches with forcing or filter (FP64); their groups' parts follow the mbarrier
    // OP: an operator launch (line_operator): no state is stored
    template <int N, typename Real, bool EXTRA, bool OP>
    __global__ void __launch_bounds__(32, LineGroup<N, Real>::MINB) line_stage_kernel(const __grid_constant__ StageArgs<Real> a)
    {
        using L = LineGroup<N, Real>;
        constexpr int ND = L::ND, G = L::G, PT = L::PT;
        extern __shared__ __align__(128) unsigned char smem[];
        Real *halo = reinterpret_cast<Real *>(smem + L::hb);
        uint32_t *codes = reinterpret_cast<uint32_t *>(smem + L::kb);
        Real *sums = reinterpret_cast<Real *>(smem + L::sb);
        uint64_t *full = reinterpret_cast<uint64_t *>(smem + L::bb);
        const int lane = threadIdx.x;
        const int e0 = a.el_begin, e1 = a.el_end > 0 ? a.el_end : a.nel;
        const int ngroups = (e1 - e0 + G - 1) / G;
        const bool has_du = (a.flags & F_READ_DU) != 0, inner = (a.flags & F_INT) != 0;
        const int limit = a.nread > 0 ? a.nread : a.nel * ND;
        const bool force = EXTRA && (a.flags & F_FORCE), filter = EXTRA && (a.flags & F_FILTER);
        unsigned char *Fs = smem + L::bytes, *As = Fs + L::ub;
        const uint64_t wlim = wait_limit(a.wait_ns);
        if (lane == 0)
        {
            mbar_init(full, 1 + 32); // the bulk copies' arrive + one cp.async arrive per lane
            fence_mbar_init();
        }
        __syncwarp();

        // an operator that only adds boundary terms leaves the groups inside the mesh alone
        const bool edges_only = OP && has_du && !(a.flags & (F_VOL | F_INT));
        uint32_t code[PT], own = 0;
        int off[PT];
        // side codes and partner offsets of group g: a lane per (element, side)
        auto tables = [&](int g)
        {
#pragma unroll
            for (int t = 0; t < PT; ++t)
            {
                const int p = lane + 32 * t, el = e0 + g * G + (p >> 2);
                code[t] = 0x80u;
                off[t] = -1;
                if (g < ngroups && p < 4 * G && el < e1)
                {
                    code[t] = (__ldg(a.fcode + el) >> (8 * (p & 3))) & 0xffu;
                    off[t] = __ldg(reinterpret_cast<const int *>(a.fbase + el) + (p & 3));
                }
            }
            own = (lane < G && g < ngroups && e0 + g * G + lane < e1) ? __ldg(a.fcode + e0 + g * G + lane) : 0u;
        };
        // this warp's first group from g on, its tables read
        auto first = [&](int g)
        {
            tables(g);
            if (OP && edges_only)
                while (g < ngroups && !__any_sync(0xffffffffu, (own & 0x80808080u) != 0))
                    tables(g += gridDim.x);
            return g;
        };
        auto shift = [](int el) { return L::size % 16 ? (int)(((size_t)el * ND * sizeof(Real)) & 15) : 0; };
        // whether the 16-byte pieces around the group's state all belong to the arrays
        auto whole = [&](int el) { return el + G <= e1 && (L::size % 16 == 0 || el + G < a.nel); };
        auto gather = [&]()
        {
            if (lane < G)
                codes[lane] = own;
#pragma unroll
            for (int t = 0; t < PT; ++t)
            {
                const int stride = partner_stride<N>(code[t]);
                int from = off[t];
                if (!inner || (code[t] & 0x80u))
                    from = -1;
                else if (from < 0 || from + (N - 1) * stride < 0 || from + 3 > limit || from + (N - 1) * stride + 3 > limit)
                {
                    atomicOr(a.err, 2u);
                    from = -1;
                }
                if constexpr (N <= 3)
                {
                    // short sides: a lane takes its side, value by value
                    Real *dst = halo + 3 * N * (lane + 32 * t);
#pragma unroll
                    for (int k = 0; k < 3 * N; ++k)
                        if (from >= 0)
                            cp_async<sizeof(Real)>(dst + k, a.u + from + (k / 3) * stride + k % 3);
                }
                else
                {
                    // the lanes of a part of the warp take a side's values
                    constexpr int W = 3 * N, GS = 32 / W, pairs = 4 * G < 32 ? 4 * G : 32;
                    const int part = lane / W, pos = lane - part * W, k = pos / 3;
#pragma unroll
                    for (int q0 = 0; q0 < pairs; q0 += GS)
                    {
                        const int q = q0 + part;
                        const int f0 = __shfl_sync(0xffffffffu, from, q & 31), st = __shfl_sync(0xffffffffu, stride, q & 31);
                        if (part < GS && q < pairs && f0 >= 0)
                            cp_async<sizeof(Real)>(halo + W * (32 * t + q) + pos, a.u + f0 + k * st + (pos - 3 * k));
                    }
                }
            }
            cp_async_mbar_arrive(full);
        };
        auto load = [&](int g)
        {
            const int el = e0 + g * G, ne = min(G, e1 - el), sh = shift(el);
            if (whole(el))
            {
                if (lane == 0)
                {
                    const uint32_t bytes = (uint32_t)((sh + L::size + 15) & ~15);
                    mbar_expect_tx(full, bytes * (1 + (has_du ? 1 : 0) + (force ? 1 : 0) + (filter ? 1 : 0)) + 64 * G);
                    bulk_g2s(smem, reinterpret_cast<const char *>(a.u + (size_t)el * ND) - sh, bytes, full);
                    if (has_du)
                        bulk_g2s(smem + L::ub, reinterpret_cast<const char *>(a.du + (size_t)el * ND) - sh, bytes, full);
                    bulk_g2s(smem + L::cb, a.corners + 8 * (size_t)el, 64 * G, full);
                    if (force)
                        bulk_g2s(Fs, reinterpret_cast<const char *>(a.F + (size_t)el * ND) - sh, bytes, full);
                    if (filter)
                        bulk_g2s(As, reinterpret_cast<const char *>(a.acc + (size_t)el * ND) - sh, bytes, full);
                }
                return;
            }
            Real *us = reinterpret_cast<Real *>(smem + sh), *dus = reinterpret_cast<Real *>(smem + L::ub + sh);
            for (int i = lane; i < ne * ND; i += 32)
            {
                us[i] = a.u[(size_t)el * ND + i];
                if (has_du)
                    dus[i] = a.du[(size_t)el * ND + i];
                if (force)
                    reinterpret_cast<Real *>(Fs + sh)[i] = a.F[(size_t)el * ND + i];
                if (filter)
                    reinterpret_cast<double *>(As + sh)[i] = a.acc[(size_t)el * ND + i];
            }
            for (int i = lane; i < ne * 8; i += 32)
                reinterpret_cast<double *>(smem + L::cb)[i] = a.corners[8 * (size_t)el + i];
            __syncwarp();
            if (lane == 0)
                mbar_arrive(full);
        };
        auto store = [&](int el, int ne)
        {
            const int sh = shift(el);
            const Real *us = reinterpret_cast<const Real *>(smem + sh), *dus = reinterpret_cast<const Real *>(smem + L::ub + sh);
            Real *out = a.out + (size_t)el * ND, *du = a.du + (size_t)el * ND;
            // the whole 16-byte pieces by bulk copies, what stands before and after them value by value
            const int total = ne * ND, head = ((16 - sh) & 15) / (int)sizeof(Real);
            int body = 0;
            if (ne == G)
            {
                body = (total - head) & ~(16 / (int)sizeof(Real) - 1);
                if (lane == 0)
                {
                    if (!OP)
                        bulk_s2g(out + head, us + head, (uint32_t)(body * sizeof(Real)));
                    bulk_s2g(du + head, dus + head, (uint32_t)(body * sizeof(Real)));
                    if (filter)
                        bulk_s2g(a.acc + (size_t)el * ND + head, reinterpret_cast<const double *>(As + sh) + head,
                                 (uint32_t)(body * sizeof(Real)));
                    bulk_commit();
                }
                if (L::size % 16 == 0)
                    return;
            }
            for (int i = lane; i < total - body; i += 32)
            {
                const int at = i < head ? i : i + body;
                if (!OP)
                    out[at] = us[at];
                du[at] = dus[at];
                if (filter)
                    a.acc[(size_t)el * ND + at] = reinterpret_cast<const double *>(As + sh)[at];
            }
        };

        WsChunk<Real> c{};
        c.u = a.u;
        c.nel = a.nel;
        c.chunk = G;
        c.flags = a.flags;
        c.rk_a = a.rk_a;
        c.rk_b = a.rk_b;
        c.dt = a.dt;
        c.fscale = a.fscale;
        c.acc_c = a.acc_c;
        const Real xm = Tab<Real>::x(N, lane % N), wm = Tab<Real>::w(N, lane % N);
        int g = first(blockIdx.x), next = g;
        if (g >= ngroups)
            return;
        if (OP || a.test_skip != 1) // test hook: group test_skip - 1 of every warp stays unloaded
            load(g);
        gather();
        for (int m = 0; g < ngroups; ++m, g = next)
        {
            next = first(g + gridDim.x);
            if (lane == 0 && next < ngroups && whole(e0 + next * G))
            {
                const int el = e0 + next * G, sh = shift(el);
                const uint32_t bytes = (uint32_t)((sh + L::size + 15) & ~15);
                bulk_prefetch(reinterpret_cast<const char *>(a.u + (size_t)el * ND) - sh, bytes);
                if (has_du)
                    bulk_prefetch(reinterpret_cast<const char *>(a.du + (size_t)el * ND) - sh, bytes);
                bulk_prefetch(a.corners + 8 * (size_t)el, 64 * G);
            }
            if (!__all_sync(0xffffffffu, mbar_wait(full, m & 1, wlim)))
            {
                if (lane == 0)
                    atomicOr(a.err, 1u);
                cp_async_wait_all(); // the gathered traces
                break;
            }
            c.el0 = e0 + g * G;
            c.ne = min(G, e1 - c.el0);
            __syncwarp(); // the side codes
            const int sh = shift(c.el0);
            const WsSlot o{L::ub, L::hb - sh, L::cb - sh, L::kb - sh, 0, 0, 0};
            c.F = reinterpret_cast<const Real *>(Fs + sh) - (size_t)c.el0 * ND;
            c.acc = reinterpret_cast<double *>(As + sh) - (size_t)c.el0 * ND;
            ws_consume<N, Real, EXTRA, false, false>(c, smem + sh, o, 1, sums, xm, wm, 0, lane);
            fence_async_smem();
            __syncwarp();
            store(c.el0, c.ne);
            if (next < ngroups)
            {
                gather();
                if (lane == 0)
                    bulk_wait_read();
                __syncwarp();
                if (OP || a.test_skip != m + 2)
                    load(next);
            }
        }
        if (lane == 0)
            bulk_wait_all();
    }

    template <int N, typename Real, bool EXTRA, bool OP>
    static cudaError_t launch_line_n(const StageArgs<Real> &a, cudaStream_t s)
    {
        using L = LineGroup<N, Real>;
        // forcing alone takes one more place, a filter (behind it) two
        const int extra = EXTRA ? ((a.flags & F_FILTER) ? 2 : 1) : 0, smem = L::bytes + extra * L::ub;
        static std::atomic<int> resident[3][64]; // CTAs of this kernel on each device, found once
        int dev = 0;
        cudaGetDevice(&dev);
        int grid = resident[extra][dev & 63].load(std::memory_order_relaxed);
        if (grid == 0)
        {
            int per_sm = 0, sms = 0;
            auto kern = line_stage_kernel<N, Real, EXTRA, OP>;
            cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 L::bytes + (EXTRA ? 2 * L::ub : 0));
            if (e == cudaSuccess)
                e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32, smem);
            if (e == cudaSuccess)
                e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            if (e != cudaSuccess)
                return e;
            grid = std::max(1, per_sm) * sms;
            resident[extra][dev & 63].store(grid, std::memory_order_relaxed);
        }
        const int ngroups = ((a.el_end > 0 ? a.el_end : a.nel) - a.el_begin + L::G - 1) / L::G;
        if (ngroups < 1)
            return cudaSuccess; // an empty range
        line_stage_kernel<N, Real, EXTRA, OP><<<std::min(grid, ngroups), 32, smem, s>>>(a);
        return cudaGetLastError();
    }
    inline bool line_aligned(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
    // Whether the launch goes to this kernel: wherever the caller left the choice and all arrays are aligned.
    // FP32 launches with forcing or filter stay with the warp-specialised kernel, which stages the FP64 filter
    // beside the FP32 state; a CTA limit is meant for its CTAs of five warps.
    template <typename Real>
    static bool line_takes(const StageArgs<Real> &a, int grid_limit)
    {
        if (!a.line || a.family != 2 || !a.use_tma || !a.tma_out || grid_limit > 0)
            return false;
        if (!a.out) // operators, FP64; the sum with a forcing has its own rounding: tiled kernel
            return sizeof(Real) == 8 && !(a.flags & F_FORCE);
        return !(a.flags & (F_FORCE | F_FILTER)) || (sizeof(Real) == 8 && (!(a.flags & F_FORCE) || line_aligned(a.F)) &&
                                                     (!(a.flags & F_FILTER) || line_aligned(a.acc)));
    }
    // An operator launch as a step of this kernel: its result is the register of a step of size 1 that starts
    // from the array it is added to (1 d + 1 r and 1 r round once, as d + r and r do) and stores no state.
    // 61 x 47, n = 6: WaveEquation::action 13 -> 8.2 us, WaveBC::action 13 -> 6.2 us against the tiled kernel, whose
    // tiles pass five CTA barriers each and which visits every element for the boundary's terms.
    template <typename Real>
    static StageArgs<Real> line_operator(StageArgs<Real> a)
    {
        a.tma_out = line_aligned(a.out);
        a.du = a.out;
        a.out = nullptr;
        a.rk_a = a.dt = 1;
        a.rk_b = 0;
        a.flags = (a.flags & ~F_ACCUM) | ((a.flags & F_ACCUM) ? F_READ_DU : 0);
        return a;
    }
    template <int N, typename Real>
    static cudaError_t launch_line(const StageArgs<Real> &a, cudaStream_t s)
    {
        if constexpr (sizeof(Real) == 8)
        {
            if (!a.out)
                return launch_line_n<N, Real, false, true>(a, s);
            if (a.flags & (F_FORCE | F_FILTER))
                return launch_line_n<N, Real, true, false>(a, s);
        }
        return launch_line_n<N, Real, false, false>(a, s);
    }
} // namespace wdg
