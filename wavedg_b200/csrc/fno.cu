// Kernels of the learned WaveHoltz warm start: a Fourier neural operator (FNO) on a
// uniform G x G grid, trained and evaluated with BF16 operands and FP32 accumulation.
//
//   gemm        C = alpha op(A) op(B) + beta C, BF16 operands, FP32 accumulate and output,
//               batched with strides, optional split-K (atomic FP32 accumulation).  Tensor
//               cores through mma.sync.m16n8k16 (BF16): every GEMM of the network has one
//               dimension of 32 (channels or retained modes), so these are bandwidth-bound
//               streams, not tensor-throughput-bound tiles.
//   layer       the two GEMMs of a Fourier layer's output (inverse DFT along x, channel mix) in one
//               pass with what follows them, forward (bias, GELU) and backward (GELU's derivative).
//   dft_y       the truncated DFT along y (retained wavenumbers 0..K/2-1 and -K/2..-1) and its
//               inverse/adjoint, FP32 on CUDA cores (small: K x KX modes per channel).
//   mix         per-mode complex channel mixing and its two adjoints.
//   pointwise   bias + GELU and its derivative, bias gradients, conversions, the MSE loss,
//               Adam, the resampling between the DG nodes and the grid, and the input
//               fields (forcing, omega, coordinates).
//
// The truncated DFT along x and the inverse real DFT along x are GEMMs against fixed
// BF16 matrices built by the host (fno.py).  All entry points are asynchronous on the
// given stream and return 0 or a negative WDG_ERR code.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <type_traits>

#include "common.hpp"

namespace
{
    using bf16 = __nv_bfloat16;

    // ------------------------------------------------------------------ GEMM
    constexpr int TM = 64, TK = 32; // TK: K per shared-memory step (two mma steps of 16, in order)

    __device__ __forceinline__ void mma_bf16(float c[4], const uint32_t a[4], const uint32_t b[2])
    {
        asm volatile(
            "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
            "{%0,%1,%2,%3};"
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
    }
    __device__ __forceinline__ uint32_t smem_at(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
    // four 8 x 8 tiles, lane l giving the row l & 7 of tile l >> 3; TRANS: each tile transposed
    template <bool TRANS>
    __device__ __forceinline__ void ldmatrix4(uint32_t r[4], const bf16 *p)
    {
        if constexpr (TRANS)
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                         : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                         : "r"(smem_at(p)));
        else
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                         : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                         : "r"(smem_at(p)));
    }

    // A ROWS x COLS tile (COLS contiguous in memory, rows ld apart) to shared memory, rows COLS + 8
    // apart (ldmatrix then reads eight rows from different banks); values past (rows, cols) are 0.
    // vec: whole 16-byte pieces by cp.async (cols a multiple of 8, everything aligned)
    template <int ROWS, int COLS>
    __device__ __forceinline__ void load_tile(bf16 *sm, const bf16 *g, long long ld, int rows, int cols, bool vec, int t)
    {
        constexpr int LD = COLS + 8;
        if (vec)
        {
#pragma unroll
            for (int i = 0; i < ROWS * COLS / 8; i += 128)
            {
                const int q = i + t, r = q / (COLS / 8), c = q % (COLS / 8) * 8;
                if (ROWS * COLS / 8 % 128 != 0 && q >= ROWS * COLS / 8)
                    break;
                const bool in = r < rows && c < cols;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_at(sm + r * LD + c)),
                             "l"(in ? g + r * ld + c : g), "r"(in ? 16 : 0)
                             : "memory");
            }
        }
        else
            for (int q = t; q < ROWS * COLS; q += 128)
            {
                const int r = q / COLS, c = q % COLS;
                sm[r * LD + c] = (r < rows && c < cols) ? g[r * ld + c] : __float2bfloat16(0.f);
            }
    }
    // acc (a warp's 32 x 32) += op(A) op(B) over one shared-memory step, K ascending; A at row m0, B at
    // column n0 of their tiles.  TA: A stored (k, m), else (m, k); TB: B stored (n, k), else (k, n)
    template <bool TA, bool TB, int LDA, int LDB>
    __device__ __forceinline__ void tile_mma(float acc[2][4][4], const bf16 *As, const bf16 *Bs, int m0, int n0, int lane)
    {
        const int r8 = lane & 7, q = lane >> 3; // row within a tile, tile
#pragma unroll
        for (int kk = 0; kk < TK; kk += 16)
        {
            uint32_t af[2][4], bfr[2][4];
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
            {
                // tiles: (m, k), (m + 8, k), (m, k + 8), (m + 8, k + 8)
                const int m = m0 + 16 * mi + 8 * (q & 1), k = kk + 8 * (q >> 1);
                ldmatrix4<TA>(af[mi], TA ? As + (k + r8) * LDA + m : As + (m + r8) * LDA + k);
            }
#pragma unroll
            for (int ni = 0; ni < 2; ++ni)
            {
                // tiles: (k, n), (k + 8, n), (k, n + 8), (k + 8, n + 8)
                const int n = n0 + 16 * ni + 8 * (q >> 1), k = kk + 8 * (q & 1);
                ldmatrix4<!TB>(bfr[ni], TB ? Bs + (n + r8) * LDB + k : Bs + (k + r8) * LDB + n);
            }
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                for (int ni = 0; ni < 4; ++ni)
                    mma_bf16(acc[mi][ni], af[mi], bfr[ni >> 1] + 2 * (ni & 1));
        }
    }

    __device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.f + erff(z * 0.70710678118654752f)); }
    __device__ __forceinline__ float gelu_grad(float z)
    {
        const float cdf = 0.5f * (1.f + erff(z * 0.70710678118654752f));
        const float pdf = 0.39894228040143268f * expf(-0.5f * z * z);
        return cdf + z * pdf;
    }

    // what a GEMM does with its result besides, or instead of, storing it
    enum
    {
        EPI_STORE = 0,    // C = alpha acc + beta C
        EPI_BIAS_ACT = 1, // v = acc + bias[row]: C = v (nullable), y = act ? gelu(v) : v in BF16 (nullable)
        EPI_ACT_BWD = 2   // v = act ? acc gelu'(z) : acc: C = v (nullable), y = v in BF16 (nullable)
    };
    struct Epilogue
    {
        const float *bias, *z;
        bf16 *y;
        int act;
    };
    // two neighbouring columns of one row; i: their place in C, z and y
    __device__ __forceinline__ void epilogue(int mode, const Epilogue &e, float *C, long long i, float bias, float v0, float v1,
                                             bool two, bool pair)
    {
        if (mode == EPI_BIAS_ACT)
        {
            v0 = v0 + bias;
            v1 = v1 + bias;
        }
        else if (e.act)
        {
            v0 = v0 * gelu_grad(e.z[i]);
            if (two)
                v1 = v1 * gelu_grad(e.z[i + 1]);
        }
        if (C)
        {
            if (pair)
                *reinterpret_cast<float2 *>(C + i) = make_float2(v0, v1);
            else
            {
                C[i] = v0;
                if (two)
                    C[i + 1] = v1;
            }
        }
        if (e.y)
        {
            if (mode == EPI_BIAS_ACT && e.act)
            {
                v0 = gelu(v0);
                v1 = gelu(v1);
            }
            if (pair)
                *reinterpret_cast<__nv_bfloat162 *>(e.y + i) = __floats2bfloat162_rn(v0, v1);
            else
            {
                e.y[i] = __float2bfloat16(v0);
                if (two)
                    e.y[i + 1] = __float2bfloat16(v1);
            }
        }
    }

    struct GemmArgs
    {
        const bf16 *A, *B;
        float *C;
        int M, N, K;
        long long lda, ldb, ldc;       // leading dimensions of the stored matrices
        long long sA, sB, sC;          // batch strides (elements)
        float alpha, beta;
        int ksplit;                    // K range per split (multiple of TK)
        int atomic;                    // accumulate with atomics (split K, or batches sharing C)
        int vecA, vecB, pairC;         // 16-byte loads of A, B; 8-byte stores of C
        Epilogue e;
    };

    // BM x BN output tile per CTA of four warps (32 x 32 each), K in steps of 32 through ST shared-memory
    // stages filled by cp.async.  These GEMMs stream one operand with hundreds of thousands of rows past
    // a matrix of at most 64 x 64: the tile shape follows the narrow side (32 x 128, 128 x 32, 64 x 64), so
    // that no half of it is padding.  Bound by HBM.
    template <int BM, int BN, int ST, bool TA, bool TB, int EPI>
    __global__ void __launch_bounds__(128) gemm_bf16_kernel(const GemmArgs g)
    {
        constexpr int LDA = (TA ? BM : TK) + 8, LDB = (TB ? TK : BN) + 8;
        constexpr int SA = (TA ? TK : BM) * LDA, SB = (TB ? BN : TK) * LDB;
        extern __shared__ __align__(16) bf16 gsm[];
        const int bz = blockIdx.z;
        const int nsplit = (g.K + g.ksplit - 1) / g.ksplit;
        const int batch = bz / nsplit, split = bz - batch * nsplit;
        const bf16 *A = g.A + batch * g.sA;
        const bf16 *B = g.B + batch * g.sB;
        const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
        const int k_begin = split * g.ksplit, k_end = min(g.K, k_begin + g.ksplit);
        const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
        constexpr int WN = BN / 32;
        const int wm = warp / WN * 32, wn = warp % WN * 32;
        const int gid = lane >> 2, tig = lane & 3;
        float acc[2][4][4] = {};
        const int nk = (k_end - k_begin + TK - 1) / TK;
        auto load = [&](int it)
        {
            bf16 *As = gsm + (it % ST) * (SA + SB), *Bs = As + SA;
            const int k0 = k_begin + it * TK, kr = k_end - k0;
            if constexpr (TA)
                load_tile<TK, BM>(As, A + (long long)k0 * g.lda + m0, g.lda, kr, g.M - m0, g.vecA, t);
            else
                load_tile<BM, TK>(As, A + (long long)m0 * g.lda + k0, g.lda, g.M - m0, kr, g.vecA, t);
            if constexpr (TB)
                load_tile<BN, TK>(Bs, B + (long long)n0 * g.ldb + k0, g.ldb, g.N - n0, kr, g.vecB, t);
            else
                load_tile<TK, BN>(Bs, B + (long long)k0 * g.ldb + n0, g.ldb, kr, g.N - n0, g.vecB, t);
        };
#pragma unroll
        for (int q = 0; q < (ST > 1 ? ST - 1 : 1); ++q)
        {
            if (q < nk)
                load(q);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        for (int it = 0; it < nk; ++it)
        {
            asm volatile("cp.async.wait_group %0;" ::"n"(ST > 1 ? ST - 2 : 0) : "memory");
            __syncthreads(); // this step has landed; every warp is done with the one before
            if constexpr (ST > 1)
            {
                if (it + ST - 1 < nk)
                    load(it + ST - 1);
                asm volatile("cp.async.commit_group;" ::: "memory");
            }
            const bf16 *As = gsm + (it % ST) * (SA + SB);
            tile_mma<TA, TB, LDA, LDB>(acc, As, As + SA, wm, wn, lane);
            if constexpr (ST == 1)
                if (it + 1 < nk)
                {
                    __syncthreads();
                    load(it + 1);
                    asm volatile("cp.async.commit_group;" ::: "memory");
                }
        }
        float *C = g.C ? g.C + batch * g.sC : nullptr;
        Epilogue e = g.e;
        if (e.z)
            e.z += batch * g.sC;
        if (e.y)
            e.y += batch * g.sC;
        // (split-K: atomic accumulation into a C that was zeroed or holds beta C)
#pragma unroll
        for (int mi = 0; mi < 2; ++mi)
#pragma unroll
            for (int hr = 0; hr < 2; ++hr)
            {
                const int r = m0 + wm + 16 * mi + gid + 8 * hr;
                if (r >= g.M)
                    continue;
                const float bias = EPI == EPI_BIAS_ACT ? g.e.bias[r] : 0.f;
#pragma unroll
                for (int ni = 0; ni < 4; ++ni)
                {
                    const int c = n0 + wn + 8 * ni + 2 * tig;
                    if (c >= g.N)
                        continue;
                    const bool two = c + 1 < g.N, pair = g.pairC && two;
                    const long long i = (long long)r * g.ldc + c;
                    float v0 = acc[mi][ni][2 * hr], v1 = acc[mi][ni][2 * hr + 1];
                    if constexpr (EPI != EPI_STORE)
                        epilogue(EPI, e, C, i, bias, v0, v1, two, pair);
                    else
                    {
                        v0 = g.alpha * v0;
                        v1 = g.alpha * v1;
                        if (g.atomic)
                        {
                            atomicAdd(C + i, v0);
                            if (two)
                                atomicAdd(C + i + 1, v1);
                        }
                        else if (pair)
                        {
                            float2 *q = reinterpret_cast<float2 *>(C + i);
                            if (g.beta != 0.f)
                            {
                                const float2 old = *q;
                                v0 = v0 + g.beta * old.x;
                                v1 = v1 + g.beta * old.y;
                            }
                            *q = make_float2(v0, v1);
                        }
                        else
                        {
                            C[i] = (g.beta == 0.f) ? v0 : v0 + g.beta * C[i];
                            if (two)
                                C[i + 1] = (g.beta == 0.f) ? v1 : v1 + g.beta * C[i + 1];
                        }
                    }
                }
            }
    }

    template <int BM, int BN, int ST, int EPI>
    void gemm_launch(const GemmArgs &g, int transA, int transB, int nz, cudaStream_t s)
    {
        const dim3 grid((g.N + BN - 1) / BN, (g.M + BM - 1) / BM, nz);
        auto run = [&](auto kern, bool ta, bool tb)
        {
            const int lda = (ta ? BM : TK) + 8, ldb = (tb ? TK : BN) + 8;
            const size_t smem = sizeof(bf16) * ST * ((ta ? TK : BM) * lda + (tb ? BN : TK) * ldb); // at most 38 KB
            kern<<<grid, 128, smem, s>>>(g);
        };
        if (transA)
            transB ? run(gemm_bf16_kernel<BM, BN, ST, true, true, EPI>, true, true)
                   : run(gemm_bf16_kernel<BM, BN, ST, true, false, EPI>, true, false);
        else
            transB ? run(gemm_bf16_kernel<BM, BN, ST, false, true, EPI>, false, true)
                   : run(gemm_bf16_kernel<BM, BN, ST, false, false, EPI>, false, false);
    }
    template <int ST, int EPI>
    void gemm_tiles(const GemmArgs &g, int transA, int transB, int nz, cudaStream_t s)
    {
        if (g.M <= 32)
            gemm_launch<32, 128, ST, EPI>(g, transA, transB, nz, s);
        else if (g.N <= 32)
            gemm_launch<128, 32, ST, EPI>(g, transA, transB, nz, s);
        else
            gemm_launch<64, 64, ST, EPI>(g, transA, transB, nz, s);
    }
    template <int EPI>
    void gemm_run(GemmArgs &g, int transA, int transB, int nz, cudaStream_t s)
    {
        auto whole = [](const void *p, long long ld, long long stride, int contiguous)
        { return (((uintptr_t)p & 15u) == 0 && ld % 8 == 0 && stride % 8 == 0 && contiguous % 8 == 0) ? 1 : 0; };
        g.vecA = whole(g.A, g.lda, g.sA, transA ? g.M : g.K);
        g.vecB = whole(g.B, g.ldb, g.sB, transB ? g.K : g.N);
        g.pairC = (((uintptr_t)g.C & 7u) == 0 && ((uintptr_t)g.e.y & 3u) == 0 && g.ldc % 2 == 0 && g.sC % 2 == 0) ? 1 : 0;
        if (std::min(g.K, g.ksplit) <= TK)
            gemm_tiles<1, EPI>(g, transA, transB, nz, s);
        else
            gemm_tiles<3, EPI>(g, transA, transB, nz, s);
    }

    // ------------------------------------------------------------ Fourier layer
    // One output tile of a layer, 32 channels x 128 grid points of row y of sample b, from its two GEMMs:
    //   forward   z = W v + U Ix  (U: the mixed spectrum after the inverse DFT along y, per channel and row;
    //             Ix: the inverse DFT along x), then bias and activation: z, y = BF16 act(z)
    //   backward  dv = W^T dz + U Ex^T  (U: the adjoint spectrum), then the derivative of the activation below:
    //             dz = dv gelu'(z) and its BF16 copy
    // In launches of their own the first result went to memory and back in FP32 and the elementwise step
    // read and wrote it again: 800 MB a layer at 4 x 32 x 512 x 512 where 270 MB are needed.  Bound by HBM.
    struct LayerArgs
    {
        const bf16 *U, *X, *W, *V;
        float *C; // z or dz (nullable)
        int Cn, K1, G;
        Epilogue e;
    };
    template <bool BACK>
    __global__ void __launch_bounds__(128) layer_kernel(const LayerArgs g)
    {
        // X: forward Ix (K1, G); backward Ex (G, K1).  W: forward (o, c), backward (c, o) read as its transpose
        constexpr int LDX = (BACK ? TK : 128) + 8, SX = (BACK ? 128 : TK) * LDX;
        __shared__ __align__(16) bf16 Us[32 * (TK + 8)], Ws[32 * (TK + 8)], Xs[SX], Vs[TK * 136];
        const int t = threadIdx.x, warp = t >> 5, lane = t & 31, gid = lane >> 2, tig = lane & 3;
        const int x0 = blockIdx.x * 128, y = blockIdx.y, b = blockIdx.z;
        const long long P = (long long)g.G * g.G, row0 = (long long)b * g.Cn;
        load_tile<32, TK>(Us, g.U + (row0 * g.G + y) * g.K1, (long long)g.G * g.K1, g.Cn, g.K1, true, t);
        load_tile<32, TK>(Ws, g.W, g.Cn, g.Cn, g.Cn, true, t);
        if constexpr (BACK)
            load_tile<128, TK>(Xs, g.X + (long long)x0 * g.K1, g.K1, g.G - x0, g.K1, true, t);
        else
            load_tile<TK, 128>(Xs, g.X + x0, g.G, g.K1, g.G - x0, true, t);
        load_tile<TK, 128>(Vs, g.V + row0 * P + (long long)y * g.G + x0, P, g.Cn, g.G - x0, true, t);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        float a1[2][4][4] = {}, a2[2][4][4] = {};
        tile_mma<false, BACK, TK + 8, LDX>(a1, Us, Xs, 0, 32 * warp, lane);
        tile_mma<BACK, false, TK + 8, 136>(a2, Ws, Vs, 0, 32 * warp, lane);
#pragma unroll
        for (int mi = 0; mi < 2; ++mi)
#pragma unroll
            for (int hr = 0; hr < 2; ++hr)
            {
                const int r = 16 * mi + gid + 8 * hr;
                if (r >= g.Cn)
                    continue;
                const float bias = BACK ? 0.f : g.e.bias[r];
#pragma unroll
                for (int ni = 0; ni < 4; ++ni)
                {
                    const int x = x0 + 32 * warp + 8 * ni + 2 * tig;
                    if (x >= g.G)
                        continue;
                    epilogue(BACK ? EPI_ACT_BWD : EPI_BIAS_ACT, g.e, g.C, (row0 + r) * P + (long long)y * g.G + x, bias,
                             a2[mi][ni][2 * hr] + a1[mi][ni][2 * hr], a2[mi][ni][2 * hr + 1] + a1[mi][ni][2 * hr + 1],
                             true, true);
                }
            }
    }

    int blocks(long long n, int threads = 256)
    {
        long long b = (n + threads - 1) / threads;
        return (int)(b < 148 * 32 ? (b < 1 ? 1 : b) : 148 * 32);
    }

    // ------------------------------------------------------------- DFT along y
    // out[bc, k, kx] = sum_y e^{s i 2 pi ky(k) y / G} in[bc, y, kx]   (forward: s = -1)
    // ky(k) = k for k < K/2, k - K otherwise; complex values as (re, im) pairs.  A CTA takes one plane bc
    // and kDftThreads pairs of outputs (k, kx) and (k + K/2, kx), so that a value read from shared memory
    // serves two sums; y runs in order, whatever the chunking.  The twiddles and a chunk of `chunk` rows
    // sit in shared memory (the twiddles of a grid too large for it stay in global memory: TAB false; so do
    // rows of which not one fits: ROWS false).  Pairs are read and written whole (VEC), or value by value, and
    // then from global memory, where an array does not lie on their boundary.
    constexpr int kDftThreads = 128, kDftRows = 128;
    constexpr size_t kDftSmem = 96 * 1024;
    constexpr long long kGridY = 65535; // blocks of a grid along y; longer work goes in several launches (`off`)
    __device__ __forceinline__ void dft_add(float2 x, float2 cs, float sign, float &re, float &im)
    {
        const float c = cs.x, s = sign * cs.y;
        // (the contraction is written out: it decides later roundings to BF16)
        re += __fmaf_rn(c, x.x, -__fmul_rn(s, x.y));
        im += __fmaf_rn(s, x.x, __fmul_rn(c, x.y));
    }
    template <bool VEC>
    __device__ __forceinline__ float2 pair_get(const float *p, long long i)
    {
        if constexpr (VEC)
            return reinterpret_cast<const float2 *>(p)[i];
        else
            return make_float2(p[2 * i], p[2 * i + 1]);
    }
    template <bool VEC>
    __device__ __forceinline__ void pair_put(float *p, long long i, float re, float im)
    {
        if constexpr (VEC)
            reinterpret_cast<float2 *>(p)[i] = make_float2(re, im);
        else
        {
            p[2 * i] = re;
            p[2 * i + 1] = im;
        }
    }
    template <bool TAB, bool ROWS, bool VEC>
    __global__ void __launch_bounds__(kDftThreads) dft_y_fwd_kernel(const float *in, float *out, const float *cs,
                                                                    const float *sn, int G, int K, int KX, float sign,
                                                                    int chunk, unsigned off)
    {
        extern __shared__ float2 dsm[];
        float2 *tab = dsm, *xs = dsm + (TAB ? G : 0); // (cos, sin) of 2 pi m / G; a chunk of rows
        auto twiddle = [&](int m) { return TAB ? tab[m] : make_float2(__ldg(cs + m), __ldg(sn + m)); };
        using index = std::conditional_t<ROWS, int, long long>; // of an output pair (the host's choice of ROWS: it fits)
        const int t = threadIdx.x, half = K / 2;
        const long long bc = blockIdx.x;
        const index q = (index)(off + blockIdx.y) * kDftThreads + t;
        const int kx = (int)(q % KX), k = (int)(q / KX);
        const bool on = k < half;
        for (int m = t; TAB && m < G; m += kDftThreads)
            tab[m] = make_float2(cs[m], sn[m]);
        const float *src = in + 2 * bc * (long long)G * KX;
        const int step0 = k % G, step1 = ((k - half) % G + G) % G; // ky of k, of k + K/2: k + K/2 - K
        float re0 = 0.f, im0 = 0.f, re1 = 0.f, im1 = 0.f;
        int p0 = 0, p1 = 0;
        for (int y0 = 0; y0 < G; y0 += chunk)
        {
            const int rows = min(chunk, G - y0);
            __syncthreads();
            for (int i = t; ROWS && i < rows * KX; i += kDftThreads)
                xs[i] = pair_get<VEC>(src, (long long)y0 * KX + i);
            __syncthreads();
            if (on)
#pragma unroll 4
                for (int y = 0; y < rows; ++y)
                {
                    const float2 x = ROWS ? xs[y * KX + kx] : pair_get<VEC>(src, (long long)(y0 + y) * KX + kx);
                    dft_add(x, twiddle(p0), sign, re0, im0);
                    dft_add(x, twiddle(p1), sign, re1, im1);
                    p0 += step0;
                    p0 -= p0 >= G ? G : 0;
                    p1 += step1;
                    p1 -= p1 >= G ? G : 0;
                }
        }
        if (on)
        {
            float *o = out + 2 * bc * (long long)K * KX;
            pair_put<VEC>(o, (long long)k * KX + kx, re0, im0);
            pair_put<VEC>(o, (long long)(k + half) * KX + kx, re1, im1);
        }
    }

    // out[bc, y, kx] = sum_k e^{s i 2 pi ky(k) y / G} in[bc, k, kx]; FP32 and/or BF16 output.  A CTA takes one
    // plane and `per` rows, kInvRows of usual length; the plane's modes and the twiddles sit in shared memory (TAB) where
    // they fit, k runs in order.
    constexpr int kInvRows = 32;
    template <bool TAB, bool VEC>
    __global__ void __launch_bounds__(kDftThreads) dft_y_inv_kernel(const float *in, float *out, bf16 *outb, const float *cs,
                                                                    const float *sn, int G, int K, int KX, float sign,
                                                                    int per, unsigned off)
    {
        extern __shared__ float2 dsm[];
        float2 *tab = dsm, *xs = dsm + G;
        const int t = threadIdx.x, half = K / 2;
        const long long bc = blockIdx.x;
        const float *src = in + 2 * bc * (long long)K * KX;
        auto twiddle = [&](int m) { return TAB ? tab[m] : make_float2(__ldg(cs + m), __ldg(sn + m)); };
        auto mode = [&](int k, int kx) { return TAB ? xs[k * KX + kx] : pair_get<VEC>(src, (long long)k * KX + kx); };
        for (int m = t; TAB && m < G; m += kDftThreads)
            tab[m] = make_float2(cs[m], sn[m]);
        for (int i = t; TAB && i < K * KX; i += kDftThreads)
            xs[i] = pair_get<VEC>(src, i);
        __syncthreads();
        const int y0 = (int)((off + blockIdx.y) * per), rows = min(per, G - y0);
        for (int i = t; i < rows * KX; i += kDftThreads)
        {
            const int kx = i % KX, y = y0 + i / KX;
            float re = 0.f, im = 0.f;
            int p = 0;
            for (int k = 0; k < half; ++k)
            {
                dft_add(mode(k, kx), twiddle(p), sign, re, im);
                p += y;
                p -= p >= G ? G : 0;
            }
            p = (G - (int)((long long)half * y % G)) % G; // ky = -K/2
            for (int k = half; k < K; ++k)
            {
                dft_add(mode(k, kx), twiddle(p), sign, re, im);
                p += y;
                p -= p >= G ? G : 0;
            }
            const long long o = (bc * G + y) * KX + kx;
            if (out)
                pair_put<VEC>(out, o, re, im);
            if (outb)
            {
                if constexpr (VEC)
                    reinterpret_cast<__nv_bfloat162 *>(outb)[o] = __floats2bfloat162_rn(re, im);
                else
                {
                    outb[2 * o] = __float2bfloat16(re);
                    outb[2 * o + 1] = __float2bfloat16(im);
                }
            }
        }
    }

    // ------------------------------------------------------------- mode mixing
    // out[b, o, m] = sum_c R[c, o, m] x[b, c, m]   (complex; m runs over the retained modes)
    __global__ void mix_fwd_kernel(const float *R, const float *x, float *out, int Bn, int Cin, int Cout, int Mm)
    {
        const long long total = (long long)Bn * Cout * Mm;
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x)
        {
            const int m = (int)(i % Mm);
            const int o = (int)((i / Mm) % Cout);
            const int b = (int)(i / ((long long)Mm * Cout));
            float re = 0.f, im = 0.f;
            for (int c = 0; c < Cin; ++c)
            {
                const float *r = R + 2 * (((long long)c * Cout + o) * Mm + m);
                const float *v = x + 2 * (((long long)b * Cin + c) * Mm + m);
                re += r[0] * v[0] - r[1] * v[1];
                im += r[0] * v[1] + r[1] * v[0];
            }
            out[2 * i] = re;
            out[2 * i + 1] = im;
        }
    }
    // dx[b, c, m] = sum_o conj(R[c, o, m]) dy[b, o, m]
    __global__ void mix_bwd_x_kernel(const float *R, const float *dy, float *dx, int Bn, int Cin, int Cout, int Mm)
    {
        const long long total = (long long)Bn * Cin * Mm;
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x)
        {
            const int m = (int)(i % Mm);
            const int c = (int)((i / Mm) % Cin);
            const int b = (int)(i / ((long long)Mm * Cin));
            float re = 0.f, im = 0.f;
            for (int o = 0; o < Cout; ++o)
            {
                const float *r = R + 2 * (((long long)c * Cout + o) * Mm + m);
                const float *d = dy + 2 * (((long long)b * Cout + o) * Mm + m);
                re += r[0] * d[0] + r[1] * d[1];
                im += r[0] * d[1] - r[1] * d[0];
            }
            dx[2 * i] = re;
            dx[2 * i + 1] = im;
        }
    }
    // dR[c, o, m] (+)= sum_b dy[b, o, m] conj(x[b, c, m])
    __global__ void mix_bwd_w_kernel(const float *x, const float *dy, float *dR, int Bn, int Cin, int Cout, int Mm,
                                     int accumulate)
    {
        const long long total = (long long)Cin * Cout * Mm;
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x)
        {
            const int m = (int)(i % Mm);
            const int o = (int)((i / Mm) % Cout);
            const int c = (int)(i / ((long long)Mm * Cout));
            float re = 0.f, im = 0.f;
            for (int b = 0; b < Bn; ++b)
            {
                const float *v = x + 2 * (((long long)b * Cin + c) * Mm + m);
                const float *d = dy + 2 * (((long long)b * Cout + o) * Mm + m);
                re += d[0] * v[0] + d[1] * v[1];
                im += d[1] * v[0] - d[0] * v[1];
            }
            if (accumulate)
            {
                dR[2 * i] += re;
                dR[2 * i + 1] += im;
            }
            else
            {
                dR[2 * i] = re;
                dR[2 * i + 1] = im;
            }
        }
    }

    // ------------------------------------------------------------- pointwise
    // z[b, c, p] += bias[c]; y = act ? gelu(z) : z (BF16 and/or FP32 copies)
    __global__ void bias_act_kernel(float *z, const float *bias, bf16 *yb, float *yf, int Bn, int Cn, long long P,
                                    int act)
    {
        const long long total = (long long)Bn * Cn * P;
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x)
        {
            const int c = (int)((i / P) % Cn);
            const float v = z[i] + bias[c];
            z[i] = v;
            const float y = act ? gelu(v) : v;
            if (yb)
                yb[i] = __float2bfloat16(y);
            if (yf)
                yf[i] = y;
        }
    }
    // dz = dy * gelu'(z) (act) or dy; FP32 and BF16 copies
    __global__ void act_bwd_kernel(const float *dy, const float *z, float *dz, bf16 *dzb, long long n, int act)
    {
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        {
            const float v = act ? dy[i] * gelu_grad(z[i]) : dy[i];
            if (dz)
                dz[i] = v;
            if (dzb)
                dzb[i] = __float2bfloat16(v);
        }
    }
    // db[c] (+)= sum_{b, p} dz[b, c, p] in a fixed summation order, in two launches so that the
    // whole GPU reads dz: block (c, slice) sums its slice of every sample's plane into part,
    // then one thread per channel adds the slices in order
    constexpr int kBiasSlices = 64;
    __global__ void bias_grad_partial_kernel(const float *__restrict__ dz, float *__restrict__ part, int Bn, int Cn,
                                             long long P)
    {
        __shared__ float red[256];
        const int c = blockIdx.x, sl = blockIdx.y;
        const long long chunk = (P + gridDim.y - 1) / gridDim.y;
        const long long p0 = sl * chunk, p1 = (p0 + chunk < P) ? p0 + chunk : P;
        float s = 0.f;
        for (int b = 0; b < Bn; ++b)
        {
            const float *row = dz + ((long long)b * Cn + c) * P;
            for (long long p = p0 + threadIdx.x; p < p1; p += blockDim.x)
                s += row[p];
        }
        red[threadIdx.x] = s;
        __syncthreads();
        for (int h = blockDim.x / 2; h > 0; h >>= 1)
        {
            if ((int)threadIdx.x < h)
                red[threadIdx.x] += red[threadIdx.x + h];
            __syncthreads();
        }
        if (threadIdx.x == 0)
            part[(long long)c * gridDim.y + sl] = red[0];
    }
    __global__ void bias_grad_final_kernel(const float *__restrict__ part, float *db, int Cn, int S, int accumulate)
    {
        const int c = blockIdx.x * blockDim.x + threadIdx.x;
        if (c >= Cn)
            return;
        float s = 0.f;
        for (int k = 0; k < S; ++k)
            s += part[(long long)c * S + k];
        db[c] = accumulate ? db[c] + s : s;
    }
    __global__ void f32_to_bf16_kernel(const float *x, bf16 *y, long long n)
    {
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
            y[i] = __float2bfloat16(x[i]);
    }
    // per-sample sum of squared errors and the gradient of the mean over everything
    __global__ void mse_kernel(const float *y, const float *t, float *dy, double *sse, long long n, float inv_count)
    {
        __shared__ double red[256];
        double s = 0.0;
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        {
            const float d = y[i] - t[i];
            s += (double)d * d;
            dy[i] = 2.f * d * inv_count;
        }
        red[threadIdx.x] = s;
        __syncthreads();
        for (int h = blockDim.x / 2; h > 0; h >>= 1)
        {
            if ((int)threadIdx.x < h)
                red[threadIdx.x] += red[threadIdx.x + h];
            __syncthreads();
        }
        if (threadIdx.x == 0)
            atomicAdd(sse, red[0]);
    }
    __global__ void adam_kernel(float *p, const float *g, float *m, float *v, long long n, float lr, float b1, float b2,
                                float eps, float c1, float c2, float wd)
    {
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        {
            const float gi = g[i] + wd * p[i];
            const float mi = b1 * m[i] + (1.f - b1) * gi;
            const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
            m[i] = mi;
            v[i] = vi;
            p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        }
    }

    // ------------------------------------------------------- grid <-> DG nodes
    // Inputs of one sample on the G x G cell-centred grid of [-1, 1]^2:
    // (gaussian forcing / amplitude, omega / omega_ref, x, y)
    __global__ void fno_inputs_kernel(float *in, int G, double cx, double cy, double sigma, double w)
    {
        const long long P = (long long)G * G;
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < P; i += (long long)gridDim.x * blockDim.x)
        {
            const int ix = (int)(i % G), iy = (int)(i / G);
            const double x = -1.0 + (ix + 0.5) * 2.0 / G, y = -1.0 + (iy + 0.5) * 2.0 / G;
            const double r2 = (x - cx) * (x - cx) + (y - cy) * (y - cy);
            in[i] = (float)exp(-r2 / (2.0 * sigma * sigma));
            in[P + i] = (float)w;
            in[2 * P + i] = (float)x;
            in[3 * P + i] = (float)y;
        }
    }
    // Lagrange basis of the n GLL nodes at t (barycentric form, FP64)
    __device__ void lagrange(int n, const double *xn, const double *wb, double t, double *phi)
    {
        for (int j = 0; j < n; ++j)
            if (t == xn[j])
            {
                for (int k = 0; k < n; ++k)
                    phi[k] = (k == j) ? 1.0 : 0.0;
                return;
            }
        double s = 0.0;
        for (int j = 0; j < n; ++j)
        {
            phi[j] = wb[j] / (t - xn[j]);
            s += phi[j];
        }
        for (int j = 0; j < n; ++j)
            phi[j] /= s;
    }
    // DG field u(d, i, j, el) on a uniform ne x ne mesh of [-1, 1]^2 (element el = ex + ne ey)
    // -> grid values out[d, iy, ix] * scale (its element's polynomial, evaluated exactly)
    __global__ void nodes_to_grid_kernel(const double *u, float *out, int ne, int n, const double *xn, const double *wb,
                                         int G, float scale)
    {
        const long long P = (long long)G * G;
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < P; i += (long long)gridDim.x * blockDim.x)
        {
            const int ix = (int)(i % G), iy = (int)(i / G);
            const double x = -1.0 + (ix + 0.5) * 2.0 / G, y = -1.0 + (iy + 0.5) * 2.0 / G;
            const double h = 2.0 / ne;
            int ex = (int)((x + 1.0) / h), ey = (int)((y + 1.0) / h);
            ex = min(max(ex, 0), ne - 1);
            ey = min(max(ey, 0), ne - 1);
            const double xi = 2.0 * (x - (-1.0 + ex * h)) / h - 1.0, eta = 2.0 * (y - (-1.0 + ey * h)) / h - 1.0;
            double px[16], py[16];
            lagrange(n, xn, wb, xi, px);
            lagrange(n, xn, wb, eta, py);
            const double *e = u + (long long)(ex + ne * ey) * 3 * n * n;
            double acc[3] = {0, 0, 0};
            for (int b = 0; b < n; ++b)
                for (int a = 0; a < n; ++a)
                {
                    const double wgt = px[a] * py[b];
                    const double *q = e + 3 * (a + n * b);
                    acc[0] += wgt * q[0];
                    acc[1] += wgt * q[1];
                    acc[2] += wgt * q[2];
                }
            for (int d = 0; d < 3; ++d)
                out[d * P + i] = (float)(acc[d] * scale);
        }
    }
    // grid field g[d, iy, ix] (cell centres) -> DG nodes (bilinear, clamped at the border) * scale
    __global__ void grid_to_nodes_kernel(const float *g, double *u, int ne, int n, const double *xn, int G, double scale)
    {
        const long long total = (long long)ne * ne * n * n;
        const long long P = (long long)G * G;
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x)
        {
            const int node = (int)(i % (n * n));
            const int el = (int)(i / (n * n));
            const int a = node % n, b = node / n, ex = el % ne, ey = el / ne;
            const double h = 2.0 / ne;
            const double x = -1.0 + ex * h + 0.5 * h * (xn[a] + 1.0), y = -1.0 + ey * h + 0.5 * h * (xn[b] + 1.0);
            const double fx = (x + 1.0) * G / 2.0 - 0.5, fy = (y + 1.0) * G / 2.0 - 0.5;
            int x0 = (int)floor(fx), y0 = (int)floor(fy);
            double tx = fx - x0, ty = fy - y0;
            if (x0 < 0) { x0 = 0; tx = 0.0; }
            if (y0 < 0) { y0 = 0; ty = 0.0; }
            if (x0 >= G - 1) { x0 = G - 2; tx = 1.0; }
            if (y0 >= G - 1) { y0 = G - 2; ty = 1.0; }
            for (int d = 0; d < 3; ++d)
            {
                const float *p = g + d * P;
                const double v = (1 - tx) * (1 - ty) * p[(long long)y0 * G + x0] + tx * (1 - ty) * p[(long long)y0 * G + x0 + 1] +
                                 (1 - tx) * ty * p[(long long)(y0 + 1) * G + x0] + tx * ty * p[(long long)(y0 + 1) * G + x0 + 1];
                u[3 * i + d] = v * scale;
            }
        }
    }

    cudaStream_t st(void *s) { return static_cast<cudaStream_t>(s); }
    int done(const char *what)
    {
        const cudaError_t e = cudaGetLastError();
        return e == cudaSuccess ? WDG_OK : wdg::cuda_fail(e, what);
    }
} // namespace

extern "C"
{
    int wdg_fno_gemm(const void *A, const void *B, float *C, int M, int N, int K, long long lda, long long ldb,
                     long long ldc, long long strideA, long long strideB, long long strideC, int batch, int transA,
                     int transB, float alpha, float beta, int ksplit, void *stream)
    {
        if (!A || !B || !C || M < 1 || N < 1 || K < 1 || batch < 1 || ksplit < 0)
            return wdg::fail(WDG_ERR_ARG, "wdg_fno_gemm: bad arguments");
        GemmArgs g{};
        g.A = static_cast<const bf16 *>(A);
        g.B = static_cast<const bf16 *>(B);
        g.C = C;
        g.M = M;
        g.N = N;
        g.K = K;
        g.lda = lda;
        g.ldb = ldb;
        g.ldc = ldc;
        g.sA = strideA;
        g.sB = strideB;
        g.sC = strideC;
        g.alpha = alpha;
        g.beta = beta;
        g.ksplit = (ksplit > 0) ? ((ksplit + TK - 1) / TK) * TK : ((K + TK - 1) / TK) * TK;
        const int nsplit = (K + g.ksplit - 1) / g.ksplit;
        // split K, or a batch that sums into one C (stride 0): accumulate atomically, beta first
        g.atomic = (nsplit > 1 || (batch > 1 && strideC == 0)) ? 1 : 0;
        if (g.atomic && beta != 1.f)
        {
            if (beta != 0.f)
                return wdg::fail(WDG_ERR_ARG, "wdg_fno_gemm: atomic accumulation needs beta 0 or 1");
            const int nb = (strideC == 0) ? 1 : batch;
            for (int b = 0; b < nb; ++b)
                if (cudaMemset2DAsync(C + b * strideC, sizeof(float) * ldc, 0, sizeof(float) * N, M, st(stream)) !=
                    cudaSuccess)
                    return done("wdg_fno_gemm");
        }
        if ((M + TM - 1) / TM > 65535 || (long long)batch * nsplit > 65535)
            return wdg::fail(WDG_ERR_ARG, "wdg_fno_gemm: problem too large for one launch");
        gemm_run<EPI_STORE>(g, transA, transB, batch * nsplit, st(stream));
        return done("wdg_fno_gemm");
    }

    // batch products op(A[b]) op(B[b]) with an epilogue instead of alpha and beta: mode 1 v = acc + bias[row],
    // out = v, y = BF16 act(v); mode 2 v = acc gelu'(z) (act) or acc, out = v, y = BF16 v; out and y nullable,
    // out, z and y of C's shape (M, ldc) per batch
    int wdg_fno_gemm_act(const void *A, const void *B, float *out, int M, int N, int K, long long lda, long long ldb,
                         long long ldc, long long strideA, long long strideB, long long strideC, int batch, int transA,
                         int transB, int mode, const float *bias, const float *z, void *y, int act, void *stream)
    {
        if (!A || !B || (!out && !y) || M < 1 || N < 1 || K < 1 || batch < 1 || batch > 65535 ||
            (M + TM - 1) / TM > 65535 || (mode != EPI_BIAS_ACT && mode != EPI_ACT_BWD) || (mode == EPI_BIAS_ACT && !bias) ||
            (mode == EPI_ACT_BWD && act && !z))
            return wdg::fail(WDG_ERR_ARG, "wdg_fno_gemm_act: bad arguments");
        GemmArgs g{};
        g.A = static_cast<const bf16 *>(A);
        g.B = static_cast<const bf16 *>(B);
        g.C = out;
        g.M = M;
        g.N = N;
        g.K = K;
        g.lda = lda;
        g.ldb = ldb;
        g.ldc = ldc;
        g.sA = strideA;
        g.sB = strideB;
        g.sC = strideC;
        g.alpha = 1.f;
        g.ksplit = ((K + TK - 1) / TK) * TK;
        g.e.bias = bias;
        g.e.z = z;
        g.e.y = static_cast<bf16 *>(y);
        g.e.act = act;
        if (mode == EPI_BIAS_ACT)
            gemm_run<EPI_BIAS_ACT>(g, transA, transB, batch, st(stream));
        else
            gemm_run<EPI_ACT_BWD>(g, transA, transB, batch, st(stream));
        return done("wdg_fno_gemm_act");
    }

    // a Fourier layer's output, forward (back = 0) or backward; see layer_kernel.  C and K1 multiples of 8, at
    // most 32; G a multiple of 8; every array 16-byte aligned
    int wdg_fno_layer(const void *U, const void *X, const void *W, const void *V, const float *bias, const float *z,
                      float *out, void *y, int B, int C, int K1, int G, int act, int back, void *stream)
    {
        if (!U || !X || !W || !V || (!out && !y) || B < 1 || B > 65535 || C < 8 || C > 32 || C % 8 || K1 < 8 || K1 > 32 ||
            K1 % 8 || G < 8 || G > 65535 || G % 8 || (back ? (act && !z) : !bias))
            return wdg::fail(WDG_ERR_ARG, "wdg_fno_layer: bad arguments");
        if ((((uintptr_t)U | (uintptr_t)X | (uintptr_t)W | (uintptr_t)V | (uintptr_t)out | (uintptr_t)y) & 15u) != 0)
            return wdg::fail(WDG_ERR_ARG, "wdg_fno_layer: arrays must be 16-byte aligned");
        LayerArgs g{};
        g.U = static_cast<const bf16 *>(U);
        g.X = static_cast<const bf16 *>(X);
        g.W = static_cast<const bf16 *>(W);
        g.V = static_cast<const bf16 *>(V);
        g.C = out;
        g.Cn = C;
        g.K1 = K1;
        g.G = G;
        g.e.bias = bias;
        g.e.z = z;
        g.e.y = static_cast<bf16 *>(y);
        g.e.act = act;
        const dim3 grid((G + 127) / 128, G, B);
        if (back)
            layer_kernel<true><<<grid, 128, 0, st(stream)>>>(g);
        else
            layer_kernel<false><<<grid, 128, 0, st(stream)>>>(g);
        return done("wdg_fno_layer");
    }

    int wdg_fno_dft_y(const float *in, float *out, void *out_bf16, const float *cos_tab, const float *sin_tab, int BC,
                      int G, int K, int KX, int inverse, float sign, void *stream)
    {
        if (!in || !cos_tab || !sin_tab || BC < 1 || G < 2 || K < 2 || (K & 1) || KX < 1 || (!out && !out_bf16))
            return wdg::fail(WDG_ERR_ARG, "wdg_fno_dft_y: bad arguments");
        const bool vec = (((uintptr_t)in | (uintptr_t)out) & 7u) == 0 && ((uintptr_t)out_bf16 & 3u) == 0;
        if (!inverse)
        {
            if (!out)
                return wdg::fail(WDG_ERR_ARG, "wdg_fno_dft_y: the forward transform writes FP32");
            const long long pairs = (long long)(K / 2) * KX;
            const bool fits = vec && pairs <= INT_MAX - kDftThreads; // the outputs are counted in an int
            const bool tab = fits && sizeof(float2) * ((size_t)G + KX) <= kDftSmem;
            const size_t left = kDftSmem / sizeof(float2) - (tab ? G : 0);
            const bool rows = fits && left >= (size_t)KX;
            const int chunk = rows ? (int)std::min<size_t>(kDftRows, left / KX) : G;
            const size_t smem = sizeof(float2) * ((tab ? (size_t)G : 0) + (rows ? (size_t)chunk * KX : 0));
            auto kern = tab    ? dft_y_fwd_kernel<true, true, true>
                        : rows ? dft_y_fwd_kernel<false, true, true>
                        : vec  ? dft_y_fwd_kernel<false, false, true>
                               : dft_y_fwd_kernel<false, false, false>;
            if (smem > 48 * 1024)
                cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDftSmem);
            const long long q = (pairs + kDftThreads - 1) / kDftThreads;
            for (long long q0 = 0; q0 < q; q0 += kGridY)
                kern<<<dim3(BC, (unsigned)std::min(kGridY, q - q0)), kDftThreads, smem, st(stream)>>>(
                    in, out, cos_tab, sin_tab, G, K, KX, sign, chunk, (unsigned)q0);
        }
        else
        {
            const size_t want = sizeof(float2) * ((size_t)G + (size_t)K * KX);
            const bool tab = vec && want <= kDftSmem;
            const int per = std::max(1, std::min(kInvRows, (INT_MAX - kDftThreads) / KX)); // their values are counted in an int
            auto kern = tab ? dft_y_inv_kernel<true, true> : vec ? dft_y_inv_kernel<false, true> : dft_y_inv_kernel<false, false>;
            if (tab && want > 48 * 1024)
                cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDftSmem);
            const long long q = ((long long)G + per - 1) / per;
            for (long long q0 = 0; q0 < q; q0 += kGridY)
                kern<<<dim3(BC, (unsigned)std::min(kGridY, q - q0)), kDftThreads, tab ? want : 0, st(stream)>>>(
                    in, out, static_cast<bf16 *>(out_bf16), cos_tab, sin_tab, G, K, KX, sign, per, (unsigned)q0);
        }
        return done("wdg_fno_dft_y");
    }

    int wdg_fno_mix(const float *R, const float *x, float *out, int B, int Cin, int Cout, int modes, void *stream)
    {
        mix_fwd_kernel<<<blocks((long long)B * Cout * modes), 256, 0, st(stream)>>>(R, x, out, B, Cin, Cout, modes);
        return done("wdg_fno_mix");
    }
    int wdg_fno_mix_bwd(const float *R, const float *x, const float *dy, float *dx, float *dR, int B, int Cin, int Cout,
                        int modes, int accumulate, void *stream)
    {
        if (dx)
            mix_bwd_x_kernel<<<blocks((long long)B * Cin * modes), 256, 0, st(stream)>>>(R, dy, dx, B, Cin, Cout, modes);
        if (dR)
            mix_bwd_w_kernel<<<blocks((long long)Cin * Cout * modes), 256, 0, st(stream)>>>(x, dy, dR, B, Cin, Cout,
                                                                                            modes, accumulate);
        return done("wdg_fno_mix_bwd");
    }
    int wdg_fno_bias_act(float *z, const float *bias, void *y_bf16, float *y_f32, int B, int C, long long P, int act,
                         void *stream)
    {
        bias_act_kernel<<<blocks((long long)B * C * P), 256, 0, st(stream)>>>(z, bias, static_cast<bf16 *>(y_bf16),
                                                                               y_f32, B, C, P, act);
        return done("wdg_fno_bias_act");
    }
    int wdg_fno_act_bwd(const float *dy, const float *z, float *dz, void *dz_bf16, long long n, int act, void *stream)
    {
        act_bwd_kernel<<<blocks(n), 256, 0, st(stream)>>>(dy, z, dz, static_cast<bf16 *>(dz_bf16), n, act);
        return done("wdg_fno_act_bwd");
    }
    int wdg_fno_bias_grad(const float *dz, float *db, int B, int C, long long P, int accumulate, void *stream)
    {
        if (B < 1 || C < 1 || P < 1)
            return wdg::fail(WDG_ERR_ARG, "wdg_fno_bias_grad: empty shape");
        // the slices' partial sums in stream-ordered scratch
        float *part = nullptr;
        const cudaError_t e = cudaMallocAsync(reinterpret_cast<void **>(&part), sizeof(float) * C * kBiasSlices, st(stream));
        if (e != cudaSuccess)
            return wdg::cuda_fail(e, "cudaMallocAsync (wdg_fno_bias_grad)");
        bias_grad_partial_kernel<<<dim3(C, kBiasSlices), 256, 0, st(stream)>>>(dz, part, B, C, P);
        bias_grad_final_kernel<<<(C + 127) / 128, 128, 0, st(stream)>>>(part, db, C, kBiasSlices, accumulate);
        cudaFreeAsync(part, st(stream));
        return done("wdg_fno_bias_grad");
    }
    int wdg_fno_to_bf16(const float *x, void *y, long long n, void *stream)
    {
        f32_to_bf16_kernel<<<blocks(n), 256, 0, st(stream)>>>(x, static_cast<bf16 *>(y), n);
        return done("wdg_fno_to_bf16");
    }
    int wdg_fno_mse(const float *y, const float *t, float *dy, double *sse, long long n, float inv_count, void *stream)
    {
        mse_kernel<<<blocks(n), 256, 0, st(stream)>>>(y, t, dy, sse, n, inv_count);
        return done("wdg_fno_mse");
    }
    int wdg_fno_adam(float *p, const float *g, float *m, float *v, long long n, float lr, float beta1, float beta2,
                     float eps, int step, float weight_decay, void *stream)
    {
        if (step < 1)
            return wdg::fail(WDG_ERR_ARG, "wdg_fno_adam: steps count from 1");
        float c1 = 1.f, c2 = 1.f;
        for (int i = 0; i < step && i < 100000; ++i)
        {
            c1 *= beta1;
            c2 *= beta2;
        }
        adam_kernel<<<blocks(n), 256, 0, st(stream)>>>(p, g, m, v, n, lr, beta1, beta2, eps, 1.f - c1, 1.f - c2,
                                                       weight_decay);
        return done("wdg_fno_adam");
    }
    int wdg_fno_inputs(float *in, int G, double cx, double cy, double sigma, double w, void *stream)
    {
        fno_inputs_kernel<<<blocks((long long)G * G), 256, 0, st(stream)>>>(in, G, cx, cy, sigma, w);
        return done("wdg_fno_inputs");
    }
    int wdg_fno_nodes_to_grid(const double *u, float *out, int ne, int n, const double *gll_x, const double *gll_bw,
                              int G, float scale, void *stream)
    {
        if (n < 2 || n > 16)
            return wdg::fail(WDG_ERR_ARG, "wdg_fno_nodes_to_grid: 2..16 nodes per direction");
        nodes_to_grid_kernel<<<blocks((long long)G * G), 256, 0, st(stream)>>>(u, out, ne, n, gll_x, gll_bw, G, scale);
        return done("wdg_fno_nodes_to_grid");
    }
    int wdg_fno_grid_to_nodes(const float *g, double *u, int ne, int n, const double *gll_x, int G, double scale,
                              void *stream)
    {
        grid_to_nodes_kernel<<<blocks((long long)ne * ne * n * n), 256, 0, st(stream)>>>(g, u, ne, n, gll_x, G, scale);
        return done("wdg_fno_grid_to_nodes");
    }
}
