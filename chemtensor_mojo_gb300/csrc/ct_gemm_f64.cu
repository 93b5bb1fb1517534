// Plain-form FP64 contraction kernel: a strided, batched SIMT GEMM.
//
// C(m,n) = alpha * sum_k A(m,k) B(k,n) + beta * C(m,n) with arbitrary element
// strides for every index and a two-level batch index, so every contraction of
// the path (dense_tensor_dot, dense_tensor.mojo:963-1328, and the permute +
// GEMM chains of dmrg.mojo:254-374 / environments.mojo:99-417) is one launch
// with the permutes folded into the operand addressing -- no physical
// transposes.  FP64 on GB300 issues at a small fraction of the FP32 rate (one
// warp instruction per 64 clocks and SM quarter), so a 64x64x16 smem tile with
// a 4x4 register block saturates the FP64 pipe of a product that fills the
// GPU; the others are spread as thin as one warp per SM quarter.  The
// tensor-core paths live in ct_tc.cu and ct_f64mod.cu.
#include <cooperative_groups.h>

#include <algorithm>

#include "ct_common.cuh"

namespace {

constexpr int BK = 16;

// One CTA computes a TBM x TBN tile of C with (TBM/4) x (TBN/4) threads, each
// holding a 4 x 4 register block.
template <int TBM, int TBN, bool A_K_CONTIG, bool B_N_CONTIG>
__global__ void __launch_bounds__((TBM / 4) * (TBN / 4)) gemm_f64_kernel(GemmDesc g) {
    ct_pdl();
    constexpr int NT = (TBM / 4) * (TBN / 4);
    constexpr int TX = TBN / 4;
    if (ct_skip(g.skip)) return;
    __shared__ double As[BK][TBM + 1];
    __shared__ double Bs[BK][TBN + 1];

    // blockIdx.z = batch * ksplit + k-chunk
    const int64_t ks = (int64_t)blockIdx.z % g.ksplit;
    const int64_t bz = (int64_t)blockIdx.z / g.ksplit;
    const int64_t b1 = bz / g.nb0, b0 = bz % g.nb0;
    const double* A = g.A + b1 * g.sA1 + b0 * g.sA0;
    const double* B = g.B + b1 * g.sB1 + b0 * g.sB0;
    double* C = g.C + b1 * g.sC1 + b0 * g.sC0;

    const int64_t m0 = (int64_t)blockIdx.y * TBM, n0 = (int64_t)blockIdx.x * TBN;
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
    if (g.tri == 1 && n0 >= m0 + TBM) return;   // tile strictly above the diagonal
    int64_t kend = (g.tri == 2 && m0 + TBM < g.K) ? m0 + TBM : g.K;
    int64_t kbeg = 0;
    if (g.ksplit > 1) {
        const int64_t chunk = ((g.K + g.ksplit - 1) / g.ksplit + BK - 1) / BK * BK;
        kbeg = ks * chunk;
        if (kbeg + chunk < kend) kend = kbeg + chunk;
    }

    double acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0;

    for (int64_t k0 = kbeg; k0 < kend; k0 += BK) {
#pragma unroll
        for (int r = 0; r < (BK * TBM) / NT; ++r) {
            const int e = tid + NT * r;
            int mm, kk;
            if (A_K_CONTIG) { kk = e % BK; mm = e / BK; }
            else            { mm = e % TBM; kk = e / TBM; }
            const int64_t gm = m0 + mm, gk = k0 + kk;
            As[kk][mm] = (gm < g.M && gk < kend) ? A[gm * g.sAm + gk * g.sAk] : 0.0;
        }
#pragma unroll
        for (int r = 0; r < (BK * TBN) / NT; ++r) {
            const int e = tid + NT * r;
            int nn, kk;
            if (B_N_CONTIG) { nn = e % TBN; kk = e / TBN; }
            else            { kk = e % BK; nn = e / BK; }
            const int64_t gn = n0 + nn, gk = k0 + kk;
            Bs[kk][nn] = (gn < g.N && gk < kend) ? B[gk * g.sBk + gn * g.sBn] : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            double a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][ty + (TBM / 4) * i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx + (TBN / 4) * j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int64_t gm = m0 + ty + (TBM / 4) * i;
        if (gm >= g.M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int64_t gn = n0 + tx + (TBN / 4) * j;
            if (gn >= g.N) continue;
            if (g.ksplit > 1) {
                g.part[(ks * g.M + gm) * g.N + gn] = acc[i][j];
                continue;
            }
            double* c = C + gm * g.sCm + gn * g.sCn;
            double v = g.alpha * acc[i][j];
            if (g.beta != 0.0) v = fma(g.beta, *c, v);
            *c = v;
        }
    }
}

// Products too small to fill the GPU with 64 x 64 tiles: an 8 x 16 tile per CTA, one element of
// C per thread, four warps.  What bounds it is a thread's own chain of FMAs, which issue at one
// per 64 clocks whether one element or sixteen are held per thread, so the elements go to as many
// SM quarters as there are (32 x 32 tiles of two warps with 4 x 4 registers before: 16 elements
// per thread in a row, on an eighth of the SMs).  The next K block is loaded to registers while
// this one is computed.  Every element adds its products in the order of k, and the K pieces in
// the order of the pieces, as the 64 x 64 kernel and splitk_reduce_kernel do; up to SP_MAXC
// pieces are one cluster, whose first CTA adds them up, without scratch memory or a second launch.
// Triangular forms keep the 32-wide granularity of what is skipped (TRI).
// Measured (us per call, 32 x 32 tiles / here): 9x17x33 33 / 16, 128x32x96 27 / 16, 64x64x512
// 29 / 20, 33x300x1000 84 / 33, 24x24x100000 414 / 152, 512x512x512 306 / 232, 1024x1024x64
// 127 / 119.
constexpr int SP_M = 8, SP_N = 16, SP_K = 32, SP_NT = SP_M * SP_N;
constexpr int SP_MAXC = 8;
constexpr int TRI = 32;

template <bool A_K_CONTIG, bool B_N_CONTIG>
__global__ void __launch_bounds__(SP_NT) gemm_f64_spread_kernel(GemmDesc g, int clustered) {
    ct_pdl();
    if (ct_skip(g.skip)) return;
    __shared__ double As[SP_K][SP_M + 1];
    __shared__ double Bs[SP_K][SP_N + 1];
    __shared__ double piece[SP_MAXC][SP_NT];
    const int ks = (int)((int64_t)blockIdx.z % g.ksplit);
    const int64_t bz = (int64_t)blockIdx.z / g.ksplit;
    const int64_t b1 = bz / g.nb0, b0 = bz % g.nb0;
    const double* A = g.A + b1 * g.sA1 + b0 * g.sA0;
    const double* B = g.B + b1 * g.sB1 + b0 * g.sB0;
    const int64_t m0 = (int64_t)blockIdx.y * SP_M, n0 = (int64_t)blockIdx.x * SP_N;
    const int64_t mt = m0 / TRI * TRI;
    if (g.tri == 1 && n0 / TRI * TRI >= mt + TRI) return;   // the whole cluster
    // the first CTA's shared memory may be written once it has started: everyone arrives here, and
    // waits before its store (the K loop covers the latency; a piece without any K comes there at once)
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    if (clustered) (void)cl.barrier_arrive();
    int64_t kend = (g.tri == 2 && mt + TRI < g.K) ? mt + TRI : g.K;
    int64_t kbeg = 0;
    if (g.ksplit > 1) {
        const int64_t chunk = ((g.K + g.ksplit - 1) / g.ksplit + BK - 1) / BK * BK;
        kbeg = ks * chunk;
        if (kbeg + chunk < kend) kend = kbeg + chunk;
    }
    const int tid = threadIdx.x, tx = tid % SP_N, ty = tid / SP_N;
    constexpr int NA = SP_M * SP_K / SP_NT, NB = SP_N * SP_K / SP_NT;
    int am[NA], ak[NA], bn[NB], bk[NB];
    const double *pa[NA], *pb[NB];
#pragma unroll
    for (int r = 0; r < NA; ++r) {
        const int e = tid + SP_NT * r;
        if (A_K_CONTIG) { ak[r] = e % SP_K; am[r] = e / SP_K; }
        else            { am[r] = e % SP_M; ak[r] = e / SP_M; }
        pa[r] = m0 + am[r] < g.M ? A + (m0 + am[r]) * g.sAm + (kbeg + ak[r]) * g.sAk : nullptr;
    }
#pragma unroll
    for (int r = 0; r < NB; ++r) {
        const int e = tid + SP_NT * r;
        if (B_N_CONTIG) { bn[r] = e % SP_N; bk[r] = e / SP_N; }
        else            { bk[r] = e % SP_K; bn[r] = e / SP_K; }
        pb[r] = n0 + bn[r] < g.N ? B + (n0 + bn[r]) * g.sBn + (kbeg + bk[r]) * g.sBk : nullptr;
    }
    double ra[NA], rb[NB];
    auto load = [&](int64_t k0) {
#pragma unroll
        for (int r = 0; r < NA; ++r) {
            ra[r] = (pa[r] && k0 + ak[r] < kend) ? *pa[r] : 0.0;
            if (pa[r]) pa[r] += SP_K * g.sAk;
        }
#pragma unroll
        for (int r = 0; r < NB; ++r) {
            rb[r] = (pb[r] && k0 + bk[r] < kend) ? *pb[r] : 0.0;
            if (pb[r]) pb[r] += SP_K * g.sBk;
        }
    };
    double acc = 0.0;
    if (kbeg < kend) load(kbeg);
    for (int64_t k0 = kbeg; k0 < kend; k0 += SP_K) {
        __syncthreads();
#pragma unroll
        for (int r = 0; r < NA; ++r) As[ak[r]][am[r]] = ra[r];
#pragma unroll
        for (int r = 0; r < NB; ++r) Bs[bk[r]][bn[r]] = rb[r];
        __syncthreads();
        if (k0 + SP_K < kend) load(k0 + SP_K);
        const int kn = kend - k0 < SP_K ? (int)(kend - k0) : SP_K;
#pragma unroll 1
        for (int kk = 0; kk < kn; kk += 8) {
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                // (the rows from kn on hold zeros)
                if (u < 4 || kk + u < kn) acc = fma(As[kk + u][ty], Bs[kk + u][tx], acc);
            }
        }
    }
    const int64_t gm = m0 + ty, gn = n0 + tx;
    if (g.ksplit > 1) {
        if (clustered) {
            cl.barrier_wait();
            *cl.map_shared_rank(&piece[ks][tid], 0) = acc;
            cl.sync();
            if (ks != 0) return;
            acc = 0.0;
            for (int64_t i = 0; i < g.ksplit; ++i) acc += piece[i][tid];
        } else if (gm < g.M && gn < g.N) {
            g.part[(ks * g.M + gm) * g.N + gn] = acc;
            return;
        }
    }
    if (gm >= g.M || gn >= g.N) return;
    double* c = g.C + b1 * g.sC1 + b0 * g.sC0 + gm * g.sCm + gn * g.sCn;
    double v = g.alpha * acc;
    if (g.beta != 0.0) v = fma(g.beta, *c, v);
    *c = v;
}

// C = alpha * sum_ks part[ks] + beta * C, the partial sums added in a fixed
// order (deterministic); tiles the GEMM kernel skips (tri == 1) stay untouched.
__global__ void splitk_reduce_kernel(GemmDesc g, int tile) {
    ct_pdl();
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < g.M * g.N;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t gm = t / g.N, gn = t % g.N;
        if (g.tri == 1 && (gn / tile) * tile >= (gm / tile) * tile + tile) continue;
        double a = 0.0;
        for (int64_t ks = 0; ks < g.ksplit; ++ks) a += g.part[(ks * g.M + gm) * g.N + gn];
        double* c = g.C + gm * g.sCm + gn * g.sCn;
        double v = g.alpha * a;
        if (g.beta != 0.0) v = fma(g.beta, *c, v);
        *c = v;
    }
}

template <int TBM, int TBN>
int launch_tiles(ct_handle* h, const GemmDesc& g, int64_t nb) {
    dim3 grid((unsigned)ct_cdiv(g.N, TBN), (unsigned)ct_cdiv(g.M, TBM), (unsigned)(nb * g.ksplit));
    if (grid.y > 65535 || grid.z > 65535) {
        ct_seterr(h, "gemm grid too large (M=%lld nb=%lld)", (long long)g.M, (long long)nb);
        return CT_ERR_UNSUPPORTED;
    }
    constexpr int nt = (TBM / 4) * (TBN / 4);
    const bool ak = (g.sAk == 1);
    const bool bn = (g.sBn == 1);
    if (ak && bn) { ct_launch(h, gemm_f64_kernel<TBM, TBN, true, true>, grid, nt, 0, g); ct_note_launch(); }
    else if (ak) { ct_launch(h, gemm_f64_kernel<TBM, TBN, true, false>, grid, nt, 0, g); ct_note_launch(); }
    else if (bn) { ct_launch(h, gemm_f64_kernel<TBM, TBN, false, true>, grid, nt, 0, g); ct_note_launch(); }
    else { ct_launch(h, gemm_f64_kernel<TBM, TBN, false, false>, grid, nt, 0, g); ct_note_launch(); }
    CT_LAUNCH_CHECK(h);
    return CT_OK;
}

int launch_spread(ct_handle* h, const GemmDesc& g, int64_t nb) {
    // (the limits of 32 x 32 tiles)
    const int64_t ym = ct_cdiv(g.M, SP_M), z = nb * g.ksplit;
    if (ym > 65535 || z > 65535) {
        ct_seterr(h, "gemm grid too large (M=%lld nb=%lld)", (long long)g.M, (long long)nb);
        return CT_ERR_UNSUPPORTED;
    }
    const bool clustered = g.ksplit > 1 && g.ksplit <= SP_MAXC;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)ct_cdiv(g.N, SP_N), (unsigned)ym, (unsigned)z);
    cfg.blockDim = dim3(SP_NT);
    cfg.stream = h->stream;
    cudaLaunchAttribute at[2]{};
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // (as ct_launch)
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim = {1, 1, (unsigned)g.ksplit};
    cfg.attrs = at;
    cfg.numAttrs = clustered ? 2 : 1;
    const bool ak = (g.sAk == 1), bn = (g.sBn == 1);
    auto* f = ak ? (bn ? gemm_f64_spread_kernel<true, true> : gemm_f64_spread_kernel<true, false>)
                 : (bn ? gemm_f64_spread_kernel<false, true> : gemm_f64_spread_kernel<false, false>);
    CT_CUDA(h, cudaLaunchKernelEx(&cfg, f, g, (int)clustered)); ct_note_launch();
    if (g.ksplit > 1 && !clustered) {
        const int64_t tot = g.M * g.N;
        int64_t blocks = ct_cdiv(tot, 256);
        if (blocks > 4 * (int64_t)h->num_sms) blocks = 4 * (int64_t)h->num_sms;
        ct_launch(h, splitk_reduce_kernel, (unsigned)blocks, 256, 0, g, TRI); ct_note_launch();
        CT_LAUNCH_CHECK(h);
    }
    return CT_OK;
}

}  // namespace

int ct_gemm_f64_launch(ct_handle* h, const GemmDesc& g) {
    if (g.M <= 0 || g.N <= 0) return CT_OK;
    const int64_t nb = g.nb1 * g.nb0;
    if (nb <= 0) return CT_OK;
    if (g.K <= 0 && g.beta == 1.0) return CT_OK;  // C unchanged; K = 0 otherwise gives C = beta*C
    GemmDesc gg = g;
    gg.ksplit = 1;
    gg.part = nullptr;
    const int64_t sms = h->num_sms;
    // 64 x 64 tiles when there are two per SM: they fill the FP64 pipes (1024 x 1024 x 64 is the
    // largest below, 127 us on 32 x 32 tiles and 119 spread); else the spread form, with K split
    // over the idle SMs when there is less than one 32 x 32 block of C for each
    // tiles that do work (tri == 1 skips those strictly above the diagonal)
    auto active = [&](int64_t t) {
        const int64_t tm = ct_cdiv(g.M, t), tn = ct_cdiv(g.N, t);
        if (g.tri != 1) return tm * tn * nb;
        int64_t a = 0;
        for (int64_t i = 0; i < tm; ++i) a += std::min<int64_t>(tn, i + 1);
        return a * nb;
    };
    if (active(64) >= 2 * sms) return launch_tiles<64, 64>(h, gg, nb);
    const int64_t tiles = active(32);
    if (nb == 1 && tiles < sms && g.K >= 64) {
        int64_t ks = ct_cdiv(sms, tiles);
        if (ks > g.K / 32) ks = g.K / 32;
        if (h->no_alloc) {
            // partials only in the caller's fixed region, as many K pieces as it holds
            const int64_t fit = (int64_t)(h->splitk_fixed_cap / (size_t)(g.M * g.N));
            if (ks > fit) ks = fit;
            if (ks > 1) {
                gg.ksplit = ks;
                gg.part = h->splitk_fixed;
            }
        } else if (ks > 1) {
            const size_t need = ks > SP_MAXC ? (size_t)(ks * g.M * g.N) : 0;
            if (h->splitk_cap < need) {
                if (h->splitk) cudaFree(h->splitk);
                h->splitk = nullptr;
                h->splitk_cap = 0;
                CT_CUDA(h, ct_malloc(h, (void**)&h->splitk, need * sizeof(double)));
                h->splitk_cap = need;
            }
            gg.ksplit = ks;
            gg.part = h->splitk;
        }
    }
    return launch_spread(h, gg, nb);
}
