// FP64-form GEMM on the BF16 tensor cores by residues (no rounding but the operands').
//
// C[M,N] = sum_k A[m,k] B[n,k] with FP64 A, B and C, for the contraction chains of the FP64
// form.  The scheme is that of K. Ozaki, Y. Uchino and T. Imamura, Ozaki Scheme II: a
// GEMM-oriented emulation of floating-point matrix multiplication using an integer modular
// technique (arXiv:2504.08009, 2025), here on tcgen05 kind::f16 with BF16 operands:
//   * every row of A and of B is scaled by a power of two and rounded to integers of b bits,
//     |X| <= 2^b (b = 62, less only beyond K = 2^15: the moduli hold 2 K 2^(2b) < P);
//   * for each of MODS pairwise coprime moduli m_i <= 256 the residues of A and B (at most
//     128 in magnitude, exact in BF16) are multiplied: a product is at most 2^14, so 1024 of K
//     add up exactly in the FP32 accumulator, which the epilogue reduces modulo m_i;
//   * the Chinese remainder theorem gives the integer product sum, below P / 2 = prod m_i / 2
//     in magnitude, exactly; it is rounded to FP64 once and scaled back.
// The only error is the operands' rounding, 2^-(b + 1) of each row's largest entry, and the
// final one.  Relative error against exact products, N(0,1) operands, 1024^3: 4.7e-17 (half an
// ulp), the SIMT kernel's 1.1e-15.  (16 moduli, b = 57, are 12% cheaper, but rows and columns
// graded in opposite directions, exp(-8 k / K) against exp(8 k / K), then lose to the SIMT
// kernel: 2.6e-15 against 3e-16 at 256^3.)
//
// What bounds it.  MODS products of full-size tensor-core tiles per FP64 product (the sliced
// scheme of ct_ozaki.cu forms 36 to 45, on 64-wide tiles that its eight accumulators leave);
// for small products the four launches.  FP64 arithmetic issues at 1/64 of the FP32 rate
// here, so the residues, the reduction and the reconstruction are integer and FP32 work.
//
// A row with an infinity or a NaN has no scale: its elements of C are computed as plain FP64
// dot products from the operands, so non-finite values go where an FP64 GEMM takes them.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <math.h>

#include <algorithm>

#include "ct_ops.cuh"
#include "ct_tc_ptx.cuh"

PFN_cuTensorMapEncodeTiled_v12000 ct_tma_encoder();

namespace {

constexpr int MODS = 18;
constexpr int GROUPS = MODS / 3;                        // reconstructed three moduli at a time
constexpr int FM_BM = 128;
constexpr int FM_BN = 128;
constexpr int FM_BK = 64;                               // BF16 of K per 128-byte row
constexpr int FM_STAGES = 4;
constexpr int FM_KCH = 16;                              // k-blocks per exact chunk (1024 of K)
constexpr int FM_NB = 512 / FM_BN;                      // accumulators in TMEM
constexpr int FM_EPW = 4;                               // epilogue warps per TMEM lane quadrant
constexpr int FM_HC = FM_BN / FM_EPW;                   // columns per epilogue thread
constexpr int FM_THREADS = 32 * (2 + 4 * FM_EPW);
constexpr int FM_A_BYTES = FM_BM * FM_BK * 2;           // 16 KB
constexpr int FM_STAGE = FM_A_BYTES + FM_BN * FM_BK * 2;
constexpr int FM_SMEM = FM_STAGES * FM_STAGE + 1024 /*align*/ + 256 /*barriers*/;
constexpr int FM_NONFINITE = 0x40000000;                // exponent of a row with an infinity or a NaN
constexpr int LIMBS = 5;                                // 32-bit limbs of P (141 bits) and of the sums

// pairwise coprime, at most 256: P = 2^140.6
constexpr int kMod[MODS] = {256, 253, 251, 249, 247, 245, 241, 239, 233, 229, 227, 223, 211, 199, 197, 193, 191, 181};

// Constants of one modulus: m, 1 / m, 2^(13 i) modulo m for i = 1 .. 4 and the inverse of P / m
// modulo m (symmetric residues: at most m / 2 in magnitude).
struct ModConst {
    float mf, rcp, p[4], inv;
};
struct ModTable {
    ModConst c[MODS];
};
// Reconstruction constants.  Group g holds the moduli 3g .. 3g + 2, G = their product: co[j] = G /
// m_j, w = P / G, rcp = round(2^40 / G); bias = 128 sum_i P / m_i, subtracted because the stored
// t_i are offset by 128.
struct CrtTable {
    unsigned co[GROUPS][3];
    unsigned w[GROUPS][LIMBS];
    unsigned rcp[GROUPS];
    unsigned P[LIMBS];
    unsigned bias[LIMBS];
    long long rbias;     // 128 sum_i 2^40 / m_i, rounded as sum of the groups' terms
};

struct Tables {
    ModTable mod;
    CrtTable crt;
};
Tables make_tables() {
    Tables t{};
    auto mul = [](unsigned (&x)[LIMBS], unsigned f) {
        unsigned long long carry = 0;
        for (int j = 0; j < LIMBS; ++j) {
            carry += (unsigned long long)x[j] * f;
            x[j] = (unsigned)carry;
            carry >>= 32;
        }
    };
    for (int i = 0; i < MODS; ++i) {
        ModConst& c = t.mod.c[i];
        const int m = kMod[i];
        c.mf = (float)m;
        c.rcp = 1.0f / (float)m;
        for (int j = 0; j < 4; ++j) {
            const int v = (int)((1ull << (13 * (j + 1))) % (unsigned long long)m);
            c.p[j] = (float)(2 * v > m ? v - m : v);
        }
        unsigned r = 1;
        for (int j = 0; j < MODS; ++j)
            if (j != i) r = r * (unsigned)kMod[j] % (unsigned)m;
        int inv = 1;
        while (inv < m && (unsigned)inv * r % (unsigned)m != 1) ++inv;
        c.inv = (float)(2 * inv > m ? inv - m : inv);
    }
    CrtTable& q = t.crt;
    q.P[0] = 1;
    for (int m : kMod) mul(q.P, (unsigned)m);
    for (int g = 0; g < GROUPS; ++g) {
        const unsigned G = (unsigned)kMod[3 * g] * (unsigned)kMod[3 * g + 1] * (unsigned)kMod[3 * g + 2];
        unsigned cosum = 0;
        for (int j = 0; j < 3; ++j) {
            q.co[g][j] = G / (unsigned)kMod[3 * g + j];
            cosum += q.co[g][j];
        }
        q.w[g][0] = 1;
        for (int i = 0; i < MODS; ++i)
            if (i / 3 != g) mul(q.w[g], (unsigned)kMod[i]);
        q.rcp[g] = (unsigned)(((1ull << 40) + G / 2) / G);
        q.rbias += 128ll * cosum * q.rcp[g];
        unsigned x[LIMBS];
        for (int l = 0; l < LIMBS; ++l) x[l] = q.w[g][l];
        mul(x, 128u * cosum);   // < 2^27
        unsigned long long carry = 0;
        for (int l = 0; l < LIMBS; ++l) {
            carry += (unsigned long long)q.bias[l] + x[l];
            q.bias[l] = (unsigned)carry;
            carry >>= 32;
        }
    }
    return t;
}
const Tables& tables() {
    static const Tables t = make_tables();
    return t;
}

// largest b with 2 K 2^(2b) < 0.98 P
int bits_for(int64_t K) {
    double lp = 0.0;
    for (int m : kMod) lp += log2((double)m);
    const int b = (int)floor((lp - 1.03 - log2((double)K)) / 2.0);
    return b < 62 ? b : 62;
}

// Element (r, k) of an operand: p[(r / R0) * s1 + (r % R0) * s0 + k * sk], r < R, k < K; its
// residues are stored [MODS][R][ldk] as BF16 (columns K..ldk-1 zero), exponents in ex[R].
struct FmSrc {
    const double* p;
    int64_t R, K, R0, s1, s0, sk;
    __nv_bfloat16* res;
    int* ex;        // the rows' exponents, and those of their pieces of FM_XK columns
    int* part;
    int64_t ldk;
    __host__ __device__ int64_t row(int64_t r) const { return (r / R0) * s1 + (r % R0) * s0; }
};

constexpr int FM_PR = 8;     // rows per block of the two operand kernels
constexpr int FM_PK = 64;    // columns per block of the residue kernel

constexpr int FM_XK = 256;   // columns per block of the exponent kernel
constexpr int FM_ZERO = -0x40000000;

// Exponents of 8 rows from r0 on over the FM_XK columns from k0 on (2^e > max |x| >= 2^(e - 1),
// FM_ZERO without a non-zero, FM_NONFINITE): true in one thread per row r0 + *row, with *e.
// sk == 1: a warp per row; else threads along the rows, which are contiguous then.
__device__ __forceinline__ bool fm_piece_exponent(const FmSrc& x, int64_t r0, int64_t k0,
                                                  unsigned long long (&part)[8][FM_PR], int* row, int* e) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // largest magnitude of each row, as bit patterns (their integer order is the order; a NaN
    // or infinity exceeds every finite value)
    constexpr unsigned long long ABS = 0x7fffffffffffffffull;
    const bool along = x.sk == 1;
    const int64_t r = r0 + (along ? warp : tid % FM_PR);
    unsigned long long m = 0;
    if (r < x.R) {
        const double* p = x.p + x.row(r);
        const int64_t k = k0 + (along ? lane : tid / FM_PR);
        unsigned long long v[FM_XK / 32];
#pragma unroll
        for (int u = 0; u < FM_XK / 32; ++u)
            v[u] = k + 32 * u < x.K ? (unsigned long long)__double_as_longlong(p[(k + 32 * u) * x.sk]) & ABS : 0ull;
#pragma unroll
        for (int u = 0; u < FM_XK / 32; ++u) m = v[u] > m ? v[u] : m;
    }
#pragma unroll
    for (int of = 16; of > 0; of >>= 1) {
        if (!along && of < FM_PR) break;
        const unsigned long long v = __shfl_xor_sync(0xffffffffu, m, of);
        m = v > m ? v : m;
    }
    if (!along) {
        if (lane < FM_PR) part[warp][lane] = m;
        __syncthreads();
        if (tid >= FM_PR) return false;
#pragma unroll
        for (int i = 0; i < 8; ++i) m = part[i][tid] > m ? part[i][tid] : m;
    } else if (lane != 0) {
        return false;
    }
    if (r >= x.R) return false;
    const int field = (int)(m >> 52);
    *e = field == 0x7ff ? FM_NONFINITE : field ? field - 1022 : m ? -1010 - __clzll((long long)m) : FM_ZERO;
    *row = (int)(r - r0);
    return true;
}

// Exponents of both operands' rows by pieces of FM_XK columns (part), for K beyond one piece.
// Blocks (x, y): 8 rows, x in [0, nba) operand A's, columns [y FM_XK, +FM_XK); every thread has
// its 8 loads in flight at once (with whole rows per block, the memory latency five times over
// and too few blocks: 12.5 us instead of 4 for the H_eff products of chi 256).
__global__ void __launch_bounds__(256) fm_rowexp_kernel(FmSrc a, FmSrc b, int nba, const int* skip) {
    ct_pdl();
    if (ct_skip(skip)) return;
    __shared__ unsigned long long part[8][FM_PR];
    const bool first = (int)blockIdx.x < nba;
    const FmSrc& x = first ? a : b;
    const int64_t r0 = (int64_t)(first ? blockIdx.x : blockIdx.x - nba) * FM_PR, k0 = (int64_t)blockIdx.y * FM_XK;
    int row, e;
    if (fm_piece_exponent(x, r0, k0, part, &row, &e)) x.part[(int64_t)blockIdx.y * x.R + r0 + row] = e;
}


// |v| 2^(bits - e) rounded to an integer (e: the row's exponent), 0 in a non-finite row
__device__ __forceinline__ unsigned long long fm_fixed(double v, int e, int bits) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v);
    int ev = (int)((u >> 52) & 0x7FF);
    unsigned long long m = u & ((1ull << 52) - 1);
    if (ev == 0) ev = 1;           // subnormal (or zero: m = 0)
    else m |= 1ull << 52;
    // v = m 2^(ev - 1075); the shift is at most bits - 53
    const int sh = ev - 1075 - e + bits;
    if (e == FM_NONFINITE) return 0;
    if (sh >= 0) return m << sh;
    return sh > -63 ? (m + (1ull << (-sh - 1))) >> (-sh) : 0;
}

// The residues of both operands in one launch: a block takes FM_PR rows x FM_PK columns, a warp
// a row, a lane two columns.  sk == 1: read along k; else through a shared-memory tile, read
// along the rows.
__global__ void __launch_bounds__(256) fm_residue_kernel(FmSrc a, FmSrc b, int nba, int bits, const ModTable tab,
                                                         const int* skip) {
    ct_pdl();
    if (ct_skip(skip)) return;
    __shared__ double tile[FM_PK][FM_PR + 1];
    const bool first = (int)blockIdx.x < nba;
    const FmSrc& x = first ? a : b;
    const int64_t r0 = (int64_t)(first ? blockIdx.x : blockIdx.x - nba) * FM_PR;
    const int64_t k0 = (int64_t)blockIdx.y * FM_PK;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t k = k0 + 2 * lane;
    double v0 = 0.0, v1 = 0.0;
    if (x.sk == 1) {
        const int64_t r = r0 + warp;
        if (r < x.R) {
            const double* p = x.p + x.row(r);
            if (k < x.K) v0 = p[k];
            if (k + 1 < x.K) v1 = p[k + 1];
        }
    } else {
        const int r = tid % FM_PR;
        const double* p = r0 + r < x.R ? x.p + x.row(r0 + r) : x.p;
#pragma unroll
        for (int kk = tid / FM_PR; kk < FM_PK; kk += 256 / FM_PR)
            tile[kk][r] = (r0 + r < x.R && k0 + kk < x.K) ? p[(k0 + kk) * x.sk] : 0.0;
        __syncthreads();
        v0 = tile[2 * lane][warp];
        v1 = tile[2 * lane + 1][warp];
    }
    __shared__ unsigned long long part[8][FM_PR];
    __shared__ int es[FM_PR];
    const bool own = x.K <= FM_XK;   // one piece: found here, 8 more loads per thread and a launch less
    if (own) {
        int row, pe;
        if (fm_piece_exponent(x, r0, 0, part, &row, &pe)) es[row] = pe;
        __syncthreads();
    }
    if (r0 + warp >= x.R) return;
    int e = FM_ZERO;   // the row's exponent, or the largest of its pieces'
    if (own) {
        e = es[warp];
    } else {
        for (int64_t c = lane; c * FM_XK < x.K; c += 32) e = max(e, x.part[c * x.R + r0 + warp]);
        e = __reduce_max_sync(0xffffffffu, e);
    }
    if (e == FM_ZERO) e = 0;
    if (blockIdx.y == 0 && lane == 0) x.ex[r0 + warp] = e;
    const unsigned long long u0 = fm_fixed(v0, e, bits), u1 = fm_fixed(v1, e, bits);
    // five 13-bit digits of each as floats with the value's sign (a digit in the low bits of
    // 2^23 + digit)
    float d[2][5];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        const float x0 = __uint_as_float(0x4B000000u | ((unsigned)(u0 >> (13 * i)) & 8191u)) - 8388608.0f;
        const float x1 = __uint_as_float(0x4B000000u | ((unsigned)(u1 >> (13 * i)) & 8191u)) - 8388608.0f;
        d[0][i] = __double2hiint(v0) < 0 ? -x0 : x0;
        d[1][i] = __double2hiint(v1) < 0 ? -x1 : x1;
    }
    const int64_t plane = x.R * x.ldk;
    __nv_bfloat16* out = x.res + (r0 + warp) * x.ldk + k;
#pragma unroll
    for (int i = 0; i < MODS; ++i) {
        const ModConst& c = tab.c[i];
        // sum of digit times 2^(13 i) mod m, below 2^23 and exact, minus m rint(sum / m): at most 128
        // in magnitude, exact in BF16 (the upper half of the FP32 word)
        constexpr float RND = 12582912.0f;   // 1.5 2^23
        uint32_t f[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            float t = d[q][0];
#pragma unroll
            for (int j = 0; j < 4; ++j) t = fmaf(d[q][j + 1], c.p[j], t);
            const float n = __fsub_rn(fmaf(t, c.rcp, RND), RND);
            f[q] = __float_as_uint(fmaf(-n, c.mf, t));
        }
        *reinterpret_cast<uint32_t*>(out + i * plane) = __byte_perm(f[0], f[1], 0x7632);
    }
}

// kind::f16 instruction descriptor: D f32, A and B bf16, both K-major.
__host__ __device__ constexpr uint32_t fm_idesc(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void fm_mma(uint32_t dtm, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        ::"r"(dtm), "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
        : "memory");
}

struct FmOut {
    unsigned char* r;    // [MODS][M][ldn]: t_i + 128 of C (ldn a multiple of FM_BN)
    int64_t ldn;
};

// The MODS residue products: one CTA per SM walks (modulus, tile) items; warp 0 issues TMA
// loads (128-byte swizzle, 4 stages of 32 KB), one thread of warp 1 the MMAs (M128 N128 K16),
// 16 epilogue warps (four per TMEM lane quadrant, 32 columns each) take a chunk's accumulator
// (512 / 128 of them in TMEM), reduce it modulo m in FP32 (x - m rint(x / m), exact below
// 2^24), add the chunks and store t = r (P / m)^-1 mod m, the reconstruction's factor.  Every wait is bounded (2 s), after which the kernel sets the
// status word, releases TMEM and returns.
__global__ void __launch_bounds__(FM_THREADS, 1)
    fm_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int M, int N,
                   int Kpad, FmOut out, const ModTable tab, const int* skip, int* status) {
    ct_pdl();
    if (ct_skip(skip)) return;
    extern __shared__ uint8_t fm_smem_raw[];
    uint8_t* smem = fm_smem_raw + ((1024u - (smem_u32(fm_smem_raw) & 1023u)) & 1023u);
    uint64_t* full = (uint64_t*)(smem + FM_STAGES * FM_STAGE);
    uint64_t* empty = full + FM_STAGES;
    uint64_t* acc_full = empty + FM_STAGES;
    uint64_t* acc_empty = acc_full + FM_NB;
    uint32_t* tmem_slot = (uint32_t*)(acc_empty + FM_NB);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_n = (N + FM_BN - 1) / FM_BN;
    const int tiles = tiles_n * ((M + FM_BM - 1) / FM_BM);
    const int items = tiles * MODS;
    const int nkb = Kpad / FM_BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < FM_STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < FM_NB; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 4 * FM_EPW);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            int g = 0;
            bool ok = true;
            for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
                const int mod = it / tiles, t = it % tiles;
                const int ya = mod * M + (t / tiles_n) * FM_BM, yb = mod * N + (t % tiles_n) * FM_BN;
                for (int kb = 0; kb < nkb; ++kb, ++g) {
                    const int s = g % FM_STAGES;
                    const uint32_t ph = (uint32_t)(g / FM_STAGES) & 1u;
                    if (g >= FM_STAGES && !mbar_wait(&empty[s], ph ^ 1u, abort_flag)) {
                        *abort_flag = 1;
                        ct_set_status(status, CT_ERR_CUDA);
                        ok = false;
                        break;
                    }
                    uint8_t* st = smem + s * FM_STAGE;
                    mbar_expect_tx(&full[s], FM_STAGE);
                    tma_load_2d(st, &tmA, kb * FM_BK, ya, &full[s]);
                    tma_load_2d(st + FM_A_BYTES, &tmB, kb * FM_BK, yb, &full[s]);
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = fm_idesc(FM_BM, FM_BN);
            int g = 0, gc = 0;
            bool ok = true;
            for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
                for (int kb0 = 0; kb0 < nkb && ok; kb0 += FM_KCH, ++gc) {
                    const int b = gc % FM_NB, u = gc / FM_NB;
                    if (u > 0 && !mbar_wait(&acc_empty[b], (uint32_t)((u - 1) & 1), abort_flag)) {
                        *abort_flag = 1;
                        ct_set_status(status, CT_ERR_CUDA);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t dt = tmem + (uint32_t)(b * FM_BN);
                    const int kb1 = kb0 + FM_KCH < nkb ? kb0 + FM_KCH : nkb;
                    for (int kb = kb0; kb < kb1; ++kb, ++g) {
                        const int s = g % FM_STAGES;
                        const uint32_t ph = (uint32_t)(g / FM_STAGES) & 1u;
                        if (!mbar_wait(&full[s], ph, abort_flag)) {
                            *abort_flag = 1;
                            ct_set_status(status, CT_ERR_CUDA);
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t a0 = smem_u32(smem + s * FM_STAGE);
#pragma unroll
                        for (int kk = 0; kk < FM_BK / 16; ++kk)
                            fm_mma(dt, sw128_desc(a0 + kk * 32), sw128_desc(a0 + FM_A_BYTES + kk * 32), idesc,
                                   (kb > kb0 || kk > 0) ? 1u : 0u);
                        mma_commit(&empty[s]);
                    }
                    if (ok) mma_commit(&acc_full[b]);
                }
            }
        }
    } else {
        const int q = warp & 3;              // TMEM lane quadrant of this warp
        const int hf = (warp - 2) >> 2;      // column group of the tile
        const int row = q * 32 + lane;
        constexpr float RND = 12582912.0f;   // 1.5 2^23: adding and subtracting it rounds to an integer
        int gc = 0;
        bool ok = true;
        for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
            const int mod = it / tiles, t = it % tiles;
            const float m = tab.c[mod].mf, rcp = tab.c[mod].rcp, inv = tab.c[mod].inv;
            float sum[FM_HC];
#pragma unroll
            for (int j = 0; j < FM_HC; ++j) sum[j] = 0.f;
            for (int kb0 = 0; kb0 < nkb; kb0 += FM_KCH, ++gc) {
                const int b = gc % FM_NB, u = gc / FM_NB;
                if (!mbar_wait(&acc_full[b], (uint32_t)(u & 1), abort_flag)) {
                    *abort_flag = 1;
                    ct_set_status(status, CT_ERR_CUDA);
                    ok = false;
                    break;
                }
                __syncwarp();
                tc_fence_after();
                const uint32_t tq = tmem + (uint32_t)(b * FM_BN + hf * FM_HC) + ((uint32_t)(q * 32) << 16);
                uint32_t r[FM_HC];
#pragma unroll
                for (int q8 = 0; q8 < FM_HC; q8 += 8)
                    tmem_ld8_nowait(tq + (uint32_t)q8, *reinterpret_cast<uint32_t(*)[8]>(&r[q8]));
                tmem_wait_ld();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[b]);
#pragma unroll
                for (int j = 0; j < FM_HC; ++j) {
                    const float x = __uint_as_float(r[j]);
                    const float k = __fsub_rn(__fadd_rn(__fmul_rn(x, rcp), RND), RND);
                    sum[j] += fmaf(-k, m, x);
                }
            }
            if (!ok) break;
            const int64_t mr = (int64_t)(t / tiles_n) * FM_BM + row;
            if (mr >= M) continue;
            // reduced once more, times the inverse (below 2^14), reduced, offset by 128 and packed, one
            // byte per element (t is at most m / 2 in magnitude; 128 occurs for m = 256 only,
            // where 256 wraps to 0, that is -128)
            uint32_t w[FM_HC / 4];
#pragma unroll
            for (int j4 = 0; j4 < FM_HC / 4; ++j4) {
                uint32_t v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float x = sum[4 * j4 + j];
                    const float k = __fsub_rn(__fadd_rn(__fmul_rn(x, rcp), RND), RND);
                    const float y = __fmul_rn(fmaf(-k, m, x), inv);
                    const float l = __fsub_rn(__fadd_rn(__fmul_rn(y, rcp), RND), RND);
                    v[j] = __float_as_uint(__fadd_rn(fmaf(-l, m, y), RND + 128.0f));   // low byte: t + 128
                }
                w[j4] = __byte_perm(__byte_perm(v[0], v[1], 0x0040), __byte_perm(v[2], v[3], 0x0040), 0x5410);
            }
            unsigned char* o = out.r + ((int64_t)mod * M + mr) * out.ldn + (t % tiles_n) * FM_BN + hf * FM_HC;
#pragma unroll
            for (int j = 0; j < FM_HC / 16; ++j)
                reinterpret_cast<uint4*>(o)[j] = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
        }
    }
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

struct FmC {
    double* p;       // row m at (m / M0) * s1 + (m % M0) * s0, columns contiguous
    int64_t M0, s1, s0;
};

// C from its residues: S = sum t_i P / m_i - k P with k = rint(sum t_i / m_i), then
// S 2^(ea + eb - 2 bits) rounded to FP64.  Three moduli at a time, u = sum t_j G / m_j (below
// 2^26), so that the multi-word sums have six terms.  A thread takes four columns of a row.
__global__ void __launch_bounds__(256) fm_crt_kernel(FmOut in, int M, int N, FmSrc a, FmSrc b, FmC c, int bits,
                                                     const CrtTable tab, const int* skip) {
    ct_pdl();
    if (ct_skip(skip)) return;
    const int64_t n0 = 4 * ((int64_t)blockIdx.x * 64 + (threadIdx.x & 63));
    const int64_t m = (int64_t)blockIdx.y * 4 + (threadIdx.x >> 6);
    if (m >= M || n0 >= N) return;
    const int em = a.ex[m];
    uint32_t r4[MODS];
#pragma unroll
    for (int i = 0; i < MODS; ++i)
        r4[i] = *reinterpret_cast<const uint32_t*>(in.r + ((int64_t)i * M + m) * in.ldn + n0);
    double* Cr = c.p + (m / c.M0) * c.s1 + (m % c.M0) * c.s0;
#pragma unroll 1
    for (int j = 0; j < 4; ++j) {
        const int64_t n = n0 + j;
        if (n >= N) break;
        const int en = b.ex[n];
        if (em == FM_NONFINITE || en == FM_NONFINITE) {
            double v = 0.0;
            const double* pa = a.p + a.row(m);
            const double* pb = b.p + b.row(n);
            for (int64_t k = 0; k < a.K; ++k) v = fma(pa[k * a.sk], pb[k * b.sk], v);
            Cr[n] = v;
            continue;
        }
        unsigned long long acc[LIMBS] = {0, 0, 0, 0, 0};
        long long frac = -tab.rbias;
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
            unsigned u = 0;
#pragma unroll
            for (int i = 0; i < 3; ++i) u += ((r4[3 * g + i] >> (8 * j)) & 0xffu) * tab.co[g][i];
            frac += (long long)((unsigned long long)u * tab.rcp[g]);
#pragma unroll
            for (int l = 0; l < LIMBS; ++l) acc[l] += (unsigned long long)u * tab.w[g][l];
        }
        // (2^40 / G to half a unit: an error below 2^-12 of the fraction)
        const int kk = (int)((frac + (1ll << 39)) >> 40);
        // S = sum - bias - kk P as a two's complement number of LIMBS limbs
        unsigned s[LIMBS];
        long long carry = 0;
#pragma unroll
        for (int l = 0; l < LIMBS; ++l) {
            const long long v = (long long)(acc[l] & 0xffffffffull) - (long long)tab.bias[l] -
                                (long long)kk * (long long)tab.P[l] + carry;
            s[l] = (unsigned)v;
            carry = (v >> 32) + (long long)(acc[l] >> 32);
        }
        const bool neg = (s[LIMBS - 1] >> 31) != 0;
        if (neg) {
            unsigned cy = 1;
#pragma unroll
            for (int l = 0; l < LIMBS; ++l) {
                const unsigned v = ~s[l];
                s[l] = v + cy;
                cy = (cy && s[l] == 0) ? 1 : 0;
            }
        }
        // magnitude (below 2^140) left-aligned in (hi, lo) and a sticky bit; the leading bit is worth
        // 2^top
        unsigned long long hi = ((unsigned long long)s[4] << 32) | s[3], lo = ((unsigned long long)s[2] << 32) | s[1];
        unsigned below = s[0];
        int top = 159;
        if (hi == 0) {
            hi = lo;
            lo = (unsigned long long)below << 32;
            below = 0;
            top -= 64;
            if (hi == 0) {
                hi = lo;
                lo = 0;
                top -= 64;
            }
        }
        double v = 0.0;
        if (hi != 0) {
            const int lz = __clzll((long long)hi);
            if (lz > 0) {
                hi = (hi << lz) | (lo >> (64 - lz));
                lo <<= lz;
            }
            top -= lz;
            // 53 bits kept, round to nearest even
            unsigned long long f = hi >> 11;
            const unsigned long long rem = hi & 0x7ff;
            f += (rem > 0x400 || (rem == 0x400 && ((lo | below) != 0 || (f & 1)))) ? 1 : 0;
            const int e = em + en - 2 * bits, ex = 1023 + top + e;   // exponent field of f's leading bit
            if (ex < 1 || ex > 2045) v = scalbn(neg ? -(double)f : (double)f, top - 52 + e);
            else v = __longlong_as_double((long long)((((unsigned long long)(ex - 1) << 52) + f) |
                                                      ((unsigned long long)neg << 63)));
        }
        Cr[n] = v;
    }
}

struct FmPlan {
    int64_t ldk, ldn, tiles;
    size_t bytes;
};
FmPlan fm_plan(int64_t M, int64_t N, int64_t K) {
    FmPlan q;
    q.ldk = ct_round_up(K, FM_BK);
    q.ldn = ct_round_up(N, FM_BN);
    q.tiles = ct_cdiv(M, FM_BM) * ct_cdiv(N, FM_BN);
    q.bytes = ct_bytes(MODS * M * q.ldk, 2) + ct_bytes(MODS * N * q.ldk, 2) + ct_bytes(MODS * M * q.ldn, 1) +
              ct_bytes(M, 4) + ct_bytes(N, 4) + ct_bytes(ct_cdiv(K, FM_XK) * M, 4) + ct_bytes(ct_cdiv(K, FM_XK) * N, 4);
    return q;
}

int fm_workspace(ct_handle* h, size_t bytes) {
    if (h->fm_ws_bytes >= bytes) return CT_OK;
    CT_CUDA(h, cudaStreamSynchronize(h->stream));
    if (h->fm_ws && h->fm_captured) h->fm_kept.push_back(h->fm_ws);   // graphs may replay on it
    else if (h->fm_ws) cudaFree(h->fm_ws);
    h->fm_captured = false;
    h->fm_ws = nullptr;
    h->fm_ws_bytes = 0;
    CT_CUDA(h, cudaMalloc(&h->fm_ws, bytes));
    h->fm_ws_bytes = bytes;
    return CT_OK;
}

int fm_map(ct_handle* h, CUtensorMap* m, const FmSrc& s, int box_rows) {
    PFN_cuTensorMapEncodeTiled_v12000 enc = ct_tma_encoder();
    if (!enc) return CT_ERR_UNSUPPORTED;
    if (((uintptr_t)s.res & 15) || (s.ldk % FM_BK)) {
        ct_seterr(h, "TMA operand misaligned (base %p, ldk %lld)", (const void*)s.res, (long long)s.ldk);
        return CT_ERR_INVALID;
    }
    cuuint64_t dims[2] = {(cuuint64_t)s.ldk, (cuuint64_t)(MODS * s.R)};
    cuuint64_t strides[1] = {(cuuint64_t)(s.ldk * 2)};
    cuuint32_t box[2] = {(cuuint32_t)FM_BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)s.res, dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        ct_seterr(h, "cuTensorMapEncodeTiled failed (%d)", (int)r);
        return CT_ERR_CUDA;
    }
    return CT_OK;
}

}  // namespace

// Whether an FP64-form product goes to the tensor cores.  Estimated times in us: the SIMT
// kernel at 85% of the FP64 pipe (2 multiply-adds per clock and SM, 1.9 GHz); here 12 us of
// launches and latencies, tile items at 1.2 us plus 0.16 us per 64 of K on each SM, and operands
// and residues written and read at 4 TB/s.  Measured (us, SIMT / here): 128x384x128 16.6 / 17.9 and
// 128x256x128 12.9 / 13.9 stay, 512x128x128 20.6 / 17.0, 640x128x128 24.0 / 18.7, 256x256x128
// 20.5 / 19.2 and 256x256x256 36.9 / 20.0 go.  Only when the scratch is there or can be had: within
// the handle's workspace limit, outside a stream capture, and with the memory available;
// otherwise the SIMT kernel, as before.
bool ct_f64_route(ct_handle* h, int64_t M, int64_t N, int64_t K) {
    if (M <= 0 || N <= 0 || K <= 0 || K > ((int64_t)1 << 20) || !ct_fp64_tc_enabled(h, M, N, K)) return false;
    const FmPlan q = fm_plan(M, N, K);
    if (MODS * M > (1ll << 30) || MODS * N > (1ll << 30) || q.tiles * MODS > (1ll << 30) || ct_cdiv(M, 4) > 65535)
        return false;
    const double simt = (double)M * (double)N * (double)K / (0.85 * 2.0 * h->num_sms * 1900.0);
    const double items = (double)ct_cdiv(q.tiles * MODS, h->num_sms) * (1.2 + 0.16 * (double)(q.ldk / FM_BK));
    const double traffic = ((double)(M + N) * (double)q.ldk * 4.0 * MODS + (double)M * (double)q.ldn * 2.0 * MODS) / 4.0e6;
    if (12.0 + items + traffic > simt) return false;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(h->stream, &cs) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    const bool capturing = cs != cudaStreamCaptureStatusNone;
    if (h->fm_ws_bytes >= q.bytes) {
        h->fm_captured |= capturing;
        return true;
    }
    if (capturing || (h->ws_limit && h->ws_cap + q.bytes > h->ws_limit)) return false;
    const std::string keep = h->err;
    if (fm_workspace(h, q.bytes) != CT_OK) {
        (void)cudaGetLastError();
        h->err = keep;
        return false;
    }
    return true;
}

// C(m,n) = sum_k A(m,k) B(n,k), operands and C with two-level row indexing (OzMat, OzOut in
// ct_ops.cuh); ct_f64_route must have accepted the size.
int ct_f64_gemm(ct_handle* h, int64_t M, int64_t N, int64_t K, const OzMat& A, const OzMat& B, const OzOut& Cout,
                const int* skip) {
    const FmPlan q = fm_plan(M, N, K);
    CT_TRY(fm_workspace(h, q.bytes));
    uint8_t* p = (uint8_t*)h->fm_ws;
    FmSrc a{A.p, M, K, A.R0 > 0 ? A.R0 : M, A.s1, A.s0, A.sk, (__nv_bfloat16*)p, nullptr, nullptr, q.ldk};
    p += ct_bytes(MODS * M * q.ldk, 2);
    FmSrc b{B.p, N, K, B.R0 > 0 ? B.R0 : N, B.s1, B.s0, B.sk, (__nv_bfloat16*)p, nullptr, nullptr, q.ldk};
    p += ct_bytes(MODS * N * q.ldk, 2);
    FmOut o{(unsigned char*)p, q.ldn};
    p += ct_bytes(MODS * M * q.ldn, 1);
    a.ex = (int*)p;
    p += ct_bytes(M, 4);
    b.ex = (int*)p;
    p += ct_bytes(N, 4);
    a.part = (int*)p;
    p += ct_bytes(ct_cdiv(K, FM_XK) * M, 4);
    b.part = (int*)p;
    CUtensorMap ta, tb;
    CT_TRY(fm_map(h, &ta, a, FM_BM));
    CT_TRY(fm_map(h, &tb, b, FM_BN));
    static int attr_dev = -1;
    if (attr_dev != h->device) {
        CT_CUDA(h, cudaFuncSetAttribute(fm_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FM_SMEM));
        attr_dev = h->device;
    }
    const Tables& t = tables();
    const int bits = bits_for(K);
    const int nba = (int)ct_cdiv(M, FM_PR);
    const dim3 grid((unsigned)(nba + ct_cdiv(N, FM_PR)), (unsigned)ct_cdiv(q.ldk, FM_PK));
    if (grid.y > 65535) return CT_ERR_UNSUPPORTED;
    if (K > FM_XK) {
        ct_launch(h, fm_rowexp_kernel, dim3(grid.x, (unsigned)ct_cdiv(K, FM_XK)), 256, 0, a, b, nba, skip); ct_note_launch();
    }
    ct_launch(h, fm_residue_kernel, grid, 256, 0, a, b, nba, bits, t.mod, skip); ct_note_launch();
    const int64_t items = q.tiles * MODS;
    const int64_t ctas = items < h->num_sms ? items : h->num_sms;
    ct_launch(h, fm_gemm_kernel, (unsigned)ctas, FM_THREADS, FM_SMEM, ta, tb, (int)M, (int)N, (int)q.ldk, o, t.mod, skip,
                                                                       h->d_status); ct_note_launch();
    const FmC c{Cout.p, Cout.M0 > 0 ? Cout.M0 : M, Cout.s1, Cout.s0};
    ct_launch(h, fm_crt_kernel, dim3((unsigned)ct_cdiv(N, 256), (unsigned)ct_cdiv(M, 4)), 256, 0, 
        o, (int)M, (int)N, a, b, c, bits, t.crt, skip); ct_note_launch();
    CT_LAUNCH_CHECK(h);
    return CT_OK;
}
