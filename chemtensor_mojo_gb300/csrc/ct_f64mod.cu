// FP64-form GEMM on the BF16 tensor cores by residues, with FP64 accuracy of every element.
//
// C[M,N] = sum_k A[m,k] B[n,k] with FP64 A, B and C, for the contraction chains of the FP64
// form.  The scheme is that of K. Ozaki, Y. Uchino and T. Imamura, Ozaki Scheme II: a
// GEMM-oriented emulation of floating-point matrix multiplication using an integer modular
// technique (arXiv:2504.08009, 2025), here on tcgen05 kind::f16, with a correction for the
// operands' rounding and a test of each element:
//   * every row of A and of B is scaled by a power of two, to a' and b' below 1, and rounded to
//     integers of b bits (b = 58 at K = 256, less for larger K: the moduli hold 2 K 2^(2b) < P);
//   * for each of MODS pairwise coprime moduli m_i <= 256 the residues of A and B (at most
//     128 in magnitude, exact in BF16) are multiplied: a product is at most 2^14, so 1024 of K
//     add up exactly in the FP32 accumulator, which the epilogue reduces modulo m_i;
//   * the Chinese remainder theorem gives the integer product sum, below P / 2 = prod m_i / 2
//     in magnitude, exactly;
//   * what the rounding took from a' and b', da and db (at most half a unit), comes back as a
//     pair of FP16 products, sum_k a' db and sum_k da b', to 2^-11 of each term;
//   * both are added as integers and rounded to FP64 once.
//
// Accuracy.  The integers are relative to a row's largest entry, so what is left of the error,
// 2^-(b + 12) T with T = sum_k |a'| [db != 0] + [da != 0] |b'|, may exceed what FP64 FMAs leave of an
// element whose S = sum_k |a'| |b'| is small (one operand falls along k and the other rises; rows of
// an identity).  So each element is tested for 2^-(b + 12) T <= 16 2^-53 S: one more BF16 product, of
// x = |a'| - theta [da != 0] and y = |b'| - theta [db != 0] with theta = 2^(37 - b), is S - theta T +
// theta^2 n, n <= K the number of k where neither is exact, and has to be theta^2 K at least.  It is
// exactly zero where no k has both, as between the blocks of a block-sparse operand (x and y of a
// non-zero entry are kept from zero): such an element passes if its product is zero too.  The
// others are computed as FP64 dot products.
// Every element is thus within 16.5 2^-53 S and the final rounding (worst case; FP64 FMAs: K 2^-53 S).
// Measured, 256^3, N(0,1) operands with A falling and B rising along k by a factor f, largest error
// in units of 2^-53 S (here, with the final rounding / FP64 FMAs): f = 1 below 0.001 / 4.0, 1e2 0.22 /
// 4.3, 1e4 0.41 / 4.0, 1e5 0.45 / 3.6, 1e6 1.1 / 4.4, 1e7 2.3 / 4.4, then all dot products, 1.2 / 4.4.  (18
// moduli alone, b = 62, without correction and test: 2e-14 of an element at f = 1e6, 1.5e-8 at 1e12.)
// Dot products of all elements, after the products here (us, and the FMA kernel without this route):
// 256^3 55 (41), 512^3 293 (231), 1280 x 1024 x 256 648 (780), 1024 x 256 x 1280 724 (570).
//
// What bounds it.  MODS + 3 products of full-size tensor-core tiles per FP64 product (the sliced
// scheme of ct_ozaki.cu forms 36 to 45, on 64-wide tiles that its eight accumulators leave);
// for small products the four launches.  FP64 arithmetic issues at 1/64 of the FP32 rate
// here, so the residues, the reduction and the reconstruction are integer and FP32 work.
//
// A row with an infinity or a NaN has no scale: its elements of C are computed as FP64
// dot products from the operands, so non-finite values go where an FP64 GEMM takes them.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math.h>

#include <algorithm>

#include "ct_ops.cuh"
#include "ct_tc_ptx.cuh"

PFN_cuTensorMapEncodeTiled_v12000 ct_tma_encoder();

namespace {

constexpr int MODS = 16;
constexpr int GROUPS = MODS / 2;                        // reconstructed two moduli at a time
// planes of an operand: the residues; a' and da of A beside db and b' of B; x or y of the test
constexpr int PL_CORR = MODS, PL_TEST = MODS + 2, PLANES = MODS + 3;
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
constexpr int LIMBS = 4;                                // 32-bit limbs of P (125 bits) and of the sums

// pairwise coprime, at most 256: P = 2^125.5
constexpr int kMod[MODS] = {256, 253, 251, 249, 247, 245, 241, 239, 233, 229, 227, 223, 211, 199, 197, 193};

// Constants of one modulus: m, 1 / m, 2^(13 i) modulo m for i = 1 .. 4 and the inverse of P / m
// modulo m (symmetric residues: at most m / 2 in magnitude).
struct ModConst {
    float mf, rcp, p[4], inv;
};
struct ModTable {
    ModConst c[MODS];
};
// Reconstruction constants.  Group g holds the moduli 2g and 2g + 1, G = their product: co[j] = G /
// m_j, w = P / G, rcp = round(2^40 / G); bias = 128 sum_i P / m_i, subtracted because the stored
// t_i are offset by 128.
struct CrtTable {
    unsigned co[GROUPS][2];
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
        const unsigned G = (unsigned)kMod[2 * g] * (unsigned)kMod[2 * g + 1];
        unsigned cosum = 0;
        for (int j = 0; j < 2; ++j) {
            q.co[g][j] = G / (unsigned)kMod[2 * g + j];
            cosum += q.co[g][j];
        }
        q.w[g][0] = 1;
        for (int i = 0; i < MODS; ++i)
            if (i / 2 != g) mul(q.w[g], (unsigned)kMod[i]);
        q.rcp[g] = (unsigned)(((1ull << 40) + G / 2) / G);
        q.rbias += 128ll * cosum * q.rcp[g];
        unsigned x[LIMBS];
        for (int l = 0; l < LIMBS; ++l) x[l] = q.w[g][l];
        mul(x, 128u * cosum);
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
    return b < 59 ? b : 59;   // (five digits of 13 bits)
}

// Element (r, k) of an operand: p[(r / R0) * s1 + (r % R0) * s0 + k * sk], r < R, k < K; its
// planes are stored [PLANES][R][ldk], 16 bits each (columns K..ldk-1 zero), exponents in ex[R].
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


// |v| 2^(bits - e) = u + d, u rounded to an integer, d to 2^-23 (e: the row's exponent; 0 in a
// non-finite row); whether d is not zero
__device__ __forceinline__ bool fm_fixed(double v, int e, int bits, unsigned long long& u, float& d) {
    const unsigned long long w = (unsigned long long)__double_as_longlong(v);
    int ev = (int)((w >> 52) & 0x7FF);
    unsigned long long m = w & ((1ull << 52) - 1);
    if (ev == 0) ev = 1;           // subnormal (or zero: m = 0)
    else m |= 1ull << 52;
    u = 0;
    d = 0.0f;
    if (e == FM_NONFINITE || m == 0) return false;
    // v = m 2^(ev - 1075); the shift is at most bits - 53
    const int s = -(ev - 1075 - e + bits);
    if (s <= 0) {
        u = m << -s;
        return false;
    }
    unsigned x;    // |d| = x 2^ex, x below 2^23
    int ex;
    bool down = false;
    if (s < 64) {
        u = (m + (1ull << (s - 1))) >> s;
        const long long rem = (long long)(m - (u << s));
        if (rem == 0) return false;
        down = rem < 0;
        const unsigned long long a = (unsigned long long)(down ? -rem : rem);
        x = (unsigned)(s > 23 ? a >> (s - 23) : a);
        ex = s > 23 ? -23 : -s;
    } else {       // u = 0
        x = (unsigned)(m >> 30);
        ex = 30 - s;
    }
    if (ex > -120) {
        d = (__uint_as_float(0x4B000000u | x) - 8388608.0f) * __uint_as_float((unsigned)(127 + ex) << 23);
        if (down) d = -d;
    }
    return true;
}

// The residues of both operands in one launch: a block takes FM_PR rows x FM_PK columns, a warp
// a row, a lane two columns.  sk == 1: read along k; else through a shared-memory tile, read
// along the rows.
__global__ void __launch_bounds__(256) fm_residue_kernel(FmSrc a, FmSrc b, int nba, int bits, float theta,
                                                         const ModTable tab, const int* skip) {
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
    unsigned long long u0, u1;
    float r0f, r1f;
    const bool inx0 = fm_fixed(v0, e, bits, u0, r0f), inx1 = fm_fixed(v1, e, bits, u1, r1f);
    const bool neg0 = __double2hiint(v0) < 0, neg1 = __double2hiint(v1) < 0;
    // five 13-bit digits of each as floats with the value's sign (a digit in the low bits of
    // 2^23 + digit)
    float d[2][5];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        const float x0 = __uint_as_float(0x4B000000u | ((unsigned)(u0 >> (13 * i)) & 8191u)) - 8388608.0f;
        const float x1 = __uint_as_float(0x4B000000u | ((unsigned)(u1 >> (13 * i)) & 8191u)) - 8388608.0f;
        d[0][i] = neg0 ? -x0 : x0;
        d[1][i] = neg1 ? -x1 : x1;
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
    // a' and da, both times 2^15 (FP16 reaches down to 2^-29 of the row's largest, or of a unit)
    const float unit = __uint_as_float((unsigned)(127 + 15 - bits) << 23);   // 2^(15 - bits)
    float hv[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        float t = d[q][4];
#pragma unroll
        for (int j = 3; j >= 0; --j) t = fmaf(t, 8192.0f, d[q][j]);
        hv[q] = t * unit;
    }
    const __half2 main2 = __floats2half2_rn(hv[0], hv[1]);
    const __half2 rest2 = __floats2half2_rn((neg0 ? -r0f : r0f) * 32768.0f, (neg1 ? -r1f : r1f) * 32768.0f);
    *reinterpret_cast<__half2*>(out + PL_CORR * plane) = first ? main2 : rest2;
    *reinterpret_cast<__half2*>(out + (PL_CORR + 1) * plane) = first ? rest2 : main2;
    // the test's x or y, in BF16 by its upper half; not zero in a non-zero entry
    float g[2] = {fabsf(hv[0]) * 0x1p-15f, fabsf(hv[1]) * 0x1p-15f};
    if (inx0) g[0] -= theta;
    if (inx1) g[1] -= theta;
    if (g[0] == 0.0f && (inx0 || u0)) g[0] = 0x1p-40f;
    if (g[1] == 0.0f && (inx1 || u1)) g[1] = 0x1p-40f;
    *reinterpret_cast<uint32_t*>(out + PL_TEST * plane) = __byte_perm(__float_as_uint(g[0]), __float_as_uint(g[1]), 0x7632);
}

// kind::f16 instruction descriptor: D f32, A and B both bf16 (type 1) or both f16 (0), K-major.
__host__ __device__ constexpr uint32_t fm_idesc(int M, int N, uint32_t type) {
    return (1u << 4) | (type << 7) | (type << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
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
    unsigned char* r;    // [MODS + 1][M][ldn]: t_i + 128 of C, then the test's answer (ldn a multiple of FM_BN)
    float* corr;         // [2][M][ldn]: the corrections times 2^30
    float limit;         // theta^2 K
    int64_t ldn;
};
constexpr unsigned FM_PASS = 0, FM_FAIL = 1, FM_NONE = 2;   // the test's answer (FM_NONE: exactly zero)

// The products of all planes: one CTA per SM walks (plane, tile) items; warp 0 issues TMA
// loads (128-byte swizzle, 4 stages of 32 KB), one thread of warp 1 the MMAs (M128 N128 K16),
// 16 epilogue warps (four per TMEM lane quadrant, 32 columns each) take a chunk's accumulator
// (512 / 128 of them in TMEM), reduce it modulo m in FP32 (x - m rint(x / m), exact below
// 2^24), add the chunks and store t = r (P / m)^-1 mod m, the reconstruction's factor.  The
// correction's chunks are added up as they are; so are the test's, which is answered in a byte.
// Every wait is bounded (2 s), after which the kernel sets the status word, releases TMEM and
// returns.
__global__ void __launch_bounds__(FM_THREADS, 1)
    fm_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int M, int N,
                   int Kpad, FmOut out, const ModTable tab, const int* skip, int* status) {
    ct_pdl_wait();
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
    const int items = tiles * PLANES;
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
                const int pl = it / tiles, t = it % tiles;
                const int ya = pl * M + (t / tiles_n) * FM_BM, yb = pl * N + (t % tiles_n) * FM_BN;
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
            drain_loads(full, FM_STAGES, g);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            int g = 0, gc = 0;
            bool ok = true;
            for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
                const int pl = it / tiles;
                const uint32_t idesc = fm_idesc(FM_BM, FM_BN, pl == PL_CORR || pl == PL_CORR + 1 ? 0u : 1u);
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
            const int pl = it / tiles, t = it % tiles, mod = pl < MODS ? pl : 0;
            const float m = tab.c[mod].mf, rcp = pl < MODS ? tab.c[mod].rcp : 0.0f, inv = tab.c[mod].inv;
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
                    const float k = __fsub_rn(__fadd_rn(__fmul_rn(x, rcp), RND), RND);   // (rcp 0: x as it is)
                    sum[j] += fmaf(-k, m, x);
                }
            }
            if (!ok) break;
            const int64_t mr = (int64_t)(t / tiles_n) * FM_BM + row;
            const int nc = (t % tiles_n) * FM_BN + hf * FM_HC;
            if (pl == PL_TEST) {
                uint32_t w[FM_HC / 4];
#pragma unroll
                for (int j = 0; j < FM_HC; ++j) {
                    const uint32_t v = sum[j] >= out.limit ? FM_PASS : sum[j] == 0.0f ? FM_NONE : FM_FAIL;
                    w[j / 4] = j % 4 ? w[j / 4] | v << (8 * (j % 4)) : v;
                }
                if (mr < M) {
                    unsigned char* o = out.r + ((int64_t)MODS * M + mr) * out.ldn + nc;
#pragma unroll
                    for (int j = 0; j < FM_HC / 16; ++j)
                        reinterpret_cast<uint4*>(o)[j] = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
                }
                continue;
            }
            if (mr >= M) continue;
            if (pl >= PL_CORR) {
                float4* o = reinterpret_cast<float4*>(out.corr + ((int64_t)(pl - PL_CORR) * M + mr) * out.ldn + nc);
#pragma unroll
                for (int j = 0; j < FM_HC / 4; ++j)
                    o[j] = make_float4(sum[4 * j], sum[4 * j + 1], sum[4 * j + 2], sum[4 * j + 3]);
                continue;
            }
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
            unsigned char* o = out.r + ((int64_t)mod * M + mr) * out.ldn + nc;
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
    // (earlier, the reconstruction's blocks would crowd on the SMs that are free first: 256^3 20.2 us for
    // the whole product, 15.5 so)
    ct_pdl_next();
}

struct FmC {
    double* p;       // row m at (m / M0) * s1 + (m % M0) * s0, columns contiguous
    int64_t M0, s1, s0;
};

constexpr int FM_CRT = 128;   // threads of the reconstruction: two rows of 128 columns

// FP64 dot products of row m of A with the rows n of B of the lanes in `mask`, v in the others.  A few
// are formed one after another by the warp, more by their lanes, at the rate of the FP64 pipe, in sums
// of 32.  (1280 x 1024 x 256 with 3% of the elements failing, in whole rows: 205 us by the warp alone, 117 so.)
__device__ __forceinline__ double fm_dots(const FmSrc& a, const FmSrc& b, int64_t m, int64_t n, unsigned mask, double v) {
    const int lane = threadIdx.x & 31;
    const double* pa = a.p + a.row(m);
    if (__popc(mask) > 6) {
        if ((mask >> lane) & 1) {
            const double* pb = b.p + b.row(n);
            v = 0.0;
            for (int64_t k0 = 0; k0 < a.K; k0 += 32) {
                double part = 0.0;
#pragma unroll
                for (int h = 0; h < 32; h += 8) {   // (eight loads of each in flight)
                    double x[8], y[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int64_t k = k0 + h + i;
                        x[i] = k < a.K ? pa[k * a.sk] : 0.0;
                        y[i] = k < a.K ? pb[k * b.sk] : 0.0;
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i) part = fma(x[i], y[i], part);
                }
                v += part;
            }
        }
        return v;
    }
    for (; mask; mask &= mask - 1) {
        const int src = __ffs(mask) - 1;
        const double* pb = b.p + b.row(__shfl_sync(0xffffffffu, n, src));
        double dot = 0.0;
        for (int64_t k0 = lane; k0 < a.K; k0 += 256) {
            double x[8], y[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int64_t k = k0 + 32 * i;
                x[i] = k < a.K ? pa[k * a.sk] : 0.0;
                y[i] = k < a.K ? pb[k * b.sk] : 0.0;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) dot = fma(x[i], y[i], dot);
        }
        dot = ct_warp_sum(dot);
        if (lane == src) v = dot;
    }
    return v;
}

// C from its residues: S = sum t_i P / m_i - k P with k = rint(sum t_i / m_i), plus the correction,
// then times 2^(ea + eb - 2 bits) and rounded to FP64.  Two moduli at a time, u = sum t_j G / m_j (below
// 2^17), so that the multi-word sums have eight terms.  A thread takes two columns of a row; the
// elements that fail the test, or have no scale, are FP64 dot products.
__global__ void __launch_bounds__(FM_CRT, 6) fm_crt_kernel(FmOut in, int M, int N, FmSrc a, FmSrc b, FmC c, int bits,
                                                     const CrtTable tab, const int* skip) {
    ct_pdl();
    if (ct_skip(skip)) return;
    const int64_t n0 = 2 * ((int64_t)blockIdx.y * 64 + (threadIdx.x & 63));
    const int64_t m = (int64_t)blockIdx.x * (FM_CRT / 64) + (threadIdx.x >> 6);   // the same for a warp
    if (m >= M) return;
    const int em = a.ex[m];
    uint32_t r2[MODS], t2 = 0;
    float2 cr = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < MODS; ++i) r2[i] = 0;
    if (n0 < N) {
#pragma unroll
        for (int i = 0; i < MODS; ++i)
            r2[i] = *reinterpret_cast<const uint16_t*>(in.r + ((int64_t)i * M + m) * in.ldn + n0);
        t2 = *reinterpret_cast<const uint16_t*>(in.r + ((int64_t)MODS * M + m) * in.ldn + n0);
        const float2 q = *reinterpret_cast<const float2*>(in.corr + m * in.ldn + n0);
        const float2 w = *reinterpret_cast<const float2*>(in.corr + ((int64_t)M + m) * in.ldn + n0);
        cr = make_float2(q.x + w.x, q.y + w.y);
    }
    double* Cr = c.p + (m / c.M0) * c.s1 + (m % c.M0) * c.s0;
    unsigned redo = 0;   // bit j: column n0 + j
#pragma unroll 1
    for (int j = 0; j < 2; ++j) {
        const int64_t n = n0 + j;
        const bool live = n < N;
        const int en = live ? b.ex[n] : 0;
        const unsigned answer = (t2 >> (8 * j)) & 0xffu;
        const float corr = j == 0 ? cr.x : cr.y;
        unsigned long long acc[LIMBS] = {};
        long long frac = -tab.rbias;
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
            unsigned u = 0;
#pragma unroll
            for (int i = 0; i < 2; ++i) u += ((r2[2 * g + i] >> (8 * j)) & 0xffu) * tab.co[g][i];
            frac += (long long)((unsigned long long)u * tab.rcp[g]);
#pragma unroll
            for (int l = 0; l < LIMBS; ++l) acc[l] += (unsigned long long)u * tab.w[g][l];
        }
        // (2^40 / G to half a unit: an error below 2^-20 of the fraction)
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
        unsigned long long hi = ((unsigned long long)s[3] << 32) | s[2], lo = ((unsigned long long)s[1] << 32) | s[0];
        const bool bad = em == FM_NONFINITE || en == FM_NONFINITE || answer == FM_FAIL ||
                         (answer == FM_NONE && ((hi | lo) != 0 || corr != 0.0f));
        {   // the correction, an integer of 2^-40 units, times 2^bits
            const long long ci = __float2ll_rn(corr * 1024.0f);
            const unsigned long long l = (unsigned long long)ci << (bits - 40);
            lo += l;
            hi += (unsigned long long)(ci >> (104 - bits)) + (lo < l ? 1 : 0);
        }
        const bool neg = (hi >> 63) != 0;
        if (neg) {
            lo = ~lo + 1;
            hi = ~hi + (lo == 0 ? 1 : 0);
        }
        // magnitude (below 2^126) left-aligned in (hi, lo); the leading bit is worth 2^top
        int top = 127;
        if (hi == 0) {
            hi = lo;
            lo = 0;
            top -= 64;
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
            f += (rem > 0x400 || (rem == 0x400 && (lo != 0 || (f & 1)))) ? 1 : 0;
            const int e = em + en - 2 * bits, ex = 1023 + top + e;   // exponent field of f's leading bit
            if (ex < 1 || ex > 2045) v = scalbn(neg ? -(double)f : (double)f, top - 52 + e);
            else v = __longlong_as_double((long long)((((unsigned long long)(ex - 1) << 52) + f) |
                                                      ((unsigned long long)neg << 63)));
        }
        if (live && bad) redo |= 1u << j;
        else if (live) Cr[n] = v;
    }
    // (apart from the loop above, whose code and registers stay few)
    if (!__any_sync(0xffffffffu, redo != 0)) return;
#pragma unroll 1
    for (int j = 0; j < 2; ++j) {
        const bool mine = (redo >> j) & 1;
        const unsigned mask = __ballot_sync(0xffffffffu, mine);
        if (mask == 0) continue;
        const double v = fm_dots(a, b, m, mine ? n0 + j : 0, mask, 0.0);
        if (mine) Cr[n0 + j] = v;
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
    q.bytes = ct_bytes(PLANES * M * q.ldk, 2) + ct_bytes(PLANES * N * q.ldk, 2) + ct_bytes((MODS + 1) * M * q.ldn, 1) +
              ct_bytes(2 * M * q.ldn, 4) + ct_bytes(M, 4) + ct_bytes(N, 4) + ct_bytes(ct_cdiv(K, FM_XK) * M, 4) + ct_bytes(ct_cdiv(K, FM_XK) * N, 4);
    return q;
}

// Room for `bytes`, with a quarter to spare for growing bonds where the limit and the memory allow it.
// Under a capture the new buffer is allocated too (in the thread's relaxed mode), so that a captured
// call computes as the same call does outside; nothing is waited for or freed then.
int fm_workspace(ct_handle* h, size_t bytes, bool capturing) {
    if (h->fm_ws_bytes >= bytes) return CT_OK;
    if (!capturing) CT_CUDA(h, cudaStreamSynchronize(h->stream));
    if (h->fm_ws && (h->fm_captured || capturing)) {   // graphs or launched kernels may run on it
        h->fm_kept.push_back(h->fm_ws);
        h->fm_kept_bytes += h->fm_ws_bytes;
    } else if (h->fm_ws) {
        cudaFree(h->fm_ws);
    }
    h->fm_captured = false;
    h->fm_ws = nullptr;
    h->fm_ws_bytes = 0;
    size_t want = bytes + bytes / 4;
    if (h->ws_limit && h->ws_cap + want > h->ws_limit) want = bytes;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    if (capturing) CT_CUDA(h, cudaThreadExchangeStreamCaptureMode(&mode));
    cudaError_t e = cudaMalloc(&h->fm_ws, want);
    if (e != cudaSuccess && want > bytes) {
        (void)cudaGetLastError();
        want = bytes;
        e = cudaMalloc(&h->fm_ws, want);
    }
    if (capturing) CT_CUDA(h, cudaThreadExchangeStreamCaptureMode(&mode));
    if (e != cudaSuccess) h->fm_ws = nullptr;
    CT_CUDA(h, e);
    h->fm_ws_bytes = want;
    return CT_OK;
}

int fm_map(ct_handle* h, CUtensorMap* m, const FmSrc& s, int box_rows) {
    PFN_cuTensorMapEncodeTiled_v12000 enc = ct_tma_encoder();
    if (!enc) return CT_ERR_UNSUPPORTED;
    if (((uintptr_t)s.res & 15) || (s.ldk % FM_BK)) {
        ct_seterr(h, "TMA operand misaligned (base %p, ldk %lld)", (const void*)s.res, (long long)s.ldk);
        return CT_ERR_INVALID;
    }
    cuuint64_t dims[2] = {(cuuint64_t)s.ldk, (cuuint64_t)(PLANES * s.R)};
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
// kernel at 85% of the FP64 pipe (2 multiply-adds per clock and SM, 1.9 GHz); here 11 us of
// launches and latencies, tile items at 1.2 us plus 0.16 us per 64 of K on each SM, and operands
// and residues written and read at 4 TB/s.  Measured (us, SIMT / here): 96x288x96 12.4 / 13.3,
// 128x256x128 12.9 / 12.2 and 128x384x128 16.9 / 14.7 stay, 128x512x128 20.7 / 14.0, 640x128x128
// 23.8 / 15.0, 256x256x128 20.9 / 13.7 and 256x256x256 36.9 / 15.5 go.  Only when the scratch is
// there or can be had: within the handle's workspace limit, beside the arena as it is, and with the
// memory available; otherwise the SIMT kernel.  (So a handle with a limit may compute a product either
// way, to the same accuracy, as its arena has grown: the arena comes first.)
bool ct_f64_route(ct_handle* h, int64_t M, int64_t N, int64_t K) {
    if (M <= 0 || N <= 0 || K <= 0 || K > ((int64_t)1 << 20) || !ct_fp64_tc_enabled(h, M, N, K)) return false;
    const FmPlan q = fm_plan(M, N, K);
    if (PLANES * M > (1ll << 30) || PLANES * N > (1ll << 30) || q.tiles * PLANES > (1ll << 30) || ct_cdiv(N, 128) > 65535)
        return false;
    const double simt = (double)M * (double)N * (double)K / (0.85 * 2.0 * h->num_sms * 1900.0);
    const double items = (double)ct_cdiv(q.tiles * PLANES, h->num_sms) * (1.2 + 0.16 * (double)(q.ldk / FM_BK));
    const double traffic = ((double)(M + N) * (double)q.ldk * 4.0 * PLANES + (double)M * (double)q.ldn * 2.0 * (MODS + 9)) / 4.0e6;
    if (11.0 + items + traffic > simt) return false;
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
    if (h->ws_limit && h->ws_cap + q.bytes > h->ws_limit) return false;
    const std::string keep = h->err;
    if (fm_workspace(h, q.bytes, capturing) != CT_OK) {
        (void)cudaGetLastError();
        h->err = keep;
        return false;
    }
    h->fm_captured |= capturing;
    return true;
}

// C(m,n) = sum_k A(m,k) B(n,k), operands and C with two-level row indexing (OzMat, OzOut in
// ct_ops.cuh); ct_f64_route must have accepted the size.
int ct_f64_gemm(ct_handle* h, int64_t M, int64_t N, int64_t K, const OzMat& A, const OzMat& B, const OzOut& Cout,
                const int* skip) {
    const FmPlan q = fm_plan(M, N, K);
    if (h->fm_ws_bytes < q.bytes) {
        ct_seterr(h, "ct_f64_gemm: no scratch for %lld x %lld x %lld", (long long)M, (long long)N, (long long)K);
        return CT_ERR_OOM;
    }
    uint8_t* p = (uint8_t*)h->fm_ws;
    FmSrc a{A.p, M, K, A.R0 > 0 ? A.R0 : M, A.s1, A.s0, A.sk, (__nv_bfloat16*)p, nullptr, nullptr, q.ldk};
    p += ct_bytes(PLANES * M * q.ldk, 2);
    FmSrc b{B.p, N, K, B.R0 > 0 ? B.R0 : N, B.s1, B.s0, B.sk, (__nv_bfloat16*)p, nullptr, nullptr, q.ldk};
    p += ct_bytes(PLANES * N * q.ldk, 2);
    const int bits = bits_for(K);
    const float theta = ldexpf(1.0f, 37 - bits);
    FmOut o{(unsigned char*)p, nullptr, theta * theta * (float)K * 1.01f, q.ldn};
    p += ct_bytes((MODS + 1) * M * q.ldn, 1);
    o.corr = (float*)p;
    p += ct_bytes(2 * M * q.ldn, 4);
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
        // the product kernel's share of the L1: an SM that changes it between the two loses time (256^3
        // 17.3 us without, 14.9 so)
        CT_CUDA(h, cudaFuncSetAttribute(fm_crt_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 60));
        attr_dev = h->device;
    }
    const Tables& t = tables();
    const int nba = (int)ct_cdiv(M, FM_PR);
    const dim3 grid((unsigned)(nba + ct_cdiv(N, FM_PR)), (unsigned)ct_cdiv(q.ldk, FM_PK));
    if (grid.y > 65535) return CT_ERR_UNSUPPORTED;
    if (K > FM_XK) {
        ct_launch(h, fm_rowexp_kernel, dim3(grid.x, (unsigned)ct_cdiv(K, FM_XK)), 256, 0, a, b, nba, skip); ct_note_launch();
    }
    ct_launch(h, fm_residue_kernel, grid, 256, 0, a, b, nba, bits, theta, t.mod, skip); ct_note_launch();
    const int64_t items = q.tiles * PLANES;
    const int64_t ctas = items < h->num_sms ? items : h->num_sms;
    ct_launch(h, fm_gemm_kernel, (unsigned)ctas, FM_THREADS, FM_SMEM, ta, tb, (int)M, (int)N, (int)q.ldk, o, t.mod, skip,
                                                                       h->d_status); ct_note_launch();
    const FmC c{Cout.p, Cout.M0 > 0 ? Cout.M0 : M, Cout.s1, Cout.s0};
    ct_launch(h, fm_crt_kernel, dim3((unsigned)ct_cdiv(M, FM_CRT / 64), (unsigned)ct_cdiv(N, 128)), FM_CRT, 0,
              o, (int)M, (int)N, a, b, c, bits, t.crt, skip); ct_note_launch();
    CT_LAUNCH_CHECK(h);
    return CT_OK;
}
