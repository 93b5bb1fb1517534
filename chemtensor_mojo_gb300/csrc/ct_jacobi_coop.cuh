// Persistent one-sided Jacobi: all round-robin rounds of all sweeps in one
// cooperative launch.  Every CTA walks the pairs of a round (k = blockIdx.x,
// += gridDim.x), each pair waiting for its two vectors; after each sweep all meet at a
// grid barrier, read the sweep's rotation flag and leave together when it is zero.  The
// waits spin at most 2 s (then sets the status word and aborts), and cooperative
// launch refuses grids that cannot be co-resident, so no wait is unbounded.
//
// What bounds it.  A warp issues one FP64 instruction every 64 cycles on this part
// (measured: 65 cycles per dependent FMA, 514 for eight independent ones of one warp; the
// four sub-partitions of an SM together one per 16), a division takes 660 cycles and a square
// root ~900.  Per pair and round the three 256-thread block sums were 120 FP64 instructions
// and nine barriers, the rotation's scalars ~4500 cycles in series.  Here the three sums
// share their instructions (tri_sum: 48, two barriers, the same additions in the same order)
// and the scalars take ~2300 cycles (rotation).
#pragma once
#include "ct_common.cuh"
#include "ct_fp64.cuh"

namespace ct_jacobi {

using namespace ct_fp64;

constexpr int NT = 256;
constexpr int MAX_SWEEPS = 48;

__device__ __forceinline__ unsigned long long gtime() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

struct Sync {
    unsigned* count;   // arrivals of all barriers of the launch, zeroed before it
    int* abort_flag;
    int* rot;          // [MAX_SWEEPS] nonzero: the sweep rotated; zeroed before launch
    int* sweeps;       // out: sweeps run
    int* status;
    unsigned* ver;     // [vectors] rounds completed of each, zeroed before the launch; null: a grid
                       // barrier after every round
};

// A round needs its vectors from two pairs of the round before, so within a sweep a pair waits
// for those alone: every vector has a count of completed rounds (a grid barrier of 128 CTAs takes
// ~2300 cycles after the stores, a release and an acquire ~1000, and no pair waits for the
// slowest).  The counts a pair waits for at round r (base: rounds of the sweeps before): r, or
// r - 1 of the vector that had no partner in the round before (odd numbers of vectors; pair 0).
__device__ __forceinline__ unsigned vec_expected(unsigned base, int r, int v, bool odd) {
    return base + (unsigned)r - (odd && v == r - 1 ? 1u : 0u);
}
// by one warp: true when both counts are there, false when the launch gives up
__device__ __forceinline__ bool vec_wait(const Sync& s, int p, unsigned ep, int q, unsigned eq) {
    const int lane = threadIdx.x & 31;
    const unsigned* at = s.ver + (lane == 0 ? p : q);
    const unsigned want = lane == 0 ? ep : eq;
    const unsigned long long t0 = gtime();
    for (;;) {
        bool ready = true, give_up = false;
        if (lane < 2) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(at) : "memory");
            ready = (int)(v - want) >= 0;
            if (!ready) {
                give_up = *(volatile int*)s.abort_flag != 0;
                if (!give_up && gtime() - t0 > 2000000000ull) {
                    atomicExch(s.abort_flag, 1);
                    ct_set_status(s.status, CT_ERR_CUDA);
                    give_up = true;
                }
            }
        }
        if (__any_sync(0xffffffffu, give_up)) return false;
        if (__all_sync(0xffffffffu, ready)) return true;
    }
}
// by one thread per vector, after a barrier of the threads that wrote it
__device__ __forceinline__ void vec_done(const Sync& s, int v, unsigned count) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(s.ver + v), "r"(count) : "memory");
}

// target: arrivals expected so far (per thread, starting at 0).  Data that crosses the
// barrier is read with __ldcg (the L1 of another SM may hold an old copy).
__device__ __forceinline__ bool grid_barrier(const Sync& s, unsigned& target) {
    __shared__ int ok;
    target += gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = 1;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(s.count) : "memory");
        const unsigned long long t0 = gtime();
        for (;;) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(s.count) : "memory");
            if ((int)(v - target) >= 0) break;
            if (*(volatile int*)s.abort_flag) { ok = 0; break; }
            if (gtime() - t0 > 2000000000ull) {
                ok = 0;
                atomicExch(s.abort_flag, 1);
                ct_set_status(s.status, CT_ERR_CUDA);
                break;
            }
        }
    }
    __syncthreads();
    return ok != 0;
}

__device__ __forceinline__ void pair_index(int P, int r, int k, int& p, int& q) {
    if (k == 0) {
        p = P - 1;
        q = r;
    } else {
        p = (r + k) % (P - 1);
        q = (r - k + (P - 1)) % (P - 1);
    }
}

// Rotation that orthogonalises two vectors with |x_p|^2=a, |x_q|^2=b, <x_p,x_q>=c.
// Vectors with |x|^2 <= floor (numerically zero next to |M|_F) are left alone:
// rotating rounding noise never converges.  The threshold |c| > tol sqrt(a b) is decided in
// FP32 on the mantissas and exponents unless the two sides agree to 1e-5.
__device__ __forceinline__ bool rotation(double a, double b, double c, double tol, double floor, double& cs,
                                         double& sn) {
    if (!(a > floor && b > floor) || c == 0.0) return false;
    {
        const int ea = exp_field(a), eb = exp_field(b), ec = exp_field(c), et = exp_field(tol);
        bool go;
        const int de = 2 * (ec - 1023) - (ea - 1023) - (eb - 1023) - 2 * (et - 1023);
        if (mid_exp(ea) && mid_exp(eb) && mid_exp(ec) && mid_exp(et)) {
            const float fc = mant_f32(c), ft = mant_f32(tol);
            // c^2 / (tol^2 a b) = ratio 2^de, ratio in (1/16, 4)
            const float ratio = __fdividef(fc * fc, ft * ft * (mant_f32(a) * mant_f32(b)));
            if (de > 6) go = true;
            else if (de < -6) go = false;
            else {
                const float z = ratio * __int_as_float((127 + de) << 23);
                go = z > 1.00001f;
                if (!go && z > 0.99999f) go = fabs(c) > tol * sqrt(a * b);
            }
        } else {
            go = fabs(c) > tol * sqrt(a * b);
        }
        if (!go) return false;
    }
    const double zeta = div_rn(b - a, 2.0 * c);
    double t;
    if (fabs(zeta) > 1e150) t = 0.5 / zeta;
    else t = copysign(div_rn(1.0, fabs(zeta) + sqrt_rn(1.0 + zeta * zeta)), zeta);
    cs = div_rn(1.0, sqrt_rn(1.0 + t * t));
    sn = cs * t;
    return true;
}

// Sums of a, b and c over the 256 threads of the CTA, each with the additions of ct_block_sum in
// its order (a warp butterfly, then the eight warp sums by the first warp), the three sharing
// instructions: per warp 6 FP64 additions instead of 15, then 3 instead of 15.  The results
// are valid in the first 24 lanes of warp 0: lanes 0-7 hold a's sum, 8-15 b's, 16-23 c's.
__device__ __forceinline__ double tri_sum(double a, double b, double c, double* sm) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // offset 16: a in lanes 0-15, b in lanes 16-31 of y; c in both halves
    const bool lo = lane < 16;
    double y = (lo ? a : b) + __shfl_xor_sync(0xffffffffu, lo ? b : a, 16);
    c += __shfl_xor_sync(0xffffffffu, c, 16);
    // offset 8: lanes 0-7 a, 8-15 b, 16-23 c
    const int src = lane < 8 ? lane : lane + 8;          // a: 0-7, b: 16-23
    const double y1 = __shfl_sync(0xffffffffu, y, src & 31), y2 = __shfl_sync(0xffffffffu, y, (src + 8) & 31);
    const double c2 = __shfl_xor_sync(0xffffffffu, c, 8);
    y = lo ? y1 + y2 : c + c2;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
    if (lane < 24 && (lane & 7) == 0) sm[(lane >> 3) * 8 + wid] = y;
    __syncthreads();
    if (wid == 0) {
        y = lane < 24 ? sm[lane] : 0.0;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
    }
    return y;
}

// x' = cs x - sn y, y' = sn x + cs y, the multiply-adds fixed (the same bits in every kernel)
template <typename T>
__device__ __forceinline__ T rot_x(T cs, T sn, T x, T y) { return fma(cs, x, -(sn * y)); }
template <typename T>
__device__ __forceinline__ T rot_y(T cs, T sn, T x, T y) { return fma(sn, x, cs * y); }

// T = float (mixed form: FP32 data, FP64 reductions) or double (plain form)
template <typename T>
__global__ void __launch_bounds__(NT) jacobi_coop_kernel(T* X, int64_t len, T* Q, int64_t nvec, double tol,
                                                        double floor_rel, const double* frob2, int max_sweeps,
                                                        Sync s) {
    ct_pdl();
    __shared__ double sm[24];
    __shared__ double rot_cs, rot_sn;
    __shared__ int do_rot, live;
    const int P = (int)(nvec + (nvec & 1));
    const double floor = floor_rel * (*frob2);
    const int tid = threadIdx.x;
    // vectors of up to 256 elements stay in a register between the sums and the rotation
    const bool held = len <= NT && nvec <= NT;
    unsigned target = 0;
    int sweep = 0;
    bool ok = true, last_rot = true;
    for (; sweep < max_sweeps && ok; ++sweep) {
        for (int r = 0; r < P - 1 && ok; ++r) {
            for (int k = blockIdx.x; k < P / 2; k += gridDim.x) {
                int p, q;
                pair_index(P, r, k, p, q);
                if (p >= nvec || q >= nvec) continue;
                const unsigned base = (unsigned)(sweep * (P - 1));
                if (s.ver && r > 0) {
                    if (tid < 32) {
                        const bool odd = nvec & 1;
                        const bool there = vec_wait(s, p, vec_expected(base, r, p, odd), q, vec_expected(base, r, q, odd));
                        if (tid == 0) live = there;
                    }
                    __syncthreads();
                    if (!live) {
                        ok = false;
                        break;
                    }
                }
                T* xp = X + (int64_t)p * len;
                T* xq = X + (int64_t)q * len;
                T* qp = Q + (int64_t)p * nvec;
                T* qq = Q + (int64_t)q * nvec;
                T x = 0, y = 0, g = 0, h = 0;
                T fa = 0, fb = 0, fc = 0;
                if (held) {
                    if (tid < len) {
                        x = __ldcg(xp + tid);
                        y = __ldcg(xq + tid);
                    }
                    if (tid < nvec) {
                        g = __ldcg(qp + tid);
                        h = __ldcg(qq + tid);
                    }
                    if (tid < len) {
                        fa += x * x;
                        fb += y * y;
                        fc += x * y;
                    }
                } else {
                    for (int64_t i = tid; i < len; i += NT) {
                        const T u = __ldcg(xp + i), v = __ldcg(xq + i);
                        fa += u * u;
                        fb += v * v;
                        fc += u * v;
                    }
                }
                const double sum = tri_sum((double)fa, (double)fb, (double)fc, sm);
                if (tid < 32) {
                    const double a = __shfl_sync(0xffffffffu, sum, 0), b = __shfl_sync(0xffffffffu, sum, 8),
                                 c = __shfl_sync(0xffffffffu, sum, 16);
                    double cs = 1.0, sn = 0.0;
                    const bool go = rotation(a, b, c, tol, floor, cs, sn);
                    if (tid == 0) {
                        rot_cs = cs;
                        rot_sn = sn;
                        if (go) s.rot[sweep] = 1;
                        do_rot = go ? 1 : 0;
                    }
                }
                __syncthreads();
                if (do_rot) {
                    const T cs = (T)rot_cs, sn = (T)rot_sn;
                    if (held) {
                        if (tid < len) {
                            xp[tid] = rot_x<T>(cs, sn, x, y);
                            xq[tid] = rot_y<T>(cs, sn, x, y);
                        }
                        if (tid < nvec) {
                            qp[tid] = rot_x<T>(cs, sn, g, h);
                            qq[tid] = rot_y<T>(cs, sn, g, h);
                        }
                    } else {
                        for (int64_t i = tid; i < len; i += NT) {
                            const T u = __ldcg(xp + i), v = __ldcg(xq + i);
                            xp[i] = rot_x<T>(cs, sn, u, v);
                            xq[i] = rot_y<T>(cs, sn, u, v);
                        }
                        for (int64_t i = tid; i < nvec; i += NT) {
                            const T u = __ldcg(qp + i), v = __ldcg(qq + i);
                            qp[i] = rot_x<T>(cs, sn, u, v);
                            qq[i] = rot_y<T>(cs, sn, u, v);
                        }
                    }
                }
                __syncthreads();
                if (s.ver && tid < 2) vec_done(s, tid ? q : p, base + (unsigned)r + 1);
            }
            if (ok && (!s.ver || r == P - 2)) ok = grid_barrier(s, target);
        }
        if (!ok) break;
        last_rot = __ldcg(s.rot + sweep) != 0;
        if (!last_rot) {
            ++sweep;
            break;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *s.sweeps = sweep;
        if (ok && sweep >= max_sweeps && last_rot) ct_set_status(s.status, CT_ERR_NOCONV);
    }
}

// Barrier and sweep scratch of a launch in d_flags: [16] count, [18] abort, [19] sweeps,
// [32 .. 32 + max_sweeps) rotation flags; zeroed on the stream.
// The vectors' counts are in d_partials, where they fit.
inline int reset_sync(ct_handle* h, int max_sweeps, int64_t nvec, Sync& s) {
    s.ver = nullptr;
    if (nvec > 0 && nvec <= 2 * (int64_t)CT_NPARTIALS) {
        s.ver = (unsigned*)h->d_partials;
        CT_CUDA(h, cudaMemsetAsync(s.ver, 0, (size_t)nvec * sizeof(unsigned), h->stream));
    }
    int* base = h->d_flags;
    CT_CUDA(h, cudaMemsetAsync(base + 16, 0, (16 + max_sweeps) * sizeof(int), h->stream));
    s.count = (unsigned*)(base + 16);
    s.abort_flag = base + 18;
    s.sweeps = base + 19;
    s.rot = base + 32;
    s.status = h->d_status;
    return CT_OK;
}

// Launches the persistent Jacobi; sync scratch comes from h->d_flags.
template <typename T>
int run(ct_handle* h, T* X, int64_t len, T* Q, int64_t nvec, double tol, double floor_rel, const double* frob2,
        int* sweeps_host) {
    if (nvec < 2) {
        if (sweeps_host) *sweeps_host = 0;
        return CT_OK;
    }
    Sync s;
    CT_TRY(reset_sync(h, MAX_SWEEPS, nvec, s));
    static int occ_dev = -1, occ = 0;
    if (occ_dev != h->device) {
        CT_CUDA(h, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, jacobi_coop_kernel<T>, NT, 0));
        occ_dev = h->device;
    }
    const int64_t pairs = (nvec + (nvec & 1)) / 2;
    int64_t grid = (int64_t)occ * h->num_sms;
    if (grid > pairs) grid = pairs;
    if (grid < 1) grid = 1;
    // the handle's sweep cap (ct_set_svd_max_sweeps) never exceeds the kernel's own
    int max_sweeps = (h->svd_max_sweeps > 0 && h->svd_max_sweeps < MAX_SWEEPS) ? h->svd_max_sweeps : MAX_SWEEPS;
    void* args[] = {&X, &len, &Q, &nvec, &tol, &floor_rel, (void*)&frob2, &max_sweeps, &s};
    CT_CUDA(h, cudaLaunchCooperativeKernel((const void*)jacobi_coop_kernel<T>, dim3((unsigned)grid), dim3(NT), args,
                                           0, h->stream));
    ct_note_launch();
    CT_TRY(ct_readback(h));
    const int sw = ct_host(h, s.sweeps);
    h->last_svd_sweeps = sw;
    h->total_svd_sweeps += sw;
    if (sweeps_host) *sweeps_host = sw;
    return CT_OK;
}

}  // namespace ct_jacobi
