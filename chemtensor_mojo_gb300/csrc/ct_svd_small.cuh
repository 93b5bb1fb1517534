// One-sided Jacobi in FP64 of up to 200 KB of vectors and rotations, in one launch, every
// round spread over many SMs.
//
// What bounds it.  A warp issues one FP64 instruction every 64 cycles on this part (see
// ct_jacobi_coop.cuh), and the algorithm is a chain of nvec - 1 dependent rounds per sweep.
// In one CTA all pairs of a round shared one SM's FP64 pipe (25 ms for 64 x 64, 106 ms for
// 112 x 112 with singular values exp(-10 k / n)).  Here a team of four warps, one per
// sub-partition, takes a pair: three of them one dot product each (in the order of a
// one-warp dot product: lane l sums elements l, l + 32, ...), then all four the rotation.
//   * up to 96 vectors: one cluster of up to 16 CTAs with one to three teams each and the
//     hardware cluster barrier (~900 cycles with the stores before it);
//   * more: one team per CTA, every pair waiting for its two vectors alone (vec_wait), with a
//     grid barrier per sweep.
// (One launch per form, us: 64 vectors 3855 as a cluster and 4178 as a grid, 96 7383 and 7342.)
// The rotations and their order are those of the one-CTA form, operation for operation, so
// the factors come out the same to the last bit (the signs of singular vectors included,
// which depend on the path: without QR preconditioning a change of 1e-16 flips some).
#pragma once
#include "ct_jacobi_coop.cuh"

namespace ct_svd_small {

constexpr int CLUSTER_MAX = 96;     // up to this many vectors: one cluster
constexpr int CLUSTER_CTAS = 16;
constexpr int MAX_SWEEPS = 60;
constexpr int TEAM = 128;           // threads of a team
constexpr int MAX_TEAMS = 3;

struct Args {
    const double* M;        // m x n, row-major
    int64_t n;              // columns of M
    int cols;               // 1: the vectors are M's columns, 0: its rows
    int nvec, len;
    double* X;              // nvec x len
    double* Q;              // nvec x nvec
    double* nsq;            // nvec: |x|^2 of the start vectors (scratch)
    double tol;
    int max_sweeps;
    ct_jacobi::Sync s;
};

__device__ __forceinline__ void team_sync(int team) {
    asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "r"(TEAM) : "memory");
}

// E: elements per thread of a team's vectors, TEAM E >= max(len, nvec), or 0: any length, the
// vectors read twice instead of held.
template <int E, bool CLUSTER>
__global__ void __launch_bounds__(CLUSTER ? TEAM * MAX_TEAMS : TEAM) svd_small_kernel(Args a) {
    ct_pdl();
    constexpr int R = E > 0 ? E : 1;
    constexpr double EPS = 2.2204460492503131e-16;
    __shared__ double dots[MAX_TEAMS][3];
    __shared__ double rot_s[MAX_TEAMS][2];
    __shared__ int go_s[MAX_TEAMS];
    __shared__ int live;
    const int lane = threadIdx.x & 31;
    // warps spread over the CTAs first, so that fewer tasks than warps still use every SM
    const int w = (int)(threadIdx.x >> 5) * (int)gridDim.x + (int)blockIdx.x;
    const int nw = (int)(blockDim.x >> 5) * (int)gridDim.x;
    const int len = a.len, nvec = a.nvec;
    unsigned target = 0;
    // Barrier of the launch.  Data that crosses it is written with plain stores and read with
    // __ldcg (the L1 of another SM may hold an old copy).
    auto barrier = [&]() -> bool {
        if constexpr (CLUSTER) {
            __syncwarp();
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
            return true;
        } else {
            return ct_jacobi::grid_barrier(a.s, target);
        }
    };

    for (int v = w; v < nvec; v += nw) {
        double f2 = 0.0;
        for (int i = lane; i < len; i += 32) {
            const double x = a.cols ? a.M[(int64_t)i * a.n + v] : a.M[(int64_t)v * a.n + i];
            a.X[(int64_t)v * len + i] = x;
            f2 = fma(x, x, f2);
        }
        f2 = ct_warp_sum(f2);
        if (lane == 0) a.nsq[v] = f2;
        for (int i = lane; i < nvec; i += 32) a.Q[(int64_t)v * nvec + i] = i == v ? 1.0 : 0.0;
    }
    if (!barrier()) return;
    double f2 = 0.0;
    for (int i = lane; i < nvec; i += 32) f2 += __ldcg(a.nsq + i);
    const double floor = EPS * EPS * ct_warp_sum(f2);

    // (the roles of a team's warps start one SM quarter later in each team, so that two teams'
    // rotations, a chain of FP64 instructions in one warp, do not share a quarter)
    const int team = (int)threadIdx.x / TEAM, tt = (int)threadIdx.x % TEAM, tw = ((tt >> 5) + 4 - team) & 3;
    const int gt = team * (int)gridDim.x + (int)blockIdx.x;
    const int teams = (int)(blockDim.x / TEAM) * (int)gridDim.x;
    // Q's elements start half a team later than X's: up to 64 of each are rotated side by side
    const int tq = (tt + TEAM / 2) % TEAM;
    const int P = nvec + (nvec & 1);
    bool converged = false;
    int sweep = 0;
    for (; sweep < a.max_sweeps && !converged; ++sweep) {
        for (int r = 0; r < P - 1; ++r) {
            for (int pr = gt; pr < P / 2; pr += teams) {
                int p, q;
                ct_jacobi::pair_index(P, r, pr, p, q);
                if (p >= nvec || q >= nvec) continue;   // the same for the whole team
                const unsigned base = (unsigned)(sweep * (P - 1));
                if constexpr (!CLUSTER) {   // (one team per CTA)
                    if (a.s.ver && r > 0) {
                        if (tt < 32) {
                            const bool odd = nvec & 1;
                            const bool there = ct_jacobi::vec_wait(a.s, p, ct_jacobi::vec_expected(base, r, p, odd), q,
                                                                   ct_jacobi::vec_expected(base, r, q, odd));
                            if (tt == 0) live = there;
                        }
                        team_sync(team);
                        if (!live) return;
                    }
                }
                double* xp = a.X + (int64_t)p * len;
                double* xq = a.X + (int64_t)q * len;
                double* qp = a.Q + (int64_t)p * nvec;
                double* qq = a.Q + (int64_t)q * nvec;
                double x[R], y[R], g[R], h[R];
                if constexpr (E > 0) {
#pragma unroll
                    for (int e = 0; e < E; ++e) {
                        const int i = e * TEAM + tt, iq = e * TEAM + tq;
                        x[e] = i < len ? __ldcg(xp + i) : 0.0;
                        y[e] = i < len ? __ldcg(xq + i) : 0.0;
                        g[e] = iq < nvec ? __ldcg(qp + iq) : 0.0;
                        h[e] = iq < nvec ? __ldcg(qq + iq) : 0.0;
                    }
                }
                // warp 0: |x_p|^2, warp 1: |x_q|^2, warp 2: <x_p, x_q>
                if (tw < 3) {
                    const double* u = tw == 1 ? xq : xp;
                    const double* v = tw == 0 ? xp : xq;
                    double s = 0.0;
                    if constexpr (E > 0) {
                        double uu[4 * R], vv[4 * R];
#pragma unroll
                        for (int e = 0; e < 4 * E; ++e) {
                            const int i = e * 32 + lane;
                            uu[e] = i < len ? __ldcg(u + i) : 0.0;
                            vv[e] = i < len ? __ldcg(v + i) : 0.0;
                        }
#pragma unroll
                        for (int e = 0; e < 4 * E; ++e)
                            if (e * 32 < len) s = fma(uu[e], vv[e], s);
                    } else {
                        for (int i = lane; i < len; i += 32) s = fma(__ldcg(u + i), __ldcg(v + i), s);
                    }
                    s = ct_warp_sum(s);
                    if (lane == 0) dots[team][tw] = s;
                }
                team_sync(team);
                if (tw == 3) {
                    double cs = 1.0, sn = 0.0;
                    const bool go = ct_jacobi::rotation(dots[team][0], dots[team][1], dots[team][2], a.tol, floor, cs, sn);
                    if (lane == 0) {
                        go_s[team] = go ? 1 : 0;
                        rot_s[team][0] = cs;
                        rot_s[team][1] = sn;
                        if (go) a.s.rot[sweep] = 1;
                    }
                }
                team_sync(team);
                const bool go = go_s[team];
                const double cs = rot_s[team][0], sn = rot_s[team][1];
                if (!go) {
                } else if constexpr (E > 0) {
#pragma unroll
                    for (int e = 0; e < E; ++e) {
                        const int i = e * TEAM + tt, iq = e * TEAM + tq;
                        if (i < len) {
                            const double u = x[e], v = y[e];
                            xp[i] = ct_jacobi::rot_x(cs, sn, u, v);
                            xq[i] = ct_jacobi::rot_y(cs, sn, u, v);
                        }
                        if (iq < nvec) {
                            const double u = g[e], v = h[e];
                            qp[iq] = ct_jacobi::rot_x(cs, sn, u, v);
                            qq[iq] = ct_jacobi::rot_y(cs, sn, u, v);
                        }
                    }
                } else {
                    for (int i = tt; i < len; i += TEAM) {
                        const double u = __ldcg(xp + i), v = __ldcg(xq + i);
                        xp[i] = ct_jacobi::rot_x(cs, sn, u, v);
                        xq[i] = ct_jacobi::rot_y(cs, sn, u, v);
                    }
                    for (int i = tq; i < nvec; i += TEAM) {
                        const double u = __ldcg(qp + i), v = __ldcg(qq + i);
                        qp[i] = ct_jacobi::rot_x(cs, sn, u, v);
                        qq[i] = ct_jacobi::rot_y(cs, sn, u, v);
                    }
                }
                if constexpr (!CLUSTER) {
                    if (a.s.ver) {
                        team_sync(team);
                        if (tt < 2) ct_jacobi::vec_done(a.s, tt ? q : p, base + (unsigned)r + 1);
                    }
                }
            }
            if (CLUSTER || !a.s.ver || r == P - 2) {
                if (!barrier()) return;
            }
        }
        // every CTA reads the same word: nothing writes rot[sweep] after the last barrier
        converged = __ldcg(a.s.rot + sweep) == 0;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *a.s.sweeps = sweep;
        if (!converged) ct_set_status(a.s.status, CT_ERR_NOCONV);
    }
}

template <int E, bool CLUSTER>
int launch(ct_handle* h, Args& a, int ctas, int teams) {
    const dim3 block((unsigned)(TEAM * teams));
    if (CLUSTER) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)ctas);
        cfg.blockDim = block;
        cfg.stream = h->stream;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)ctas;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        CT_CUDA(h, cudaLaunchKernelEx(&cfg, svd_small_kernel<E, CLUSTER>, a));
    } else {
        void* args[] = {&a};
        cudaError_t e;
        do {   // (fewer CTAs where the handle has not the whole device)
            e = cudaLaunchCooperativeKernel((const void*)svd_small_kernel<E, CLUSTER>, dim3((unsigned)ctas), block, args, 0,
                                            h->stream);
        } while (e == cudaErrorCooperativeLaunchTooLarge && cudaGetLastError() == e && (ctas /= 2) > 0);
        CT_CUDA(h, e);
    }
    ct_note_launch();
    return CT_OK;
}

// Jacobi of the vectors of M (nvec >= 2): X, Q and nsq in the fields set by the caller; the
// sweeps run go to d_flags[19].
inline int run(ct_handle* h, Args& a) {
    CT_TRY(ct_jacobi::reset_sync(h, MAX_SWEEPS, a.nvec, a.s));
    a.max_sweeps = (h->svd_max_sweeps > 0 && h->svd_max_sweeps < MAX_SWEEPS) ? h->svd_max_sweeps : MAX_SWEEPS;
    const int pairs = (a.nvec + 1) / 2;
    const int big = a.len > a.nvec ? a.len : a.nvec;
    if (a.nvec <= CLUSTER_MAX) {
        int ctas = 1;
        while (ctas < pairs && ctas < CLUSTER_CTAS) ctas *= 2;
        // the largest cluster that can run here; the rotations are the same in any
        const auto kernel = big <= TEAM       ? svd_small_kernel<1, true>
                            : big <= 2 * TEAM ? svd_small_kernel<2, true>
                                              : svd_small_kernel<0, true>;
        while (ctas > 1 && !ct_cluster_fits(h, kernel, (unsigned)ctas, TEAM * MAX_TEAMS)) ctas /= 2;
        const int teams = std::min((pairs + ctas - 1) / ctas, MAX_TEAMS);
        if (big <= TEAM) return launch<1, true>(h, a, ctas, teams);
        if (big <= 2 * TEAM) return launch<2, true>(h, a, ctas, teams);
        return launch<0, true>(h, a, ctas, teams);
    }
    const int ctas = pairs < h->num_sms ? pairs : h->num_sms;
    if (big <= TEAM) return launch<1, false>(h, a, ctas, 1);
    if (big <= 2 * TEAM) return launch<2, false>(h, a, ctas, 1);
    return launch<0, false>(h, a, ctas, 1);
}

}  // namespace ct_svd_small
