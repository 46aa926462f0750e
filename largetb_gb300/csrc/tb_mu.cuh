// tb_mu.cuh -- the chemical potential's multisection (runKPM's mu search,
// withSP2_deltaH.cpp:1640-1712, on the electron count): DOS at the quadrature
// nodes, electron count of a candidate, end of a round; and the mixing's small
// linear system.  Shared by the single-structure and the batched kernels.
#pragma once

#include <cuda_runtime.h>
#include <math.h>

#include "tb_internal.h"

namespace tb {

// Above this beta_x the multisection evaluates the Fermi function node by node;
// below it e^{beta x} e^{-beta mu} stays far inside the FP64 range (|t| <= 600).
constexpr double kEtabBeta = 300.0;
constexpr int kDosSlices = 8;  // lanes that share a node's sum
constexpr int kDosGroup = 32 / kDosSlices;  // nodes of a warp, whose sum is kept beside them
constexpr int kDosBlock = 8 * kDosGroup;    // nodes of a CTA of 256 threads

__device__ __forceinline__ double fermi(double x, double mu_x, double beta_x)
{
    const double t = beta_x * (x - mu_x);
    if (t > 0) {
        const double e = exp(-t);
        return e / (1.0 + e);
    }
    return 1.0 / (1.0 + exp(t));
}

// rho_q = g_0 mu_0 + 2 sum_{k>=1} g_k mu_k cos(k theta_q): the damped DOS at
// the Chebyshev-Gauss nodes (times pi sin theta), e^{beta_x x_q} beside it and
// the sums of kDosGroup nodes, for the CTAs blockIdx.x of one structure (256
// threads; wk: M doubles of shared memory).  Eight neighbouring lanes share a
// node: one thread a node walks M dependent table loads on a handful of CTAs
// (nq = 2048, M = 300: 45 us).
__device__ __forceinline__ void dos_nodes(const double *__restrict__ g, const double *__restrict__ mom, int M,
                                          double beta_x, int nq, int nq_cap, const double *__restrict__ tab, double *wk,
                                          double *__restrict__ rho, double *__restrict__ ebx, double *__restrict__ gsum)
{
    for (int k = threadIdx.x; k < M; k += blockDim.x) wk[k] = k == 0 ? g[0] * mom[0] : 2.0 * g[k] * mom[k];
    __syncthreads();
    const int r = nq > 0 ? nq_cap / nq : 1;
    const size_t cmask = 4 * (size_t)nq_cap - 1;  // keeps every table index in range
    const unsigned mask = 4u * (unsigned)nq - 1u;
    const int sl = threadIdx.x % kDosSlices;
    const int len = (M + kDosSlices - 1) / kDosSlices, k0 = sl * len, k1 = min(M, k0 + len);
    for (int q0 = blockIdx.x * kDosBlock; q0 < nq; q0 += gridDim.x * kDosBlock) {  // nq is a multiple of kDosBlock
        const int q = q0 + threadIdx.x / kDosSlices;
        const unsigned step = 2u * (unsigned)q + 1u;
        unsigned j = ((unsigned)k0 * step) & mask;
        double s = 0.0;
#pragma unroll 8
        for (int k = k0; k < k1; k++) {
            s += wk[k] * tab[((size_t)j * r) & cmask];
            j = (j + step) & mask;
        }
        for (int o = 1; o < kDosSlices; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (sl == 0) {
            rho[q] = s;
            // e^{beta_x x_q} for the multisection; unused above kEtabBeta
            ebx[q] = beta_x <= kEtabBeta ? exp(beta_x * tab[((size_t)step * r) & cmask]) : 0.0;
        }
        for (int o = kDosSlices; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if ((threadIdx.x & 31) == 0) gsum[q / kDosGroup] = s;
    }
}

// sum_q f(x_q) rho_q at candidate p of P equispaced ones in [lo, hi], by a CTA
// of 256 threads; thread 0 has the sum.  FP64 issues two operations a clock
// and SM, so what all threads repeat costs more than the sum: the Fermi
// function is evaluated within 40 kT of mu only -- beyond it is nought or one
// to 4e-18 -- with the nodes further below entering by their group sums (2048
// nodes at beta_x = 45: some 1200 divisions), the window is found in FP32 with
// nodes to spare, and one thread evaluates mu and e^{-beta mu}.
// Measured (M = 120, nq = 2048): 17.3 -> 10.7 us a round.
__device__ __forceinline__ double fermi_count(const double *__restrict__ rho, const double *__restrict__ ebx,
                                              const double *__restrict__ gsum, const double *__restrict__ tab, int nq,
                                              int nq_cap, double lo, double hi, int p, int P, double beta_x)
{
    __shared__ double s_mu, s_c, s_w[8];
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid == 0) {
        const double mu = lo + (hi - lo) * (double)p / (double)(P - 1);
        s_mu = mu;
        // f(x_q) = 1 / (1 + e^{beta x_q} e^{-beta mu}): one exp per candidate,
        // the node factors from dos_nodes (no overflow below kEtabBeta)
        s_c = beta_x <= kEtabBeta ? exp(-beta_x * mu) : 0.0;
    }
    const int r = nq > 0 ? nq_cap / nq : 1;
    const size_t cmask = 4 * (size_t)nq_cap - 1;  // keeps every table index in range
    // Nodes x_q = cos(pi (q + 1/2) / nq) fall with q: [qa, qb) holds mu +- w.
    // FP32 arguments are off by 3e-7, which near +-1 is 8e-4 in the angle, or
    // nq / 4000 nodes.
    const float mu32 = (float)lo + (float)(hi - lo) * (float)p / (float)(P - 1), w = 40.f / (float)beta_x;
    const float per = (float)nq * 0.318309886f;  // nodes per radian
    const int spare = 2 + (nq >> 11);
    int qa = 0, qb = nq;
    if (mu32 + w < 1.f) qa = max(0, (int)(acosf(fmaxf(mu32 + w, -1.f)) * per) - spare);
    if (mu32 - w > -1.f) qb = min(nq, (int)(acosf(fminf(mu32 - w, 1.f)) * per) + spare);
    qb = (qb + kDosGroup - 1) / kDosGroup * kDosGroup;
    double s = 0.0;
    for (int u = qb / kDosGroup + tid; u < nq / kDosGroup; u += blockDim.x) s += gsum[u];
    int q = qa + tid;
    double d = q < qb ? rho[q] : 0.0, e = q < qb ? ebx[q] : 0.0;
    __syncthreads();
    if (beta_x <= kEtabBeta) {
        const double C = s_c;
        while (q < qb) {
            s += d / (1.0 + e * C);
            q += blockDim.x;
            if (q < qb) {
                d = rho[q];
                e = ebx[q];
            }
        }
    } else {
        const double mu = s_mu;
        for (; q < qb; q += blockDim.x) s += fermi(tab[((size_t)(2 * q + 1) * r) & cmask], mu, beta_x) * rho[q];
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) s_w[tid >> 5] = s;
    __syncthreads();
    if (tid < 32) {
        s = lane < 8 ? s_w[lane] : 0.0;
        for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    }
    return s;
}

// Narrow [lo, hi] from the electron counts vc[0 .. kBisectCand) of equispaced
// candidates, or record the solution (the nearest candidate, within tol_n) or
// a bracketing failure.  Called by every thread of the round's last CTA (at
// least kBisectCand threads, whole warps): one thread scanning the candidates
// through dependent L2 loads took 30 us of a 36 us round.
__device__ __forceinline__ void bisect_narrow(const double *vc, double lo, double hi, double n_elec, double tol_n,
                                              int round, int last_round, DevState *st)
{
    static_assert(kBisectCand == 128, "four warps of candidates");
    __shared__ double s_dv[4];
    __shared__ int s_best[4], s_ge[4];
    const int P = kBisectCand, i = threadIdx.x, lane = i & 31;
    if (i < P) {
        const double v = __ldcg(vc + i), dev = fabs(v - n_elec);
        double dv = dev == dev ? dev : INFINITY;
        int best = i, ge = v >= n_elec ? i : P - 1;
        for (int o = 16; o > 0; o >>= 1) {  // smallest deviation, the first of equals
            const double od = __shfl_xor_sync(0xffffffffu, dv, o);
            const int ob = __shfl_xor_sync(0xffffffffu, best, o);
            if (od < dv || (od == dv && ob < best)) {
                dv = od;
                best = ob;
            }
        }
        ge = __reduce_min_sync(0xffffffffu, ge);
        if (lane == 0) {
            s_dv[i >> 5] = dv;
            s_best[i >> 5] = best;
            s_ge[i >> 5] = ge;
        }
    }
    __syncthreads();
    if (i != 0) return;
    st->ticket = 0u;
    st->bisect_rounds = round + 1;
    if (round == 0 && !(__ldcg(vc) <= n_elec && n_elec <= __ldcg(vc + P - 1))) {
        st->status = TB_ERR_BISECTION;
        st->bisect_done = 1;
        st->mu_x = 0.0;
        return;
    }
    double bd = s_dv[0];
    int best = s_best[0], first_ge = s_ge[0];
    for (int w = 1; w < 4; w++) {
        if (s_dv[w] < bd) {
            bd = s_dv[w];
            best = s_best[w];
        }
        first_ge = min(first_ge, s_ge[w]);
    }
    const double h = (hi - lo) / (double)(P - 1);
    if (bd <= tol_n) {
        st->mu_x = lo + h * best;
        st->bisect_done = 1;
        return;
    }
    const double nlo = (first_ge > 0) ? lo + h * (first_ge - 1) : lo;
    const double nhi = lo + h * first_ge;
    st->lo = nlo;
    st->hi = nhi;
    if (round == last_round) {
        st->mu_x = 0.5 * (nlo + nhi);
        st->bisect_done = 1;
    }
}

// Gaussian elimination with partial pivoting of the m x m normal equations
// A x = rhs (both overwritten) by one warp, x in gam, *solved = 0 where a
// pivot vanishes; m <= kMaxHistory, everything in shared memory.  The order of
// operations is that of the plain loops, which one thread runs in 25 us at
// m = 8 (dependent FP64 divisions and shared loads).
__device__ __forceinline__ void anderson_solve(double *A, double *rhs, double *gam, double *fac, int m, int *solved)
{
    const int lane = threadIdx.x & 31;
    int use = m > 0;
    if (lane < m) A[lane * m + lane] *= (1.0 + 1e-10);
    __syncwarp();
    for (int k = 0; k < m; k++) {
        int piv = k;
        for (int i = k + 1; i < m; i++)
            if (fabs(A[i * m + k]) > fabs(A[piv * m + k])) piv = i;
        if (!(fabs(A[piv * m + k]) > 1e-300)) {
            use = 0;
            break;
        }
        __syncwarp();
        if (piv != k) {
            double *x = lane < m ? A + k * m + lane : rhs + k, *y = lane < m ? A + piv * m + lane : rhs + piv;
            if (lane <= m) {
                const double t = *x;
                *x = *y;
                *y = t;
            }
        }
        __syncwarp();
        for (int i = k + 1 + lane; i < m; i += 32) fac[i] = A[i * m + k] / A[k * m + k];
        __syncwarp();
        const int cols = m - k + 1;  // columns k .. m - 1 and the right-hand side
        for (int e = lane; e < (m - k - 1) * cols; e += 32) {
            const int i = k + 1 + e / cols, j = k + e % cols;
            if (j < m)
                A[i * m + j] -= fac[i] * A[k * m + j];
            else
                rhs[i] -= fac[i] * rhs[k];
        }
        __syncwarp();
    }
    if (lane == 0) {
        if (use)
            for (int k = m - 1; k >= 0; k--) {
                double v = rhs[k];
                for (int j = k + 1; j < m; j++) v -= A[k * m + j] * gam[j];
                gam[k] = v / A[k * m + k];
            }
        *solved = use;
    }
}

}  // namespace tb
