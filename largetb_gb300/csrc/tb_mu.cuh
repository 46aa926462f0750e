// tb_mu.cuh -- end of a multisection round of the chemical potential (runKPM's
// mu search, withSP2_deltaH.cpp:1640-1712, on the electron count), shared by
// the single-structure and the batched kernels.
#pragma once

#include <cuda_runtime.h>

#include "tb_internal.h"

namespace tb {

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

}  // namespace tb
