// tb_fixed.cu -- the FP64 form's Chebyshev recurrence in 64-bit fixed point
// (tb_fixed.cuh) over identity column slabs: the recurrence of getKPE,
// withSP2_deltaH.cpp:1134-1168, with the moments from
//   T_{2k} = 2 T_k^2 - 1,  T_{2k+1} = 2 T_k T_{k+1} - X
// (column dot products), so M moments need (M + 2)/2 steps.
//
// Used whenever X is scaled by its own Gershgorin interval; a caller's own
// interval (tb_params.bounds_lo/hi) may not hold the spectrum, and T_k then
// grows past any fixed range: those calls keep the FP64 kernel k_cheb_f64.
//
// Against an 80-bit recurrence the moments d[k][i] have 2.3e-17 (rms, 2x2x2
// cell, M = 200), 2.1e-17 (1152 atoms, M = 300) and 2.5e-16 (1x1x1, M = 6000)
// where the FP64 recurrence has 2.8e-16, 8.4e-17 and 6.5e-15: X is formed to
// 2^-61 from the unrounded quotient, and the sums round once.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "tb_fixed.cuh"
#include "tb_internal.h"

namespace tb {

namespace {

// X = (H0 + diag(shift) - b)/a (fx_scaled), a thread an entry.
__global__ void k_build_x_fixed(int64_t nnzb, const int32_t *__restrict__ blkrow, const int32_t *__restrict__ colidx,
                                const double *__restrict__ h0, const double *__restrict__ shift, DevState *st,
                                int32_t *__restrict__ xfx, int64_t *__restrict__ xdfx)
{
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nnzb * 16) return;
    const int64_t t = e >> 4;
    const int r = (int)(e >> 2) & 3, c = (int)e & 3, I = blkrow[t];
    const bool diag = colidx[t] == I && r == c;
    const int64_t x = fx_scaled(h0[e], diag && shift ? shift[4 * I + r] : 0.0, diag, st);
    int32_t hi, lo;
    fx_split(x, hi, lo);
    xfx[t * 32 + 8 * r + c] = hi;
    xfx[t * 32 + 8 * r + 4 + c] = lo;
    if (diag) xdfx[4 * I + r] = x;
}

// Identity columns c0 .. c0+B-1, (hi, lo) pairs, row-major [n][B].
__global__ void k_fixed_identity(int2 *__restrict__ T0, int n, int B, int c0)
{
    const int64_t tot = (int64_t)n * B;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(e / B), j = (int)(e - (int64_t)i * B);
        T0[e] = make_int2(i == c0 + j ? 1 << kFxLimb : 0, 0);
    }
}

// One step on a slab, for matrices whose columns do not fit on chip
// (tb_resident.cu) and pinned slab widths: Tout = X Tin (first) or
// 2 X Tin - Tout, in place over T_{k-1}.  A warp takes kRPW consecutive block
// rows x 64 columns, a lane two columns: a block costs a lane four 16-byte
// loads of T (two (hi, lo) pairs each), eight broadcast 16-byte loads of X and
// 96 mad.wide, so the integer pipe is its floor (7 clocks per block row and
// column of an SM at 3.67 blocks a row).  Measured on a whole density of 1152
// atoms, M = 300: 236 (FP64 kernel) -> 42.9 ms: the warps wait for the next
// block's index and rows.  The columns' dot products are integers: they are
// added up with atomics in any order and come out the same.
constexpr int kFxWarps = 8;

template <int kRPW>
__global__ void __launch_bounds__(32 * kFxWarps, 2)
    k_cheb_fixed(int nb, const int32_t *__restrict__ rowptr, const int32_t *__restrict__ colidx,
                 const int4 *__restrict__ xfx, const int2 *__restrict__ Tin, int2 *__restrict__ Tout, int B, int first,
                 unsigned long long *__restrict__ dsum)
{
    __shared__ unsigned long long red[kFxWarps][2][64];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int col = blockIdx.y * 64 + lane * 2;
    const int I0 = (blockIdx.x * kFxWarps + w) * kRPW;
    FxDots dots[2];
#pragma unroll 1
    for (int rr = 0; rr < kRPW; rr++) {
        const int I = I0 + rr;
        if (I >= nb) break;
        FxAcc acc[4][2];
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int c = 0; c < 2; c++) acc[q][c] = FxAcc{0, 0};
        const int t0 = rowptr[I], t1 = rowptr[I + 1];
#pragma unroll 1
        for (int t = t0; t < t1; t++) {
            const int J = __ldg(colidx + t);
            int4 tv[4];
#pragma unroll
            for (int m = 0; m < 4; m++)
                tv[m] = __ldg(reinterpret_cast<const int4 *>(Tin + (int64_t)(4 * J + m) * B + col));
            const int4 *xb = xfx + (int64_t)t * 8;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int4 xh = __ldg(xb + 2 * q), xl = __ldg(xb + 2 * q + 1);
                const int32_t h[4] = {xh.x, xh.y, xh.z, xh.w}, l[4] = {xl.x, xl.y, xl.z, xl.w};
#pragma unroll
                for (int m = 0; m < 4; m++) {
                    fx_mul_add(acc[q][0], h[m], l[m], tv[m].x, tv[m].y);
                    fx_mul_add(acc[q][1], h[m], l[m], tv[m].z, tv[m].w);
                }
            }
            if (((t - t0) & (kFxFlush - 1)) == kFxFlush - 1) {
#pragma unroll
                for (int q = 0; q < 4; q++)
#pragma unroll
                    for (int c = 0; c < 2; c++) fx_flush(acc[q][c]);
            }
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int64_t at = (int64_t)(4 * I + q) * B + col;
            const int4 own = __ldg(reinterpret_cast<const int4 *>(Tin + at));
            int4 *dst = reinterpret_cast<int4 *>(Tout + at);
            int64_t o0, o1;
            if (first) {
                o0 = fx_sum(acc[q][0]);
                o1 = fx_sum(acc[q][1]);
            } else {
                const int4 p = *dst;
                o0 = fx_twice(acc[q][0]) - fx_join(p.x, p.y);
                o1 = fx_twice(acc[q][1]) - fx_join(p.z, p.w);
            }
            int4 o;
            fx_split(o0, o.x, o.y);
            fx_split(o1, o.z, o.w);
            *dst = o;
            dots[0].add(own.x, own.y, o.x, o.y);
            dots[1].add(own.z, own.w, o.z, o.w);
        }
    }
#pragma unroll
    for (int c = 0; c < 2; c++) {
        red[w][0][2 * lane + c] = (unsigned long long)dots[c].even();
        red[w][1][2 * lane + c] = (unsigned long long)dots[c].odd();
    }
    __syncthreads();
    if (threadIdx.x < 128) {
        const int which = threadIdx.x >> 6, j = threadIdx.x & 63;
        unsigned long long s = 0;
#pragma unroll
        for (int q = 0; q < kFxWarps; q++) s += red[q][which][j];
        atomicAdd(dsum + (int64_t)which * B + blockIdx.y * 64 + j, s);
    }
}

// d[2k][j] = 2 <T_k,T_k>_j - 1 and d[2k+1][j] = 2 <T_k,T_{k+1}>_j - X_jj.
__global__ void k_fixed_finalize(const unsigned long long *__restrict__ dsum, int B, int c0, int n,
                                 const int64_t *__restrict__ xdfx, const DevState *__restrict__ st,
                                 double *__restrict__ d, int M)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y, i = c0 + j;
    if (j >= B || i >= n) return;
    const int64_t e = (int64_t)dsum[(int64_t)(2 * k) * B + j], o = (int64_t)dsum[(int64_t)(2 * k + 1) * B + j];
    const double bad = st->poison ? NAN : 0.0;
    if (2 * k <= M) d[(int64_t)(2 * k) * n + i] = (double)(2 * e - kFxOne) * (1.0 / kFxScale) + bad;
    if (2 * k + 1 <= M) d[(int64_t)(2 * k + 1) * n + i] = (double)(2 * o - xdfx[i]) * (1.0 / kFxScale) + bad;
}

}  // namespace

void launch_build_x_fixed(cudaStream_t st, const DevMatrix &m, const double *shift, DevState *state)
{
    const int64_t tot = m.nnzb * 16;
    k_build_x_fixed<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(m.nnzb, m.blkrow, m.colidx, m.h0, shift, state,
                                                                  reinterpret_cast<int32_t *>(m.xfx), m.xdfx);
}

void launch_fixed_identity(cudaStream_t st, int2 *T0, int n, int B, int c0)
{
    const int64_t tot = (int64_t)n * B;
    k_fixed_identity<<<(int)std::min<int64_t>((tot + 255) / 256, 152 * 16), 256, 0, st>>>(T0, n, B, c0);
}

void launch_cheb_fixed(cudaStream_t st, const DevMatrix &m, const int2 *Tin, int2 *Tout, int B, int first,
                       unsigned long long *dsum)
{
    const dim3 blk(32 * kFxWarps);
    // several block rows a warp keep the column sums' atomics rare; one a warp
    // where the grid would not fill the device
    const int64_t wide = (int64_t)((m.nb + 4 * kFxWarps - 1) / (4 * kFxWarps)) * (B / 64);
    if (wide >= 2 * 152)
        k_cheb_fixed<4><<<dim3((m.nb + 4 * kFxWarps - 1) / (4 * kFxWarps), B / 64), blk, 0, st>>>(
            m.nb, m.rowptr, m.colidx, m.xfx, Tin, Tout, B, first, dsum);
    else
        k_cheb_fixed<1><<<dim3((m.nb + kFxWarps - 1) / kFxWarps, B / 64), blk, 0, st>>>(
            m.nb, m.rowptr, m.colidx, m.xfx, Tin, Tout, B, first, dsum);
}

void launch_fixed_finalize(cudaStream_t st, const DevMatrix &m, const unsigned long long *dsum, int K, int B, int c0,
                           const DevState *state, double *d, int M)
{
    k_fixed_finalize<<<dim3((B + 127) / 128, K), 128, 0, st>>>(dsum, B, c0, m.n, m.xdfx, state, d, M);
}

// Columns of a slab: both buffers (16 bytes an entry) stay in L2 together
// with X, in equal slabs.
int fixed_slab_width(int n)
{
    const int n64 = (n + 63) / 64 * 64;
    const int64_t cap = std::max<int64_t>(64, (int64_t)(72.0e6 / (16.0 * n)) / 64 * 64);
    const int ns = (int)((n64 + cap - 1) / cap);
    return ((n + ns - 1) / ns + 63) / 64 * 64;
}

}  // namespace tb
