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

#include "tb_chain.cuh"
#include "tb_fixed.cuh"
#include "tb_internal.h"

namespace tb {

namespace {

// X = (H0 + diag(shift) - b)/a (fx_scaled), a thread an entry.
__global__ void k_build_x_fixed(int64_t nnzb, const int32_t *__restrict__ blkrow, const int32_t *__restrict__ colidx,
                                const double *__restrict__ h0, const double *__restrict__ shift, double most,
                                DevState *st, int32_t *__restrict__ xfx, int64_t *__restrict__ xdfx)
{
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nnzb * 16) return;
    const int64_t t = e >> 4;
    const int r = (int)(e >> 2) & 3, c = (int)e & 3, I = blkrow[t];
    const bool diag = colidx[t] == I && r == c;
    const int64_t x = fx_scaled(h0[e], diag && shift ? shift[4 * I + r] : 0.0, diag, st, most);
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
// (tb_resident.cu), pinned slab widths and probe vectors: Tout = X Tin (first)
// or 2 X Tin - Tout, in place over T_{k-1}.
//
// A warp takes `rpw` consecutive block rows x 32 W columns, a lane W columns
// (W = 1 for up to 32 probes, so that fewer lanes are padding).  Its work is a
// stream of items of four rows: a row's referenced rows of T_k, then its old
// row of T_{k-1} and the row to multiply the new one with.  Every lane copies
// its own columns of the items kFxAhead ahead of their use into a ring of
// shared memory (cp.async: no registers, no barrier, nothing shared between
// lanes), and the row's blocks of X come coalesced a row ahead and are handed
// round through shared memory.  That leaves 48 W mad.wide a block and lane as
// the bound (3.75 clocks per 4x4 block and column of an SM); measured at 0.6
// of it.  The reference's logged DOS (18432 orbitals, 500 probes, 1000
// moments): 307 ms with the FP64 kernel, 70 with plain loads of T and X, 48.5
// now (50.6 with each step launched after the one before); 20 probes on 108000
// orbitals: 250 -> 24 ms.
//
// Column sums (kTrace, kMoments): <T_k,T_k> and <T_k,T_{k+1}> of every column,
// integers added up with atomics (low and high halves apart: probes have norms
// beyond one), the same in any order.  Row sums (kDensity): num_i += weight
// sum_t R_it (T_{k+1})_it, num one row per 32 W columns of the slab.
//
// Probes (kMoments, kDensity) start with entries of at most 1/4, and an entry
// beyond 1/2 raises *over: the call then starts again in FP64.  Up to there
// nothing leaves its range, whatever X's interval (rows of |X| below three):
// a new entry is below 2 * 3 / 2 + 1/2, and the middle sums of kFxChunk blocks
// stay below 24 * 2^59 / 2 + 3 * 2^59.  Entries of unit variance then come in
// steps of 2^-55: against an 80-bit run the density's error (rms over diagP, 20
// probes, M = 100 to 200, quartz cells of 324 to 675 atoms) is 1.7e-16 to
// 3.7e-16, the FP64 pass's 3.2e-16 to 5.8e-16.
enum FxMode { kTrace, kMoments, kDensity };
constexpr int kFxWarps = 8, kFxAhead = 3, kFxChunk = 6;  // kFxChunk: blocks of X handed round at once
constexpr int64_t kFxMost = kFxOne / 2;

template <int W>
__device__ __forceinline__ void fx_copy(int2 *dst, const int2 *src)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
    if (W == 2)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(src) : "memory");
}

template <int W>
constexpr size_t fx_smem()
{
    return (size_t)kFxWarps * (kFxAhead + 1) * 4 * 32 * W * sizeof(int2);
}

template <int W, int kMode>
__global__ void __launch_bounds__(32 * kFxWarps, 2)
    k_cheb_fixed(int nb, int n, int rpw, const int32_t *__restrict__ rowptr, const int32_t *__restrict__ colidx,
                 const int4 *__restrict__ xfx, const int2 *__restrict__ Tin, int2 *__restrict__ Tout, int B, int first,
                 unsigned long long *__restrict__ dsum, const int2 *__restrict__ R, const double *__restrict__ weight,
                 double *__restrict__ num, int32_t *__restrict__ over)
{
    constexpr bool kDens = kMode == kDensity;
    constexpr int CW = 32 * W;
    extern __shared__ __align__(16) int2 ring_all[];
    __shared__ int4 xs[kFxWarps][64];
    __shared__ unsigned long long red[kDens ? 1 : kFxWarps][4][CW];  // low halves of both sums, then high
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int Ia = min(nb, (blockIdx.x * kFxWarps + w) * rpw), Ib = min(nb, Ia + rpw);
    const int64_t col = (int64_t)blockIdx.y * CW + lane * W;
    int2 *ring = ring_all + (size_t)w * (kFxAhead + 1) * 4 * CW + lane * W;  // [slot][4 rows][CW]
    const int2 *with = kDens ? R : Tin;
    // the lane's own column sums stay in shared memory, for want of registers
    if (!kDens) {
#pragma unroll
        for (int v = 0; v < 4; v++)
#pragma unroll
            for (int c = 0; c < W; c++) red[w][v][lane * W + c] = 0;
    }
    chain_release();
    if (Ia < Ib) {
        // ---- the copies' side of the stream: item fb of row fI, its block row fJ known one item early ----
        int fI = Ia, fb = 0, ft = rowptr[Ia], fe = rowptr[Ia + 1], fslot = 0, fJ = colidx[ft];
        auto issue = [&]() {
            if (fI < Ib) {
                const int L = fe - ft;
                const int2 *src = (fb < L ? Tin : fb == L ? Tout : with) + (int64_t)(4 * fJ) * B + col;
                int2 *dst = ring + (size_t)fslot * 4 * CW;
#pragma unroll
                for (int m = 0; m < 4; m++) fx_copy<W>(dst + m * CW, src + (int64_t)m * B);
                if (++fb == L + 2) {
                    fb = 0;
                    fI++;
                    ft = fe;
                    if (fI < Ib) fe = __ldg(rowptr + fI + 1);
                }
                fJ = fI;
                if (fI < Ib && fb < fe - ft) fJ = __ldg(colidx + ft + fb);
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
            fslot = fslot == kFxAhead ? 0 : fslot + 1;
        };
        chain_wait();
#pragma unroll 1
        for (int i = 0; i < kFxAhead; i++) issue();
        int slot = 0;
        auto next = [&]() {  // the next item has landed; its slot
            asm volatile("cp.async.wait_group %0;\n" ::"n"(kFxAhead - 1) : "memory");
            const int2 *p = ring + (size_t)slot * 4 * CW;
            slot = slot == kFxAhead ? 0 : slot + 1;
            return p;
        };
        // ---- X: two 16-byte registers a lane hold the next kFxChunk blocks ----
        int4 xn[2];
        auto fetch = [&](int t, int te) {
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int e = lane + 32 * i, tt = t + e / 8;
                if (e < 8 * kFxChunk && tt < te) xn[i] = __ldg(xfx + (int64_t)tt * 8 + (e & 7));
            }
        };
        int t = rowptr[Ia], te = rowptr[Ia + 1];
        fetch(t, te);
#pragma unroll 1
        for (int I = Ia; I < Ib; I++) {
            const int tn = te, ten = I + 1 < Ib ? __ldg(rowptr + I + 2) : te;
            FxAcc acc[4][W];
#pragma unroll
            for (int q = 0; q < 4; q++)
#pragma unroll
                for (int c = 0; c < W; c++) acc[q][c] = FxAcc{0, 0};
#pragma unroll 1
            for (int t0 = t; t0 < te; t0 += kFxChunk) {
                __syncwarp();
                xs[w][lane] = xn[0];
                xs[w][lane + 32] = xn[1];
                __syncwarp();
                if (t0 + kFxChunk < te)
                    fetch(t0 + kFxChunk, te);
                else
                    fetch(tn, ten);
                const int nblk = min(kFxChunk, te - t0);
#pragma unroll 1
                for (int bk = 0; bk < nblk; bk++) {
                    const int2 *src = next();
                    int2 tv[4][W];
#pragma unroll
                    for (int m = 0; m < 4; m++) {
                        if (W == 2) {
                            const int4 v = *reinterpret_cast<const int4 *>(src + m * CW);
                            tv[m][0] = make_int2(v.x, v.y);
                            tv[m][W - 1] = make_int2(v.z, v.w);
                        } else {
                            tv[m][0] = src[m * CW];
                        }
                    }
                    issue();  // into the slot read before this one
                    const int4 *xb = &xs[w][bk * 8];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const int4 xh = xb[2 * q], xl = xb[2 * q + 1];
                        const int32_t h[4] = {xh.x, xh.y, xh.z, xh.w}, l[4] = {xl.x, xl.y, xl.z, xl.w};
#pragma unroll
                        for (int m = 0; m < 4; m++)
#pragma unroll
                            for (int c = 0; c < W; c++) fx_mul_add(acc[q][c], h[m], l[m], tv[m][c].x, tv[m][c].y);
                    }
                }
                if (t0 + kFxChunk < te) {
#pragma unroll
                    for (int q = 0; q < 4; q++)
#pragma unroll
                        for (int c = 0; c < W; c++) fx_flush(acc[q][c]);
                }
            }
            {
                const int2 *old = next();
                int2 *dst = Tout + (int64_t)(4 * I) * B + col;
                int2 o[4][W];
#pragma unroll
                for (int q = 0; q < 4; q++) {
#pragma unroll
                    for (int c = 0; c < W; c++) {
                        const int2 p = old[q * CW + c];
                        const int64_t v = first ? fx_sum(acc[q][c]) : fx_twice(acc[q][c]) - fx_join(p.x, p.y);
                        fx_split(v, o[q][c].x, o[q][c].y);
                        if (kMode != kTrace && (v > kFxMost || v < -kFxMost)) *over = 1;
                    }
                    if (W == 2)
                        *reinterpret_cast<int4 *>(dst + (int64_t)q * B) =
                            make_int4(o[q][0].x, o[q][0].y, o[q][W - 1].x, o[q][W - 1].y);
                    else
                        dst[(int64_t)q * B] = o[q][0];
                }
                issue();
                const int2 *own = next();
                if constexpr (kDens) {
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        int64_t row = 0;
#pragma unroll
                        for (int c = 0; c < W; c++) {
                            FxDots d;
                            const int2 p = own[q * CW + c];
                            d.add(p.x, p.y, o[q][c].x, o[q][c].y);
                            row += d.odd();
                        }
                        for (int s = 16; s > 0; s >>= 1) row += __shfl_xor_sync(0xffffffffu, (long long)row, s);
                        if (lane == q) num[(int64_t)blockIdx.y * n + 4 * I + q] += *weight * (double)row;
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < W; c++) {
                        FxDots d;
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const int2 p = own[q * CW + c];
                            d.add(p.x, p.y, o[q][c].x, o[q][c].y);
                        }
                        const int64_t e = d.even(), f = d.odd();
                        unsigned long long *r = &red[w][0][lane * W + c];
                        r[0] += (uint32_t)e;
                        r[CW] += (uint32_t)f;
                        r[2 * CW] += (unsigned long long)(e >> 32);
                        r[3 * CW] += (unsigned long long)(f >> 32);
                    }
                }
                issue();
            }
            t = tn;
            te = ten;
        }
    }
    if constexpr (!kDens) {
        __syncthreads();
        for (int e = threadIdx.x; e < 4 * CW; e += blockDim.x) {
            const int which = e / CW, j = e % CW;
            unsigned long long s = 0;
#pragma unroll
            for (int q = 0; q < kFxWarps; q++) s += red[q][which][j];
            atomicAdd(dsum + (int64_t)which * B + blockIdx.y * CW + j, s);
        }
    }
}

// The column sum of a step's dsum ([lo <T_k,T_k>][lo <T_k,T_{k+1}>][hi][hi], B each).
__device__ __forceinline__ __int128 fx_colsum(const unsigned long long *dk, int B, int which, int j)
{
    return (__int128)(int64_t)dk[(int64_t)which * B + j] + ((__int128)(int64_t)dk[(int64_t)(2 + which) * B + j] << 32);
}

// ---- probe vectors, scaled by 2^-shift so that every entry is at most 1/4 ----
__global__ void __launch_bounds__(256) k_fx_probe_max(const double *__restrict__ R, int64_t tot, uint32_t *__restrict__ most)
{
    float m = 0.f;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x)
        m = fmaxf(m, __double2float_ru(fabs(R[e])));
    const unsigned u = __reduce_max_sync(0xffffffffu, __float_as_uint(m));  // non-negative floats order as integers
    if ((threadIdx.x & 31) == 0) atomicMax(most, u);
}

// *most: the largest entry's bits in, the shift out
__global__ void k_fx_probe_shift(uint32_t *__restrict__ most)
{
    const float m = 4.f * __uint_as_float(*most);
    int s = 0;
    while (s < 40 && ldexpf(1.f, s) < m) s++;
    *most = (uint32_t)s;
}

__global__ void k_fx_probe_quantise(const double *__restrict__ R, int64_t tot, const int32_t *__restrict__ shift,
                                    int2 *__restrict__ T0, int2 *__restrict__ keep)
{
    const double sc = ldexp(1.0, kFxBits - *shift);
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
        int2 v;
        fx_split((int64_t)rint(R[e] * sc), v.x, v.y);
        T0[e] = v;
        if (keep) keep[e] = v;
    }
}

// mu_2k += sum_t 2 <T_k r,T_k r> - <r,r>, mu_{2k+1} += sum_t 2 <T_k r,T_{k+1} r> - <r,T_1 r>
// over the columns of one slab, in column order.
__global__ void k_fx_probe_moments(const unsigned long long *__restrict__ dsum, int B, int nr, int nmom,
                                   const int32_t *__restrict__ shift, double *__restrict__ mom)
{
    const int kk = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32, lane = threadIdx.x & 31;
    if (kk >= nmom) return;
    const int k = kk / 2, which = kk & 1;
    double s = 0.0;
    for (int t = lane; t < nr; t += 32)
        s += (double)(2 * fx_colsum(dsum + (int64_t)k * 4 * B, B, which, t) - fx_colsum(dsum, B, which, t));
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) mom[kk] += ldexp(s, 2 * *shift - kFxBits);
}

// den_i += sum_t R_it^2 over a slab and num_i += weight of that (the k = 0
// term), in units of 2^-60: every slab has a shift of its own, so its squares
// count 2^(2 shift) times what the fixed point holds.  A warp an orbital.
__global__ void k_fx_probe_den(const int2 *__restrict__ R, int n, int B, const int32_t *__restrict__ shift,
                               const double *__restrict__ weight, double *__restrict__ num, double *__restrict__ den)
{
    const int lane = threadIdx.x & 31;
    const int i = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (i >= n) return;
    int64_t part = 0;  // at most 32 squares of at most 1/16
    for (int t = lane; t < B; t += 32) {
        const int2 v = R[(int64_t)i * B + t];
        FxDots d;
        d.add(v.x, v.y, 0, 0);
        part += d.even();
    }
    double s = (double)part;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
        s = ldexp(s, 2 * *shift);
        num[i] += *weight * s;
        den[i] += s;
    }
}

// num_i += the slab's column groups' sums, in order and in k_fx_probe_den's
// units, and clears them
__global__ void k_fx_probe_num(double *__restrict__ part, int n, int groups, const int32_t *__restrict__ shift,
                               double *__restrict__ num)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double unit = ldexp(1.0, 2 * *shift);
    double s = num[i];
    for (int g = 0; g < groups; g++) {
        s += unit * part[(int64_t)g * n + i];
        part[(int64_t)g * n + i] = 0.0;
    }
    num[i] = s;
}

__global__ void k_fx_weights(const double *__restrict__ c, const double *__restrict__ g, int M, double *__restrict__ w)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < M) w[k] = c[k] * g[k];
}

// d[2k][j] = 2 <T_k,T_k>_j - 1 and d[2k+1][j] = 2 <T_k,T_{k+1}>_j - X_jj.
__global__ void k_fixed_finalize(const unsigned long long *__restrict__ dsum, int B, int c0, int n,
                                 const int64_t *__restrict__ xdfx, const DevState *__restrict__ st,
                                 double *__restrict__ d, int M)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y, i = c0 + j;
    if (j >= B || i >= n) return;
    const int64_t e = (int64_t)fx_colsum(dsum + (int64_t)k * 4 * B, B, 0, j),
                  o = (int64_t)fx_colsum(dsum + (int64_t)k * 4 * B, B, 1, j);
    const double bad = st->poison ? NAN : 0.0;
    if (2 * k <= M) d[(int64_t)(2 * k) * n + i] = (double)(2 * e - kFxOne) * (1.0 / kFxScale) + bad;
    if (2 * k + 1 <= M) d[(int64_t)(2 * k + 1) * n + i] = (double)(2 * o - xdfx[i]) * (1.0 / kFxScale) + bad;
}

}  // namespace

void launch_build_x_fixed(cudaStream_t st, const DevMatrix &m, const double *shift, DevState *state, double most)
{
    const int64_t tot = m.nnzb * 16;
    k_build_x_fixed<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(m.nnzb, m.blkrow, m.colidx, m.h0, shift, most, state,
                                                                  reinterpret_cast<int32_t *>(m.xfx), m.xdfx);
}

void launch_fixed_identity(cudaStream_t st, int2 *T0, int n, int B, int c0)
{
    const int64_t tot = (int64_t)n * B;
    k_fixed_identity<<<(int)std::min<int64_t>((tot + 255) / 256, 152 * 16), 256, 0, st>>>(T0, n, B, c0);
}

int fixed_probe_width(int nr) { return nr <= 32 ? 32 : (nr + 63) / 64 * 64; }

int fixed_groups(int B) { return B / (B % 64 ? 32 : 64); }

template <int W, int kMode>
static void launch_fixed_t(cudaStream_t st, const DevMatrix &m, const int2 *Tin, int2 *Tout, int B, int first,
                           unsigned long long *dsum, const int2 *R, const double *weight, double *num, int32_t *over)
{
    const auto fn = k_cheb_fixed<W, kMode>;
    // for the current device; a refusal shows as the launch's error
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fx_smem<W>());
    // Rows a warp: the count whose waves of CTAs (two an SM) take least, a
    // stream's start (its first index, copies and blocks of X come one after
    // the other) costing about 1.5 rows.  Two rows a warp took 59 us a step of
    // the reference's 4608-atom DOS.
    const int ny = B / (32 * W);
    int rpw = 1;
    double best = 1e300;
    for (int r = 1; r <= 32; r++) {
        const int64_t ctas = (int64_t)((m.nb + kFxWarps * r - 1) / (kFxWarps * r)) * ny;
        const double cost = (double)((ctas + 303) / 304) * (r + 1.5);
        if (cost < best) {
            best = cost;
            rpw = r;
        }
    }
    launch_chained(fn, dim3((m.nb + kFxWarps * rpw - 1) / (kFxWarps * rpw), ny), 32 * kFxWarps, fx_smem<W>(), st, m.nb,
                   m.n, rpw, m.rowptr, m.colidx, m.xfx, Tin, Tout, B, first, dsum, R, weight, num, over);
}

void launch_cheb_fixed(cudaStream_t st, const DevMatrix &m, const int2 *Tin, int2 *Tout, int B, int first,
                       unsigned long long *dsum, int32_t *over)
{
    if (over && B % 64)
        launch_fixed_t<1, kMoments>(st, m, Tin, Tout, B, first, dsum, nullptr, nullptr, nullptr, over);
    else if (over)
        launch_fixed_t<2, kMoments>(st, m, Tin, Tout, B, first, dsum, nullptr, nullptr, nullptr, over);
    else
        launch_fixed_t<2, kTrace>(st, m, Tin, Tout, B, first, dsum, nullptr, nullptr, nullptr, nullptr);
}

void launch_cheb_fixed_rows(cudaStream_t st, const DevMatrix &m, const int2 *Tin, int2 *Tout, int B, int first,
                            const int2 *R, const double *weight, double *part, int32_t *over)
{
    if (B % 64)
        launch_fixed_t<1, kDensity>(st, m, Tin, Tout, B, first, nullptr, R, weight, part, over);
    else
        launch_fixed_t<2, kDensity>(st, m, Tin, Tout, B, first, nullptr, R, weight, part, over);
}

void launch_fx_probe_num(cudaStream_t st, double *part, int n, int groups, const int32_t *shift, double *num)
{
    k_fx_probe_num<<<(n + 255) / 256, 256, 0, st>>>(part, n, groups, shift, num);
}

void launch_fx_probes(cudaStream_t st, const double *R, int n, int B, int32_t *shift, int2 *T0, int2 *keep)
{
    const int64_t tot = (int64_t)n * B;
    const int blocks = (int)std::min<int64_t>((tot + 255) / 256, 152 * 16);
    auto *bits = reinterpret_cast<uint32_t *>(shift);
    cudaMemsetAsync(shift, 0, sizeof(*shift), st);
    k_fx_probe_max<<<blocks, 256, 0, st>>>(R, tot, bits);
    k_fx_probe_shift<<<1, 1, 0, st>>>(bits);
    k_fx_probe_quantise<<<blocks, 256, 0, st>>>(R, tot, shift, T0, keep);
}

void launch_fx_probe_moments(cudaStream_t st, const unsigned long long *dsum, int B, int nr, int nmom,
                             const int32_t *shift, double *mom)
{
    k_fx_probe_moments<<<(nmom + 7) / 8, 256, 0, st>>>(dsum, B, nr, nmom, shift, mom);
}

void launch_fx_probe_den(cudaStream_t st, const int2 *R, int n, int B, const int32_t *shift, const double *weight,
                         double *num, double *den)
{
    k_fx_probe_den<<<(unsigned)(((int64_t)n * 32 + 255) / 256), 256, 0, st>>>(R, n, B, shift, weight, num, den);
}

void launch_fx_weights(cudaStream_t st, const double *c, const double *g, int M, double *w)
{
    k_fx_weights<<<(M + 127) / 128, 128, 0, st>>>(c, g, M, w);
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
    const int64_t cap = std::max<int64_t>(64, (int64_t)(80.0e6 / (16.0 * n)) / 64 * 64);
    const int ns = (int)((n64 + cap - 1) / cap);
    return ((n + ns - 1) / ns + 63) / 64 * 64;
}

}  // namespace tb
