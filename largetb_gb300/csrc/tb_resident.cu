// tb_resident.cu -- Chebyshev recurrence with the columns held on chip (K2 of
// the density-matrix path: the recurrence of getKPE, withSP2_deltaH.cpp:
// 1134-1168, over identity columns), in FP32 or in the FP64 form's 64-bit
// fixed point (tb_fixed.cuh).
//
// The columns of T_k(X) do not depend on one another, so one CTA takes a few
// of them through all K steps: T_k and T_{k-1} stay in shared memory, the only
// traffic per step is X (from L2, or L1 where it fits), a step ends with one
// CTA barrier instead of a launch, and no flag or neighbour is ever waited
// for.  Moments come from the column dot products, d[2k] = 2 <T_k,T_k> - 1 and
// d[2k+1] = 2 <T_k,T_{k+1}> - X_jj, written straight to d.
//
// Layout.  A unit is 16 bytes of one row: four FP32 columns or two fixed-point
// ones (hi, lo).  A buffer is [4 rows m of a block][position] units; a lane
// owns one unit of all four rows of a block row, so a block costs it four
// 16-byte shared loads and its 4x4 values (small structures in fixed point: of
// one row, res_split).  X is stored for 32 positions at a
// time, slot by slot (ELL; rows are ordered by their number of blocks, so
// padding is rare), [slot][row q][32 lanes] x 16 bytes: coalesced.  Block rows
// are further ordered so that the rows of one sublattice follow each other
// (plan_order): the neighbours that eight lanes read at once are then mostly
// at consecutive positions too, which is what keeps 16-byte shared loads free
// of bank conflicts.
//
// Bounds.  FP32: shared memory and L1, about 46 wavefronts of 128 bytes per 32
// blocks x 4 columns (16 for X, 16 for T, the row's own, old and new units);
// measured at 0.76 of that.  Fixed point: mad.wide (96 a block and lane), 0.75
// of its rate.  One density, before (one launch a step) and now: FP32, 768
// orbitals, M = 200: 0.80 -> 0.18 ms; 3456, M = 200: 2.97 -> 1.90; 5760, M = 300:
// 10.6 -> 8.0; 6144, M = 400: 15.9 -> 11.8.  Fixed point, 768 orbitals, M = 200:
// 1.15 -> 0.63 ms; 4608, M = 300: 42.6 -> 26.6.
//
// A block row's products run in column order and round as in the slab kernels
// (staged, pipelined): T_k is the same to the bit, only the column sums are
// added in another order.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <numeric>

#include "tb_f32x2.cuh"
#include "tb_fixed.cuh"
#include "tb_internal.h"

namespace tb {

namespace {

constexpr int kResMaxWarps = 16;
// Rows of a block that a lane takes: all four; one in fixed point where a
// structure has up to kResSplitChunks chunks, whose few warps would each carry
// a long chain (144 orbitals: 2.7 us a step with four rows a lane, 1.4 with
// one; 768 orbitals: 6.2 and 7.1, T being read four times).
constexpr int kResSplitChunks = 3;
__host__ __device__ constexpr int res_split(int nch, bool fx) { return fx && nch <= kResSplitChunks ? 4 : 1; }

__device__ __forceinline__ void pair_merge(float &h, float &l, float h2, float l2)
{
    pair_add(h, l, h2);
    l += l2;
}

template <bool kFx>
struct ResSums;  // a lane's column sums: 2 W values (W columns' <T_k,T_k>, then <T_k,T_{k+1}>)

template <>
struct ResSums<false> {
    static constexpr int W = 4, kVals = 8;
    typedef float2 Word;
    float2 h2[4], l2[4];  // <T_k,T_k> of columns 0-1, 2-3, then <T_k,T_{k+1}>, as (hi, lo) pairs
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int i = 0; i < 4; i++) h2[i] = l2[i] = make_float2(0.f, 0.f);
    }
    // sum over the warp, halving the values a lane carries while there are
    // several; returns the lane's value index
    __device__ __forceinline__ int reduce(int lane)
    {
        float h[8], l[8];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            h[2 * i] = h2[i].x;
            h[2 * i + 1] = h2[i].y;
            l[2 * i] = l2[i].x;
            l[2 * i + 1] = l2[i].y;
        }
        int v = 0;
#pragma unroll
        for (int s = 0; s < 3; s++) {
            const int off = 16 >> s, half = 4 >> s;
            const bool up = lane & off;
#pragma unroll
            for (int i = 0; i < half; i++) {
                const float sh = up ? h[i] : h[i + half], sl = up ? l[i] : l[i + half];
                const float rh = __shfl_xor_sync(0xffffffffu, sh, off), rl = __shfl_xor_sync(0xffffffffu, sl, off);
                h[i] = up ? h[i + half] : h[i];
                l[i] = up ? l[i + half] : l[i];
                pair_merge(h[i], l[i], rh, rl);
            }
            v += up ? half : 0;
        }
#pragma unroll
        for (int off = 2; off > 0; off >>= 1) {
            const float rh = __shfl_xor_sync(0xffffffffu, h[0], off), rl = __shfl_xor_sync(0xffffffffu, l[0], off);
            pair_merge(h[0], l[0], rh, rl);
        }
        h2[0].x = h[0];
        l2[0].x = l[0];
        return v;
    }
    static __device__ __forceinline__ bool writes(int lane) { return (lane & 3) == 0; }
    __device__ __forceinline__ Word word() const { return make_float2(h2[0].x, l2[0].x); }
    // over the warps' words, by one warp: lanes 8 apart share a value
    static __device__ __forceinline__ double total(const Word *w, int lane, int nw)
    {
        float hs = 0.f, ls = 0.f;
        for (int i = lane / kVals; i < nw; i += 32 / kVals) {
            const Word v = w[i * kVals + lane % kVals];
            pair_merge(hs, ls, v.x, v.y);
        }
        for (int o = kVals; o < 32; o <<= 1) {
            const float rh = __shfl_down_sync(0xffffffffu, hs, o), rl = __shfl_down_sync(0xffffffffu, ls, o);
            pair_merge(hs, ls, rh, rl);
        }
        return (double)hs + (double)ls;
    }
};

template <>
struct ResSums<true> {
    static constexpr int W = 2, kVals = 4;
    typedef long long Word;
    int64_t s[4];
    __device__ __forceinline__ void clear() { s[0] = s[1] = s[2] = s[3] = 0; }
    __device__ __forceinline__ int reduce(int lane)
    {
        int v = 0;
#pragma unroll
        for (int st = 0; st < 2; st++) {
            const int off = 16 >> st, half = 2 >> st;
            const bool up = lane & off;
#pragma unroll
            for (int i = 0; i < half; i++) {
                const int64_t snd = up ? s[i] : s[i + half];
                const int64_t rcv = __shfl_xor_sync(0xffffffffu, (long long)snd, off);
                s[i] = (up ? s[i + half] : s[i]) + rcv;
            }
            v += up ? half : 0;
        }
#pragma unroll
        for (int off = 4; off > 0; off >>= 1) s[0] += __shfl_xor_sync(0xffffffffu, (long long)s[0], off);
        return v;
    }
    static __device__ __forceinline__ bool writes(int lane) { return (lane & 7) == 0; }
    __device__ __forceinline__ Word word() const { return s[0]; }
    // the 64-bit integer, in a double's bits
    static __device__ __forceinline__ double total(const Word *w, int lane, int nw)
    {
        int64_t t = 0;
        for (int i = lane / kVals; i < nw; i += 32 / kVals) t += w[i * kVals + lane % kVals];
        for (int o = kVals; o < 32; o <<= 1) t += __shfl_xor_sync(0xffffffffu, (long long)t, o);
        return __longlong_as_double(t);
    }
};

// One CTA: the W columns from c0 on of one structure through all K steps.  A
// warp takes the chunks of 32 block rows that the plan gave it (they are
// numbered warp by warp, so that its slots form one stream of memory: each
// row of X is fetched one slot ahead, into the registers just used, with
// nothing but a pointer increment), a lane one block row at a time.
template <bool kFx, int kSplit>
__global__ void __launch_bounds__(32 * kResMaxWarps, 1)
    k_cheb_resident(const ResJob *__restrict__ jobs, const int2 *__restrict__ tasks, int K, int M)
{
    extern __shared__ __align__(16) uint4 smem[];
    typedef ResSums<kFx> Sums;
    constexpr int W = Sums::W, kVals = Sums::kVals, kQ = kFx ? 8 : 4;  // kQ: 16-byte rows of X a slot
    constexpr int QS = 4 / kSplit, kX = kQ / kSplit;
    const int2 task = tasks ? tasks[blockIdx.x] : make_int2(0, (int)blockIdx.x);
    const ResJob jb = jobs[task.x];
    if (jb.active && !*jb.active) return;
    const int c0 = task.y * W, n = jb.n, plane = jb.nch * 32;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nt = blockDim.x;
    const int nw = min(nt >> 5, jb.nw * kSplit);  // warps past the structure's own idle
    const int q0 = w % kSplit * QS;               // this warp's rows of a block
    uint4 *cur = smem, *prv = smem + 4 * plane;
    typename Sums::Word *red = reinterpret_cast<typename Sums::Word *>(smem + 8 * plane);  // [2][warps][kVals]
    for (int i = tid; i < 8 * plane; i += nt) smem[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    if (tid < W && c0 + tid < n) {  // T_0: the identity's columns
        const int col = c0 + tid, u = (col & 3) * plane + jb.posof[col >> 2];
        if (kFx)
            reinterpret_cast<int2 *>(cur + u)[tid] = make_int2(1 << kFxLimb, 0);
        else
            reinterpret_cast<float *>(cur + u)[tid] = 1.f;
    }
    __syncthreads();
    const int ch0 = w < nw ? __ldg(jb.wchunk + w / kSplit) : 0, ch1 = w < nw ? __ldg(jb.wchunk + w / kSplit + 1) : 0;
    const int sb0 = ch1 > ch0 ? __ldg(jb.sbase + ch0) : 0;
    for (int k = 0; k < K; k++) {
        Sums sums;
        sums.clear();
        const uint4 *xp = reinterpret_cast<const uint4 *>(jb.x) + (int64_t)sb0 * kQ * 32 + w % kSplit * kX * 32 + lane;
        const int32_t *cp = jb.colpos + sb0 * 32 + lane;
        uint4 xr[kX];
        int j = 0, sb = sb0;
        if (ch1 > ch0) {
            j = __ldg(cp);
#pragma unroll
            for (int q = 0; q < kX; q++) xr[q] = __ldg(xp + q * 32);
        }
        for (int ch = ch0; ch < ch1; ch++) {
            const int L = __ldg(jb.sbase + ch + 1) - sb;
            sb += L;
            const int u = ch * 32 + lane;
            if constexpr (kFx) {
                FxAcc fa[QS][2];
#pragma unroll
                for (int q = 0; q < QS; q++) fa[q][0] = fa[q][1] = FxAcc{0, 0};
#pragma unroll 1
                for (int s = 0; s < L; s++) {
                    uint4 v[4];
#pragma unroll
                    for (int m = 0; m < 4; m++) v[m] = cur[m * plane + j];
                    cp += 32;
                    xp += kQ * 32;
                    j = __ldg(cp);
#pragma unroll
                    for (int q = 0; q < QS; q++) {
                        const uint32_t h[4] = {xr[2 * q].x, xr[2 * q].y, xr[2 * q].z, xr[2 * q].w},
                                       l[4] = {xr[2 * q + 1].x, xr[2 * q + 1].y, xr[2 * q + 1].z, xr[2 * q + 1].w};
#pragma unroll
                        for (int m = 0; m < 4; m++) {
                            fx_mul_add(fa[q][0], (int)h[m], (int)l[m], (int)v[m].x, (int)v[m].y);
                            fx_mul_add(fa[q][1], (int)h[m], (int)l[m], (int)v[m].z, (int)v[m].w);
                        }
                        xr[2 * q] = __ldg(xp + 2 * q * 32);
                        xr[2 * q + 1] = __ldg(xp + (2 * q + 1) * 32);
                    }
                    if ((s & (kFxFlush - 1)) == kFxFlush - 1) {
#pragma unroll
                        for (int q = 0; q < QS; q++) {
                            fx_flush(fa[q][0]);
                            fx_flush(fa[q][1]);
                        }
                    }
                }
                FxDots dots[2];
#pragma unroll
                for (int q = 0; q < QS; q++) {
                    const int at = (q0 + q) * plane + u;
                    const uint4 own = cur[at], old = prv[at];
                    int64_t o0, o1;
                    if (k == 0) {
                        o0 = fx_sum(fa[q][0]);
                        o1 = fx_sum(fa[q][1]);
                    } else {
                        o0 = fx_twice(fa[q][0]) - fx_join((int)old.x, (int)old.y);
                        o1 = fx_twice(fa[q][1]) - fx_join((int)old.z, (int)old.w);
                    }
                    int32_t h0, l0, h1, l1;
                    fx_split(o0, h0, l0);
                    fx_split(o1, h1, l1);
                    prv[at] = make_uint4(h0, l0, h1, l1);
                    dots[0].add((int)own.x, (int)own.y, h0, l0);
                    dots[1].add((int)own.z, (int)own.w, h1, l1);
                }
                sums.s[0] += dots[0].even();
                sums.s[1] += dots[1].even();
                sums.s[2] += dots[0].odd();
                sums.s[3] += dots[1].odd();
            } else {
                float acc[4][4];
#pragma unroll
                for (int q = 0; q < 4; q++) acc[q][0] = acc[q][1] = acc[q][2] = acc[q][3] = 0.f;
#pragma unroll 1
                for (int s = 0; s < L; s++) {
                    uint4 v[4];
#pragma unroll
                    for (int m = 0; m < 4; m++) v[m] = cur[m * plane + j];
                    cp += 32;
                    xp += kQ * 32;
                    j = __ldg(cp);
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const float xm[4] = {__uint_as_float(xr[q].x), __uint_as_float(xr[q].y),
                                             __uint_as_float(xr[q].z), __uint_as_float(xr[q].w)};
#pragma unroll
                        for (int m = 0; m < 4; m++) {
                            acc[q][0] = fmaf(xm[m], __uint_as_float(v[m].x), acc[q][0]);
                            acc[q][1] = fmaf(xm[m], __uint_as_float(v[m].y), acc[q][1]);
                            acc[q][2] = fmaf(xm[m], __uint_as_float(v[m].z), acc[q][2]);
                            acc[q][3] = fmaf(xm[m], __uint_as_float(v[m].w), acc[q][3]);
                        }
                        xr[q] = __ldg(xp + q * 32);
                    }
                }
                float2 ee[2], eo[2];
                ee[0] = ee[1] = eo[0] = eo[1] = make_float2(0.f, 0.f);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int at = q * plane + u;
                    float2 nv[2] = {make_float2(acc[q][0], acc[q][1]), make_float2(acc[q][2], acc[q][3])};
                    if (k > 0) {
                        const float4 old = reinterpret_cast<const float4 *>(prv)[at];
                        nv[0] = cheb_next2(nv[0], make_float2(old.x, old.y));
                        nv[1] = cheb_next2(nv[1], make_float2(old.z, old.w));
                    }
                    reinterpret_cast<float4 *>(prv)[at] = make_float4(nv[0].x, nv[0].y, nv[1].x, nv[1].y);
                    const float4 own = reinterpret_cast<const float4 *>(cur)[at];
                    const float2 ov[2] = {make_float2(own.x, own.y), make_float2(own.z, own.w)};
#pragma unroll
                    for (int c = 0; c < 2; c++) {
                        ee[c] = __ffma2_rn(ov[c], ov[c], ee[c]);
                        eo[c] = __ffma2_rn(ov[c], nv[c], eo[c]);
                    }
                }
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    pair_add2(sums.h2[c], sums.l2[c], ee[c]);
                    pair_add2(sums.h2[2 + c], sums.l2[2 + c], eo[c]);
                }
            }
        }
        // ---- the step's column sums: over the warp, then (after the barrier) over the warps ----
        typename Sums::Word *rk = red + (k & 1) * kResMaxWarps * kVals;
        if (w < nw) {
            const int v = sums.reduce(lane);
            if (Sums::writes(lane)) rk[w * kVals + v] = sums.word();
        }
        __syncthreads();  // T_{k+1} and the warps' sums are complete
        if (w == k % (nt >> 5)) {  // the warps in turn: 32 / kVals lanes a value
            const int vi = lane % kVals, which = vi / W, col = c0 + vi % W, kk = 2 * k + which;
            const double total = Sums::total(rk, lane, nw);
            if (lane < kVals && col < n && kk <= M) {
                double *dst = jb.d + (int64_t)kk * jb.dstride + col;
                if constexpr (kFx) {
                    const int64_t less = which ? reinterpret_cast<const int64_t *>(jb.xdiag)[col] : kFxOne;
                    *dst = (double)(2 * __double_as_longlong(total) - less) * (1.0 / kFxScale) +
                           (jb.st->poison ? NAN : 0.0);
                } else {
                    *dst = 2.0 * total - (which ? (double)reinterpret_cast<const float *>(jb.xdiag)[col] : 1.0);
                }
            }
        }
        uint4 *t = cur;
        cur = prv;
        prv = t;
    }
}

// X = (H0 + diag(shift) - b)/a straight into the ELL layout, a thread an
// entry, slots of every structure concatenated; padding is zero.
template <bool kFx>
__global__ void k_build_x_ell(const ResJob *__restrict__ jobs, const int32_t *__restrict__ slotjob,
                              const int32_t *__restrict__ src, int64_t nent, const int32_t *__restrict__ blkrow,
                              const int32_t *__restrict__ colidx, const double *__restrict__ h0,
                              const double *__restrict__ shift, void *__restrict__ xe, void *__restrict__ xdiag)
{
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;  // ((slot 4 + q) 32 + lane) 4 + c
    if (e >= nent) return;
    const int64_t slot = e >> 9;
    const int q = (int)(e >> 7) & 3, ln = (int)(e >> 2) & 31, c = (int)e & 3;
    const ResJob &jb = jobs[slotjob ? slotjob[slot] : 0];
    if (jb.active && !*jb.active) return;
    const int t = src[slot * 32 + ln];
    double v = 0.0, s0 = 0.0;
    bool diag = false;
    int I = 0;
    DevState *st = jb.st;
    if (t >= 0) {
        I = blkrow[t];
        v = h0[(int64_t)t * 16 + q * 4 + c];
        diag = colidx[t] == I && q == c;
        if (diag && shift) s0 = shift[4 * I + q];
    }
    if constexpr (kFx) {
        const int64_t x = t >= 0 ? fx_scaled(v, s0, diag, st) : 0;
        int32_t hi, lo;
        fx_split(x, hi, lo);
        int32_t *d = reinterpret_cast<int32_t *>(xe) + ((slot * 8 + 2 * q) * 32 + ln) * 4 + c;
        d[0] = hi;
        d[128] = lo;
        if (diag) reinterpret_cast<int64_t *>(xdiag)[4 * I + q] = x;
    } else {
        if (t >= 0) v = (diag ? v + s0 - st->b : v) / st->a;
        reinterpret_cast<float *>(xe)[e] = (float)v;
        if (diag) reinterpret_cast<float *>(xdiag)[4 * I + q] = (float)v;
    }
}

// Order of the block rows: by their number of blocks, most first, then (if the
// pattern repeats after `per` rows, as a lattice given cell by cell does: row
// I + per references the columns of row I plus per) sublattice by sublattice.
void plan_order(int nb, const int32_t *brow, const int32_t *bcol, std::vector<int32_t> &order)
{
    int per = 1, best = 0;
    for (int p = 1; p <= std::min(64, nb - 1); p++) {
        int same = 0;
        for (int I = 0; I + p < nb; I++) {
            const int L = brow[I + 1] - brow[I];
            if (brow[I + p + 1] - brow[I + p] != L) continue;
            const int32_t *x = bcol + brow[I], *y = bcol + brow[I + p];
            int s = 0;
            while (s < L && y[s] == x[s] + p) s++;
            same += s == L;
        }
        if (same > best && 4 * same >= nb) {
            best = same;
            per = p;
        }
    }
    order.resize(nb);
    std::iota(order.begin(), order.end(), 0);
    std::sort(order.begin(), order.end(), [&](int a, int b) {
        const int la = brow[a + 1] - brow[a], lb = brow[b + 1] - brow[b];
        if (la != lb) return la > lb;
        if (a % per != b % per) return a % per < b % per;
        return a < b;
    });
}

template <bool kFx, int kSplit>
int configure()
{
    return (int)cudaFuncSetAttribute(k_cheb_resident<kFx, kSplit>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     smem_optin_max((const void *)k_cheb_resident<kFx, kSplit>));
}

}  // namespace

void resident_plan_rows(int nb, const int32_t *brow, const int32_t *bcol, int64_t blk0, int warps, ResPlanHost &out)
{
    std::vector<int32_t> order;
    plan_order(nb, brow, bcol, order);
    const int nch = (nb + 31) / 32;
    // chunks (32 rows of the order, the first the longest) to warps, longest
    // first to the warp with the least; then numbered warp by warp
    const int nw = std::min(warps, nch);
    std::vector<int> load(nw, 0), len(nch), warp_of(nch);
    for (int c = 0; c < nch; c++) len[c] = brow[order[c * 32] + 1] - brow[order[c * 32]];
    for (int c = 0; c < nch; c++) {
        const int w = (int)(std::min_element(load.begin(), load.end()) - load.begin());
        warp_of[c] = w;
        load[w] += len[c] + 1;  // a row's end costs about one more block
    }
    std::vector<int> chunk_at;
    for (int w = 0; w < nw; w++) {
        out.wchunk.push_back((int32_t)chunk_at.size());
        for (int c = 0; c < nch; c++)
            if (warp_of[c] == w) chunk_at.push_back(c);
    }
    out.wchunk.push_back(nch);
    const size_t p0 = out.posof.size(), e0 = out.colpos.size();
    out.posof.resize(p0 + nb);
    int slots = 0;
    for (int ch = 0; ch < nch; ch++) {
        out.sbase.push_back(slots);
        slots += len[chunk_at[ch]];
        for (int ln = 0; ln < 32 && chunk_at[ch] * 32 + ln < nb; ln++)
            out.posof[p0 + order[chunk_at[ch] * 32 + ln]] = ch * 32 + ln;
    }
    out.sbase.push_back(slots);
    // one slot more than used: the stream is read one slot ahead
    out.colpos.resize(e0 + (size_t)(slots + 1) * 32, 0);
    out.src.resize(e0 + (size_t)(slots + 1) * 32, -1);
    size_t at = e0;
    for (int ch = 0; ch < nch; ch++) {
        const int c = chunk_at[ch];
        for (int s = 0; s < len[c]; s++)
            for (int ln = 0; ln < 32; ln++, at++) {
                const int p = c * 32 + ln, I = p < nb ? order[p] : -1, L = I >= 0 ? brow[I + 1] - brow[I] : 0;
                out.colpos[at] = ch * 32 + ln;
                if (s >= L) continue;
                out.colpos[at] = out.posof[p0 + bcol[brow[I] + s]];
                out.src[at] = (int32_t)(blk0 + brow[I] + s);
            }
    }
    out.nch = nch;
    out.nw = nw;
    out.slots = slots + 1;
}

size_t resident_smem(int nch, bool fx)
{
    return (size_t)8 * nch * 32 * 16 + (size_t)2 * kResMaxWarps * (fx ? 4 : 8) * 8;
}

bool resident_fits(int nb, bool fx)
{
    return resident_smem((nb + 31) / 32, fx) <= 227 * 1024 &&
           (fx ? configure<true, 1>() : configure<false, 1>()) == (int)cudaSuccess &&
           (!fx || configure<true, 4>() == (int)cudaSuccess);
}

int resident_columns(bool fx) { return fx ? 2 : 4; }

// Warps of the plan (lists of chunks, each walked by res_split warps): an SM's
// register file holds kResMaxWarps warps, shared between the CTAs that its
// shared memory and the launch have for it.
int resident_warps(int nb, bool fx)
{
    const int nch = (nb + 31) / 32, cols = resident_columns(fx), split = res_split(nch, fx);
    const int fit = (int)(227 * 1024 / resident_smem(nch, fx)), want = ((4 * nb + cols - 1) / cols + 151) / 152;
    return std::max(1, kResMaxWarps / split / std::max(1, std::min(fit, want)));
}

void launch_build_x_ell(cudaStream_t st, const ResPlan &rp, bool fx, const int32_t *blkrow, const int32_t *colidx,
                        const double *h0, const double *shift)
{
    const int64_t nent = rp.slots * 512;
    const unsigned grid = (unsigned)((nent + 255) / 256);
    if (fx)
        k_build_x_ell<true><<<grid, 256, 0, st>>>(rp.jobs, rp.slotjob, rp.src, nent, blkrow, colidx, h0, shift, rp.x,
                                                 rp.xdiag);
    else
        k_build_x_ell<false><<<grid, 256, 0, st>>>(rp.jobs, rp.slotjob, rp.src, nent, blkrow, colidx, h0, shift, rp.x,
                                                  rp.xdiag);
}

void launch_cheb_resident(cudaStream_t st, const ResJob *jobs, const int2 *tasks, int ntasks, int max_nch, int warps,
                          bool fx, int K, int M)
{
    const size_t smem = resident_smem(max_nch, fx);
    const int split = res_split(max_nch, fx);
    if (!fx)
        k_cheb_resident<false, 1><<<ntasks, 32 * warps, smem, st>>>(jobs, tasks, K, M);
    else if (split == 1)
        k_cheb_resident<true, 1><<<ntasks, 32 * warps, smem, st>>>(jobs, tasks, K, M);
    else
        k_cheb_resident<true, 4><<<ntasks, 32 * warps * split, smem, st>>>(jobs, tasks, K, M);
}

}  // namespace tb
