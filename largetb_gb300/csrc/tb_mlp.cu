// tb_mlp.cu -- learned SCC starting charges: per-atom radial features and a
// small MLP (32 -> 64 -> 64 -> 1, SiLU), trained and evaluated on the GPU by
// these kernels.  No counterpart in the reference, which always starts its
// SCC loop from the neutral charges (withSP2_deltaH.cpp:1725-1740, 1804-1812).
//
// Features of atom i: 16 Gaussians exp(-eta (r_ij - mu_k)^2) f_c(r_ij) summed
// over Si neighbours j, then 16 over O neighbours, mu_k = 0.8 + 0.28 k A,
// eta = 12.5 A^-2, f_c(r) = (cos(pi r / 5 A) + 1)/2 inside 5 A, minimum image
// in an orthorhombic box.
//
// Network: y = w3 . silu(W2 silu(W1 x~ + b1) + b2) + b3 with
// x~ = (x - mean) * istd (feature normalisation fixed from the first
// training set).  Weights are used in BF16 (a round-to-nearest-even copy of
// FP32 master weights), activations and accumulation in FP32; training is
// minibatch Adam on the mean squared error.  Each CTA takes tiles of 64 atoms
// with the weights (transposed where a warp reads along output units) in
// shared memory; weight gradients accumulate in registers across tiles and
// are added to global memory once per CTA.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <new>
#include <numeric>
#include <string>
#include <vector>

#include "tb_cells.cuh"
#include "tb_internal.h"

namespace tb {
namespace {

constexpr int kF = TB_MLP_NFEAT;  // 32
constexpr int kH = 64;
constexpr int kW1 = 0, kB1 = kW1 + kH * kF, kW2 = kB1 + kH, kB2 = kW2 + kH * kH, kW3 = kB2 + kH,
              kB3 = kW3 + kH, kNP = kB3 + 1;
static_assert(kNP == TB_MLP_NPARAM, "parameter layout");
constexpr int kTile = 64;
constexpr double kBohrPerAng = 1.88973;

__device__ __forceinline__ float sigm(float z) { return 1.f / (1.f + __expf(-z)); }

// ---- features --------------------------------------------------------------
__constant__ double c_gauss[16] = {1, 0.37531109885139957, 0.019841094744370288, 0.00014774836023203364, 1.5497531357028967e-07, 2.289734845645553e-11, 4.7653047352990878e-16, 1.3969439431471091e-21, 5.7683299612478847e-28, 3.3550888562311458e-35, 2.7487850079102147e-43, 3.1721983574449558e-52, 5.1565913268420381e-62, 1.1807226845823849e-72, 3.8081663925605564e-84, 1.7300822096825899e-96};  // e^{-12.5 (0.28 k)^2}

// The pair (i, j) in FP64: its 16 Gaussians times the cutoff, in FP32, or false
// beyond the cutoff.  e^{-12.5 (r - mu_k)^2} = e^{-12.5 x^2} (e^{7 x})^k
// e^{-0.98 k^2} with x = r - 0.8: two exponentials a pair instead of sixteen;
// the powers stay within 1e-98 .. 1e193 up to the cutoff, 1e-13 off.
__device__ __forceinline__ bool pair_features(const double *__restrict__ xyz, int i, int j, const double box[3],
                                              const double inv[3], float v[16])
{
    double r2 = 0.0;
#pragma unroll
    for (int q = 0; q < 3; q++) {
        double t = xyz[3 * j + q] - xyz[3 * i + q];
        if (box[q] > 0) t -= box[q] * rint(t * inv[q]);
        r2 = fma(t, t, r2);
    }
    const double rc = 5.0 * kBohrPerAng;
    if (r2 >= rc * rc) return false;
    const double r = sqrt(r2) * (1.0 / kBohrPerAng), x = r - 0.8;  // angstrom
    const double fc = 0.5 * (cospi(r * 0.2) + 1.0), a = exp(7.0 * x);
    double t = exp(-12.5 * x * x) * fc;
#pragma unroll
    for (int k = 0; k < 16; k++) {
        v[k] = (float)(t * c_gauss[k]);
        t *= a;
    }
    return true;
}

// FP32 prefilter of the pair distance (minimum image by a multiply with the
// inverse box), with a 1 % margin on rc^2 that covers its rounding; a NaN passes.
__device__ __forceinline__ bool pair_near(const float4 p, const float fi[3], const float fbox[3], const float finv[3])
{
    const float t0[3] = {p.x - fi[0], p.y - fi[1], p.z - fi[2]};
    float r2 = 0.f;
#pragma unroll
    for (int q = 0; q < 3; q++) {
        const float t = t0[q] - fbox[q] * rintf(t0[q] * finv[q]);
        r2 = fmaf(t, t, r2);
    }
    return !(r2 >= (float)(25.0 * kBohrPerAng * kBohrPerAng * 1.01));
}

// Eight lanes an atom (atoms in cell order): they gather the near atoms of the
// cells around it into a list, sort it, and evaluate eight pairs at a time, so
// that the FP64 work -- the bound -- runs on full groups.  Lane l sums features
// 4 l .. 4 l + 3 over the pairs in ascending order of j (the order in which a
// walk over all atoms meets them).  An atom with more than kFeatList near ones
// walks all atoms.  12288 atoms: 6.64 ms with every thread looking at every
// atom and 16 exponentials a pair, 0.25 ms now.
constexpr int kFeatLanes = 8, kFeatList = 128, kFeatThreads = 128, kFeatGroups = kFeatThreads / kFeatLanes;

__global__ void __launch_bounds__(kFeatThreads)
    k_features(int natoms, const double *__restrict__ xyz, const int32_t *__restrict__ sp, const CellGrid g,
               float *__restrict__ feat)
{
    __shared__ int32_t found[kFeatGroups][kFeatList], sorted[kFeatGroups][kFeatList];
    __shared__ __align__(16) float val[kFeatGroups][kFeatLanes][16];
    const int grp = threadIdx.x / kFeatLanes, l = threadIdx.x % kFeatLanes, lane = threadIdx.x & 31;
    const unsigned mask = 0xffu << (lane & 24);
    const int at = blockIdx.x * kFeatGroups + grp;
    if (at >= natoms) return;  // whole groups
    const int i = g.atom[at];
    const double x[3] = {xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]};
    double inv[3];
    float fi[3], fbox[3], finv[3];
#pragma unroll
    for (int q = 0; q < 3; q++) {
        inv[q] = g.box[q] > 0 ? 1.0 / g.box[q] : 0.0;
        fi[q] = (float)x[q];
        fbox[q] = (float)g.box[q];
        finv[q] = (float)inv[q];
    }
    float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
    auto evaluate = [&](const int32_t *list, int n) {
        __syncwarp(mask);
        for (int h0 = 0; h0 < n; h0 += kFeatLanes) {
            int kind = -1;  // 0: Si, 1: O
            if (h0 + l < n) {
                const int j = list[h0 + l];
                float v[16];
                if (pair_features(xyz, i, j, g.box, inv, v)) {
                    kind = sp[j] == 14 ? 0 : 1;
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        reinterpret_cast<float4 *>(val[grp][l])[k] =
                            make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
                }
            }
            __syncwarp(mask);
#pragma unroll
            for (int h = 0; h < kFeatLanes; h++) {
                const int kd = __shfl_sync(mask, kind, h, kFeatLanes);
                if (kd != (l >> 2)) continue;
                const float4 v = reinterpret_cast<const float4 *>(val[grp][h])[l & 3];
                f.x += v.x;
                f.y += v.y;
                f.z += v.z;
                f.w += v.w;
            }
            __syncwarp(mask);
        }
    };
    // candidate j (or i itself: none) of each lane into the list, n in all
    auto add = [&](int n, int j) {
        const unsigned hit = __ballot_sync(mask, j != i) >> (lane & 24);
        const int to = n + __popc(hit & ((1u << l) - 1u));
        if (j != i && to < kFeatList) found[grp][to] = j;
        return n + __popc(hit);
    };
    int n = 0;
    cell_around(g, x, [&](int s, int e) {
        for (int b = s; b < e; b += kFeatLanes) {
            int j = i;
            if (b + l < e && pair_near(g.pos[b + l], fi, fbox, finv)) j = g.atom[b + l];
            n = add(n, j);
        }
    });
    __syncwarp();  // the groups together again
    if (n <= kFeatList) {
        for (int h = l; h < n; h += kFeatLanes) {
            const int j = found[grp][h];
            int to = 0;
            for (int k = 0; k < n; k++) to += found[grp][k] < j;
            sorted[grp][to] = j;
        }
        evaluate(sorted[grp], n);
    } else {
        n = 0;
        for (int b = 0; b < natoms; b += kFeatLanes) {
            int j = i;
            if (b + l < natoms) {
                const float4 p = make_float4((float)xyz[3 * (b + l)], (float)xyz[3 * (b + l) + 1],
                                             (float)xyz[3 * (b + l) + 2], 0.f);
                if (pair_near(p, fi, fbox, finv)) j = b + l;
            }
            n = add(n, j);
            if (n > kFeatList - kFeatLanes) {
                evaluate(found[grp], n);
                n = 0;
            }
        }
        evaluate(found[grp], n);
    }
    reinterpret_cast<float4 *>(feat + (int64_t)i * kF)[l] = f;
}

// ---- forward / backward over tiles of 64 atoms ---------------------------------
constexpr int kSX = kF + 4, kSH = kH + 4;  // row strides: 16-byte rows, two rows 4 apart on different banks
constexpr size_t kFbSmem = sizeof(float) * (kF * kH + 2 * kH * kH + 3 * kH + 2 * kF + kTile * kSX + 2 * kTile * kSH);

// Gradients are added up in kCopies copies, by blockIdx.x, and the losses
// beside them: chains of some 40 additions instead of 300, which keeps the FP32
// error of the sum below that of the products (131072 samples: 5.8e-7 with one
// copy, 7.4e-8 with eight).
constexpr int kCopies = 8, kGStride = (kNP + 3) / 4 * 4;

__device__ __forceinline__ float copies_sum(const float *g, int stride)
{
    static_assert(kCopies == 8, "pairwise");
    return ((g[0] + g[stride]) + (g[2 * stride] + g[3 * stride])) +
           ((g[4 * stride] + g[5 * stride]) + (g[6 * stride] + g[7 * stride]));
}

// sum: the gradient, then the loss
__global__ void k_grad_sum(const float *__restrict__ g, const float *__restrict__ loss, float *__restrict__ sum)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kNP) sum[i] = copies_sum(g + i, kGStride);
    if (i == kNP) sum[i] = copies_sum(loss, 1);
}

// acc[r][c] += sum_k A[a0 + r][k] B[k][u0 + c], k ascending; A and B in shared
// memory with rows of SA and kH floats.
template <int K, int SA>
__device__ __forceinline__ void tile_product(float (&acc)[4][4], const float *A, const float *B)
{
#pragma unroll 4
    for (int k = 0; k < K; k += 4) {
        float4 x[4];
#pragma unroll
        for (int r = 0; r < 4; r++) x[r] = *reinterpret_cast<const float4 *>(A + r * SA + k);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float4 w = *reinterpret_cast<const float4 *>(B + (k + j) * kH);
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const float v = j == 0 ? x[r].x : j == 1 ? x[r].y : j == 2 ? x[r].z : x[r].w;
                acc[r][0] = fmaf(w.x, v, acc[r][0]);
                acc[r][1] = fmaf(w.y, v, acc[r][1]);
                acc[r][2] = fmaf(w.z, v, acc[r][2]);
                acc[r][3] = fmaf(w.w, v, acc[r][3]);
            }
        }
    }
}

// Wq: BF16-rounded parameters (FP32 storage).  idx (optional) maps sample
// positions to rows of X / target.  With target == nullptr only the forward
// pass runs and y goes to out.
//
// FP32 products on the CUDA cores (gradients hold 32 bits): 1 M of them a tile.
// A thread takes 4 atoms x 4 units of each layer, and 4 x 4 (4 x 2) entries of
// the weight gradients, so that two 16-byte shared loads feed 16 products (one
// product a load pair: 65536 samples 267 us; now 84 us, 0.40 of the FP32
// rate, bound by shared-memory loads); activations and their derivatives stay in its registers between the
// passes.  W2 is kept in both orders: two CTAs an SM.
__global__ void __launch_bounds__(256, 2)
    k_mlp_fb(int n, const int32_t *__restrict__ idx, const float *__restrict__ X,
             const float *__restrict__ mean, const float *__restrict__ istd, const float *__restrict__ Wq,
             const float *__restrict__ target, float inv_n, float *__restrict__ out,
             float *__restrict__ grad, float *__restrict__ loss)
{
    extern __shared__ __align__(16) float ms[];
    float *W1T = ms;                 // [i][u]   32 x 64
    float *W2T = W1T + kF * kH;      // [v][u]   64 x 64 (u = output unit)
    float *W2 = W2T + kH * kH;       // [u][v]
    float *b1 = W2 + kH * kH;
    float *b2 = b1 + kH;
    float *w3 = b2 + kH;
    float *nm = w3 + kH;             // mean, istd
    float *Xs = nm + 2 * kF;         // [a][i]
    float *H1 = Xs + kTile * kSX;    // [a][u], then dZ1
    float *G = H1 + kTile * kSH;     // [a][u]: dZ2
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, u0 = 4 * tx, a0 = 4 * ty;
    // a lane reads 16 bytes of its unit's row: no bank conflicts in the transposed stores
    for (int e = tid; e < kH * kF / 4; e += 256) {
        const int u = e % kH, i = e / kH * 4;
        const float4 x = *reinterpret_cast<const float4 *>(Wq + kW1 + u * kF + i);
        const float xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int j = 0; j < 4; j++) W1T[(i + j) * kH + u] = xv[j];
    }
    for (int e = tid; e < kH * kH / 4; e += 256) {
        const int u = e % kH, v = e / kH * 4;
        const float4 x = *reinterpret_cast<const float4 *>(Wq + kW2 + u * kH + v);
        const float xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int j = 0; j < 4; j++) W2T[(v + j) * kH + u] = xv[j];
    }
    for (int e = tid; e < kH * kH; e += 256) W2[e] = Wq[kW2 + e];
    if (tid < kH) {
        b1[tid] = Wq[kB1 + tid];
        b2[tid] = Wq[kB2 + tid];
        w3[tid] = Wq[kW3 + tid];
    } else if (tid < kH + kF) {
        nm[tid - kH] = mean[tid - kH];
        nm[tid - kH + kF] = istd[tid - kH];
    }
    const float b3 = Wq[kB3];
    const bool bwd = target != nullptr;
    float gW2[4][4] = {}, gW1[4][2] = {}, gb1[4] = {}, gb2[4] = {}, gw3[4] = {}, gb3 = 0.f, lsum = 0.f;
    __syncthreads();
    for (int tile = blockIdx.x; tile * kTile < n; tile += gridDim.x) {
        const int base = tile * kTile;
        for (int e = tid; e < kTile * kF / 4; e += 256) {
            const int a = e / (kF / 4), i = e % (kF / 4) * 4, s = base + a;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (s < n) {
                const int64_t row = idx ? idx[s] : s;
                v = __ldg(reinterpret_cast<const float4 *>(X + row * kF + i));
                v.x = (v.x - nm[i]) * nm[kF + i];
                v.y = (v.y - nm[i + 1]) * nm[kF + i + 1];
                v.z = (v.z - nm[i + 2]) * nm[kF + i + 2];
                v.w = (v.w - nm[i + 3]) * nm[kF + i + 3];
            }
            *reinterpret_cast<float4 *>(Xs + a * kSX + i) = v;
        }
        __syncthreads();
        // layer 1: z, silu(z) to shared memory, silu'(z) kept
        float z[4][4], d1[4][4];
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) z[r][c] = b1[u0 + c];
        tile_product<kF, kSX>(z, Xs + a0 * kSX, W1T + u0);
#pragma unroll
        for (int r = 0; r < 4; r++) {
            float h[4];
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const float sg = sigm(z[r][c]);
                h[c] = z[r][c] * sg;
                d1[r][c] = sg * (1.f + z[r][c] * (1.f - sg));
            }
            *reinterpret_cast<float4 *>(H1 + (a0 + r) * kSH + u0) = make_float4(h[0], h[1], h[2], h[3]);
        }
        __syncthreads();
        // layer 2 and output: the 16 threads of an atom add up w3 . silu(z)
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) z[r][c] = b2[u0 + c];
        tile_product<kH, kSH>(z, H1 + a0 * kSH, W2T + u0);
#pragma unroll
        for (int r = 0; r < 4; r++) {
            float h[4], sg[4], y = 0.f;
#pragma unroll
            for (int c = 0; c < 4; c++) {
                sg[c] = sigm(z[r][c]);
                h[c] = z[r][c] * sg[c];
                y = fmaf(w3[u0 + c], h[c], y);
            }
            for (int o = 8; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
            y += b3;
            const int s = base + a0 + r;
            if (out && tx == 0 && s < n) out[s] = y;
            if (!bwd) continue;
            float g = 0.f;
            if (s < n) {
                const float err = y - target[idx ? idx[s] : s];
                g = 2.f * err * inv_n;
                if (tx == 0) {
                    lsum += err * err * inv_n;
                    gb3 += g;
                }
            }
#pragma unroll
            for (int c = 0; c < 4; c++) {
                gw3[c] = fmaf(g, h[c], gw3[c]);
                z[r][c] = g * w3[u0 + c] * sg[c] * (1.f + z[r][c] * (1.f - sg[c]));
                gb2[c] += z[r][c];
            }
            *reinterpret_cast<float4 *>(G + (a0 + r) * kSH + u0) = make_float4(z[r][0], z[r][1], z[r][2], z[r][3]);
        }
        if (!bwd) continue;
        __syncthreads();
        // dZ1 of the thread's atoms and units of layer 1, dW2 of its units
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) z[r][c] = 0.f;
        tile_product<kH, kSH>(z, G + a0 * kSH, W2 + u0);
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) {
                z[r][c] *= d1[r][c];
                gb1[c] += z[r][c];
            }
#pragma unroll 4
        for (int a = 0; a < kTile; a++) {
            const float4 d = *reinterpret_cast<const float4 *>(G + a * kSH + u0);
            const float4 h = *reinterpret_cast<const float4 *>(H1 + a * kSH + a0);
            const float dv[4] = {d.x, d.y, d.z, d.w}, hv[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
            for (int c = 0; c < 4; c++)
#pragma unroll
                for (int j = 0; j < 4; j++) gW2[c][j] = fmaf(dv[c], hv[j], gW2[c][j]);
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 4; r++)
            *reinterpret_cast<float4 *>(H1 + (a0 + r) * kSH + u0) = make_float4(z[r][0], z[r][1], z[r][2], z[r][3]);
        __syncthreads();
#pragma unroll 4
        for (int a = 0; a < kTile; a++) {
            const float4 d = *reinterpret_cast<const float4 *>(H1 + a * kSH + u0);
            const float2 x = *reinterpret_cast<const float2 *>(Xs + a * kSX + 2 * ty);
            const float dv[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
            for (int c = 0; c < 4; c++) {
                gW1[c][0] = fmaf(dv[c], x.x, gW1[c][0]);
                gW1[c][1] = fmaf(dv[c], x.y, gW1[c][1]);
            }
        }
        __syncthreads();
    }
    if (!bwd) return;
    grad += blockIdx.x % kCopies * kGStride;
    loss += blockIdx.x % kCopies;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        atomicAdd(reinterpret_cast<float4 *>(grad + kW2 + (u0 + c) * kH + a0),
                  make_float4(gW2[c][0], gW2[c][1], gW2[c][2], gW2[c][3]));
        atomicAdd(reinterpret_cast<float2 *>(grad + kW1 + (u0 + c) * kF + 2 * ty), make_float2(gW1[c][0], gW1[c][1]));
    }
    // the units' sums over the atoms: two halves of a warp, then the warps
    const int lane = tid & 31, w = tid >> 5;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const float v[3] = {gb1[c], gb2[c], gw3[c]};
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const float t = v[q] + __shfl_xor_sync(0xffffffffu, v[q], 16);
            if (lane < 16) Xs[(q * 8 + w) * kH + u0 + c] = t;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
        gb3 += __shfl_xor_sync(0xffffffffu, gb3, o);
    }
    if (lane == 0) {
        Xs[24 * kH + w] = lsum;
        Xs[24 * kH + 8 + w] = gb3;
    }
    __syncthreads();
    if (tid < 3 * kH) {
        const int q = tid / kH, u = tid % kH;
        float t = 0.f;
        for (int i = 0; i < 8; i++) t += Xs[(q * 8 + i) * kH + u];
        atomicAdd(grad + (q == 0 ? kB1 : q == 1 ? kB2 : kW3) + u, t);
    } else if (tid < 3 * kH + 2) {  // one addition a CTA: the loss is a long sum
        const float *x = Xs + 24 * kH + 8 * (tid - 3 * kH);
        float t = 0.f;
        for (int i = 0; i < 8; i++) t += x[i];
        atomicAdd(tid == 3 * kH ? loss : grad + kB3, t);
    }
}
static_assert(24 * kH + 16 <= kTile * kSX, "the units' sums fit where the features were");
static_assert(kW1 % 4 == 0 && kW2 % 4 == 0, "16-byte loads and atomics");

// Adam on the FP32 master weights, then the BF16 working copy.
__global__ void k_adam(int np, float *__restrict__ W, float *__restrict__ Wq, float *__restrict__ m1,
                       float *__restrict__ m2, const float *__restrict__ g, float lr, float c1, float c2)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= np) return;
    const float gi = copies_sum(g + i, kGStride);
    const float a = 0.9f * m1[i] + 0.1f * gi, b = 0.999f * m2[i] + 0.001f * gi * gi;
    m1[i] = a;
    m2[i] = b;
    const float w = W[i] - lr * (a * c1) / (sqrtf(b * c2) + 1e-8f);
    W[i] = w;
    Wq[i] = __bfloat162float(__float2bfloat16_rn(w));
}

__global__ void k_round_bf16(int np, const float *__restrict__ W, float *__restrict__ Wq)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < np) Wq[i] = __bfloat162float(__float2bfloat16_rn(W[i]));
}

uint64_t mix64(uint64_t z)
{
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

}  // namespace
}  // namespace tb

using namespace tb;

struct tb_mlp {
    int device = 0;
    cudaStream_t stream = nullptr;
    float *W = nullptr, *Wq = nullptr, *m1 = nullptr, *m2 = nullptr;
    float *g = nullptr, *loss = nullptr, *sum = nullptr;  // kCopies gradients, kCopies losses, their sums (kNP + 1)
    float *mean = nullptr, *istd = nullptr;
    int32_t *err = nullptr;  // bounded-wait flag of the tensor-core forward
    bool have_norm = false;
    int64_t step = 0;
    // every call on the handle holds `mu` from its first look at the members to
    // its last: weights, gradients and device space are one set for all threads
    mutable std::mutex mu;
    // device space of one grad or predict call and its pinned results: a
    // cudaMalloc and cudaFree of 8 MB take 90 us, as long as the copy into it
    char *work = nullptr;
    size_t work_bytes = 0;
    float *host = nullptr;  // kNP + 1 floats
    cudaStream_t copy = nullptr;
    cudaEvent_t copied = nullptr;
};

namespace {

int mlp_alloc(tb_mlp *m)
{
    if (cudaMalloc(&m->W, sizeof(float) * kNP) || cudaMalloc(&m->Wq, sizeof(float) * kNP) ||
        cudaMalloc(&m->m1, sizeof(float) * kNP) || cudaMalloc(&m->m2, sizeof(float) * kNP) ||
        cudaMalloc(&m->g, sizeof(float) * (kCopies * (kGStride + 1) + kNP + 1)) || cudaMallocHost(&m->host, sizeof(float) * (kNP + 1)) ||
        cudaMalloc(&m->mean, sizeof(float) * kF) || cudaMalloc(&m->istd, sizeof(float) * kF) ||
        cudaMalloc(&m->err, sizeof(int32_t)) || cudaMemset(m->err, 0, sizeof(int32_t)))
        return TB_ERR_OUT_OF_MEMORY;
    m->loss = m->g + kCopies * kGStride;
    m->sum = m->loss + kCopies;
    return TB_OK;
}

// The handle's device space, at least `bytes`; up to kWorkKept stays with the
// handle until it is destroyed, more goes back at the end of the call.
constexpr size_t kWorkKept = 64u << 20;

struct MlpWork {
    tb_mlp *m;
    std::lock_guard<std::mutex> lock;
    explicit MlpWork(tb_mlp *m_) : m(m_), lock(m_->mu) {}
    int reserve(size_t bytes)
    {
        if (m->work_bytes >= bytes) return TB_OK;
        cudaFree(m->work);
        m->work = nullptr;
        m->work_bytes = 0;
        if (cudaMalloc(&m->work, bytes)) {
            cudaGetLastError();
            return TB_ERR_OUT_OF_MEMORY;
        }
        m->work_bytes = bytes;
        return TB_OK;
    }
    ~MlpWork()
    {
        if (m->work_bytes <= kWorkKept) return;
        cudaFree(m->work);
        m->work = nullptr;
        m->work_bytes = 0;
    }
};

// Upload features (and targets) and launch(s0, count) on them.  Beyond two
// chunks the upload of one runs beside the kernel on the one before (65536
// samples: 64 us to copy, 84 us of kernel).
constexpr int kChunk = 32768;

template <class F>
void in_chunks(tb_mlp *m, int n, const float *feat, const float *target, float *dX, float *dT, F launch)
{
    const int step = n >= 2 * kChunk ? kChunk : n;
    cudaStream_t up = step < n ? m->copy : m->stream;
    for (int64_t s0 = 0; s0 < n; s0 += step) {
        const int c = (int)std::min<int64_t>(step, n - s0);
        cudaMemcpyAsync(dX + s0 * kF, feat + s0 * kF, sizeof(float) * (size_t)c * kF, cudaMemcpyHostToDevice, up);
        if (target) cudaMemcpyAsync(dT + s0, target + s0, sizeof(float) * c, cudaMemcpyHostToDevice, up);
        if (up != m->stream) {
            cudaEventRecord(m->copied, up);
            cudaStreamWaitEvent(m->stream, m->copied, 0);
        }
        launch(s0, c);
    }
}

// Upload host features (and targets); returns device pointers owned by the caller.
int upload_set(cudaStream_t st, int n, const float *feat, const float *target, float **dX, float **dT)
{
    *dX = nullptr;
    if (dT) *dT = nullptr;
    if (cudaMalloc(dX, sizeof(float) * (size_t)n * kF)) return TB_ERR_OUT_OF_MEMORY;
    cudaMemcpyAsync(*dX, feat, sizeof(float) * (size_t)n * kF, cudaMemcpyHostToDevice, st);
    if (dT && target) {
        if (cudaMalloc(dT, sizeof(float) * n)) return TB_ERR_OUT_OF_MEMORY;
        cudaMemcpyAsync(*dT, target, sizeof(float) * n, cudaMemcpyHostToDevice, st);
    }
    return TB_OK;
}

// Sets weights and normalisation; the handle's lock is held.
int mlp_set(tb_mlp *m, const float *params, const float *norm)
{
    if (params) {
        for (int i = 0; i < kNP; i++)
            if (!std::isfinite(params[i])) return TB_ERR_NONFINITE;
        cudaMemcpy(m->W, params, sizeof(float) * kNP, cudaMemcpyHostToDevice);
        k_round_bf16<<<(kNP + 255) / 256, 256, 0, m->stream>>>(kNP, m->W, m->Wq);
    }
    if (norm) {
        cudaMemcpy(m->mean, norm, sizeof(float) * kF, cudaMemcpyHostToDevice);
        cudaMemcpy(m->istd, norm + kF, sizeof(float) * kF, cudaMemcpyHostToDevice);
        m->have_norm = true;
    }
    return cudaStreamSynchronize(m->stream) == cudaSuccess ? TB_OK : TB_ERR_CUDA;
}

int fb_grid(int n)
{
    const int tiles = (n + kTile - 1) / kTile;
    return std::max(1, std::min(tiles, 152 * 2));
}

}  // namespace

extern "C" {

int tb_mlp_features(int32_t natoms, const double *xyz, const int32_t *species, const double *box, float *feat)
{
    TB_ABI_TRY
    if (natoms <= 0 || !xyz || !species || !box || !feat) return TB_ERR_INVALID_ARG;
    CellGrid g;
    cell_grid(natoms, xyz, box, 5.0 * kBohrPerAng, g);
    // one allocation: features, positions, cells, species
    const size_t fb = sizeof(float) * (size_t)natoms * kF, xb = (sizeof(double) * 3 * natoms + 15) / 16 * 16,
                 cb = (cell_bytes(natoms, g) + 15) / 16 * 16;
    char *mem = nullptr;
    if (cudaMalloc(&mem, fb + xb + cb + sizeof(int32_t) * natoms)) {
        cudaGetLastError();
        return TB_ERR_OUT_OF_MEMORY;
    }
    float *df = reinterpret_cast<float *>(mem);
    double *dx = reinterpret_cast<double *>(mem + fb);
    int32_t *ds = reinterpret_cast<int32_t *>(mem + fb + xb + cb);
    cudaMemcpy(dx, xyz, sizeof(double) * 3 * natoms, cudaMemcpyHostToDevice);
    cudaMemcpy(ds, species, sizeof(int32_t) * natoms, cudaMemcpyHostToDevice);
    cell_build(0, natoms, dx, ds, g, mem + fb + xb);
    k_features<<<(natoms + kFeatGroups - 1) / kFeatGroups, kFeatThreads>>>(natoms, dx, ds, g, df);
    const int rc = cudaMemcpy(feat, df, fb, cudaMemcpyDeviceToHost) == cudaSuccess ? TB_OK : TB_ERR_CUDA;
    cudaFree(mem);
    return rc;
    TB_ABI_CATCH
}

int tb_mlp_create(int32_t device, uint64_t seed, tb_mlp **out)
{
    TB_ABI_TRY
    if (!out) return TB_ERR_INVALID_ARG;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
        cudaGetLastError();
        return TB_ERR_NO_DEVICE;
    }
    tb_mlp *m = new (std::nothrow) tb_mlp();
    if (!m) return TB_ERR_OUT_OF_MEMORY;
    m->device = device;
    cudaSetDevice(device);
    if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaStreamCreateWithFlags(&m->copy, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreateWithFlags(&m->copied, cudaEventDisableTiming) != cudaSuccess || mlp_alloc(m)) {
        tb_mlp_destroy(m);
        return TB_ERR_CUDA;
    }
    // He-style uniform initialisation from splitmix64, zero biases
    std::vector<float> w(kNP, 0.f);
    uint64_t k = 0;
    auto uni = [&](double lim) {
        const double u = (double)(mix64(seed + (++k) * 0x9E3779B97F4A7C15ull) >> 11) / 9007199254740992.0;
        return (float)((2.0 * u - 1.0) * lim);
    };
    for (int i = 0; i < kH * kF; i++) w[kW1 + i] = uni(std::sqrt(6.0 / kF));
    for (int i = 0; i < kH * kH; i++) w[kW2 + i] = uni(std::sqrt(6.0 / kH));
    for (int i = 0; i < kH; i++) w[kW3 + i] = uni(std::sqrt(3.0 / kH));
    std::vector<float> zero(kNP, 0.f), mean(kF, 0.f), one(kF, 1.f);
    cudaMemcpy(m->W, w.data(), sizeof(float) * kNP, cudaMemcpyHostToDevice);
    cudaMemcpy(m->m1, zero.data(), sizeof(float) * kNP, cudaMemcpyHostToDevice);
    cudaMemcpy(m->m2, zero.data(), sizeof(float) * kNP, cudaMemcpyHostToDevice);
    cudaMemcpy(m->mean, mean.data(), sizeof(float) * kF, cudaMemcpyHostToDevice);
    cudaMemcpy(m->istd, one.data(), sizeof(float) * kF, cudaMemcpyHostToDevice);
    k_round_bf16<<<(kNP + 255) / 256, 256, 0, m->stream>>>(kNP, m->W, m->Wq);
    if (cudaFuncSetAttribute(k_mlp_fb, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFbSmem) != cudaSuccess ||
        cudaStreamSynchronize(m->stream) != cudaSuccess) {
        tb_mlp_destroy(m);
        return TB_ERR_CUDA;
    }
    *out = m;
    return TB_OK;
    TB_ABI_CATCH
}

int tb_mlp_destroy(tb_mlp *m)
{
    TB_ABI_TRY
    if (!m) return TB_OK;
    cudaSetDevice(m->device);
    if (m->stream) cudaStreamSynchronize(m->stream);
    cudaFree(m->W);
    cudaFree(m->Wq);
    cudaFree(m->m1);
    cudaFree(m->m2);
    cudaFree(m->g);
    cudaFree(m->work);
    cudaFreeHost(m->host);
    if (m->copied) cudaEventDestroy(m->copied);
    if (m->copy) cudaStreamDestroy(m->copy);
    cudaFree(m->mean);
    cudaFree(m->istd);
    cudaFree(m->err);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
    return TB_OK;
    TB_ABI_CATCH
}

int tb_mlp_get(const tb_mlp *m, float *params, float *norm)
{
    TB_ABI_TRY
    if (!m) return TB_ERR_INVALID_ARG;
    cudaSetDevice(m->device);
    std::lock_guard<std::mutex> lock(m->mu);
    if (params && cudaMemcpy(params, m->W, sizeof(float) * kNP, cudaMemcpyDeviceToHost)) return TB_ERR_CUDA;
    if (norm && (cudaMemcpy(norm, m->mean, sizeof(float) * kF, cudaMemcpyDeviceToHost) ||
                 cudaMemcpy(norm + kF, m->istd, sizeof(float) * kF, cudaMemcpyDeviceToHost)))
        return TB_ERR_CUDA;
    return TB_OK;
    TB_ABI_CATCH
}

int tb_mlp_set(tb_mlp *m, const float *params, const float *norm)
{
    TB_ABI_TRY
    if (!m) return TB_ERR_INVALID_ARG;
    cudaSetDevice(m->device);
    std::lock_guard<std::mutex> lock(m->mu);
    return mlp_set(m, params, norm);
    TB_ABI_CATCH
}

int tb_mlp_grad(tb_mlp *m, int32_t n, const float *feat, const float *target, float *grad, float *loss)
{
    TB_ABI_TRY
    if (!m || n <= 0 || !feat || !target || !grad) return TB_ERR_INVALID_ARG;
    cudaSetDevice(m->device);
    MlpWork work(m);
    int rc = work.reserve(sizeof(float) * (size_t)n * (kF + 1));
    if (rc == TB_OK) {
        float *dX = reinterpret_cast<float *>(m->work), *dT = dX + (size_t)n * kF;
        cudaMemsetAsync(m->g, 0, sizeof(float) * kCopies * (kGStride + 1), m->stream);
        in_chunks(m, n, feat, target, dX, dT, [&](int64_t s0, int c) {
            k_mlp_fb<<<fb_grid(c), 256, kFbSmem, m->stream>>>(c, nullptr, dX + s0 * kF, m->mean, m->istd, m->Wq, dT + s0,
                                                              1.f / n, nullptr, m->g, m->loss);
        });
        k_grad_sum<<<(kNP + 256) / 256, 256, 0, m->stream>>>(m->g, m->loss, m->sum);
        cudaMemcpyAsync(m->host, m->sum, sizeof(float) * (kNP + 1), cudaMemcpyDeviceToHost, m->stream);
        if (cudaStreamSynchronize(m->stream) != cudaSuccess || cudaGetLastError() != cudaSuccess) rc = TB_ERR_CUDA;
        if (rc == TB_OK) {
            std::memcpy(grad, m->host, sizeof(float) * kNP);
            if (loss) *loss = m->host[kNP];
        }
    }
    return rc;
    TB_ABI_CATCH
}

int tb_mlp_predict(tb_mlp *m, int32_t n, const float *feat, float *out)
{
    TB_ABI_TRY
    if (!m || n <= 0 || !feat || !out) return TB_ERR_INVALID_ARG;
    cudaSetDevice(m->device);
    MlpWork work(m);
    int rc = work.reserve(sizeof(float) * (size_t)n * (kF + 1));
    if (rc == TB_OK) {
        float *dX = reinterpret_cast<float *>(m->work), *dY = dX + (size_t)n * kF;
        in_chunks(m, n, feat, nullptr, dX, nullptr, [&](int64_t s0, int c) {
            launch_mlp_forward_tc(m->stream, c, dX + s0 * kF, m->mean, m->istd, m->Wq, dY + s0, m->err);
        });
        cudaMemcpyAsync(out, dY, sizeof(float) * n, cudaMemcpyDeviceToHost, m->stream);
        cudaMemcpyAsync(m->host, m->err, sizeof(int32_t), cudaMemcpyDeviceToHost, m->stream);
        if (cudaStreamSynchronize(m->stream) != cudaSuccess || cudaGetLastError() != cudaSuccess) rc = TB_ERR_CUDA;
        if (rc == TB_OK && *reinterpret_cast<int32_t *>(m->host)) {
            cudaMemsetAsync(m->err, 0, sizeof(int32_t), m->stream);
            rc = TB_ERR_CUDA;
        }
    }
    return rc;
    TB_ABI_CATCH
}

int tb_mlp_predict_fp32(tb_mlp *m, int32_t n, const float *feat, float *out)
{
    TB_ABI_TRY
    if (!m || n <= 0 || !feat || !out) return TB_ERR_INVALID_ARG;
    cudaSetDevice(m->device);
    std::lock_guard<std::mutex> lock(m->mu);
    float *dX = nullptr, *dY = nullptr;
    int rc = upload_set(m->stream, n, feat, nullptr, &dX, nullptr);
    if (rc == TB_OK && cudaMalloc(&dY, sizeof(float) * n)) rc = TB_ERR_OUT_OF_MEMORY;
    if (rc == TB_OK) {
        k_mlp_fb<<<fb_grid(n), 256, kFbSmem, m->stream>>>(n, nullptr, dX, m->mean, m->istd, m->Wq, nullptr, 0.f,
                                                         dY, nullptr, nullptr);
        cudaMemcpyAsync(out, dY, sizeof(float) * n, cudaMemcpyDeviceToHost, m->stream);
        if (cudaStreamSynchronize(m->stream) != cudaSuccess || cudaGetLastError() != cudaSuccess) rc = TB_ERR_CUDA;
    }
    cudaFree(dX);
    cudaFree(dY);
    return rc;
    TB_ABI_CATCH
}

int tb_mlp_train(tb_mlp *m, int32_t n, const float *feat, const float *target, int32_t epochs, int32_t batch,
                 float lr, uint64_t seed, float *loss_per_epoch)
{
    TB_ABI_TRY
    if (!m || n <= 0 || !feat || !target || epochs < 1 || batch < 1 || !(lr > 0)) return TB_ERR_INVALID_ARG;
    cudaSetDevice(m->device);
    std::lock_guard<std::mutex> lock(m->mu);
    cudaStream_t st = m->stream;
    if (!m->have_norm) {
        // fix the feature normalisation from this training set
        std::vector<double> mu(kF, 0.0), var(kF, 0.0);
        for (int64_t s = 0; s < n; s++)
            for (int i = 0; i < kF; i++) mu[i] += feat[s * kF + i];
        for (int i = 0; i < kF; i++) mu[i] /= n;
        for (int64_t s = 0; s < n; s++)
            for (int i = 0; i < kF; i++) {
                const double d = feat[s * kF + i] - mu[i];
                var[i] += d * d;
            }
        std::vector<float> norm(2 * kF);
        for (int i = 0; i < kF; i++) {
            norm[i] = (float)mu[i];
            const double sd = std::sqrt(var[i] / n);
            norm[kF + i] = (float)(sd > 1e-6 ? 1.0 / sd : 1.0);
        }
        mlp_set(m, nullptr, norm.data());
    }
    float *dX, *dT;
    int32_t *dI = nullptr;
    int rc = upload_set(st, n, feat, target, &dX, &dT);
    if (rc == TB_OK && cudaMalloc(&dI, sizeof(int32_t) * n)) rc = TB_ERR_OUT_OF_MEMORY;
    std::vector<int32_t> perm(n);
    std::iota(perm.begin(), perm.end(), 0);
    uint64_t rs = seed;
    for (int ep = 0; ep < epochs && rc == TB_OK; ep++) {
        for (int i = n - 1; i > 0; i--) {  // Fisher-Yates with splitmix64
            rs += 0x9E3779B97F4A7C15ull;
            const int j = (int)(mix64(rs) % (uint64_t)(i + 1));
            std::swap(perm[i], perm[j]);
        }
        cudaMemcpyAsync(dI, perm.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice, st);
        cudaMemsetAsync(m->loss, 0, sizeof(float) * kCopies, st);
        for (int b0 = 0; b0 < n; b0 += batch) {
            const int nb = std::min(batch, n - b0);
            cudaMemsetAsync(m->g, 0, sizeof(float) * kCopies * kGStride, st);
            k_mlp_fb<<<fb_grid(nb), 256, kFbSmem, st>>>(nb, dI + b0, dX, m->mean, m->istd, m->Wq, dT,
                                                        1.f / nb, nullptr, m->g, m->loss);
            m->step++;
            const float c1 = 1.f / (1.f - std::pow(0.9f, (float)m->step));
            const float c2 = 1.f / (1.f - std::pow(0.999f, (float)m->step));
            k_adam<<<(kNP + 255) / 256, 256, 0, st>>>(kNP, m->W, m->Wq, m->m1, m->m2, m->g, lr, c1, c2);
        }
        float part[kCopies] = {}, l = 0.f;
        cudaMemcpyAsync(part, m->loss, sizeof(part), cudaMemcpyDeviceToHost, st);
        if (cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess) rc = TB_ERR_CUDA;
        for (float x : part) l += x;
        // the per-batch losses are batch means: average over the batches
        if (loss_per_epoch) loss_per_epoch[ep] = l * (float)batch / (float)n;
    }
    cudaFree(dX);
    cudaFree(dT);
    cudaFree(dI);
    return rc;
    TB_ABI_CATCH
}

}  // extern "C"
