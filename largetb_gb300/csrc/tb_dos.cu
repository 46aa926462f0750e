// tb_dos.cu -- stochastic KPM density of states (runKPM's DOS,
// withSP2_deltaH.cpp:1579-1648) on the GPU.
//
// n_random Gaussian probe vectors r (counter-based splitmix64 + Box-Muller:
// entry i of vector t is deviate t*n + i of the stream seeded with `seed`)
// form the columns of slabs; mu_k = sum_t r_t^T T_k(X) r_t comes from the
// fixed-point step's column sums (tb_fixed.cu) or, on a caller's interval, from
// the FP64 step and k_probe_dot (block shares summed in block order): the
// moments are the same from run to run.
// The DOS at the Chebyshev nodes x_q = cos(pi (q+1/2)/npts) is
//   rho(x_q) = [g_0 mu_0 + 2 sum_{k>=1} g_k mu_k cos(k acos x_q)] / (pi sqrt(1 - x_q^2))
// with the closed-form Jackson g_k (N = n_moments), at energies a x_q + b.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <vector>

#include "tb_internal.h"

namespace tb {

namespace {

constexpr double kPi = 3.141592653589793238463;

__device__ __forceinline__ uint64_t splitmix_at(uint64_t seed, uint64_t k)
{
    uint64_t z = seed + (k + 1ull) * 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__device__ __forceinline__ double gauss_at(uint64_t seed, uint64_t idx)
{
    const double two53 = 1.0 / 9007199254740992.0;
    const double u1 = ((double)(splitmix_at(seed, 2ull * idx) >> 11) + 1.0) * two53;
    const double u2 = (double)(splitmix_at(seed, 2ull * idx + 1ull) >> 11) * two53;
    return sqrt(-2.0 * log(u1)) * cos(2.0 * kPi * u2);
}

__global__ void k_probe_init(double *__restrict__ T0, double *__restrict__ R, int n, int B, int nr,
                             uint64_t seed)
{
    const int64_t tot = (int64_t)n * B;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < tot;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(e / B), t = (int)(e % B);
        const double v = t < nr ? gauss_at(seed, (uint64_t)t * n + i) : 0.0;
        T0[e] = v;
        R[e] = v;
    }
}

// part_k[block] = this block's share of sum_{i,t} R[i][t] T_k[i][t]; the
// shares are summed in block order by k_sum_parts, so the moments do not
// depend on the order in which blocks finish.
__global__ void __launch_bounds__(256) k_probe_dot(const double *__restrict__ R,
                                                   const double *__restrict__ Tk, int64_t tot,
                                                   double *__restrict__ part_k)
{
    __shared__ double sh[8];
    double s = 0.0;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < tot;
         e += (int64_t)gridDim.x * blockDim.x)
        s = fma(R[e], Tk[e], s);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < 8; w++) t += sh[w];
        part_k[blockIdx.x] = t;
    }
}

// mom[k] = sum over blocks of part[k][block], one CTA per moment, a fixed
// tree order.
__global__ void __launch_bounds__(256) k_sum_parts(const double *__restrict__ part, int nparts,
                                                   double *__restrict__ mom)
{
    __shared__ double sh[8];
    const double *p = part + (int64_t)blockIdx.x * nparts;
    double s = 0.0;
    for (int b = threadIdx.x; b < nparts; b += blockDim.x) s += p[b];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < 8; w++) t += sh[w];
        mom[blockIdx.x] = t;
    }
}

// rho(x_q) on the nodes, eight neighbouring lanes a node.  With the table
// tab[j] = cos(pi j / (2 npts)), j < 4 npts, cos(k theta_q) is entry
// k (2q + 1) mod 4 npts; without one (npts above kDosTabMax) it is evaluated.
// One thread a node with a cosine a term took 2.5 ms at 1000 moments and 2000
// nodes.
constexpr int kDosTabMax = 1 << 20, kDosLanes = 8;

__global__ void k_dos_table(int npts, double *__restrict__ tab)
{
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < 4 * npts; j += gridDim.x * blockDim.x)
        tab[j] = cos(kPi * j / (2.0 * npts));
}

__global__ void __launch_bounds__(256)
    k_dos_eval(const double *__restrict__ g, const double *__restrict__ mom, int nmom, int npts,
               const double *__restrict__ tab, const DevState *__restrict__ st, double *__restrict__ E,
               double *__restrict__ dos)
{
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int q = (int)(tid / kDosLanes), sl = (int)(tid % kDosLanes);
    const bool on = q < npts;
    const uint32_t period = 4u * (uint32_t)npts;
    const double th = kPi * (q + 0.5) / npts;
    double s = 0.0;
    if (on) {
        const int len = (nmom + kDosLanes - 1) / kDosLanes, k0 = sl * len, k1 = min(nmom, k0 + len);
        const uint32_t step = 2u * (uint32_t)q + 1u;
        uint32_t j = tab ? (uint32_t)((uint64_t)k0 * step % period) : 0u;
        for (int k = k0; k < k1; k++) {
            const double c = tab ? tab[j] : cos(k * th);
            s += (k == 0 ? 1.0 : 2.0) * g[k] * mom[k] * c;
            if (tab) {
                j += step;
                if (j >= period) j -= period;
            }
        }
    }
    for (int o = 1; o < kDosLanes; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (on && sl == 0) {
        const double x = cos(th);
        dos[q] = s / (kPi * sqrt(1.0 - x * x));
        E[q] = x * st->a + st->b;
    }
}

// Chemical potential and refined spectral interval from the DOS on the
// nodes (runKPM, withSP2_deltaH.cpp:1663-1703), written into the state for
// the density pass: trapezoid area from the bottom of the spectrum up to
// N_e / (2n) of the total gives mu = E[index]; the interval is where
// DOS/n >= 0.001 first holds from either end (-10, 10 when it never does).
// One CTA: every thread sums a run of trapezoids (node npts - 1 downwards),
// and the thread whose run crosses the area walks it again; a sequential scan
// with its two cosines a node took milliseconds.  Also sets beta_x = a/kT
// and the quadrature size of the new interval (the Gershgorin rule).
__global__ void __launch_bounds__(256)
    k_dos_mu(const double *__restrict__ E, const double *__restrict__ dos, int npts, int n, double n_elec, double kT,
             int M, int nq_cap, DevState *st)
{
    __shared__ double part[256];
    __shared__ int s_mi, s_lo, s_hi;
    const int t = threadIdx.x, len = (npts - 1 + 255) / 256;
    // trapezoid u = 0 .. npts - 2 lies between nodes npts - 1 - u and npts - 2 - u
    const int u0 = min(npts - 1, t * len), u1 = min(npts - 1, u0 + len);
    auto trap = [&](int u) {
        const int i = npts - 1 - u;
        const double xi = cos(kPi * (i + 0.5) / npts), xm = cos(kPi * (i - 0.5) / npts);
        return (xm - xi) * (dos[i] + dos[i - 1]) / 2;
    };
    double s = 0.0;
    for (int u = u0; u < u1; u++) s += trap(u);
    part[t] = s;
    int lo = -1, hi = npts;  // the support's last and first nodes
    for (int i = t; i < npts; i += 256)
        if (dos[i] / n >= 0.001) {
            if (i > 0) lo = max(lo, i);
            hi = min(hi, i);
        }
    if (t == 0) {
        s_mi = -1;
        s_lo = -1;
        s_hi = npts;
    }
    __syncthreads();
    atomicMax(&s_lo, lo);
    atomicMin(&s_hi, hi);
    double before = 0.0, all = 0.0;
    for (int w = 0; w < 256; w++) {
        if (w == t) before = all;
        all += part[w];
    }
    const double area = n_elec * all / (2.0 * n);
    double cum = before;
    for (int u = u0; u < u1; u++) {
        cum += trap(u);
        if (cum >= area) {
            atomicMax(&s_mi, npts - 1 - u);  // the first from the bottom
            break;
        }
    }
    __syncthreads();
    if (t != 0) return;
    const int mi = s_mi < 0 ? 0 : s_mi;
    const double emin = s_lo >= 0 ? E[s_lo] : -10.0, emax = s_hi < npts ? E[s_hi] : 10.0;
    const double a = (emax - emin) / 2, b = (emax + emin) / 2;
    st->a = a;
    st->b = b;
    st->mu = E[mi];
    st->mu_x = (E[mi] - b) / a;
    st->status = (a > 0 && isfinite(a)) ? 0 : TB_ERR_SPECTRUM;
    st->beta_x = kT > 0 ? a / kT : 0.0;
    double need = 4.0 * M;
    if (st->beta_x > 0 && 13.0 * st->beta_x > need) need = 13.0 * st->beta_x;
    if (need < 256) need = 256;
    int nq = 256;
    while (nq < need && nq < (1 << 22)) nq *= 2;
    if (nq > nq_cap) st->status = TB_ERR_SPECTRUM;
    st->nq = nq > nq_cap ? nq_cap : nq;
    st->bisect_done = 1;
}

// Probe slab of the density pass: columns t < nr of probes t0 .. t0+nr-1 of
// the stream `seed` (deviate index (t0 + t) n + i), zero beyond; to T0 as well
// where it is given.
__global__ void k_probe_slab(double *__restrict__ T0, double *__restrict__ R, int n, int B, int nr, int t0,
                             uint64_t seed)
{
    const int64_t tot = (int64_t)n * B;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < tot;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(e / B), t = (int)(e % B);
        const double v = t < nr ? gauss_at(seed, (uint64_t)(t0 + t) * n + i) : 0.0;
        if (T0) T0[e] = v;
        R[e] = v;
    }
}

// computeDiagonalElements' accumulation for step k: one warp per orbital i,
// num_i += c_k g_k sum_t R[i][t] T_k[i][t]; at k = 0 also den_i += sum_t R[i][t]^2.
__global__ void k_probe_rowacc(const double *__restrict__ R, const double *__restrict__ Tk, int n, int B,
                               const double *__restrict__ c, const double *__restrict__ g, int k,
                               double *__restrict__ num, double *__restrict__ den)
{
    const int lane = threadIdx.x & 31;
    const int i = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (i >= n) return;
    double s = 0.0, s2 = 0.0;
    for (int t = lane; t < B; t += 32) {
        const double r = R[(int64_t)i * B + t];
        s = fma(r, Tk[(int64_t)i * B + t], s);
        s2 = fma(r, r, s2);
    }
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    if (lane == 0) {
        num[i] += c[k] * g[k] * s;
        if (k == 0) den[i] += s2;
    }
}

// diagP_i = num_i / den_i; q_a = 2 sum over the atom's four orbitals.
__global__ void k_probe_diag(const double *__restrict__ num, const double *__restrict__ den, int natoms,
                             double *__restrict__ diagP, double *__restrict__ q)
{
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= natoms) return;
    double s = 0.0;
    for (int r = 0; r < 4; r++) {
        const double d = num[4 * a + r] / den[4 * a + r];
        diagP[4 * a + r] = d;
        s += d;
    }
    q[a] = 2.0 * s;
}

// Device scratch of the stochastic paths, carved in 256-byte steps: up to
// kDosKept stays with the context between calls and goes back with its matrix,
// more goes back at the end of the call (slabs in FP64 hold all probes: 4096 of
// 108000 orbitals take 11 GB).
constexpr size_t kDosKept = 512u << 20;

struct DosKeep {
    tb_ctx *ctx;
    ~DosKeep()
    {
        if (ctx->dos_bytes <= kDosKept) return;
        cudaFree(ctx->dos_scratch);
        ctx->dos_scratch = nullptr;
        ctx->dos_bytes = 0;
    }
};

struct Carve {
    char *base;
    size_t used = 0;
    template <typename T>
    T *take(size_t n)
    {
        T *p = reinterpret_cast<T *>(base + used);
        used += (n * sizeof(T) + 255) / 256 * 256;
        return p;
    }
};

int ensure_scratch(tb_ctx *ctx, size_t bytes)
{
    if (ctx->dos_bytes >= bytes) return TB_OK;
    if (ctx->dos_scratch) cudaFree(ctx->dos_scratch);
    ctx->dos_scratch = nullptr;
    ctx->dos_bytes = 0;
    const cudaError_t e = cudaMalloc(&ctx->dos_scratch, bytes);
    if (e != cudaSuccess) {
        ctx->dos_scratch = nullptr;
        cudaGetLastError();
        ctx->err = std::string("cudaMalloc(stochastic scratch): ") + cudaGetErrorString(e);
        return e == cudaErrorMemoryAllocation ? TB_ERR_OUT_OF_MEMORY : TB_ERR_CUDA;
    }
    ctx->dos_bytes = bytes;
    return TB_OK;
}

template <typename T>
int ensure_x(tb_ctx *ctx, T *&p, size_t n)
{
    if (p) return TB_OK;
    if (cudaMalloc(&p, sizeof(T) * n) == cudaSuccess) return TB_OK;
    cudaGetLastError();
    p = nullptr;
    ctx->err = "cudaMalloc(X)";
    return TB_ERR_OUT_OF_MEMORY;
}

// Probes of one slab: as many as keep both fixed-point buffers in L2.
int probe_slab(int n, int nr)
{
    const int cap = std::min(1024, std::max(64, (int)(80.0e6 / (16.0 * n)) / 64 * 64));
    const int ns = (nr + cap - 1) / cap;
    return fixed_probe_width((nr + ns - 1) / ns);
}

// Scratch of the moments and the DOS.
struct DosScratch {
    int B = 0;         // probes a slab
    bool fixed = false;
    double *T0 = nullptr, *T1 = nullptr, *R = nullptr, *mom = nullptr, *g = nullptr, *E = nullptr, *dos = nullptr;
    double *part = nullptr, *tab = nullptr, *num = nullptr, *den = nullptr, *wts = nullptr, *rows = nullptr;
    int2 *keep = nullptr;
    unsigned long long *sums = nullptr;
    int32_t *shift = nullptr, *over = nullptr;
    int blocks = 0;
    std::vector<double> gh;  // host copy of g: the call waits for the stream before it ends

    // the widest slab of the call is B x n; for the density, its pass's arrays too
    void carve(Carve &c, int n, int nr, int nmom, int npts, int M, bool density)
    {
        const size_t slab = (size_t)n * B;
        blocks = (int)std::min<int64_t>(((int64_t)slab + 255) / 256, 152 * 8);
        T0 = c.take<double>(slab);
        T1 = c.take<double>(slab);
        R = c.take<double>(slab);
        mom = c.take<double>(nmom);
        g = c.take<double>(nmom);
        E = c.take<double>(npts);
        dos = c.take<double>(npts);
        tab = npts <= kDosTabMax ? c.take<double>(4 * (size_t)npts) : nullptr;
        shift = c.take<int32_t>(1);
        over = c.take<int32_t>(1);
        sums = c.take<unsigned long long>(fixed ? (size_t)((nmom + 1) / 2) * 4 * B : 1);
        part = c.take<double>(fixed ? 1 : (size_t)blocks * nmom);
        if (density) {
            num = c.take<double>(n);
            den = c.take<double>(n);
            wts = c.take<double>(M);
            keep = c.take<int2>(slab);
            rows = c.take<double>((size_t)n * fixed_groups(B));
        }
    }
};

// mu_k = sum_t r_t^T T_k(X) r_t of nr probes, k < nmom, and the DOS on npts
// nodes; the state holds the interval.
//
// In fixed point (slabs that stay in L2) the moments come from <T_k r, T_k r>
// and <T_k r, T_{k+1} r>, nmom / 2 steps; on a caller's interval, which may not
// hold the spectrum, from r . T_k r in FP64.
void run_moments(tb_ctx *ctx, DosScratch &w, const double *d_shift, DevState *state, int nr, uint64_t seed, int nmom,
                int npts, int64_t *nl)
{
    DevMatrix &m = ctx->m;
    cudaStream_t st = ctx->stream;
    // closed-form Jackson damping with N = nmom (runKPM, withSP2_deltaH.cpp:1593-1595)
    std::vector<double> &gh = w.gh;
    gh.resize(nmom);
    const double N = nmom, cotv = std::cos(kPi / (N + 1)) / std::sin(kPi / (N + 1));
    for (int k = 0; k < nmom; k++)
        gh[k] = ((N - k + 1) * std::cos(kPi * k / (N + 1)) + std::sin(kPi * k / (N + 1)) * cotv) / (N + 1);
    cudaMemcpyAsync(w.g, gh.data(), sizeof(double) * nmom, cudaMemcpyHostToDevice, st);
    if (w.fixed) {
        launch_build_x_fixed(st, m, d_shift, state);
        cudaMemsetAsync(w.mom, 0, sizeof(double) * nmom, st);
        cudaMemsetAsync(w.over, 0, sizeof(int32_t), st);
        const int K = (nmom + 1) / 2;
        for (int t0 = 0; t0 < nr; t0 += w.B) {
            const int nrs = std::min(w.B, nr - t0), B = std::min(w.B, fixed_probe_width(nrs));
            const int64_t tot = (int64_t)m.n * B;
            k_probe_slab<<<(int)std::min<int64_t>((tot + 255) / 256, 152 * 8), 256, 0, st>>>(nullptr, w.R, m.n, B, nrs,
                                                                                             t0, seed);
            int2 *A = reinterpret_cast<int2 *>(w.T0), *C = reinterpret_cast<int2 *>(w.T1);
            launch_fx_probes(st, w.R, m.n, B, w.shift, A, nullptr);
            cudaMemsetAsync(w.sums, 0, sizeof(*w.sums) * (size_t)K * 4 * B, st);
            for (int k = 0; k < K; k++)
                launch_cheb_fixed(st, m, k & 1 ? C : A, k & 1 ? A : C, B, k == 0, w.sums + (size_t)k * 4 * B,
                                  w.over);
            launch_fx_probe_moments(st, w.sums, B, nrs, nmom, w.shift, w.mom);
            *nl += 5 + K;
        }
        *nl += 1;
    } else {
        const int64_t tot = (int64_t)m.n * w.B;
        launch_build_x(st, m, d_shift, TB_PREC_FP64, state);
        k_probe_init<<<w.blocks, 256, 0, st>>>(w.T0, w.R, m.n, w.B, nr, seed);
        k_probe_dot<<<w.blocks, 256, 0, st>>>(w.R, w.T0, tot, w.part);
        for (int kout = 1; kout < nmom; kout++) {
            const bool odd = kout & 1;
            double *in = odd ? w.T0 : w.T1, *out = odd ? w.T1 : w.T0;
            // c0 = n: no identity diagonal to gather for probe vectors
            launch_cheb_step_f64(st, m, in, out, w.B, m.n, kout == 1, nullptr, kout);
            k_probe_dot<<<w.blocks, 256, 0, st>>>(w.R, out, tot, w.part + (int64_t)kout * w.blocks);
            *nl += (kout == 1) ? 3 : 2;
        }
        k_sum_parts<<<nmom, 256, 0, st>>>(w.part, w.blocks, w.mom);
        *nl += 4;
    }
    if (w.tab) k_dos_table<<<std::min((4 * npts + 255) / 256, 1024), 256, 0, st>>>(npts, w.tab);
    k_dos_eval<<<(unsigned)(((int64_t)npts * kDosLanes + 255) / 256), 256, 0, st>>>(w.g, w.mom, nmom, npts, w.tab,
                                                                                   state, w.E, w.dos);
    *nl += w.tab ? 2 : 1;
}

}  // namespace

int run_density_stochastic(tb_ctx *ctx, const double *d_shift, int nr, uint64_t seed, int nmom_dos, int npts,
                           int64_t *launches)
{
    DevMatrix &m = ctx->m;
    DevWork &w = ctx->w;
    cudaStream_t st = ctx->stream;
    const int M = ctx->p.M;
    cudaError_t e = cudaSuccess;
    int64_t nl = 0;
    DosKeep keep{ctx};
    DosScratch ws;
    const int Bdens = std::min((nr + 63) / 64 * 64, 256);  // FP64 density slabs
    int Bpass = 0, rc = TB_OK;
    DevState hs;
    for (bool want = !(ctx->p.bounds_hi > ctx->p.bounds_lo);; want = false) {
        ws.fixed = want;
        Bpass = ws.fixed ? probe_slab(m.n, nr) : (nr + 63) / 64 * 64;
        ws.B = std::max(Bpass, Bdens);  // room for either density pass
        Carve size{nullptr};
        ws.carve(size, m.n, nr, nmom_dos, npts, M, true);
        if ((rc = ensure_scratch(ctx, size.used)) || (rc = ensure_x(ctx, m.xfx, (size_t)m.nnzb * 8)) ||
            (rc = ensure_x(ctx, m.xdfx, (size_t)m.n)) || (!ws.fixed && (rc = ensure_x(ctx, m.x64, (size_t)m.nnzb * 16))))
            return rc;
        Carve arena{(char *)ctx->dos_scratch};
        ws.carve(arena, m.n, nr, nmom_dos, npts, M, true);
        ws.B = Bpass;
        // ---- runKPM: stochastic moments of X on the Gershgorin interval ----
        launch_gershgorin(st, m, d_shift, ctx->p.spectral_pad, ctx->p.kT, M, w.nq_cap, w.state, ctx->p.bounds_lo,
                          ctx->p.bounds_hi);
        run_moments(ctx, ws, d_shift, w.state, nr, seed, nmom_dos, npts, &nl);
        // ---- mu and the refined interval; the expansion coefficients ----
        k_dos_mu<<<1, 256, 0, st>>>(ws.E, ws.dos, npts, m.n, ctx->p.n_electrons, ctx->p.kT, M, w.nq_cap, w.state);
        launch_fermi_coeffs(st, M, w.state, w.nq_cap, w.costab, w.fq, w.c);
        nl += 4;
        int32_t over = 0;
        if (ws.fixed) cudaMemcpyAsync(&over, ws.over, sizeof(over), cudaMemcpyDeviceToHost, st);
        cudaMemcpyAsync(&hs, w.state, sizeof(hs), cudaMemcpyDeviceToHost, st);
        if ((e = cudaStreamSynchronize(st)) != cudaSuccess || (e = cudaGetLastError()) != cudaSuccess) {
            ctx->err = std::string("stochastic density: ") + cudaGetErrorString(e);
            return TB_ERR_CUDA;
        }
        if (!over && !(ws.fixed && hs.poison)) break;  // else again, in FP64
    }
    // The refined interval may leave some of the spectrum outside, and T_k x
    // then grows.  Fixed point holds while every row of |X| sums to less than
    // three (rho, from Gershgorin's bounds), no entry of X passes 1.9 (a limb
    // holds less than two; such an entry is left out of X and raises the
    // state's poison) and no entry of T_k x passes twice the largest of x, of
    // which the step keeps watch; else the pass is made again in FP64.
    const double rho = std::max(hs.lmax - hs.b, hs.b - hs.lmin) / hs.a;
    bool fixed = hs.status == 0 && rho < 2.9;
    // ---- computeDiagonalElements: fresh probes (stream seed + 1), in slabs ----
    if (fixed) {
        cudaMemsetAsync(ws.num, 0, sizeof(double) * m.n, st);
        cudaMemsetAsync(ws.den, 0, sizeof(double) * m.n, st);
        cudaMemsetAsync(ws.rows, 0, sizeof(double) * m.n * fixed_groups(ws.B), st);
        cudaMemsetAsync(ws.over, 0, sizeof(int32_t), st);
        launch_build_x_fixed(st, m, d_shift, w.state, 1.9);
        launch_fx_weights(st, w.c, w.g, M, ws.wts);
        const int Bf = ws.fixed ? Bpass : Bdens;
        for (int t0 = 0; t0 < nr; t0 += Bf) {
            const int nrs = std::min(Bf, nr - t0), B = std::min(Bf, fixed_probe_width(nrs));
            const int64_t tot = (int64_t)m.n * B;
            k_probe_slab<<<(int)std::min<int64_t>((tot + 255) / 256, 152 * 8), 256, 0, st>>>(nullptr, ws.R, m.n, B, nrs,
                                                                                             t0, seed + 1);
            int2 *A = reinterpret_cast<int2 *>(ws.T0), *C = reinterpret_cast<int2 *>(ws.T1);
            launch_fx_probes(st, ws.R, m.n, B, ws.shift, A, ws.keep);
            launch_fx_probe_den(st, ws.keep, m.n, B, ws.shift, ws.wts, ws.num, ws.den);
            for (int k = 0; k + 1 < M; k++)
                launch_cheb_fixed_rows(st, m, k & 1 ? C : A, k & 1 ? A : C, B, k == 0, ws.keep, ws.wts + k + 1, ws.rows,
                                       ws.over);
            launch_fx_probe_num(st, ws.rows, m.n, fixed_groups(B), ws.shift, ws.num);
            nl += 6 + M - 1;
        }
        nl += 2;
        int32_t over = 0, poison = 0;
        cudaMemcpyAsync(&over, ws.over, sizeof(over), cudaMemcpyDeviceToHost, st);
        cudaMemcpyAsync(&poison, &w.state->poison, sizeof(poison), cudaMemcpyDeviceToHost, st);
        if ((e = cudaStreamSynchronize(st)) != cudaSuccess) {
            ctx->err = std::string("stochastic density: ") + cudaGetErrorString(e);
            return TB_ERR_CUDA;
        }
        fixed = !over && !poison;
    }
    if (!fixed) {
        cudaMemsetAsync(ws.num, 0, sizeof(double) * m.n, st);
        cudaMemsetAsync(ws.den, 0, sizeof(double) * m.n, st);
        if ((rc = ensure_x(ctx, m.x64, (size_t)m.nnzb * 16))) return rc;
        launch_build_x(st, m, d_shift, TB_PREC_FP64, w.state);
        nl++;
        const int rblocks = (int)((((int64_t)m.n * 32) + 255) / 256), B = Bdens;
        for (int t0 = 0; t0 < nr; t0 += B) {
            const int nrs = std::min(B, nr - t0);
            const int64_t ts = (int64_t)m.n * B;
            k_probe_slab<<<(int)std::min<int64_t>((ts + 255) / 256, 152 * 8), 256, 0, st>>>(ws.T0, ws.R, m.n, B, nrs, t0,
                                                                                             seed + 1);
            k_probe_rowacc<<<rblocks, 256, 0, st>>>(ws.R, ws.T0, m.n, B, w.c, w.g, 0, ws.num, ws.den);
            nl += 2;
            for (int kout = 1; kout < M; kout++) {
                const bool odd = kout & 1;
                double *in = odd ? ws.T0 : ws.T1, *out = odd ? ws.T1 : ws.T0;
                launch_cheb_step_f64(st, m, in, out, B, m.n, kout == 1, nullptr, kout);
                k_probe_rowacc<<<rblocks, 256, 0, st>>>(ws.R, out, m.n, B, w.c, w.g, kout, ws.num, ws.den);
                nl += (kout == 1) ? 3 : 2;
            }
        }
    }
    k_probe_diag<<<(m.natoms + 127) / 128, 128, 0, st>>>(ws.num, ws.den, m.natoms, w.diagP, w.q);
    nl++;
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess || (e = cudaGetLastError()) != cudaSuccess) {
        ctx->err = std::string("stochastic density: ") + cudaGetErrorString(e);
        rc = TB_ERR_CUDA;
    }
    if (launches) *launches = nl;
    return rc;
}

int run_kpm_dos(tb_ctx *ctx, int nmom, int nr, uint64_t seed, int npts, double *mom_h, double *E_h,
                double *dos_h, double *a_out, double *b_out, int64_t *launches)
{
    DevMatrix &m = ctx->m;
    cudaStream_t st = ctx->stream;
    cudaError_t e = cudaSuccess;
    int64_t nl = 0;
    DosKeep keep{ctx};
    DosScratch ws;
    int rc = TB_OK;
    for (bool want = !(ctx->p.bounds_hi > ctx->p.bounds_lo);; want = false) {
        ws.fixed = want;
        ws.B = ws.fixed ? probe_slab(m.n, nr) : (nr + 63) / 64 * 64;
        Carve size{nullptr};
        size.take<DevState>(1);
        ws.carve(size, m.n, nr, nmom, npts, 0, false);
        if ((rc = ensure_scratch(ctx, size.used)) ||
            (ws.fixed && ((rc = ensure_x(ctx, m.xfx, (size_t)m.nnzb * 8)) || (rc = ensure_x(ctx, m.xdfx, (size_t)m.n)))) ||
            (!ws.fixed && (rc = ensure_x(ctx, m.x64, (size_t)m.nnzb * 16))))
            return rc;
        Carve arena{(char *)ctx->dos_scratch};
        DevState *state = arena.take<DevState>(1);
        ws.carve(arena, m.n, nr, nmom, npts, 0, false);
        launch_gershgorin(st, m, nullptr, 0.0, 0.0, 2, 1 << 22, state, ctx->p.bounds_lo, ctx->p.bounds_hi);
        nl++;
        run_moments(ctx, ws, nullptr, state, nr, seed, nmom, npts, &nl);
        DevState hs;
        int32_t over = 0;
        if (ws.fixed) cudaMemcpyAsync(&over, ws.over, sizeof(over), cudaMemcpyDeviceToHost, st);
        cudaMemcpyAsync(mom_h, ws.mom, sizeof(double) * nmom, cudaMemcpyDeviceToHost, st);
        cudaMemcpyAsync(E_h, ws.E, sizeof(double) * npts, cudaMemcpyDeviceToHost, st);
        cudaMemcpyAsync(dos_h, ws.dos, sizeof(double) * npts, cudaMemcpyDeviceToHost, st);
        cudaMemcpyAsync(&hs, state, sizeof(hs), cudaMemcpyDeviceToHost, st);
        if ((e = cudaStreamSynchronize(st)) != cudaSuccess || (e = cudaGetLastError()) != cudaSuccess) {
            ctx->err = std::string("kpm dos: ") + cudaGetErrorString(e);
            rc = TB_ERR_CUDA;
            break;
        }
        if (over || (ws.fixed && hs.poison)) continue;  // again, in FP64
        if (hs.status) {
            ctx->err = "Gershgorin interval collapsed";
            rc = TB_ERR_SPECTRUM;
        }
        if (a_out) *a_out = hs.a;
        if (b_out) *b_out = hs.b;
        break;
    }
    if (launches) *launches = nl;
    return rc;
}

}  // namespace tb
