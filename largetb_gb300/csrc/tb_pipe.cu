// tb_pipe.cu -- FP32 Chebyshev recurrence, pipelined form (K2 of the
// density-matrix path: the recurrence of getKPE, withSP2_deltaH.cpp:1134-1168,
// over identity columns, with the moments taken from column dot products as in
// k_cheb_f32_staged).
//
// Slab layout: chunk-major, [B/64][n][64] floats, so that a block row of one
// 64-column chunk is 1 KB contiguous and consecutive block rows are
// contiguous too.
//
// One CTA per SM loops over tiles (row group g of R block rows x one
// 64-column chunk).  A producer warp gathers each tile into a ring of
// shared-memory stages with bulk asynchronous copies (cp.async.bulk,
// completion counted in bytes on the stage's "full" mbarrier): the group's
// distinct referenced block rows of T_k as runs of consecutive rows (one copy
// per run), its own rows of T_{k-1} (one copy), its X blocks (one copy) and a
// packed index record (one copy).  Twelve consumer warps compute the tile from
// shared memory while the producer fills the next stages.  The header and
// copy runs of the next tile are loaded while the producer waits for a free
// stage, so no global load latency sits on its path.
//
// Three launch modes share the kernel:
//  - one launch per step (steps = 1);
//  - one cooperative launch per slab running all K steps.  A tile publishes
//    its step count in flags[tile] (release, after an mbarrier that every
//    consumer warp arrives on after its stores); before the producer copies
//    tile (chunk, g) of step k >= 1 it waits (acquire) until every group g'
//    whose rows g references, g itself included, has published step k in the
//    same chunk.  That covers both the T_k rows it reads and the T_{k-1} rows
//    it overwrites: the block pattern is symmetric, so the groups that read
//    rows of g at step k-1 are exactly those neighbours.  Each CTA runs its
//    tiles in step order and all CTAs are co-resident, so the oldest
//    unfinished step can always proceed.  The pipeline never drains between
//    steps;
//  - the batched form (k_cheb_f32_pipe<true, ...>, one launch per step): tiles
//    come from a list over many structures, each tile naming its row group
//    and carrying the offset of its chunk in that structure's slabs and of
//    its column sums; a group's header holds its first (structure-local)
//    block row.
//
// Column dot products <T_k,T_k> and <T_k,T_{k+1}> accumulate in FP32 over one
// block row and then as unevaluated FP32 pairs (hi, lo) across rows and warps:
// every addition is Knuth's TwoSum (s = a + b, e = (a - (s - b')) + (b - b'),
// b' = s - a), its exact rounding error collected in lo.  GB300 issues FP64 at
// about 2 operations per clock per SM, so per-row FP64 accumulation would cost
// as much as the rest of the step; the pairs keep ~44 significant bits with
// FP32 arithmetic only.  The recurrence itself and the per-row products use
// packed FP32 pair instructions (fma.f32x2 / add.f32x2: two columns per
// instruction, each rounded as the scalar operation).  Each consumer warp
// hands its pairs over in a shared array and arrives on an mbarrier; four
// consumer warps, in rotation from tile to tile, wait for all twelve and sum
// them in warp order, giving partial[k][g][col][2] as float2 (hi, lo), while
// the other warps go on with the next tile.  k_f32_finalize_pairs converts to
// FP64.
//
// Every wait is bounded: after kPipeSpin unsuccessful polls the thread raises
// a block-wide abort flag and the device error flag; every later wait in the
// CTA then returns at once, the warps run out their tile sequence skipping
// the work, other CTAs waiting on this one's flags time out the same way, and the
// producer, before it returns, waits (again bounded) for the copies it has
// issued.  The host turns the error flag into TB_ERR_TIMEOUT (1: a stage
// mbarrier wait, 2: a neighbour-flag wait ran out).
//
// Two environment variables, read at each one-launch-per-slab launch, let a
// test make a neighbour wait run out without any fault: LARGETB_TEST_WAIT_LIMIT
// (neighbour-flag polls before giving up; default 2^22) and
// LARGETB_TEST_STALL_TILE (a tile whose step flags are never published, so
// every tile that reads its rows waits for a flag that nothing sets).
#include <cuda_runtime.h>

#include <algorithm>
#include <functional>
#include <cstdlib>

#include "tb_chain.cuh"
#include "tb_f32x2.cuh"
#include "tb_internal.h"

namespace tb {

namespace {

constexpr int kPipeCols = 64;
constexpr int kPipeCW = 12;  // consumer warps; then one producer and one publisher warp
constexpr int kPipeThreads = 32 * (kPipeCW + 2);
constexpr int kPubSlots = 4;  // tiles the publisher may lag behind the consumers
constexpr int kRedWarps = 4;  // consumer warps that reduce one tile's column sums, in rotation
static_assert(kPipeCW % kRedWarps == 0 && kRedWarps * 32 == 2 * kPipeCols, "reducer split");
constexpr uint32_t kPipeSpin = 1u << 22;  // mbarrier polls
constexpr uint32_t kFlagSpin = 1u << 22;  // neighbour-flag polls (~128 ns apart)

struct PipeArgs {
    int n, nb, R, G, nchunk, stages, stage_bytes, maxU, maxBlk, B, run_stride;
    int k0, steps;     // steps k0 .. k0+steps-1 (k = 0 computes T_1 = X T_0)
    const int4 *hdr;   // per group: {nu, tb0, nbk, rec_off}, {rec_len, -, nruns, nr}
    const int4 *runs;  // run_stride per group: {first block row, rows, first slot, 0}
    const int32_t *rec;
    const int32_t *nbr_ptr, *nbr;  // neighbouring groups of each group (itself included)
    const float *x32;
    float *T0, *T1;    // step k reads T_k from (k even ? T0 : T1) and writes T_{k+1} to the other
    float2 *partial;   // [steps][G][B][2] pairs; step k writes block k - k0
    int32_t *flags;    // [G * nchunk] completed steps per tile (multi-step launch), or null
    int32_t *err;
    const PipeBatchTile *tiles;  // batched form: the tile list (slab and partial offsets per tile)
    int ntiles;
    // symmetric half (kSymRows > 0)
    const int32_t *symtiles;  // runs of computed tiles: (chunks - 1) << 29 | first chunk << 16 | group,
    const int32_t *symstart;  // CTA b's from symstart[b] to symstart[b + 1]
    int symlog, symsplit;     // a run has 2^symlog chunks, from chunk symsplit on one
    const int2 *mirror;       // per block column: the chunks (of the row) whose mirror tile is not computed
                              // start at .x; a mirrored copy is needed up to .y
    const int64_t *rowoff;    // per set of a run's chunks: index of block row 0 in a step's row sums
    float2 *rowpart;          // row sums of the step, 8 pairs per (set of chunks, block row)
    uint32_t flag_spin;  // neighbour-flag polls before a wait gives up (kFlagSpin unless a test lowers it)
    int stall_tile;      // test knob: this tile never publishes its step flags (-1: none)
};

__device__ __forceinline__ uint32_t sm_addr(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(sm_addr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(sm_addr(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(sm_addr(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n"
        " .reg .pred p;\n"
        " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(sm_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// global -> shared bulk copy; both addresses 16-byte aligned, bytes % 16 == 0
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
            sm_addr(dst)),
        "l"(src), "r"(bytes), "r"(sm_addr(bar))
        : "memory");
}

__device__ __forceinline__ int ld_acquire(const int32_t *p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release(int32_t *p, int v)
{
    asm volatile("st.release.gpu.global.b32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory");
}

// orders generic-proxy accesses to global memory with the bulk (async-proxy)
// copies that follow
__device__ __forceinline__ void fence_proxy_async_global()
{
    asm volatile("fence.proxy.async.global;\n" ::: "memory");
}

// Poll until the phase of the given parity completes; false on abort or
// after kPipeSpin polls (then the abort and device error flags are raised).
// Each lane polls on its own; lanes may leave on an abort at different polls,
// so a caller uses it only where a lane's answer governs that lane's own work.
__device__ __forceinline__ bool wait_phase(uint64_t *bar, uint32_t parity, volatile int *s_abort,
                                           int32_t *err)
{
    uint32_t n = 0;
    while (!mbar_try_wait(bar, parity)) {
        if (*s_abort) return false;
        if (++n >= kPipeSpin) {
            *s_abort = 1;
            atomicExch(err, 1);
            return false;
        }
    }
    return true;
}

// wait_phase with the warp's answer: every lane of the warp calls it and all
// get the same result, so a warp never splits over an abort.  For the
// producer (its copy issue is one warp-wide step), the publisher and the
// publisher hand-off.
__device__ __forceinline__ bool wait_phase_warp(uint64_t *bar, uint32_t parity, volatile int *s_abort,
                                                int32_t *err)
{
    return __all_sync(0xffffffffu, wait_phase(bar, parity, s_abort, err));
}

// The consumers' wait for tile i's stage (per lane, like wait_phase).  A tile
// the producer issued is always waited for (its bulk copies must land before
// the stage is refilled or the CTA exits), abort or not; a tile the producer
// never issued (*s_issued: -1 while it runs, then the count it issued) is
// given up, and so is every later one (gave_up): once a lane has passed over
// a phase that never completed, a later poll of that stage could name a
// parity that an older, completed phase had, and try_wait would report a
// never-filled stage as full.  Until then no phase was skipped, so a poll
// that succeeds is the tile's own phase.  Every lane reaches the same verdict
// (a never-issued tile never completes, an issued one always does).  The
// issue count is looked at once every 64 unsuccessful polls, keeping the
// common path to the poll alone.  Bounded by kPipeSpin polls like every wait.
__device__ __forceinline__ bool wait_full(uint64_t *bar, uint32_t parity, int i, volatile int *s_abort,
                                          volatile int *s_issued, int32_t *err, bool &gave_up)
{
    if (gave_up) return false;
    uint32_t n = 0;
    while (!mbar_try_wait(bar, parity)) {
        if ((++n & 63u) == 0u) {
            const int iss = *s_issued;
            if (iss >= 0 && i >= iss) {
                gave_up = true;
                return false;
            }
        }
        if (n >= kPipeSpin) {
            *s_abort = 1;
            atomicExch(err, 1);
            gave_up = true;
            return false;
        }
    }
    return true;
}

// Producer warp: the flag word lane q watches for tile (chunk, g): neighbour
// q of g (q < 32), or null.
__device__ __forceinline__ const int32_t *neighbour_flag(const PipeArgs &a, int chunk, int g, int q)
{
    const int p0 = a.nbr_ptr[g], p1 = a.nbr_ptr[g + 1];
    return p0 + q < p1 ? a.flags + (int64_t)chunk * a.G + a.nbr[p0 + q] : nullptr;
}

// Producer warp: wait until every neighbour tile of (chunk, g) has published
// step k.  seen: this lane's flag as read (acquire) before the stage wait, so
// that an already satisfied wait costs no further round trip.  Otherwise the
// lanes poll the neighbours in parallel with acquire loads; false on abort /
// timeout.
__device__ __forceinline__ bool wait_neighbours(const PipeArgs &a, int chunk, int g, int k, int lane, int seen,
                                                volatile int *s_abort)
{
    const int p0 = a.nbr_ptr[g], p1 = a.nbr_ptr[g + 1];
    const int32_t *fl = a.flags + (int64_t)chunk * a.G;
    if (p1 - p0 <= 32 && __all_sync(0xffffffffu, seen >= k)) return true;
    for (int base = p0; base < p1; base += 32) {
        const int q = base + lane;
        const int32_t *f = q < p1 ? fl + a.nbr[q] : nullptr;
        uint32_t n = 0;
        while (!__all_sync(0xffffffffu, f == nullptr || ld_acquire(f) >= k)) {
            if (__any_sync(0xffffffffu, *s_abort != 0)) return false;
            if (++n >= a.flag_spin) {
                if (lane == 0) {
                    *s_abort = 1;
                    atomicExch(a.err, 2);
                }
                __syncwarp();
                return false;
            }
            __nanosleep(128);
        }
    }
    return true;
}

// Tile of this CTA's i-th task.  One-launch-per-step launches sweep the
// tiles backwards on odd steps, so a step starts on the rows of T_{k+1} and
// T_k that the previous step touched last and that are still in L2.
template <bool kMulti>
__device__ __forceinline__ int tile_of_task(const PipeArgs &a, int ntiles, int i, int mine)
{
    const int t = (int)blockIdx.x + (i % mine) * (int)gridDim.x;
    const int k = a.k0 + i / mine;
    return (!kMulti && (k & 1)) ? ntiles - 1 - t : t;
}

// Tiles of the symmetric half, in the CTA's order: runs of up to 2^a.symlog
// chunks of one row group, so that the row sums (warp_pairs8, a fifth of a
// tile's instructions) are reduced once a run.  A step goes through them
// forwards or backwards, from the tiles that the step before touched last.
struct SymCursor {
    int run, end, dir, sub, word;
    __device__ void load(const PipeArgs &a) { word = run != end ? __ldg(a.symtiles + run) : -1; }
    __device__ void start(const PipeArgs &a)
    {
        const int b = __ldg(a.symstart + blockIdx.x), e = __ldg(a.symstart + blockIdx.x + 1);
        dir = a.k0 & 1 ? -1 : 1;
        run = dir > 0 ? b : e - 1;
        end = dir > 0 ? e : b - 1;
        sub = 0;
        load(a);
    }
    __device__ void next(const PipeArgs &a)
    {
        if (++sub <= (int)((unsigned)word >> 29)) return;
        sub = 0;
        run += dir;
        load(a);
    }
    __device__ bool valid() const { return word != -1; }
    __device__ int group() const { return word & 0xffff; }
    __device__ int first() const { return (word >> 16) & 0x1fff; }
    __device__ int chunk() const { return first() + sub; }
    __device__ int set(const PipeArgs &a) const  // of its chunks, in the row sums
    {
        return first() < a.symsplit ? first() >> a.symlog : (a.symsplit >> a.symlog) + first() - a.symsplit;
    }
};

// Sum over the warp of 8 (hi, lo) values a lane, packed by twos, halving the
// values a lane carries.  Lanes 4v .. 4v + 3 end with value v.
__device__ __forceinline__ float2 warp_pairs8(const float2 (&rh)[4], const float2 (&rl)[4], int lane)
{
    float h[8], l[8];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        h[2 * i] = rh[i].x;
        h[2 * i + 1] = rh[i].y;
        l[2 * i] = rl[i].x;
        l[2 * i + 1] = rl[i].y;
    }
#pragma unroll
    for (int s = 0; s < 5; s++) {
        const int off = 16 >> s, half = s < 3 ? 4 >> s : 1;
        const bool up = s < 3 && (lane & off);
#pragma unroll
        for (int i = 0; i < half; i++) {
            const float sh = s >= 3 || up ? h[i] : h[i + half], sl = s >= 3 || up ? l[i] : l[i + half];
            const float gh = __shfl_xor_sync(0xffffffffu, sh, off), gl = __shfl_xor_sync(0xffffffffu, sl, off);
            if (up) {
                h[i] = h[i + half];
                l[i] = l[i + half];
            }
            pair_add(h[i], l[i], gh);
            l[i] += gl;
        }
    }
    return make_float2(h[0], l[0]);
}

// (h, l) += x for |x| <= |h| on both components: the rounding error of h + x is
// then x - ((h + x) - h), in two operations less than TwoSum.  The row sums are
// kept so from kRowBase on where every sum of squares is at most one (and every
// <T_k,T_{k+1}> between minus one and one): h stays between two and four, its
// last place 2^-22, and l holds what lies below to 2^-44.
constexpr float kRowBase = 3.f;

__device__ __forceinline__ void based_add2(float2 &h, float2 &l, float2 x)
{
    const float2 m1 = make_float2(-1.f, -1.f);
    const float2 t = __fadd2_rn(h, x);
    l = __fadd2_rn(l, __ffma2_rn(m1, __ffma2_rn(m1, h, t), x));
    h = t;
}

// kBatch: tiles come from a.tiles (row groups of many structures, each
// structure its own chunk-major slabs and partial block); else tile t is
// (chunk t / G, group t % G) of one slab.  kMulti: the one-launch-per-slab
// mode (step flags, neighbour waits, the publisher warp); the per-step and
// batched instantiations carry none of that code.
//
// kSymRows > 0: one slab of all columns, of which only the tiles from the diagonal
// down are computed (a.symtiles): T_k is symmetric, so an element above them
// is the mirror image of a computed one.  Half the copies, products and
// stores.  Two things come from the mirror: the rows above the computed tiles
// that a computed tile references (a frontier of a few per cent: the lane that
// computes T[a][r] also stores it as T[r][a], at its own place, where the next
// step's copies find it), and the column sums' share above (the row sums of
// the computed tiles, over the columns whose mirror is not computed).  One
// density of the 20736-orbital cell at M = 400: 164.6 ms over the whole slab
// (0.94 of HBM), 93.3 ms over the half (0.82 of HBM; 111 ms while the row sums
// were reduced tile by tile).
//
// The row sums are pairs like the column sums: two products of a lane in FP32,
// then an addition that keeps its error, chunk by chunk.  Shared memory, HBM and
// the instructions are all near their limits here, so it shows: 90.0 ms with 32
// products in plain FP32 before the first pair, 93.3 with based_add2, 95.8 with
// TwoSum; 99.9 and 102 with a third block row's sums in registers.  So kSymRows
// is 2 for groups of up to 2 kPipeCW block rows and 3 beyond, and kUnit
// (based_add2) is for Gershgorin's interval, where T_k is bounded by one; on a
// caller's interval it may grow.
template <bool kBatch, bool kMulti, int kSymRows = 0, bool kUnit = false>
__global__ void __launch_bounds__(kPipeThreads, 1) k_cheb_f32_pipe(const PipeArgs a)
{
    constexpr bool kSym = kSymRows > 0;
    extern __shared__ __align__(128) unsigned char smem[];
    // [CW][2][32][4]: consumer warp w, lane l, column 2l + h at ((2w + h) 32 + l) 4,
    // holding (<T_k,T_k> hi, lo, <T_k,T_{k+1}> hi, lo); each 16-byte store of a
    // warp covers 512 contiguous bytes (no bank conflict)
    float *red = reinterpret_cast<float *>(smem + (size_t)a.stages * a.stage_bytes);
    uint64_t *full = reinterpret_cast<uint64_t *>(red + kPipeCW * kPipeCols * 4);
    uint64_t *empty = full + a.stages;
    uint64_t *pub = empty + a.stages;       // consumers -> publisher: tile done
    uint64_t *pubfree = pub + kPubSlots;    // publisher -> consumers: slot free again
    uint64_t *redfull = pubfree + kPubSlots;  // consumer warps -> reducers: red[] holds the tile's sums
    uint64_t *redfree = redfull + 1;          // reducers -> consumer warps: red[] read
    volatile int *s_abort = reinterpret_cast<volatile int *>(redfree + 1);
    volatile int *s_issued = s_abort + 1;  // tiles the producer issued, -1 while it runs
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < a.stages; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kPipeCW);
        }
        for (int s = 0; s < kPubSlots; s++) {
            mbar_init(&pub[s], 1);
            mbar_init(&pubfree[s], 1);
        }
        mbar_init(redfull, kPipeCW);
        mbar_init(redfree, kRedWarps);
        *s_abort = 0;
        *s_issued = -1;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    const int ntiles = kBatch || kSym ? a.ntiles : a.G * a.nchunk;
    const int mine = ntiles > (int)blockIdx.x ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int total = mine * a.steps;  // this CTA's tiles over all steps, step-major
    const int oT = 0, oP = a.maxU * 4 * kPipeCols, oX = oP + a.R * 4 * kPipeCols,
              oRec = oX + a.maxBlk * 16;  // float offsets inside a stage
    const int64_t chunk_floats = (int64_t)a.n * kPipeCols;

    if (warp == kPipeCW + 1) {
        // ---------------- publisher ----------------
        // Publishes each finished tile's step count: a GPU-scope fence makes
        // the consumers' T_{k+1} stores (ordered before the slot's mbarrier
        // arrival) visible before the release store of the flag.  The fence
        // stalls only this warp.
        if constexpr (!kMulti) return;
        for (int i = 0; i < total; ++i) {
            const int s = i % kPubSlots;
            if (!wait_phase_warp(&pub[s], (uint32_t)(i / kPubSlots) & 1u, s_abort, a.err)) break;
            if (lane == 0) {
                const int k = a.k0 + i / mine;
                const int t = tile_of_task<kMulti>(a, ntiles, i, mine);
                __threadfence();
                fence_proxy_async_global();
                if (t != a.stall_tile) st_release(a.flags + t, k + 1);
                mbar_arrive(&pubfree[s]);
            }
            __syncwarp();
        }
        return;
    }

    if (warp == kPipeCW) {
        // ---------------- producer ----------------
        int i = 0;
        int4 ha = make_int4(0, 0, 0, 0), hb = ha, run = ha;
        int gnext = 0;          // group of the next tile
        int64_t cnext = 0;      // batched form and symmetric half: its chunk offset
        SymCursor sym{0, 0, 0, 0, -1};
        if constexpr (kSym) sym.start(a);
        bool more = kSym ? sym.valid() : total > 0;
        if (more) {
            if constexpr (kBatch) {
                const int t0 = tile_of_task<kMulti>(a, ntiles, 0, mine);
                gnext = a.tiles[t0].g;
                cnext = a.tiles[t0].coff;
            } else if constexpr (kSym) {
                gnext = sym.group();
                cnext = sym.chunk() * chunk_floats;
            } else {
                gnext = tile_of_task<kMulti>(a, ntiles, 0, mine) % a.G;
            }
            ha = __ldg(a.hdr + 2 * gnext);
            hb = __ldg(a.hdr + 2 * gnext + 1);
            run = __ldg(a.runs + (int64_t)gnext * a.run_stride + lane);
        }
        if constexpr (kSym) {
            chain_release();
            chain_wait();
            fence_proxy_async_global();
        }
        int s = 0, lap = 0;  // i % stages, i / stages
        for (; more; ++i) {
            const int k = kSym ? a.k0 : a.k0 + i / mine;
            const int t = kSym ? 0 : tile_of_task<kMulti>(a, ntiles, i, mine);
            const int g = gnext;
            const int chunk = kBatch || kSym ? 0 : t / a.G;
            const int64_t coff = kBatch || kSym ? cnext : (int64_t)chunk * chunk_floats;
            const int nu = ha.x, tb0 = ha.y, nbk = ha.z, r0 = ha.w;
            const int rl = hb.x, I0 = hb.y, nruns = hb.z, nr = hb.w;
            const int4 cur = run;
            if constexpr (kSym) sym.next(a);
            more = kSym ? sym.valid() : i + 1 < total;
            if (more) {  // header and runs of the next tile
                const int tn = kSym ? 0 : tile_of_task<kMulti>(a, ntiles, i + 1, mine);
                if constexpr (kBatch) {
                    gnext = a.tiles[tn].g;
                    cnext = a.tiles[tn].coff;
                } else if constexpr (kSym) {
                    gnext = sym.group();
                    cnext = sym.chunk() * chunk_floats;
                } else {
                    gnext = tn % a.G;
                }
                ha = __ldg(a.hdr + 2 * gnext);
                hb = __ldg(a.hdr + 2 * gnext + 1);
                run = __ldg(a.runs + (int64_t)gnext * a.run_stride + lane);
            }
            // this tile's neighbour flags, read before the stage wait
            int seen = 0x7fffffff;
            if (kMulti && k > 0) {
                const int32_t *f = neighbour_flag(a, chunk, g, lane);
                if (f) seen = ld_acquire(f);
            }
            if (lap > 0 && !wait_phase_warp(&empty[s], (uint32_t)(lap - 1) & 1u, s_abort, a.err)) break;
            if (kMulti && k > 0) {
                if (!wait_neighbours(a, chunk, g, k, lane, seen, s_abort)) break;
                fence_proxy_async_global();
            }
            const float *Tin = (k & 1) ? a.T1 : a.T0;
            const float *Tprev = (k & 1) ? a.T0 : a.T1;
            float *stg = reinterpret_cast<float *>(smem + (size_t)s * a.stage_bytes);
            if (lane == 0)
                mbar_arrive_expect_tx(&full[s], (uint32_t)nu * 1024u + (k == 0 ? 0u : (uint32_t)nr * 1024u) +
                                                    (uint32_t)nbk * 64u + (uint32_t)rl * 4u);
            __syncwarp();
            const float *srcT = Tin + coff;
            if (lane < nruns)
                bulk_g2s(stg + oT + cur.z * 4 * kPipeCols, srcT + (int64_t)cur.x * 4 * kPipeCols,
                         (uint32_t)cur.y * 1024u, &full[s]);
            for (int q = lane + 32; q < nruns; q += 32) {
                const int4 rr = __ldg(a.runs + (int64_t)g * a.run_stride + q);
                bulk_g2s(stg + oT + rr.z * 4 * kPipeCols, srcT + (int64_t)rr.x * 4 * kPipeCols,
                         (uint32_t)rr.y * 1024u, &full[s]);
            }
            if (lane == 0) {
                bulk_g2s(stg + oX, a.x32 + (int64_t)tb0 * 16, (uint32_t)nbk * 64u, &full[s]);
                bulk_g2s(stg + oRec, a.rec + r0, (uint32_t)rl * 4u, &full[s]);
                if (k > 0)
                    bulk_g2s(stg + oP, Tprev + coff + (int64_t)I0 * 4 * kPipeCols, (uint32_t)nr * 1024u, &full[s]);
            }
            if (++s == a.stages) {
                s = 0;
                lap++;
            }
        }
        // the consumers wait for every tile issued (i of them) and give up the rest
        __syncwarp();
        if (lane == 0) {
            __threadfence_block();
            *s_issued = i;
        }
        if (*s_abort) {
            // let the copies already issued land before the CTA exits
            for (int j = max(0, i - a.stages); j < i; j++) {
                uint32_t n = 0;
                while (!mbar_try_wait(&full[j % a.stages], (uint32_t)(j / a.stages) & 1u) && ++n < kPipeSpin) {
                }
            }
        }
        return;
    }

    // ---------------- consumers ----------------
    const int c = 2 * lane;
    bool gave_up = false;  // this warp has passed over a tile that was never issued
    // batched form: the next tile's descriptor and group header, loaded one
    // tile ahead so that their latency overlaps the current tile
    PipeBatchTile bt_next{};
    int4 hb_next = make_int4(0, 0, 0, 0);
    if (kBatch && total > 0) {
        bt_next = a.tiles[tile_of_task<kMulti>(a, ntiles, 0, mine)];
        hb_next = __ldg(a.hdr + 2 * bt_next.g + 1);
    }
    // symmetric half: the next tile and its mirror bounds, likewise
    SymCursor sym{0, 0, 0, 0, -1};
    int2 mir_next = make_int2(0, 0);
    // of the warp's block rows, over the run's chunks so far: row q's <T_k,T_k>
    // and <T_k,T_{k+1}> over the lane's columns, as (hi, lo) pairs
    float2 rowh[kSym ? kSymRows : 1][4], rowl[kSym ? kSymRows : 1][4];
    uint32_t seen = 0;  // rows that have any
    if constexpr (kSym) {
        sym.start(a);
        if (sym.valid()) mir_next = __ldg(a.mirror + sym.chunk() * (kPipeCols / 4) + (lane >> 1));
        chain_wait();
    }
    bool more = kSym ? sym.valid() : total > 0;
    int s = -1, lap = 0;  // i % stages, i / stages
    for (int i = 0; more; ++i) {
        if (++s == a.stages) {
            s = 0;
            lap++;
        }
        const int k = kSym ? a.k0 : a.k0 + i / mine;
        const int t = kSym ? 0 : tile_of_task<kMulti>(a, ntiles, i, mine);
        int g, I0, nr;
        int64_t coff, pbase;  // slab offset of the tile's chunk; float2 offset of its column sums
        if constexpr (kBatch) {
            const PipeBatchTile bt = bt_next;
            const int4 hb = hb_next;
            if (i + 1 < total) {
                bt_next = a.tiles[tile_of_task<kMulti>(a, ntiles, i + 1, mine)];
                hb_next = __ldg(a.hdr + 2 * bt_next.g + 1);
            }
            g = bt.g;
            coff = bt.coff;
            pbase = bt.pbase;
            I0 = hb.y;
            nr = hb.w;
        } else if constexpr (kSym) {
            g = sym.group();
            I0 = g * a.R;
            nr = min(a.nb, I0 + a.R) - I0;
            coff = sym.chunk() * chunk_floats;
            pbase = ((int64_t)g * a.B + sym.chunk() * kPipeCols) * 2;
        } else {
            const int chunk = t / a.G;
            g = t - chunk * a.G;
            I0 = g * a.R;
            nr = min(a.nb, I0 + a.R) - I0;
            coff = (int64_t)chunk * chunk_floats;
            pbase = (((int64_t)(k - a.k0) * a.G + g) * a.B + chunk * kPipeCols) * 2;
        }
        const int2 mir = mir_next;
        const int rchunk = sym.chunk(), rset = sym.set(a);  // this tile's chunk of columns, its run's place
        bool run_ends = false;
        if constexpr (kSym) {
            if (sym.sub == 0) {
                seen = 0;
#pragma unroll
                for (int u = 0; u < kSymRows; u++)
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        rowh[u][q] = kUnit ? make_float2(kRowBase, kRowBase) : make_float2(0.f, 0.f);
                        rowl[u][q] = make_float2(0.f, 0.f);
                    }
            }
            sym.next(a);
            run_ends = sym.sub == 0;
            if (sym.valid()) mir_next = __ldg(a.mirror + sym.chunk() * (kPipeCols / 4) + (lane >> 1));
        }
        more = kSym ? sym.valid() : i + 1 < total;
        float *out = ((k & 1) ? a.T0 : a.T1) + coff + (int64_t)I0 * 4 * kPipeCols + c;
        // pairs (hi, lo), packed over columns (c, c+1): <T_k,T_k> in (eh, el),
        // <T_k,T_{k+1}> in (oh, ol)
        float2 eh = make_float2(0.f, 0.f), el = eh, oh = eh, ol = eh;
        if (wait_full(&full[s], (uint32_t)lap & 1u, i, s_abort, s_issued, a.err, gave_up)) {
            const float *stg = reinterpret_cast<const float *>(smem + (size_t)s * a.stage_bytes);
            const float *sT = stg + oT, *sP = stg + oP, *sX = stg + oX;
            const int32_t *sRp = reinterpret_cast<const int32_t *>(stg + oRec);
            const int32_t *sLc = sRp + nr + 1;
            const int32_t *sLs = sLc + sRp[nr];
            auto block_row = [&](int r, int u) {  // u: r's place among the warp's rows
                // acc[q] = row q of the block row, columns (c, c+1)
                float2 acc[4];
#pragma unroll
                for (int q = 0; q < 4; q++) acc[q] = make_float2(0.f, 0.f);
                const int ta = sRp[r], te = sRp[r + 1];
                for (int tt = ta; tt < te; tt++) {
                    const float *tv = sT + sLc[tt] * 4 * kPipeCols + c;
                    const float4 *xb = reinterpret_cast<const float4 *>(sX + tt * 16);
                    float2 v[4];
#pragma unroll
                    for (int m = 0; m < 4; m++) v[m] = *reinterpret_cast<const float2 *>(tv + m * kPipeCols);
                    block_fma2(acc, xb, v);
                }
                const float *own = sT + sLs[r] * 4 * kPipeCols + c;
                float2 ee = make_float2(0.f, 0.f), eo = ee, ow[4];
                const int ca = (int)((unsigned)(I0 + r) / (kPipeCols / 4));  // the chunk of columns that row block I0 + r heads
                const bool above = kSym && ca >= mir.x;     // the mirror tile is not computed
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const float2 ov = *reinterpret_cast<const float2 *>(own + q * kPipeCols);
                    float2 o = acc[q];
                    if (k > 0) o = cheb_next2(acc[q], *reinterpret_cast<const float2 *>(sP + (r * 4 + q) * kPipeCols + c));
                    *reinterpret_cast<float2 *>(out + (r * 4 + q) * kPipeCols) = o;
                    ee = __ffma2_rn(ov, ov, ee);
                    eo = __ffma2_rn(ov, o, eo);
                    if constexpr (kSym) {
                        ow[q] = ov;
                        acc[q] = o;
                    }
                }
                if constexpr (kSym) {
                    if (above) {
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const float2 ov = ow[q], o = acc[q],
                                         x = make_float2(fmaf(ov.x, ov.x, ov.y * ov.y), fmaf(ov.x, o.x, ov.y * o.y));
                            if (kUnit)
                                based_add2(rowh[u][q], rowl[u][q], x);
                            else
                                pair_add2(rowh[u][q], rowl[u][q], x);
                        }
                    }
                    if (above && ca <= mir.y) {
                        // T[4 a + q][c], q = 0..3, as row c's columns 4 a + q: one 16-byte store a column
                        float *m = ((k & 1) ? a.T0 : a.T1) + (int64_t)ca * chunk_floats +
                                   ((int64_t)rchunk * kPipeCols + c) * kPipeCols +
                                   ((unsigned)(I0 + r) % (kPipeCols / 4)) * 4;
                        *reinterpret_cast<float4 *>(m) = make_float4(acc[0].x, acc[1].x, acc[2].x, acc[3].x);
                        *reinterpret_cast<float4 *>(m + kPipeCols) = make_float4(acc[0].y, acc[1].y, acc[2].y, acc[3].y);
                    }
                    if (__any_sync(0xffffffffu, above)) seen |= 1u << u;
                    if (run_ends && (seen >> u & 1u)) {
                        if (kUnit)
#pragma unroll
                            for (int q = 0; q < 4; q++) {  // exact
                                rowh[u][q].x -= kRowBase;
                                rowh[u][q].y -= kRowBase;
                            }
                        const float2 s = warp_pairs8(rowh[u], rowl[u], lane);
                        if ((lane & 3) == 0)
                            a.rowpart[(__ldg(a.rowoff + rset) + I0 + r) * 8 + (lane >> 2)] = s;
                    }
                }
                pair_add2(eh, el, ee);
                pair_add2(oh, ol, eo);
            };
            if constexpr (kSym) {
#pragma unroll
                for (int u = 0; u < kSymRows; u++)  // at most kSymRows kPipeCW rows a group
                    if (warp + u * kPipeCW < nr) block_row(warp + u * kPipeCW, u);
            } else {
                for (int r = warp; r < nr; r += kPipeCW) block_row(r, 0);
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);  // stage s may be refilled
        // Hand this warp's sums over in red[warp]; the buffer is free again once
        // the previous tile's reducers have read it.  Neither phase below can
        // complete twice before it is polled: the next phase of redfull needs
        // this tile's redfree, and the next phase of redfree needs this warp's
        // arrival on redfull.
        if (i == 0 || wait_phase(redfree, (uint32_t)(i - 1) & 1u, s_abort, a.err)) {
            float4 *rb = reinterpret_cast<float4 *>(red + ((size_t)(2 * warp) * 32 + lane) * 4);
            rb[0] = make_float4(eh.x, el.x, oh.x, ol.x);   // column c
            rb[32] = make_float4(eh.y, el.y, oh.y, ol.y);  // column c + 1
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(redfull);  // after this warp's T_{k+1} stores of the tile
        const int rw = warp - kRedWarps * (i % (kPipeCW / kRedWarps));
        if (rw >= 0 && rw < kRedWarps) {
            // this tile's reducers: (column, which) pairs summed over the
            // consumer warps in warp order
            if (wait_phase(redfull, (uint32_t)i & 1u, s_abort, a.err)) {
                // reducer lane q reads float2 q of every warp's [2][32][4] block:
                // half h = q / 64, consumer lane l, sum `which` (consecutive lanes,
                // consecutive addresses); its column is j = 2 l + h
                const int q = rw * 32 + lane, h = q >> 6, l = (q & 63) >> 1, which = q & 1, j = 2 * l + h;
                float hsum = 0.f, lsum = 0.f;
#pragma unroll
                for (int w = 0; w < kPipeCW; w++) {
                    const float2 v = *reinterpret_cast<const float2 *>(red + (size_t)w * 256 + 2 * q);
                    pair_add(hsum, lsum, v.x);
                    lsum += v.y;
                }
                a.partial[pbase + j * 2 + which] = make_float2(hsum, lsum);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(redfree);
            // the first reducer hands the tile to the publisher: it has seen every
            // consumer warp's arrival, so all stores of the tile precede this
            if (kMulti && rw == 0) {
                const int ps = i % kPubSlots;
                if (i < kPubSlots ||
                    wait_phase_warp(&pubfree[ps], (uint32_t)((i / kPubSlots) - 1) & 1u, s_abort, a.err)) {
                    if (lane == 0) mbar_arrive(&pub[ps]);
                }
            }
        }
    }
}

// Identity columns c0 .. c0+B-1 in the chunk-major layout [B/64][n][64].
__global__ void k_slab_identity_cm(float *__restrict__ T0, int n, int B, int c0)
{
    const int64_t tot = (int64_t)n * B, per = (int64_t)n * kPipeCols;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
        const int chunk = (int)(e / per);
        const int64_t rem = e - (int64_t)chunk * per;
        const int row = (int)(rem / kPipeCols), j = (int)(rem % kPipeCols);
        T0[e] = (row == c0 + chunk * kPipeCols + j) ? 1.f : 0.f;
    }
}

// Sum of (hi, lo) pairs over groups g = 0 .. G-1 at p[g * stride], in group
// order, eight 16-byte loads in flight before their additions.
__device__ __forceinline__ void sum_group_pairs(const float4 *__restrict__ p, int64_t stride, int G, float &eh,
                                                float &el, float &oh, float &ol)
{
    int g = 0;
    for (; g + 8 <= G; g += 8) {
        float4 v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) v[u] = __ldg(p + (g + u) * stride);
#pragma unroll
        for (int u = 0; u < 8; u++) {
            pair_add(eh, el, v[u].x);
            el += v[u].y;
            pair_add(oh, ol, v[u].z);
            ol += v[u].w;
        }
    }
    for (; g < G; g++) {
        const float4 v = __ldg(p + g * stride);
        pair_add(eh, el, v.x);
        el += v.y;
        pair_add(oh, ol, v.z);
        ol += v.w;
    }
}

// The symmetric half's moments: column j's sums over the computed groups (from
// g0 of its chunk on) and, for its share above them, the row sums of block row
// j / 4 over the runs of chunks that have some of it.
__global__ void k_f32_finalize_sym(const float2 *__restrict__ partial, const float2 *__restrict__ rowpart, int64_t rowtot,
                                   const int64_t *__restrict__ rowoff, const int2 *__restrict__ span, int K, int G, int B,
                                   int n, const float *__restrict__ xdiag32, double *__restrict__ d, int M)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
    if (j >= n || k >= K) return;
    const int2 s = span[j >> 2];  // first computed group of the column, runs with row sums of the row
    float eh = 0.f, el = 0.f, oh = 0.f, ol = 0.f;
    const float4 *p = reinterpret_cast<const float4 *>(partial + (int64_t)k * G * B * 2) + j;
    sum_group_pairs(p + (int64_t)s.x * B, B, G - s.x, eh, el, oh, ol);
    const float4 *r = reinterpret_cast<const float4 *>(rowpart + (int64_t)k * rowtot * 8);
    int c = 0;
    for (; c + 8 <= s.y; c += 8) {
        float4 v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) v[u] = __ldg(r + (rowoff[c + u] + (j >> 2)) * 4 + (j & 3));
#pragma unroll
        for (int u = 0; u < 8; u++) {
            pair_add(eh, el, v[u].x);
            el += v[u].y;
            pair_add(oh, ol, v[u].z);
            ol += v[u].w;
        }
    }
    for (; c < s.y; c++) {
        const float4 v = __ldg(r + (rowoff[c] + (j >> 2)) * 4 + (j & 3));
        pair_add(eh, el, v.x);
        el += v.y;
        pair_add(oh, ol, v.z);
        ol += v.w;
    }
    const double se = (double)eh + (double)el, so = (double)oh + (double)ol;
    if (2 * k <= M) d[(int64_t)(2 * k) * n + j] = 2.0 * se - 1.0;
    if (2 * k + 1 <= M) d[(int64_t)(2 * k + 1) * n + j] = 2.0 * so - (double)xdiag32[j];
}

// Sum the per-group (hi, lo) pairs of a slab in FP32 pairs, convert once to
// FP64 and form the moments d[2k][j] = 2 <T_k,T_k>_j - 1,
// d[2k+1][j] = 2 <T_k,T_{k+1}>_j - X_jj.
__global__ void k_f32_finalize_pairs(const float2 *__restrict__ partial, int K, int rowgroups, int B, int c0,
                                     int n, const float *__restrict__ xdiag32, double *__restrict__ d, int M)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int k = blockIdx.y;
    if (j >= B || k >= K) return;
    const int i = c0 + j;
    if (i >= n) return;
    float eh = 0.f, el = 0.f, oh = 0.f, ol = 0.f;
    // (e, o) of column j in group g: one 16-byte load at [g][B][2] float2
    const float4 *p = reinterpret_cast<const float4 *>(partial + (int64_t)k * rowgroups * B * 2) + j;
    sum_group_pairs(p, B, rowgroups, eh, el, oh, ol);
    const double se = (double)eh + (double)el, so = (double)oh + (double)ol;
    if (2 * k <= M) d[(int64_t)(2 * k) * n + i] = 2.0 * se - 1.0;
    if (2 * k + 1 <= M) d[(int64_t)(2 * k + 1) * n + i] = 2.0 * so - (double)xdiag32[i];
}

}  // namespace

size_t cheb_f32_pipe_stage_bytes(int R, int maxU, int maxBlk, int rec_cap)
{
    const size_t b = (size_t)(maxU + R) * 4 * kPipeCols * sizeof(float) + (size_t)maxBlk * 16 * sizeof(float) +
                     (size_t)rec_cap * sizeof(int32_t);
    return (b + 127) / 128 * 128;
}

size_t cheb_f32_pipe_smem(size_t stage_bytes, int stages)
{
    return (size_t)stages * stage_bytes + (size_t)kPipeCW * kPipeCols * 4 * sizeof(float) +
           (size_t)(2 * stages + 2 * kPubSlots + 2) * sizeof(uint64_t) + 16;
}

int cheb_f32_pipe_max_rows() { return kPipeCW * 3; }

int cheb_f32_pipe_configure(size_t smem, int *ctas_per_sm, bool batch)
{
    const void *fn = batch ? (const void *)k_cheb_f32_pipe<true, false> : (const void *)k_cheb_f32_pipe<false, false>;
    const int lim = smem_optin_max(fn);
    if ((int)smem > lim) return (int)cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
    if (e != cudaSuccess) return (int)e;
    if (!batch) {
        const void *fm = (const void *)k_cheb_f32_pipe<false, true>;
        if ((e = cudaFuncSetAttribute(fm, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin_max(fm))))
            return (int)e;
        for (const void *fs : {(const void *)k_cheb_f32_pipe<false, false, 2, true>,
                               (const void *)k_cheb_f32_pipe<false, false, 2, false>,
                               (const void *)k_cheb_f32_pipe<false, false, 3, false>})
            if ((e = cudaFuncSetAttribute(fs, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin_max(fs))))
                return (int)e;
    }
    *ctas_per_sm = 0;
    return (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, fn, kPipeThreads, smem);
}

void launch_f32_finalize_pairs(cudaStream_t st, const DevMatrix &m, const float2 *partial, int K, int rowgroups,
                               int B, int c0, double *d, int M)
{
    dim3 grid((B + 127) / 128, K);
    k_f32_finalize_pairs<<<grid, 128, 0, st>>>(partial, K, rowgroups, B, c0, m.n, m.xdiag32, d, M);
}

void launch_slab_identity_cm(cudaStream_t st, float *T0, int n, int B, int c0)
{
    const int64_t tot = (int64_t)n * B;
    const int blocks = (int)std::min<int64_t>((tot + 255) / 256, 152 * 16);
    k_slab_identity_cm<<<blocks, 256, 0, st>>>(T0, n, B, c0);
}

// Plan of the symmetric half.  With groups of R block rows and chunks of 16
// block columns, tile (group g, chunk c) is computed if the group reaches the
// chunk's first row or beyond, g >= 16 c / R; so the mirror (group r / R, chunk
// a / 16) of an element (row a, column r) is not computed from chunk
// lo = ceil(R (r / R + 1) / 16) of the row on, and row r there is needed by the
// groups that are computed and reference it, up to the last chunk computed for
// the furthest of them.
void pipe_sym_plan(int nb, int R, int grid, const int32_t *brow, const int32_t *bcol, PipeSymHost &out)
{
    constexpr int A = kPipeCols / 4;  // block columns a chunk
    const int G = (nb + R - 1) / R, nchunk = (nb + A - 1) / A;
    auto lo_of = [&](int r) { return (R * (r / R + 1) + A - 1) / A; };
    // Runs in the order of their chunks, each to the CTA with the least so far;
    // the last chunks, two tiles a CTA or so, go tile by tile and level them
    // (5760 orbitals, some 18 tiles a CTA: 7.2 ms in runs of four to the end).
    int64_t single = 0, tiles = 0;
    for (int c = 0; c < nchunk; c++) tiles += G - A * c / R;
    // longer runs where a CTA has many (M = 200, runs of four and eight chunks, ms:
    // 18 tiles a CTA 4.35, 4.61; 32: 7.37, 7.41; 35: 7.94, 8.34; 46: 10.26, 10.13;
    // 72: 15.6, 15.1; 232: 48.8, 47.2; runs of one and two took 1.16 and 1.05 of four's)
    out.log = tiles >= 40 * (int64_t)grid ? 3 : 2;
    const int len = 1 << out.log;
    int split = nchunk;
    while (split > 0 && single < 2 * grid) single += G - A * --split / R;
    out.split = split = split / len * len;
    std::vector<std::vector<int32_t>> runs(grid);
    std::vector<std::pair<int, int>> load(grid);  // a heap: tiles so far, CTA
    for (int b = 0; b < grid; b++) load[b] = {0, b};
    const auto less = std::greater<std::pair<int, int>>();
    for (int c = 0; c < nchunk; c += c < split ? len : 1)
        for (int g = A * c / R; g < G; g++) {
            int e = c + 1;  // the group's run ends at its last computed chunk
            while (c < split && e < c + len && A * e / R <= g) e++;
            std::pop_heap(load.begin(), load.end(), less);
            runs[load.back().second].push_back((int32_t)((uint32_t)(e - c - 1) << 29 | (uint32_t)c << 16 | (uint32_t)g));
            load.back().first += e - c;
            std::push_heap(load.begin(), load.end(), less);
        }
    out.tiles.clear();
    out.start.assign(1, 0);
    for (const auto &r : runs) {
        out.tiles.insert(out.tiles.end(), r.begin(), r.end());
        out.start.push_back((int32_t)out.tiles.size());
    }
    out.mirror.assign((size_t)nchunk * A * 2, 1 << 30);
    for (int r = 0; r < nb; r++) {
        int hi = -1;
        for (int t = brow[r]; t < brow[r + 1]; t++)  // the pattern is symmetric: the rows that reference r
            hi = std::max(hi, (R * (bcol[t] / R + 1) + A - 1) / A - 1);
        out.mirror[2 * (size_t)r] = lo_of(r);
        out.mirror[2 * (size_t)r + 1] = hi;
    }
    // row sums: a block per (run, row) with a column whose mirror is not
    // computed, i.e. for the rows of the chunks from lo of the run's first
    // column on
    const int nset = split / len + nchunk - split;
    auto first_of = [&](int q) { return q < split / len ? len * q : split + q - split / len; };
    out.rowoff.assign(nset, 0);
    out.span.assign((size_t)nb * 2, 0);
    int64_t tot = 0;
    for (int c = 0; c < nset; c++) {
        const int64_t first = std::min<int64_t>(nb, (int64_t)A * lo_of(A * first_of(c)));
        out.rowoff[c] = tot - first;
        tot += nb - first;
    }
    out.rowtot = tot;
    int rows = 0;
    for (int a = 0; a < nb; a++) {
        while (rows < nset && lo_of(A * first_of(rows)) <= a / A) rows++;
        out.span[2 * (size_t)a] = A * (a / A) / R;
        out.span[2 * (size_t)a + 1] = rows;
    }
}

void launch_cheb_f32_sym(cudaStream_t st, const DevMatrix &m, const PipePlan &pl, float *T0, float *T1, int B, int k,
                         bool unit, float2 *partial, float2 *rowpart)
{
    PipeArgs a{};
    a.n = m.n;
    a.nb = m.nb;
    a.R = pl.R;
    a.G = pl.G;
    a.nchunk = B / kPipeCols;
    a.stages = pl.stages;
    a.stage_bytes = (int)pl.stage_bytes;
    a.maxU = pl.maxU;
    a.maxBlk = pl.maxBlk;
    a.B = B;
    a.run_stride = pl.run_stride;
    a.k0 = k;
    a.steps = 1;
    a.hdr = reinterpret_cast<const int4 *>(pl.hdr);
    a.runs = reinterpret_cast<const int4 *>(pl.runs);
    a.rec = pl.rec;
    a.x32 = m.x32;
    a.T0 = T0;
    a.T1 = T1;
    a.partial = partial;
    a.err = pl.err;
    a.symtiles = pl.symtiles;
    a.symstart = pl.symstart;
    a.symlog = pl.symlog;
    a.symsplit = pl.symsplit;
    a.mirror = reinterpret_cast<const int2 *>(pl.mirror);
    a.rowoff = pl.rowoff;
    a.rowpart = rowpart;
    a.flag_spin = kFlagSpin;
    a.stall_tile = -1;
    auto fn = k_cheb_f32_pipe<false, false, 3, false>;
    if (pl.R <= 2 * kPipeCW) fn = unit ? k_cheb_f32_pipe<false, false, 2, true> : k_cheb_f32_pipe<false, false, 2, false>;
    launch_chained(fn, dim3(pl.nsm), kPipeThreads, cheb_f32_pipe_smem(pl.stage_bytes, pl.stages), st, a);
}

void launch_f32_finalize_sym(cudaStream_t st, const DevMatrix &m, const PipePlan &pl, const float2 *partial,
                             const float2 *rowpart, int K, int B, double *d, int M)
{
    k_f32_finalize_sym<<<dim3((m.n + 127) / 128, K), 128, 0, st>>>(partial, rowpart, pl.rowtot, pl.rowoff,
                                                                  reinterpret_cast<const int2 *>(pl.span), K, pl.G, B,
                                                                  m.n, m.xdiag32, d, M);
}

int launch_cheb_f32_pipe(cudaStream_t st, const DevMatrix &m, const PipePlan &pl, float *T0, float *T1, int B,
                         int k0, int steps, float2 *partial, bool multi)
{
    PipeArgs a{};
    a.n = m.n;
    a.nb = m.nb;
    a.R = pl.R;
    a.G = pl.G;
    a.nchunk = B / kPipeCols;
    a.stages = pl.stages;
    a.stage_bytes = (int)pl.stage_bytes;
    a.maxU = pl.maxU;
    a.maxBlk = pl.maxBlk;
    a.B = B;
    a.run_stride = pl.run_stride;
    a.k0 = k0;
    a.steps = steps;
    a.hdr = reinterpret_cast<const int4 *>(pl.hdr);
    a.runs = reinterpret_cast<const int4 *>(pl.runs);
    a.rec = pl.rec;
    a.nbr_ptr = pl.nbr_ptr;
    a.nbr = pl.nbr;
    a.x32 = m.x32;
    a.T0 = T0;
    a.T1 = T1;
    a.partial = partial;
    a.flags = multi ? pl.flags : nullptr;
    a.err = pl.err;
    a.tiles = nullptr;
    a.ntiles = 0;
    a.flag_spin = kFlagSpin;
    a.stall_tile = -1;
    if (multi) {
        if (const char *v = std::getenv("LARGETB_TEST_WAIT_LIMIT")) {
            const unsigned long x = std::strtoul(v, nullptr, 10);
            if (x > 0 && x < kFlagSpin) a.flag_spin = (uint32_t)x;
        }
        if (const char *v = std::getenv("LARGETB_TEST_STALL_TILE")) a.stall_tile = (int)std::strtol(v, nullptr, 10);
    }
    const int ntiles = pl.G * a.nchunk;
    const int grid = std::min(ntiles, pl.nsm);
    const size_t smem = cheb_f32_pipe_smem(pl.stage_bytes, pl.stages);
    if (!multi) {
        k_cheb_f32_pipe<false, false><<<grid, kPipeThreads, smem, st>>>(a);
        return (int)cudaSuccess;
    }
    cudaError_t e = cudaMemsetAsync(pl.flags, 0, sizeof(int32_t) * (size_t)ntiles, st);
    if (e != cudaSuccess) return (int)e;
    void *args[] = {&a};
    return (int)cudaLaunchCooperativeKernel((const void *)k_cheb_f32_pipe<false, true>, dim3(grid), dim3(kPipeThreads), args,
                                            smem, st);
}

void launch_cheb_f32_pipe_batch(cudaStream_t st, const PipePlan &pl, const PipeBatchTile *tiles, int ntiles,
                                const float *x32, float *T0, float *T1, int k, float2 *partial)
{
    PipeArgs a{};
    a.R = pl.R;
    a.G = pl.G;
    a.stages = pl.stages;
    a.stage_bytes = (int)pl.stage_bytes;
    a.maxU = pl.maxU;
    a.maxBlk = pl.maxBlk;
    a.run_stride = pl.run_stride;
    a.k0 = k;
    a.steps = 1;
    a.hdr = reinterpret_cast<const int4 *>(pl.hdr);
    a.runs = reinterpret_cast<const int4 *>(pl.runs);
    a.rec = pl.rec;
    a.x32 = x32;
    a.T0 = T0;
    a.T1 = T1;
    a.partial = partial;
    a.flags = nullptr;
    a.err = pl.err;
    a.tiles = tiles;
    a.ntiles = ntiles;
    a.flag_spin = kFlagSpin;
    a.stall_tile = -1;
    const int grid = std::min(ntiles, pl.nsm);
    if (grid < 1) return;
    k_cheb_f32_pipe<true, false><<<grid, kPipeThreads, cheb_f32_pipe_smem(pl.stage_bytes, pl.stages), st>>>(a);
}

}  // namespace tb
