// Batched ensembles in one persistent kernel: the initial force evaluation and,
// per KDK step, the force at the drifted positions of every realisation, each
// pair of particles evaluated once (sym_r3.cuh).
//
// Warps take (stage, task) pairs from one counter, stage by stage. A stage's
// tasks are the pair items of every realisation, largest first -- (group,
// chunk), as in pair_sym.cu -- and then their finish tasks, 32 particles each. A
// finish task adds the slabs of its particles in order (deterministic), writes
// F, applies the kick of the step that the stage ends (StePS/src/step.cc:256-262),
// then the next step's kick and drift (step.cc:131-149); the last of a tile
// rebuilds it. Pair items of stage s wait for the finish tasks of stage s - 1 of
// their realisation, finish tasks for its pair items. Listed behind all pair
// items, finish tasks rarely wait, and the next stage begins with the
// realisation that was finished first (listed one realisation later instead,
// every warp ends up waiting for the few items of a realisation: 16.4 -> 15.9 ms
// for three stages of the set below). A task waits only for tasks taken before
// it, so the earliest unfinished one always progresses. Every wait is bounded (a
// second, more for very large items): one that gives up records STEPS_E_TIMEOUT,
// and every warp then stops taking tasks.
//
// Particles keep the order of the initial sort for the whole run (the forces do
// not depend on it). What other warps rewrite during the run (tile data,
// positions, velocities, slabs) is read through L2.
//
// FP32 sums are half as long as in pair_sym.cu (SHORT in sym_r3.cuh), and rows
// are 128 particles: against the one-sided kernel that this one replaced
// (tiles of 128; 24 sets of 4,736 to 27,000 particles, relative errors against
// FP64, median / 99th percentile: 2.55e-7 / 1.41e-6) the error was 4-7 % larger
// with the longer sums and 16-22 % with rows of 256; it is 2.36e-7 / 1.37e-6.
// The short sums cost 0.5 % (12 x 8,192 particles) to 1.5 % (3 x 20,000); rows
// of 256 were the slower ones at every size tried (500 to 250,000).
//
// Measured (12 realisations of 4,736 to 65,024 particles, 1 + 4 stages, 6.4e10
// ordered pairs): whole batch call with the data 34.9 ms with the one-sided
// kernel, 27.8 with this one; 4.8 ms a stage, 2.7e12 pairs/s, of which the
// finish tasks are 3 %. Four blocks an SM, as in pair_sym.cu: 24.1 ms for the run
// against 24.5 with 6 blocks.
#include <algorithm>

#include "context.cuh"
#include "ensemble.cuh"
#include "sym_r3.cuh"
#include "tile.cuh"

namespace steps {

namespace {

using namespace mixed;

// Bounded spin on a counter that other warps increment: true once it reaches
// target; false after `limit` cycles or as soon as the status word is set.
__device__ __forceinline__ bool wait_counter(const unsigned long long *cnt, unsigned long long target, long long limit,
                                             const int *status)
{
    const volatile unsigned long long *c = cnt;
    const volatile int *st = status;
    if (*c >= target) return true;
    const long long t0 = clock64();
    while (*c < target) {
        if (*st != 0 || clock64() - t0 > limit) return false;
        __nanosleep(200);
    }
    return true;
}

// Tile `tile` rebuilt by one warp from its particles' new positions: the
// arithmetic of build_tile (tile.cuh). Masses, softening and indices do not
// change.
__device__ __forceinline__ void rebuild_tile(const EnsembleArgs &e, int tile)
{
    const int lane = threadIdx.x & 31;
    double xn[4][3];
    bool valid[4];
#pragma unroll
    for (int r = 0; r < 4; r++) {
        uint32_t o = __ldg(e.idx + (size_t)tile * SYM_T + 32 * r + lane);
        valid[r] = o != PAD_J;
        if (valid[r]) STEPS_CHECK_IDX(o, e.n, CK_PERM);
#pragma unroll
        for (int k = 0; k < 3; k++) xn[r][k] = valid[r] ? __ldcg(e.x + 3 * (size_t)o + k) : 0.0;
    }
    float c[3], h[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        unsigned long long lo = ~0ull, nhi = ~0ull;
#pragma unroll
        for (int r = 0; r < 4; r++)
            if (valid[r]) extend_box(xn[r][k], lo, nhi);
        lo = warp_min(lo);
        nhi = warp_min(nhi);
        const bool some = lo <= ~nhi;  // else an empty tile
        const double mn = some ? from_ordered_bits(lo) : 0.0, mx = some ? from_ordered_bits(~nhi) : 0.0;
        c[k] = __double2float_rn(0.5 * (mn + mx));
        const double ext = fmax(mx - (double)c[k], (double)c[k] - mn);
        h[k] = __double2float_ru(ext * (1.0 + 1e-6)) + 1e-30f;
    }
    if (lane == 0) {
        const float emax = __ldcg(e.meta + 2 * tile).w;
        e.meta[2 * tile] = make_float4(c[0], c[1], c[2], emax);
        e.meta[2 * tile + 1] = make_float4(h[0], h[1], h[2], 0.0f);
    }
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const size_t q = (size_t)tile * SYM_T + 32 * r + lane;
        float p[3] = {0.0f, 0.0f, 0.0f}, l[3] = {0.0f, 0.0f, 0.0f};
        if (valid[r])
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const double o = xn[r][k] - (double)c[k];
                p[k] = __double2float_rn(o);
                l[k] = __double2float_rn(o - p[k]);
            }
        e.pack[q] = make_float4(p[0], p[1], p[2], __ldcg(e.pack + q).w);
        e.resid[q] = make_float4(l[0], l[1], l[2], 0.0f);
        // boxes of the SUBTILE particles of each half warp
        float lo[3], hi[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            lo[k] = hi[k] = p[k];
#pragma unroll
            for (int o = SUBTILE / 2; o > 0; o >>= 1) {
                lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
                hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
            }
        }
        if ((lane & (SUBTILE - 1)) == 0) {
            float cc[3], ww[3];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                cc[k] = 0.5f * (lo[k] + hi[k]);
                const float w = fmaxf(hi[k] - cc[k], cc[k] - lo[k]);
                ww[k] = w * 1.000001f + 1e-6f * (fabsf(cc[k]) + w) + 1e-30f;
            }
            float4 *d = e.sub + 2 * ((size_t)tile * SYM_NSUB + 2 * r + (lane >> 4));
            d[0] = make_float4(cc[0], cc[1], cc[2], __ldcg(d).w);
            d[1] = make_float4(ww[0], ww[1], ww[2], 0.0f);
        }
    }
}

// Finish task of 32 particles (block b of realisation k). The warp that ends the
// last of a tile's four blocks rebuilds the tile and counts it done. Not
// inlined: its registers would be taken from the pair loop.
__device__ __noinline__ void finish_block(const EnsembleArgs &e, int k, int b, int stage)
{
    const int lane = threadIdx.x & 31;
    const EnsRel R = e.rel[k];
    const bool kick2 = stage >= 1, kick1 = stage < e.nsteps;
    const double h2 = e.h / 2.0;
    const double *pi = e.part + R.part, *pj = pi + 3 * (size_t)R.C * R.npad;
    const int q = b * 32 + lane, tile = R.tile0 + (b >> 2);
    uint32_t o = __ldg(e.idx + (size_t)R.tile0 * SYM_T + q);
    const bool valid = o != PAD_J;
    if (valid) STEPS_CHECK_IDX(o, e.n, CK_PERM);
    double f[3] = {0.0, 0.0, 0.0};
#pragma unroll 8
    for (int s = 0; s < R.C; s++)
#pragma unroll
        for (int c = 0; c < 3; c++) f[c] += __ldcg(pi + ((size_t)s * 3 + c) * R.npad + q);
    const int row = q / SYM_T;
    int ng = row > 0 ? (row - 1) / R.G + 1 : 0;
    STEPS_CHECK_IDX(ng, R.npair / R.C + 1, CK_SLOT);
#pragma unroll 8
    for (int A = 0; A < ng; A++) {
        const size_t start = (size_t)A * R.step, len = R.npad - start;
        const double *p = pj + 3 * sym_slab(A, R.step, 1, R.npad) + (q - start);
#pragma unroll
        for (int c = 0; c < 3; c++) f[c] -= __ldcg(p + c * len);
    }
    if (valid)
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const size_t p = 3 * (size_t)o + c;
            e.F[p] = f[c];
            if (e.hold) continue;
            double vv = __ldcg(e.v + p);
            // acceleration g F a^-3 - 2 H v at g = 1, a = 1, H = 0, as the batch's KDK kernels evaluate it
            if (kick2) vv += (1.0 * f[c] * 1.0 - 2.0 * 0.0 * vv) * h2;
            if (kick1) {
                vv = vv + (1.0 * f[c] * 1.0 - 2.0 * 0.0 * vv) * h2;
                e.x[p] = __ldcg(e.x + p) + vv * e.h;
            }
            e.v[p] = vv;
        }
    __threadfence();
    __syncwarp();
    unsigned c = 0;
    if (lane == 0) c = atomicAdd(e.tile_cnt + tile, 1u);
    if ((__shfl_sync(0xffffffffu, c, 0) & 3u) != 3u) return;
    __threadfence();
    if (kick1) rebuild_tile(e, tile);
    __threadfence();
    __syncwarp();
    if (lane == 0 && !(stage == 0 && k == e.stall_rel)) atomicAdd(e.fin_done + k, 1ull);
}

__global__ void __launch_bounds__(SYM_THREADS, SYM_R3_BLOCKS) k_ensemble(EnsembleArgs e)
{
    __shared__ __align__(16) SymWarp<ENS_NP> shw[SYM_WARPS];
    __shared__ SymArgs sha[SYM_WARPS];  // each warp's item, out of the pair loop's registers
    const int lane = threadIdx.x & 31;
    SymArgs &a = sha[threadIdx.x >> 5];
    const long long total = (long long)e.ntasks * (e.nsteps + 1LL);
    for (;;) {
        int stage = -1, which = 0;
        if (lane == 0) {
            const volatile int *st = e.status;
            const long long task = *st != 0 ? total : (long long)atomicAdd(e.queue, 1ull);
            if (task < total) {
                stage = (int)(task / e.ntasks);
                which = (int)(task % e.ntasks);
                const int4 d = __ldg(e.tasks + which);
                const EnsRel *R = e.rel + d.x;
                const bool ok = d.w ? wait_counter(e.pair_done + d.x, __ldg(&R->npair) * (stage + 1ull), e.wait_cycles, e.status)
                                    : wait_counter(e.fin_done + d.x, __ldg(&R->ntiles) * (unsigned long long)stage,
                                                   e.wait_cycles, e.status);
                if (!ok) {
                    atomicExch(e.status, STEPS_E_TIMEOUT);
                    stage = -1;
                }
            }
            __threadfence();
        }
        stage = __shfl_sync(0xffffffffu, stage, 0);
        if (stage < 0) return;
        const int4 d = __ldg(e.tasks + __shfl_sync(0xffffffffu, which, 0));
        int k = d.x;
        STEPS_CHECK_IDX(k, e.nrel, CK_I_TILE);
        if (d.w) {
            finish_block(e, k, d.y, stage);
        } else {
            if (lane == 0) {
                const EnsRel R = e.rel[k];
                const size_t q0 = (size_t)R.tile0 * SYM_T;
                a.pack = e.pack + q0;
                a.resid = e.resid + q0;
                a.meta = e.meta + 2 * R.tile0;
                a.sub = e.sub + 2 * (size_t)R.tile0 * SYM_NSUB;
                a.eps = e.eps + q0;
                a.idx = e.idx + q0;
                a.njt = R.ntiles;
                a.nrows = R.ntiles;
                a.G = R.G;
                a.C = R.C;
                a.step = R.step;
                a.npad = R.npad;
                a.pi = e.part + R.part;
                a.pj = a.pi + 3 * (size_t)R.C * R.npad;
                a.guard2 = e.guard2;
            }
            __syncwarp();
            sym_item<ENS_NP, true, true>(a, shw[threadIdx.x >> 5], d.y, d.z);
            __threadfence();
            __syncwarp();
            if (lane == 0) atomicAdd(e.pair_done + k, 1ull);
        }
    }
}

}  // namespace

int ensemble_blocks()
{
    int occ = 0;
    STEPS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_ensemble, SYM_THREADS, 0));
    return std::max(occ, 1);
}

void ensemble_launch(const EnsembleArgs &e, cudaStream_t st)
{
    k_ensemble<<<ctx().nsm * ensemble_blocks(), SYM_THREADS, 0, st>>>(e);
    note_launch("k_ensemble");
}

}  // namespace steps
