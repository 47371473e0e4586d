// The persistent ensemble kernel (ensemble.cu): every force evaluation and KDK
// step of a batch of R^3 realisations in one launch.
#pragma once

#include "common.cuh"
#include "sym.cuh"

namespace steps {

constexpr int ENS_NP = 2;  // rows of 64 ENS_NP particles
static_assert(64 * ENS_NP == SYM_T, "a row of the ensemble kernel is a tile");

// One realisation: its tiles, the split of its pairs (SymPlan) and its slabs of
// partial sums.
struct EnsRel {
    int tile0, ntiles;  // first tile of the batch arrays; tiles (rows)
    int G, C, step;     // as in SymArgs / SymPlan
    int npair;          // pair tasks of a stage; finish tasks: 4 ntiles
    size_t npad;
    size_t part;                  // first double of its slabs
};

struct EnsembleArgs {
    const EnsRel *rel;
    const int4 *tasks;      // of one stage: (realisation, group, chunk, 0) or (realisation, 32 particles, 0, 1)
    int ntasks, nsteps, nrel;  // nsteps + 1 stages
    float4 *pack, *resid, *meta, *sub;
    const float *eps;       // softening (constant over the run)
    const uint32_t *idx;    // original index of each padded position (constant)
    double *part;
    // 64 bits: a stage of 64 realisations of 8,192 particles is up to 242,000
    // tasks, 2^31 of them fewer than 9,000 steps.
    unsigned long long *queue;                 // task counter, over all stages
    unsigned long long *pair_done, *fin_done;  // per realisation: items, tiles done, over all stages
    unsigned *tile_cnt;     // per tile: finish tasks done, over all stages, modulo 2^32 (read modulo 4)
    double *x, *v, *F;      // caller-order FP64 positions, velocities, forces
    bool hold;              // stages are evaluated and tiles rebuilt, x and v left as they are (timing)
    double h;               // fixed step; acceleration g F a^-3 - 2 H v with g = 1, a = 1, H = 0
    float guard2;
    int n;                  // particles of all realisations (bounds checks)
    long long wait_cycles;  // SM clock cycles after which a wait gives up
    int *status;            // STEPS_E_TIMEOUT when a wait gave up
    int stall_rel;          // test hook: this realisation's stage-0 tiles are never reported done (-1: none)
};

void ensemble_launch(const EnsembleArgs &e, cudaStream_t st);
int ensemble_blocks();  // resident blocks per SM

}  // namespace steps
