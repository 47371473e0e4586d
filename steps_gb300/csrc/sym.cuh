// Shared pieces of the pairwise kernels (pair_sym.cu, pair_box.cu): the tile
// size, the argument block and the slabs of FP64 partial sums.
#pragma once

#include "common.cuh"
#include "context.cuh"

namespace steps {

constexpr int SYM_T = 128;                 // particles per tile
constexpr int SYM_WARPS = 4;               // per block; each works on its own
constexpr int SYM_THREADS = 32 * SYM_WARPS;
constexpr int SYM_R3_BLOCKS = 4;  // per SM asked of the register allocator: 128 registers a thread
constexpr int SYM_HALF = SYM_T / 2;
constexpr int SYM_NSUB = SYM_T / SUBTILE;  // 8 sub-tile boxes per tile

struct SymArgs {
    const float4 *pack, *resid, *meta, *sub;
    const float *eps;
    const uint32_t *idx;
    int njt;     // tiles that hold particles (arrays are padded to whole rows)
    int nrows;
    int G, C;    // granules per group, j chunks per group
    int step, tri;  // particles per group, triangular j slabs (sym_slab)
    int nitems;  // groups x C
    unsigned *counter;
    double *pi, *pj;  // partial sums [C][3][npad] and [groups][3][npad]
    size_t npad;
    float guard2;
};

// The split of a call. A group is `step` consecutive particles in curve order,
// made of granules: rows (64 NP particles, pair_sym.cu) or blocks (32,
// pair_box.cu). Particles of a granule get j-side sums from every group that
// begins before it.
struct SymPlan {
    int NP, ntiles, nrows, G, groups, C;  // G granules to a group
    int gran, step, tri;                  // particles per granule, per group; triangular j slabs
    size_t npad, doubles;                 // padded particles; partial sums
};

// The j slabs: slab A covers the padded particles from the start of its group
// on (tri; groups are whole tiles), or all of them (small sets, whose groups
// are parts of tiles). Particles in the slabs before A:
__host__ __device__ inline size_t sym_slab(int A, int step, int tri, size_t npad)
{
    return (size_t)A * npad - (tri ? (size_t)step * ((size_t)A * (A - 1) / 2) : 0);
}

// Bounds-checked builds: whether the padded particles [i0, i1) and [j0, j1) of
// item (A, ch), the i slab ch and the words of the j slab A that it writes lie
// in their arrays; the first that does not is recorded and the item is left out.
__device__ __forceinline__ bool check_item(int A, int groups, int ch, int C, long long i0, long long i1, long long j0,
                                           long long j1, int step, int tri, size_t npad, long long nj)
{
#ifdef STEPS_CHECK
    const long long slab = 3 * (long long)sym_slab(A, step, tri, npad), end = 3 * (long long)sym_slab(A + 1, step, tri, npad);
    const long long jlo = tri ? (long long)A * step : 0, jlen = (long long)npad - jlo;
    return check_span(A, A, groups, CK_I_TILE) && check_span(ch, ch, C, CK_CHUNK) &&
           (i0 >= i1 || check_span(i0, i1 - 1, (long long)npad, CK_I_TILE)) &&
           (j0 >= j1 || (check_span(j0, j1 - 1, nj, CK_J_TILE) && check_span(j0 - jlo, j1 - 1 - jlo, jlen, CK_J_TILE) &&
                         check_span(slab + j0 - jlo, slab + 2 * jlen + j1 - 1 - jlo, end, CK_SLOT)));
#else
    return true;
#endif
}

// Adds to a partial sum that only this thread writes: the first contribution
// is stored, later ones are added in the memory system, in program order, so
// the sum is deterministic.
__device__ __forceinline__ void add_slab(double *o, double v, bool first)
{
    if (first) *o = v;
    else asm volatile("red.global.add.f64 [%0], %1;" ::"l"(o), "d"(v) : "memory");
}

// pair_sym.cu: groups and chunks of a plan whose granules are set (groups that
// are whole tiles of `tile` particles get triangular slabs); the reduction of
// the slabs into F (perm: curve order to the caller's, NULL: the same).
bool sym_split(SymPlan &p, int tile = SYM_T);
void sym_reduce(const SymPlan &p, const double *part, const uint32_t *perm, int n, const double *x, const Background &bg,
                double *F);
bool box_plan(int n, SymPlan &p);
// pair_box.cu: whether a periodic call can take the pairwise kernel (its kind,
// and a correction table that is odd in the separation), and the launch.
bool box_supported(const KParams &kp, const Tables &tb);
// The same for FP64: a table that is odd to the last bits, or none.
bool fp64_odd(const KParams &kp, const Tables &tb);
void box_launch(const KParams &kp, const Tables &tb, const SymArgs &s);

}  // namespace steps
