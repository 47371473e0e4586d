// Mixed-precision R^3 forces of all particles with every pair of particles
// evaluated once and added to both (Newton's third law).
//
// The one-sided kernels (pair_mixed.cu, pair_r3x2.cu) evaluate each pair
// twice, once from either side, at 12 FP32 FMA-pipe instructions, and are
// bound by that pipe. Once evaluated, a pair costs 16 (3 for d, 3 for r^2, 2
// for r^-3, and a weight and 3 accumulations for either particle): 8 a force
// contribution instead of 12. What makes the second accumulation cheap:
//
//   * A lane holds 2 NP i particles as NP packed FP32x2 pairs (a warp's row is
//     64 NP particles) and one j particle of 32 at a time. In step s lane l
//     works on j particle (l + s) mod 32 of the group, read from shared memory
//     (stored twice in a row, so the index never wraps), and the j sums move
//     one lane on after each step, so each is back in its own lane after 32:
//     6 shuffles and one LDS.128 for 2 NP pairs, beside the FMA pipe. Packing
//     two j to an instruction instead would need the i particles as broadcast
//     pairs (twice the registers) and rotate twice the sums.
//   * Warps work on their own, with no block-wide barrier: a block-row variant
//     whose 4 warps shared a j tile lost 15 % of its warps' time at barriers,
//     since near pairs make the warps' times uneven.
//
// Work: rows are gathered into groups of G. A group meets the j tiles from its
// own first tile on, cut into C chunks of equal length; an item is (group,
// chunk). Later groups have shorter chunks, so the queue runs from long items
// to short ones and ends evenly. With 64 x 64 items the last wave cost up to
// 40 % at n = 2^17; 256 x 128 is within 1 % of finer splits, whose partial
// sums cost the reduction more than they gain. A row's own particles are met
// one-sided (both orders of a pair occur there).
//
// Partial sums are FP64 slabs: one per chunk for the i side, one per group for
// the j side, the latter written by the one warp that owns the (group, chunk)
// part and added in row order; the reduction adds slabs in a fixed order.
// Results are deterministic.
//
// Near pairs (inside the softening support, or with FP32 offsets that are
// coarse for their distance) are found per (64 i, 16 j) box pair with the rule
// of the one-sided kernels and take the double-float path, after the far ones.
//
// Measured (GB300, clustered compactified sets, pair kernel, one-sided packed
// kernel -> this one): n = 32,768: 628 (tuned 525) -> 416 us; 262,144:
// 28.3 -> 19.0 ms; 2^20: 404 -> 291 ms, 16 instructions a pair at 77 % of the
// measured FMA issue rate (counted by ncu at 131,072: pipe 70 % active, 5.1 ms).
// Scalar instead of packed sums and a single rotated sum instead of two
// measured within 3 % or slower: the FMA pipe with its operand reads is the
// limit. 16 warps an SM with 128 registers a thread (NP = 2 fits, NP = 4 spills
// 12 bytes) do better than more:
// NP = 2, 6 blocks of 80 registers 433 us at n = 32,768 and 648 at 39,999, 5
// blocks 422 and 624, 4 blocks 416 and 613 (3: 449 and 650). The rotation is
// unrolled 16 times (8 / 16 / 32 times: NP = 2, n = 32,768 420 / 416 / 449 us;
// NP = 4, n = 262,144 19.37 / 19.02 / 25.1 ms).
#include <algorithm>

#include "common.cuh"
#include "context.cuh"
#include "mixed.cuh"
#include "sym.cuh"
#include "sym_r3.cuh"


namespace steps {

namespace {

using namespace mixed;

template <int NP>
__global__ void __launch_bounds__(SYM_THREADS, SYM_R3_BLOCKS) k_sym_r3(SymArgs a)
{
    __shared__ __align__(16) SymWarp<NP> shw[SYM_WARPS];
    const int lane = threadIdx.x & 31;
    for (;;) {
        int item = 0;
        if (lane == 0) item = (int)atomicAdd(a.counter, 1u);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= a.nitems) return;
        const int A = item / a.C;
        sym_item<NP, false, false>(a, shw[threadIdx.x >> 5], A, item - A * a.C);
    }
}

// F of one particle component: its chunk slabs in order, less the slabs of
// the groups that met it from the i side; then the background term, scattered
// to the caller's order. A block takes 32 particles; its 8 warps sum every 8th
// slab in order, and the first adds the 8 sums in order. The sums of a few
// hundred slabs are latency-bound with one thread per component at small n.
constexpr int RED_PARTS = 8;
__global__ void __launch_bounds__(32 * RED_PARTS) k_sym_reduce(const double *__restrict__ pi,
                                                               const double *__restrict__ pj, SymPlan p,
                                                               const uint32_t *__restrict__ perm, int count,
                                                               const double *__restrict__ x, Background bg,
                                                               double *__restrict__ F)
{
    __shared__ double part[RED_PARTS][3][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int q = blockIdx.x * 32 + lane;  // < npad
    double f[3] = {0.0, 0.0, 0.0};
#pragma unroll 4
    for (int s = w; s < p.C; s += RED_PARTS)
#pragma unroll
        for (int c = 0; c < 3; c++) f[c] += pi[((size_t)s * 3 + c) * p.npad + q];
    const int r = q / p.gran;  // met from the i side by the granules before its own
    int ng = r > 0 ? (r - 1) / p.G + 1 : 0;
    STEPS_CHECK_IDX(ng, p.groups + 1, CK_SLOT);
#pragma unroll 4
    for (int A = w; A < ng; A += RED_PARTS) {
        const size_t start = p.tri ? (size_t)A * p.step : 0, len = p.npad - start;
        const double *o = pj + 3 * sym_slab(A, p.step, p.tri, p.npad) + (q - start);
#pragma unroll
        for (int c = 0; c < 3; c++) f[c] -= o[c * len];
    }
#pragma unroll
    for (int c = 0; c < 3; c++) part[w][c][lane] = f[c];
    __syncthreads();
    if (w != 0 || q >= count) return;
#pragma unroll
    for (int v = 1; v < RED_PARTS; v++)
#pragma unroll
        for (int c = 0; c < 3; c++) f[c] += part[v][c][lane];
    long long o = perm ? (long long)perm[q] : q;
    STEPS_CHECK_IDX(o, count, CK_OUTPUT);
    add_background(bg, x + 3 * (size_t)o, f);
#pragma unroll
    for (int c = 0; c < 3; c++) F[3 * (size_t)o + c] = f[c];
}

}  // namespace

// Groups and chunks of a plan whose granules are set: at most 256 groups and
// 128 chunks, the slabs within the partial-sum budget.
bool sym_split(SymPlan &p, int tile)
{
    const long long slabs = std::max<long long>(SYM_PARTIAL_BYTES / (24 * (long long)p.npad), 1);
    p.G = div_up(p.nrows, (int)std::min<long long>(256, slabs));
    p.tri = (long long)p.gran * p.G % tile == 0;
    p.step = p.gran * p.G;
    p.groups = div_up(p.nrows, p.G);
    p.C = (int)std::min<long long>(std::min(128, p.ntiles), std::max<long long>(slabs / 2, 1));
    p.doubles = 3 * ((size_t)p.C * p.npad + sym_slab(p.groups, p.step, p.tri, p.npad));
    return slabs >= 160;
}

namespace {

// Row width for n particles. Narrow rows give small sets enough items, wide ones
// amortise the rotation (pair kernel and reduction, NP = 2 / 4: n = 48,000
// 0.894 / 0.911 ms; 72,000 1.821 / 1.883; 90,000 2.710 / 2.727; 110,000
// 3.897 / 3.867; 131,072 5.41 / 5.29).
bool sym_plan(int n, SymPlan &p)
{
    p.NP = n >= SYM_NP4_N ? 4 : 2;
    p.ntiles = div_up(n, SYM_T);
    p.nrows = div_up(2 * p.ntiles, p.NP);
    p.npad = (size_t)div_up(p.nrows * p.NP, 2) * SYM_T;
    p.gran = SYM_HALF * p.NP;
    return sym_split(p);
}

template <int NP>
void sym_launch(const SymArgs &a)
{
    Ctx &c = ctx();
    int occ = 0;
    STEPS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_sym_r3<NP>, SYM_THREADS, 0));
    const int grid = std::min(div_up(a.nitems, SYM_WARPS), c.nsm * std::max(occ, 1));
    k_sym_r3<NP><<<grid, SYM_THREADS, 0, c.stream>>>(a);
    note_launch("k_sym_r3");
}

}  // namespace

void sym_reduce(const SymPlan &p, const double *part, const uint32_t *perm, int n, const double *x, const Background &bg,
                double *F)
{
    k_sym_reduce<<<div_up(n, 32), 32 * RED_PARTS, 0, ctx().stream>>>(part, part + 3 * (size_t)p.C * p.npad, p, perm, n, x,
                                                                    bg, F);
    note_launch("k_sym_reduce");
}

bool sym_supported(const KParams &kp, const Tables &tb, int n)
{
    SymPlan p;
    const bool ok = kp.topology == STEPS_R3 ? n >= SYM_MIN_N && sym_plan(n, p)
                                            : n >= BOX_MIN_N && box_plan(n, p) && box_supported(kp, tb);
    return ok && ctx().partial.fits(p.doubles * sizeof(double));
}

void forces_sym(const KParams &kp, const Tables &tb, const double *x, const double *m64, const double *eps64, int n,
                double *F, bool reuse_order)
{
    Ctx &c = ctx();
    cudaStream_t st = c.stream;
    SymPlan p;
    const bool box = kp.topology != STEPS_R3;
    if (!(box ? box_plan(n, p) : sym_plan(n, p))) fail(STEPS_E_ARG, "pairwise kernel: too many particles");
    STEPS_CUDA(cudaEventRecord(c.phase[0], st));
    build_tiles(c.tj, x, m64, eps64, 0, n, SYM_T, reuse_order, st, c.bbox.ensure<unsigned long long>(8), PAD_J,
                (int)(p.npad / SYM_T));
    STEPS_CUDA(cudaEventRecord(c.phase[1], st));
    SymArgs a{};
    a.pack = c.tj.pack.as<float4>();
    a.resid = c.tj.resid.as<float4>();
    a.meta = c.tj.meta.as<float4>();
    a.sub = c.tj.sub.as<float4>();
    a.eps = c.tj.eps.as<float>();
    a.idx = c.tj.idx.as<uint32_t>();
    a.njt = p.ntiles;
    a.nrows = p.nrows;
    a.G = p.G;
    a.C = p.C;
    a.step = p.step;
    a.tri = p.tri;
    a.nitems = p.groups * p.C;
    a.counter = c.counter.ensure<unsigned>(4);
    a.npad = p.npad;
    a.pi = c.partial.ensure<double>(p.doubles);
    a.pj = a.pi + 3 * (size_t)p.C * p.npad;
    a.guard2 = c.shape.guard * c.shape.guard;
    STEPS_CUDA(cudaMemsetAsync(a.counter, 0, sizeof(unsigned), st));
    const Background bg = background_of(kp, tb);
    if (box) box_launch(kp, tb, a);
    else if (p.NP == 4) sym_launch<4>(a);
    else sym_launch<2>(a);
    STEPS_CUDA(cudaEventRecord(c.phase[2], st));
    sym_reduce(p, a.pi, c.tj.perm(), n, x, bg, F);
    STEPS_CUDA(cudaEventRecord(c.phase[3], st));
    c.phase_valid = true;
    c.last_pairs = (double)n * (double)n;
}

}  // namespace steps
