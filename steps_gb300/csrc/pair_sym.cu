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
// kernel -> this one): n = 32,768: 628 (tuned 525) -> 421 us; 262,144:
// 28.3 -> 19.4 ms; 2^20: 404 -> 297 ms, the FMA pipe 77 % busy.
// Further warps per SM (fewer registers, NP = 2), scalar instead of packed
// sums, other unrollings and a single rotated sum instead of two all measured
// within 3 % or slower: the FMA pipe with its operand reads is the limit.
#include <algorithm>

#include "common.cuh"
#include "context.cuh"
#include "mixed.cuh"
#include "sym.cuh"


namespace steps {

namespace {

using namespace mixed;

// A warp's shared memory; NP packed i pairs per lane.
template <int NP>
struct SymWarp {
    double acc[3][2 * NP][32];  // FP64 i sums; each entry is its lane's own
    float4 q[64];               // 32 j particles, stored twice in a row
};

__device__ __forceinline__ f2 f2_shfl(f2 v, int src)
{
    float lo, hi;
    f2_unpack(v, lo, hi);
    lo = __shfl_sync(0xffffffffu, lo, src);
    hi = __shfl_sync(0xffffffffu, hi, src);
    return f2_pack(lo, hi);
}

// Box (centre, half extents) and largest softening of 64 consecutive i
// particles from their 4 sub-tile boxes, in their tile's frame.
__device__ __forceinline__ void quad_box(const float4 *sub, float4 &c, float4 &h, float &emax)
{
    float lo[3] = {3e38f, 3e38f, 3e38f}, hi[3] = {-3e38f, -3e38f, -3e38f};
    emax = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float4 s = __ldg(sub + 2 * k), w = __ldg(sub + 2 * k + 1);
        lo[0] = fminf(lo[0], s.x - w.x); hi[0] = fmaxf(hi[0], s.x + w.x);
        lo[1] = fminf(lo[1], s.y - w.y); hi[1] = fmaxf(hi[1], s.y + w.y);
        lo[2] = fminf(lo[2], s.z - w.z); hi[2] = fmaxf(hi[2], s.z + w.z);
        emax = fmaxf(emax, s.w);
    }
    float cc[3], hh[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        cc[d] = 0.5f * (lo[d] + hi[d]);
        hh[d] = fmaxf(hi[d] - cc[d], cc[d] - lo[d]) * 1.000001f + 1e-6f * fabsf(cc[d]);
    }
    c = make_float4(cc[0], cc[1], cc[2], 0.0f);
    h = make_float4(hh[0], hh[1], hh[2], 0.0f);
}

// The far loop's weights are r^-3 times either mass, so r^-3 itself must be a
// normal FP32 number: boxes further apart or nearer than these bounds take the
// near path, whose products start with a mass.
constexpr float SYM_FAR2_MAX = 1e23f, SYM_GAP2_MIN = 1e-24f;

// d_O + e_O = centre of tile J less the centre of half tile H's tile, exactly.
__device__ __forceinline__ void frame_offset(const SymArgs &a, int J, int H, float *dO, float *eO)
{
    const float4 mJ = __ldg(a.meta + 2 * J), mI = __ldg(a.meta + 2 * (H >> 1));
    dO[0] = two_diff(mJ.x, mI.x, eO[0]);
    dO[1] = two_diff(mJ.y, mI.y, eO[1]);
    dO[2] = two_diff(mJ.z, mI.z, eO[2]);
}

// One group of 32 j particles (lane l's own is j0 + l) against the slots 2h,
// 2h + 1 of this warp, pair by pair in double-float coordinates with the
// softening spline: the exact path of r3x2_tile, rotated like the far loop.
// near = false runs the far arithmetic instead (a far slot pair of a group
// that has near ones). The i sums go to the FP64 accumulators, the j sums to
// (jx, jy, jz).
template <int NP>
__device__ __forceinline__ void r3_slots(const SymArgs &a, SymWarp<NP> &sh, int H, int h, int J, int g, bool near,
                                         const float *dO, const float *eO, float &jx, float &jy, float &jz)
{
    const int lane = threadIdx.x & 31, nxt = (lane + 1) & 31;
    const size_t qi0 = (size_t)H * SYM_HALF + lane;
    const size_t qj0 = (size_t)J * SYM_T + g * 32;
    float ph[2][3], pl[2][3], mi[2], ei[2], f[2][3];
    uint32_t ii[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const float4 p = __ldg(a.pack + qi0 + 32 * k), l = __ldg(a.resid + qi0 + 32 * k);
        frame_split(p.x, l.x, dO[0], eO[0], ph[k][0], pl[k][0]);
        frame_split(p.y, l.y, dO[1], eO[1], ph[k][1], pl[k][1]);
        frame_split(p.z, l.z, dO[2], eO[2], ph[k][2], pl[k][2]);
        mi[k] = p.w;
        ei[k] = __ldg(a.eps + qi0 + 32 * k);
        ii[k] = __ldg(a.idx + qi0 + 32 * k);
        f[k][0] = f[k][1] = f[k][2] = 0.0f;
    }
#pragma unroll 1
    for (int s = 0; s < 32; s++) {
        const size_t qj = qj0 + ((lane + s) & 31);
        const float4 q = __ldg(a.pack + qj);
        if (near) {
            const float4 ql = __ldg(a.resid + qj);
            const float ej = __ldg(a.eps + qj);
            const uint32_t jid = __ldg(a.idx + qj);
#pragma unroll
            for (int k = 0; k < 2; k++) {
                // the self pair gets d = 0 exactly, padding (whose ids are equal too) weight 0
                const bool self = jid == ii[k], none = jid == PAD_J || ii[k] == PAD_J;
                const float dx = self ? 0.0f : (q.x - ph[k][0]) + (ql.x - pl[k][0]);
                const float dy = self ? 0.0f : (q.y - ph[k][1]) + (ql.y - pl[k][1]);
                const float dz = self ? 0.0f : (q.z - ph[k][2]) + (ql.z - pl[k][2]);
                const float b = ei[k] + ej;
                const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                const float ri = rsqrt_mufu(r2), ri2 = ri * ri;
                float wi = (q.w * ri) * ri2, wj = (mi[k] * ri) * ri2;
                if (r2 < b * b) {
                    const float w = spline_inner_f32(r2, b);
                    wi = w * q.w;
                    wj = w * mi[k];
                }
                if (none) wi = wj = 0.0f;
                f[k][0] = fmaf(wi, dx, f[k][0]);
                f[k][1] = fmaf(wi, dy, f[k][1]);
                f[k][2] = fmaf(wi, dz, f[k][2]);
                jx = fmaf(wj, dx, jx);
                jy = fmaf(wj, dy, jy);
                jz = fmaf(wj, dz, jz);
            }
        } else {
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const float dx = q.x - (ph[k][0] + pl[k][0]), dy = q.y - (ph[k][1] + pl[k][1]),
                            dz = q.z - (ph[k][2] + pl[k][2]);
                const float ri = rsqrt_mufu(fmaf(dx, dx, fmaf(dy, dy, dz * dz)));
                const float w = ri * ri * ri, wi = w * q.w, wj = w * mi[k];
                f[k][0] = fmaf(wi, dx, f[k][0]);
                f[k][1] = fmaf(wi, dy, f[k][1]);
                f[k][2] = fmaf(wi, dz, f[k][2]);
                jx = fmaf(wj, dx, jx);
                jy = fmaf(wj, dy, jy);
                jz = fmaf(wj, dz, jz);
            }
        }
        jx = __shfl_sync(0xffffffffu, jx, nxt);
        jy = __shfl_sync(0xffffffffu, jy, nxt);
        jz = __shfl_sync(0xffffffffu, jz, nxt);
    }
#pragma unroll
    for (int k = 0; k < 2; k++)
#pragma unroll
        for (int c = 0; c < 3; c++) sh.acc[c][2 * h + k][lane] += (double)f[k][c];
}

template <int NP>
__global__ void __launch_bounds__(SYM_THREADS, NP == 4 ? 4 : 6) k_sym_r3(SymArgs a)
{
    constexpr unsigned BITS = (unsigned)((1ull << (8 * NP)) - 1), GROUP_BITS = 0x03030303u & BITS;
    __shared__ __align__(16) SymWarp<NP> shw[SYM_WARPS];
    const int lane = threadIdx.x & 31, nxt = (lane + 1) & 31;
    SymWarp<NP> &sh = shw[threadIdx.x >> 5];

    for (;;) {
        int item = 0;
        if (lane == 0) item = (int)atomicAdd(a.counter, 1u);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= a.nitems) return;
        const int A = item / a.C, ch = item - A * a.C;
        const int row0 = A * a.G, row1 = min(a.nrows, row0 + a.G);
        const int first = row0 * NP / 2, tiles = a.njt - first;
        const int J0 = first + (int)((long long)tiles * ch / a.C);
        const int J1 = first + (int)((long long)tiles * (ch + 1) / a.C);

        // this group's j slab: the padded particles from its first tile on
        const size_t jlo = (size_t)first * SYM_T, jlen = a.npad - jlo;
        double *pj = a.pj + 3 * sym_slab(A, a.step, 1, a.npad);

        for (int r = row0; r < row1; r++) {
            int H0 = r * NP;  // this row's half tiles: H0 .. H0 + NP - 1
            STEPS_CHECK_IDX(H0, a.nrows * NP, CK_I_TILE);
            const int Ja = max(J0, H0 / 2);
#pragma unroll
            for (int c = 0; c < 3; c++)
#pragma unroll
                for (int k = 0; k < 2 * NP; k++) sh.acc[c][k][lane] = 0.0;
            // lane l classifies slot pair l / 8 against sub-tile l % 8 of the j tile
            const int hl = min(lane >> 3, NP - 1);
            float4 wc, wh;
            float wemax;
            quad_box(a.sub + (size_t)(H0 + hl) * (SYM_NSUB / 2) * 2, wc, wh, wemax);

            for (int J = Ja; J < J1; ++J) {
                const float4 mJ = __ldg(a.meta + 2 * J);
                unsigned near;
                {
                    const float4 mI = __ldg(a.meta + 2 * ((H0 + hl) >> 1));
                    const float ox = mJ.x - mI.x, oy = mJ.y - mI.y, oz = mJ.z - mI.z;
                    const float4 *sj = a.sub + ((size_t)J * SYM_NSUB + (lane & 7)) * 2;
                    const float4 s = __ldg(sj), hs = __ldg(sj + 1);
                    bool f = warp_full_sub(ox, oy, oz, s, hs, wc, wh, wemax, a.guard2);
                    const float ex = (ox - wc.x) + s.x, ey = (oy - wc.y) + s.y, ez = (oz - wc.z) + s.z;
                    const float gx = axis_gap(ex, wh.x, hs.x), gy = axis_gap(ey, wh.y, hs.y),
                                gz = axis_gap(ez, wh.z, hs.z);
                    const float fx = fabsf(ex) + wh.x + hs.x, fy = fabsf(ey) + wh.y + hs.y,
                                fz = fabsf(ez) + wh.z + hs.z;
                    f = f || !(fx * fx + fy * fy + fz * fz < SYM_FAR2_MAX) ||
                        !(gx * gx + gy * gy + gz * gz > SYM_GAP2_MIN);
                    near = __ballot_sync(0xffffffffu, f) & BITS;
                }
                // i positions in J's frame, two slots to a packed pair
                f2 PX[NP], PY[NP], PZ[NP], PM[NP], AX[NP], AY[NP], AZ[NP];
#pragma unroll
                for (int h = 0; h < NP; h++) {
                    float v[2][4], dO[3], eO[3];
                    frame_offset(a, J, H0 + h, dO, eO);
#pragma unroll
                    for (int k = 0; k < 2; k++) {
                        const size_t q = (size_t)H0 * SYM_HALF + (2 * h + k) * 32 + lane;
                        const float4 p = __ldg(a.pack + q), l = __ldg(a.resid + q);
                        v[k][0] = ((p.x - dO[0]) - eO[0]) + l.x;
                        v[k][1] = ((p.y - dO[1]) - eO[1]) + l.y;
                        v[k][2] = ((p.z - dO[2]) - eO[2]) + l.z;
                        v[k][3] = p.w;
                    }
                    PX[h] = f2_pack(v[0][0], v[1][0]);
                    PY[h] = f2_pack(v[0][1], v[1][1]);
                    PZ[h] = f2_pack(v[0][2], v[1][2]);
                    PM[h] = f2_pack(v[0][3], v[1][3]);
                    AX[h] = AY[h] = AZ[h] = 0ull;
                }
                const size_t qj = (size_t)J * SYM_T + lane;
                double *oj = pj + (qj - jlo);
                const bool firstrow = r == row0;
                float4 nq = __ldg(a.pack + qj);
#pragma unroll 1
                for (int g = 0; g < 4; g++) {
                    const float4 q0 = nq;
                    if (g < 3) nq = __ldg(a.pack + qj + (g + 1) * 32);
                    if ((near >> (2 * g)) & GROUP_BITS) continue;  // some slot pair is near: below
                    const int Hj = 2 * J + (g >> 1);
                    if (Hj < H0) continue;  // an earlier row's
                    const bool both = Hj >= H0 + NP;  // the row's own half tiles: one-sided
                    __syncwarp();
                    sh.q[lane] = sh.q[32 + lane] = q0;
                    __syncwarp();
                    f2 JX = 0ull, JY = 0ull, JZ = 0ull;
#pragma unroll 8
                    for (int s = 0; s < 32; s++) {
                        const float4 q = sh.q[lane + s];
                        const f2 qx = f2_bcast(q.x), qy = f2_bcast(q.y), qz = f2_bcast(q.z), qm = f2_bcast(q.w);
#pragma unroll
                        for (int h = 0; h < NP; h++) {
                            const f2 dx = f2_sub(qx, PX[h]), dy = f2_sub(qy, PY[h]), dz = f2_sub(qz, PZ[h]);
                            const f2 r2 = f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx)));
                            float r2a, r2b;
                            f2_unpack(r2, r2a, r2b);
                            const f2 ri = f2_pack(rsqrt_mufu(r2a), rsqrt_mufu(r2b));
                            const f2 ri3 = f2_mul(f2_mul(ri, ri), ri);
                            const f2 wi = f2_mul(ri3, qm), wj = f2_mul(ri3, PM[h]);
                            AX[h] = f2_fma(wi, dx, AX[h]);
                            AY[h] = f2_fma(wi, dy, AY[h]);
                            AZ[h] = f2_fma(wi, dz, AZ[h]);
                            JX = f2_fma(wj, dx, JX);
                            JY = f2_fma(wj, dy, JY);
                            JZ = f2_fma(wj, dz, JZ);
                        }
                        JX = f2_shfl(JX, nxt);
                        JY = f2_shfl(JY, nxt);
                        JZ = f2_shfl(JZ, nxt);
                    }
                    if (both) {
                        float v[3][2];
                        f2_unpack(JX, v[0][0], v[0][1]);
                        f2_unpack(JY, v[1][0], v[1][1]);
                        f2_unpack(JZ, v[2][0], v[2][1]);
#pragma unroll
                        for (int c = 0; c < 3; c++)
                            add_slab(oj + c * jlen + g * 32, (double)(v[c][0] + v[c][1]), firstrow);
                    }
                }
#pragma unroll
                for (int h = 0; h < NP; h++) {
                    float lo, hi;
                    f2_unpack(AX[h], lo, hi);
                    sh.acc[0][2 * h][lane] += (double)lo;
                    sh.acc[0][2 * h + 1][lane] += (double)hi;
                    f2_unpack(AY[h], lo, hi);
                    sh.acc[1][2 * h][lane] += (double)lo;
                    sh.acc[1][2 * h + 1][lane] += (double)hi;
                    f2_unpack(AZ[h], lo, hi);
                    sh.acc[2][2 * h][lane] += (double)lo;
                    sh.acc[2][2 * h + 1][lane] += (double)hi;
                }
                if (near)
#pragma unroll 1
                    for (int g = 0; g < 4; g++) {
                        const unsigned nm = (near >> (2 * g)) & GROUP_BITS;
                        const int Hj = 2 * J + (g >> 1);
                        if (!nm || Hj < H0) continue;
                        const bool both = Hj >= H0 + NP;
                        double jd[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
                        for (int h = 0; h < NP; h++) {
                            float dO[3], eO[3];
                            frame_offset(a, J, H0 + h, dO, eO);
                            float jx = 0.0f, jy = 0.0f, jz = 0.0f;
                            r3_slots(a, sh, H0 + h, h, J, g, (nm >> (8 * h)) & 3u, dO, eO, jx, jy, jz);
                            jd[0] += (double)jx;
                            jd[1] += (double)jy;
                            jd[2] += (double)jz;
                        }
                        if (both)
#pragma unroll
                            for (int c = 0; c < 3; c++) add_slab(oj + c * jlen + g * 32, jd[c], firstrow);
                    }
            }
#pragma unroll
            for (int k = 0; k < 2 * NP; k++)
#pragma unroll
                for (int c = 0; c < 3; c++)
                    a.pi[((size_t)ch * 3 + c) * a.npad + (size_t)H0 * SYM_HALF + k * 32 + lane] = sh.acc[c][k][lane];
        }
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
    const int ng = r > 0 ? (r - 1) / p.G + 1 : 0;
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

// Row width for n particles. Narrow rows
// give small sets enough warps, wide ones amortise the rotation (pair kernel,
// NP = 1 / 2 / 4: n = 32,768 439 / 421 / 456 us; 65,536 1566 / 1445 / 1400 us).
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
    if (kp.topology == STEPS_R3) return n >= SYM_MIN_N && sym_plan(n, p);
    return n >= BOX_MIN_N && box_plan(n, p) && box_supported(kp, tb);
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
