// Device code of the R^3 pairwise kernel, shared by the single-set kernel
// (pair_sym.cu, which explains it) and the persistent ensemble (ensemble.cu).
#pragma once

#include "common.cuh"
#include "context.cuh"
#include "mixed.cuh"
#include "sym.cuh"

namespace steps {
namespace mixed {

template <bool COH>
__device__ __forceinline__ float4 ld_tile(const float4 *p)
{
    return COH ? __ldcg(p) : __ldg(p);
}

// A warp's shared memory; NP packed i pairs per lane.
template <int NP>
struct SymWarp {
    double acc[3][2 * NP][32];  // FP64 i sums; each entry is its lane's own
    float4 q[64];               // 32 j particles, stored twice in a row
    float jhalf[3][32];         // far path: j sums over the first half of a rotation, each its lane's own
    union {
        struct {
            float4 ql[64];  // near path: their residuals, softening lengths and ids
            float2 qe[64];
        };
        float half[3][2 * NP][32];  // far path: i sums over the tile's earlier j particles, each its lane's own
    };
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
template <bool COH>
__device__ __forceinline__ void quad_box(const float4 *sub, float4 &c, float4 &h, float &emax)
{
    float lo[3] = {3e38f, 3e38f, 3e38f}, hi[3] = {-3e38f, -3e38f, -3e38f};
    emax = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float4 s = ld_tile<COH>(sub + 2 * k), w = ld_tile<COH>(sub + 2 * k + 1);
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
template <bool COH>
__device__ __forceinline__ void frame_offset(const SymArgs &a, int J, int H, float *dO, float *eO)
{
    const float4 mJ = ld_tile<COH>(a.meta + 2 * J), mI = ld_tile<COH>(a.meta + 2 * (H >> 1));
    dO[0] = two_diff(mJ.x, mI.x, eO[0]);
    dO[1] = two_diff(mJ.y, mI.y, eO[1]);
    dO[2] = two_diff(mJ.z, mI.z, eO[2]);
}

// The group of 32 j particles in shared memory (lane l's own is entry l)
// against the slots 2h, 2h + 1 of this warp, pair by pair in double-float
// coordinates with the softening spline: the exact path of r3x2_tile, rotated
// like the far loop. Lane l starts at entry l and moves on by one entry a step.
// near = false runs the far arithmetic instead (a far slot pair of a group that
// has near ones). The i sums go to the FP64 accumulators, the j sums to
// (jx, jy, jz).
template <int NP, bool COH>
__device__ __forceinline__ void r3_slots(const SymArgs &a, SymWarp<NP> &sh, int H, int h, bool near,
                                         const float *dO, const float *eO, float &jx, float &jy, float &jz)
{
    const int lane = threadIdx.x & 31, nxt = (lane + 1) & 31;
    const size_t qi0 = (size_t)H * SYM_HALF + lane;
    float ph[2][3], pl[2][3], mi[2], ei[2], f[2][3];
    uint32_t ii[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const float4 p = ld_tile<COH>(a.pack + qi0 + 32 * k), l = ld_tile<COH>(a.resid + qi0 + 32 * k);
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
        const float4 q = sh.q[lane + s];
        if (near) {
            const float4 ql = sh.ql[lane + s];
            const float2 qe = sh.qe[lane + s];
            const float ej = qe.x;
            const uint32_t jid = __float_as_uint(qe.y);
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

// v added to two FP32 sums.
__device__ __forceinline__ void add_half(f2 v, float &a, float &b)
{
    float lo, hi;
    f2_unpack(v, lo, hi);
    a += lo;
    b += hi;
}

// Item (A, ch) of the R^3 pairwise kernel: the rows of group A against its chunk
// ch, by one warp. COH: tile data through L2 (other warps of the same launch
// rewrite it between the stages of an ensemble). SHORT: FP32 sums of at most 32
// terms on either side before partial sums are added (else 64 on the i side and
// 32 NP on the j side).
template <int NP, bool COH, bool SHORT>
__device__ __forceinline__ void sym_item(const SymArgs &a, SymWarp<NP> &sh, int A, int ch)
{
    constexpr unsigned BITS = (unsigned)((1ull << (8 * NP)) - 1), GROUP_BITS = 0x03030303u & BITS;
    const int lane = threadIdx.x & 31, nxt = (lane + 1) & 31;
    const int row0 = A * a.G, row1 = min(a.nrows, row0 + a.G);
    const int first = row0 * NP / 2, tiles = a.njt - first;
    const int J0 = first + (int)((long long)tiles * ch / a.C);
    const int J1 = first + (int)((long long)tiles * (ch + 1) / a.C);

    if (!check_item(A, div_up(a.nrows, a.G), ch, a.C, (long long)row0 * NP * SYM_HALF, (long long)row1 * NP * SYM_HALF,
                    (long long)J0 * SYM_T, (long long)J1 * SYM_T, a.step, 1, a.npad, (long long)a.njt * SYM_T))
        return;

    // this group's j slab: the padded particles from its first tile on
    const size_t jlo = (size_t)first * SYM_T, jlen = a.npad - jlo;
    double *pj = a.pj + 3 * sym_slab(A, a.step, 1, a.npad);

    for (int r = row0; r < row1; r++) {
        const int H0 = r * NP;  // this row's half tiles: H0 .. H0 + NP - 1
        const int Ja = max(J0, H0 / 2);
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
            for (int k = 0; k < 2 * NP; k++) sh.acc[c][k][lane] = 0.0;
        // lane l classifies slot pair l / 8 against sub-tile l % 8 of the j tile
        const int hl = min(lane >> 3, NP - 1);
        float4 wc, wh;
        float wemax;
        quad_box<COH>(a.sub + (size_t)(H0 + hl) * (SYM_NSUB / 2) * 2, wc, wh, wemax);

        for (int J = Ja; J < J1; ++J) {
            const float4 mJ = ld_tile<COH>(a.meta + 2 * J);
            unsigned near;
            {
                const float4 mI = ld_tile<COH>(a.meta + 2 * ((H0 + hl) >> 1));
                const float ox = mJ.x - mI.x, oy = mJ.y - mI.y, oz = mJ.z - mI.z;
                const float4 *sj = a.sub + ((size_t)J * SYM_NSUB + (lane & 7)) * 2;
                const float4 s = ld_tile<COH>(sj), hs = ld_tile<COH>(sj + 1);
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
                frame_offset<COH>(a, J, H0 + h, dO, eO);
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const size_t q = (size_t)H0 * SYM_HALF + (2 * h + k) * 32 + lane;
                    const float4 p = ld_tile<COH>(a.pack + q), l = ld_tile<COH>(a.resid + q);
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
            float4 nq = ld_tile<COH>(a.pack + qj);
            // FP32 i sums run over 64 j particles (SHORT: 32), the parts of a tile are
            // added in FP32, and the tile's sum goes to FP64 (in one sum over whole
            // tiles the median error at n = 2^20 was 3 % above the one-sided
            // kernel's).
#pragma unroll 1
            for (int g = 0; g < 4; g++) {
                if (SHORT ? g > 0 : g == 2)
#pragma unroll
                    for (int h = 0; h < NP; h++) {
                        if (SHORT && g > 1) {
                            add_half(AX[h], sh.half[0][2 * h][lane], sh.half[0][2 * h + 1][lane]);
                            add_half(AY[h], sh.half[1][2 * h][lane], sh.half[1][2 * h + 1][lane]);
                            add_half(AZ[h], sh.half[2][2 * h][lane], sh.half[2][2 * h + 1][lane]);
                        } else {
                            f2_unpack(AX[h], sh.half[0][2 * h][lane], sh.half[0][2 * h + 1][lane]);
                            f2_unpack(AY[h], sh.half[1][2 * h][lane], sh.half[1][2 * h + 1][lane]);
                            f2_unpack(AZ[h], sh.half[2][2 * h][lane], sh.half[2][2 * h + 1][lane]);
                        }
                        AX[h] = AY[h] = AZ[h] = 0ull;
                    }
                const float4 q0 = nq;
                if (g < 3) nq = ld_tile<COH>(a.pack + qj + (g + 1) * 32);
                if ((near >> (2 * g)) & GROUP_BITS) continue;  // some slot pair is near: below
                const int Hj = 2 * J + (g >> 1);
                if (Hj < H0) continue;  // an earlier row's
                const bool both = Hj >= H0 + NP;  // the row's own half tiles: one-sided
                __syncwarp();
                sh.q[lane] = sh.q[32 + lane] = q0;
                __syncwarp();
                f2 JX = 0ull, JY = 0ull, JZ = 0ull;
                auto step = [&](int s) {
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
                };
                auto jsum = [&](float *v) {
                    float lo, hi;
                    f2_unpack(JX, lo, hi);
                    v[0] = lo + hi;
                    f2_unpack(JY, lo, hi);
                    v[1] = lo + hi;
                    f2_unpack(JZ, lo, hi);
                    v[2] = lo + hi;
                };
                float v[3];
                if constexpr (SHORT) {
#pragma unroll 1
                    for (int s0 = 0; s0 < 32; s0 += 16) {
#pragma unroll
                        for (int s = 0; s < 16; s++) step(s0 + s);
                        jsum(v);
                        if (s0 == 0) {  // of j particle (lane + 16) mod 32
#pragma unroll
                            for (int c = 0; c < 3; c++) sh.jhalf[c][(lane + 16) & 31] = v[c];
                            JX = JY = JZ = 0ull;
                            __syncwarp();
                        }
                    }
#pragma unroll
                    for (int c = 0; c < 3; c++) v[c] += sh.jhalf[c][lane];
                } else {
#pragma unroll 16
                    for (int s = 0; s < 32; s++) step(s);
                    jsum(v);
                }
                if (both)
#pragma unroll
                    for (int c = 0; c < 3; c++) add_slab(oj + c * jlen + g * 32, (double)v[c], firstrow);
            }
#pragma unroll
            for (int h = 0; h < NP; h++) {
                float lo, hi;
                f2_unpack(AX[h], lo, hi);
                sh.acc[0][2 * h][lane] += (double)(sh.half[0][2 * h][lane] + lo);
                sh.acc[0][2 * h + 1][lane] += (double)(sh.half[0][2 * h + 1][lane] + hi);
                f2_unpack(AY[h], lo, hi);
                sh.acc[1][2 * h][lane] += (double)(sh.half[1][2 * h][lane] + lo);
                sh.acc[1][2 * h + 1][lane] += (double)(sh.half[1][2 * h + 1][lane] + hi);
                f2_unpack(AZ[h], lo, hi);
                sh.acc[2][2 * h][lane] += (double)(sh.half[2][2 * h][lane] + lo);
                sh.acc[2][2 * h + 1][lane] += (double)(sh.half[2][2 * h + 1][lane] + hi);
            }
            if (near)
#pragma unroll 1
                for (int g = 0; g < 4; g++) {
                    const unsigned nm = (near >> (2 * g)) & GROUP_BITS;
                    const int Hj = 2 * J + (g >> 1);
                    if (!nm || Hj < H0) continue;
                    const bool both = Hj >= H0 + NP;
                    {
                        const size_t q = qj + g * 32;
                        const float4 p = ld_tile<COH>(a.pack + q), l = ld_tile<COH>(a.resid + q);
                        const float2 ei = make_float2(__ldg(a.eps + q), __uint_as_float(__ldg(a.idx + q)));
                        __syncwarp();
                        sh.q[lane] = sh.q[32 + lane] = p;
                        sh.ql[lane] = sh.ql[32 + lane] = l;
                        sh.qe[lane] = sh.qe[32 + lane] = ei;
                        __syncwarp();
                    }
                    double jd[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
                    for (int h = 0; h < NP; h++) {
                        float dO[3], eO[3];
                        frame_offset<COH>(a, J, H0 + h, dO, eO);
                        float jx = 0.0f, jy = 0.0f, jz = 0.0f;
                        r3_slots<NP, COH>(a, sh, H0 + h, h, (nm >> (8 * h)) & 3u, dO, eO, jx, jy, jz);
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

}  // namespace mixed
}  // namespace steps
