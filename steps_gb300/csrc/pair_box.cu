// Mixed-precision forces of all particles on T^3 and S1xR2 with every pair of
// particles evaluated once and added to both (Newton's third law): the
// periodic counterpart of pair_sym.cu, with its items, slabs and reduction.
//
// The table kernels are bound by the L1 path of their table gathers, the image
// sum by FP32 and MUFU issue, so evaluating a pair once halves what bounds
// them. The correction must be odd in the separation for that (for the (rho, z)
// table: D_rho even and D_z odd in z); the host checks the table.
//
// A warp evaluates blocks of 32 i x 32 j particles with 8 consecutive i times 4
// consecutive j across its lanes: lane (a, b) = (lane / 4, lane % 4) holds the
// i particles 8 A + a of the block for A = 0..3 and meets the j particles
// 4 B + b for B = 0..7. A gather of 32 such pairs touches fewer table records
// than one of 32 i against one j: counted on the T^3 workload, 13.7 distinct
// cells against 17.3 at n = 120,000 and 9.7 against 13.6 at 2^19 (24.7 and 19.8
// for the rotation of pair_sym.cu). The j sums of one or two B are added over
// the lanes of equal b (9 shuffles per 4 or 8 pairs); the i sums over the lanes of equal
// a once per j tile.
//
// Per block the kernel knows whether any pair can be near (the double-float
// path), which axes can cross half a period, whether the table's stencils stay
// inside its halo, and which images can lie inside the cut; one lane per block
// of a 128 x 128 tile pair works that out. Images outside the cut are left out
// rather than evaluated at a distance where they vanish.
#include <string.h>

#include <algorithm>

#include "common.cuh"
#include "context.cuh"
#include "mixed.cuh"
#include "sym.cuh"
#include "table.cuh"

namespace steps {

namespace {

using namespace mixed;

enum BoxKind { B_T3_NEAR = 0, B_T3_LIN, B_T3_CUB, B_S1_NEAR, B_S1_CIC, B_S1_TSC, B_S1_IMG };

constexpr bool is_t3(int K) { return K <= B_T3_CUB; }
constexpr int t3_order(int K) { return K == B_T3_LIN ? 2 : K == B_T3_CUB ? 4 : 0; }
constexpr int s1_order(int K) { return K == B_S1_CIC ? 2 : K == B_S1_TSC ? 4 : 0; }

struct BoxArgs {
    SymArgs s;
    MixedArgs t;  // periods, tolerances and tables
};

// Block flags, made by one lane and read by the warp.
constexpr unsigned F_WRAP = 7u;            // axes on which a pair can cross half a period
constexpr unsigned F_HALO = 8u;            // every stencil inside the table's halo
constexpr unsigned F_NEAR = 0x80000000u;   // double-float path
// Images: first and last inside or straddling the cut, and those entirely
// inside, as m + 64 in 7 bits each.
__device__ __forceinline__ unsigned pack_images(int m0, int m1, int i0, int i1)
{
    return (unsigned)(m0 + 64) | (unsigned)(m1 + 64) << 7 | (unsigned)(i0 + 64) << 14 | (unsigned)(i1 + 64) << 21;
}

// d_O + e_O: centre of tile J (its image nearest to I's) less that of tile I.
template <int K>
__device__ __forceinline__ void box_frame(const BoxArgs &a, int I, int J, float *dO, float *eO)
{
    const float4 mJ = __ldg(a.s.meta + 2 * J), mI = __ldg(a.s.meta + 2 * I);
    dO[0] = two_diff(mJ.x, mI.x, eO[0]);
    dO[1] = two_diff(mJ.y, mI.y, eO[1]);
    dO[2] = two_diff(mJ.z, mI.z, eO[2]);
    if (is_t3(K)) {
        shift_frame(dO[0], eO[0], a.t.L, a.t.L_lo);
        shift_frame(dO[1], eO[1], a.t.L, a.t.L_lo);
    }
    if (K != B_S1_IMG) shift_frame(dO[2], eO[2], a.t.L, a.t.L_lo);
}

// Box of 32 consecutive particles from their 2 sub-tile boxes: centre (largest
// softening in w) and half extents.
__device__ __forceinline__ void pair_box(const float4 *sub, float4 &c, float4 &h)
{
    const float4 s0 = __ldg(sub), w0 = __ldg(sub + 1), s1 = __ldg(sub + 2), w1 = __ldg(sub + 3);
    auto join = [](float c0, float h0, float c1, float h1, float &cc, float &hh) {
        const float lo = fminf(c0 - h0, c1 - h1), hi = fmaxf(c0 + h0, c1 + h1);
        cc = 0.5f * (lo + hi);
        hh = fmaxf(hi - cc, cc - lo) * 1.000001f + 1e-6f * fabsf(cc);
    };
    join(s0.x, w0.x, s1.x, w1.x, c.x, h.x);
    join(s0.y, w0.y, s1.y, w1.y, c.y, h.y);
    join(s0.z, w0.z, s1.z, w1.z, c.z, h.z);
    c.w = fmaxf(s0.w, s1.w);
    h.w = 0.0f;
}

// Flags of i block ib of tile I against j block g of tile J.
template <int K>
__device__ __forceinline__ unsigned classify(const BoxArgs &a, int I, int J, int ib, int g)
{
    float dO[3], eO[3];
    box_frame<K>(a, I, J, dO, eO);
    float4 ci, hi, cj, hj;
    pair_box(a.s.sub + ((size_t)I * SYM_NSUB + 2 * ib) * 2, ci, hi);
    pair_box(a.s.sub + ((size_t)J * SYM_NSUB + 2 * g) * 2, cj, hj);
    const float e[3] = {dO[0] - ci.x, dO[1] - ci.y, dO[2] - ci.z};
    const float d[3] = {e[0] + cj.x, e[1] + cj.y, e[2] + cj.z};
    // half extents of the i box, widened by the rounding of the box offset
    const float w[3] = {hi.x + 1e-6f * (fabsf(e[0]) + fabsf(cj.x) + fabsf(ci.x)),
                        hi.y + 1e-6f * (fabsf(e[1]) + fabsf(cj.y) + fabsf(ci.y)),
                        hi.z + 1e-6f * (fabsf(e[2]) + fabsf(cj.z) + fabsf(ci.z))};
    const float h[3] = {w[0] + hj.x, w[1] + hj.y, w[2] + hj.z};
    unsigned flags = 0;
    float g2 = 0.0f;
    if (K == B_S1_IMG) {
        const float gx = fmaxf(fabsf(d[0]) - h[0], 0.0f), gy = fmaxf(fabsf(d[1]) - h[1], 0.0f);
        const float g2xy = gx * gx + gy * gy, lo = d[2] - h[2], up = d[2] + h[2];
        const float cin = a.t.cutL * (1.0f - 1e-6f), cout = a.t.cutL * (1.0f + 1e-6f);
        int m0 = 1, m1 = 0, i0 = 1, i1 = 0;
        g2 = 3e38f;
        for (int m = -a.t.emax; m <= a.t.emax; m++) {
            const float sh = (float)m * a.t.L, l = lo + sh, u = up + sh;
            if (l > cout || u < -cout) continue;  // entirely outside the cut
            if (m0 > m1) m0 = m;
            m1 = m;
            if (fmaxf(fabsf(l), fabsf(u)) <= cin) {  // entirely inside
                if (i0 > i1) i0 = m;
                i1 = m;
            }
            const float gz = (l <= 0.0f && u >= 0.0f) ? 0.0f : fminf(fabsf(l), fabsf(u));
            g2 = fminf(g2, g2xy + gz * gz);
        }
        flags = pack_images(m0, m1, i0, i1);
    } else {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const bool periodic = is_t3(K) || c == 2;
            float ad = fabsf(d[c]);
            if (periodic) {
                if (ad + h[c] > a.t.halfL - a.t.wrap_tol) flags |= 1u << c;
                ad = fminf(ad, a.t.L - ad);
            }
            const float gc = fmaxf(ad - h[c], 0.0f);
            g2 += gc * gc;
        }
        if (t3_order(K)) {
            constexpr int NT = t3_order(K), OFF = NT == 4 ? 1 : 0;
            bool halo = true;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const int w0 = (int)floorf((d[c] - h[c]) * a.t.ih + a.t.u0 - 1e-3f) - OFF;
                const int w1 = (int)floorf((d[c] + h[c]) * a.t.ih + a.t.u0 + 1e-3f) - OFF + NT;
                halo = halo && w0 >= -a.t.halo && w1 <= a.t.ng + a.t.halo;
            }
            if (halo) flags |= F_HALO;
        }
    }
    const float bmax = ci.w + cj.w;
    const float sc = sqrtf(e[0] * e[0] + e[1] * e[1] + e[2] * e[2]) + sqrtf(w[0] * w[0] + w[1] * w[1] + w[2] * w[2]) +
                     sqrtf(cj.x * cj.x + cj.y * cj.y + cj.z * cj.z) + sqrtf(hj.x * hj.x + hj.y * hj.y + hj.z * hj.z);
    if (!(g2 > bmax * bmax * 1.0001f + 1e-30f) || !(sc * sc <= a.t.guard2 * g2)) flags |= F_NEAR;
    return flags;
}

// A pair as the exact decisions need it: position qi of tile I, qj of tile J.
struct PairAt {
    int I, J;
    size_t qi, qj;
};

// The nearest-image decision |d| > L/2 along axis c on the exact separation.
template <int K>
__device__ __noinline__ bool wraps_exactly(const BoxArgs &a, PairAt p, int c)
{
    float dO[3], eO[3], ph, pl;
    box_frame<K>(a, p.I, p.J, dO, eO);
    const float *x = reinterpret_cast<const float *>(a.s.pack + p.qi), *xl = reinterpret_cast<const float *>(a.s.resid + p.qi);
    const float *q = reinterpret_cast<const float *>(a.s.pack + p.qj), *ql = reinterpret_cast<const float *>(a.s.resid + p.qj);
    frame_split(x[c], xl[c], dO[c], eO[c], ph, pl);
    const float d = (q[c] - ph) + (ql[c] - pl);
    return nearest_image(d, q[c], ph, ql[c], pl, a.t.L, a.t.halfL, a.t.halfL_lo, a.t.wrap_tol) != d;
}

// The image cut |dz + sh| <= cutL on the exact separation.
__device__ __noinline__ bool in_cut_exactly(const BoxArgs &a, PairAt p, float sh)
{
    float dO[3], eO[3], ph, pl;
    box_frame<B_S1_IMG>(a, p.I, p.J, dO, eO);
    frame_split(a.s.pack[p.qi].z, a.s.resid[p.qi].z, dO[2], eO[2], ph, pl);
    return cut_in_exact(a.s.pack[p.qj].z, a.s.resid[p.qj].z, ph, pl, sh, a.t.cutL);
}

// d moved to the nearest image along axis c of a block that can wrap there.
template <int K>
__device__ __forceinline__ float wrap_far(const BoxArgs &a, float d, int c, const PairAt &p)
{
    const float ad = fabsf(d);
    bool w = ad > a.t.halfL;
    if (fabsf(ad - a.t.halfL) < a.t.wrap_tol) w = wraps_exactly<K>(a, p, c);
    return w ? d - copysignf(a.t.L, d) : d;
}

// Correction D of the separation d (unwrapped on T^3, nearest image on S1xR2),
// to be subtracted; zero for kinds without a table.
template <int K>
__device__ __forceinline__ void correction(const BoxArgs &a, unsigned flags, float dx, float dy, float dz, float rho2,
                                           float &Dx, float &Dy, float &Dz)
{
    Dx = Dy = Dz = 0.0f;
    if constexpr (t3_order(K) != 0) t3_correction<t3_order(K)>(a.t, flags & F_HALO, dx, dy, dz, Dx, Dy, Dz);
    if constexpr (s1_order(K) != 0) {
        const float rho = sqrt_mufu(rho2);
        float Dr;
        s1r2_interp_f32<s1_order(K)>(a.t.s1tab, a.t.s1rec, a.t.nrho, a.t.nz, a.t.irho, a.t.rho_max, a.t.iz, a.t.halfL, rho, dz, Dr, Dz);
        const float er = rho > 0.0f ? Dr * rcp_mufu(rho) : 0.0f;
        Dx = er * dx;
        Dy = er * dy;
    }
}

// Image sums of the far pairs of one j particle with the lane's four i
// particles: sum of w and of w (dz + m L) over the images of the block that can
// lie inside the cut, in order; p0: the first pair, the others have qi + 8 k.
__device__ __forceinline__ void far_images(const BoxArgs &a, unsigned flags, const PairAt &p0, const f2 *dx, const f2 *dy,
                                           const f2 *dz, f2 *sw, f2 *sz)
{
    const int m0 = (int)(flags & 127u), m1 = (int)(flags >> 7 & 127u), i0 = (int)(flags >> 14 & 127u),
              i1 = (int)(flags >> 21 & 127u);  // + 64
    f2 rho2[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        rho2[h] = f2_fma(dx[h], dx[h], f2_mul(dy[h], dy[h]));
        sw[h] = sz[h] = 0ull;
    }
    auto image = [&](float fm, bool straddles) {
        const float sh = fm * a.t.L;
        const f2 s2 = f2_bcast(sh);
        f2 dzm[2], w[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            float r0, r1;
            dzm[h] = f2_add(dz[h], s2);
            f2_unpack(f2_fma(dzm[h], dzm[h], rho2[h]), r0, r1);
            const f2 ri = f2_pack(rsqrt_mufu(r0), rsqrt_mufu(r1));
            w[h] = f2_mul(f2_mul(ri, ri), ri);
        }
        if (straddles) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                float z[2], v[2];
                f2_unpack(dzm[h], z[0], z[1]);
                f2_unpack(w[h], v[0], v[1]);
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const float t = fabsf(z[k]) - a.t.cutL;
                    bool in = t <= 0.0f;
                    if (fabsf(t) < a.t.cut_tol) in = in_cut_exactly(a, PairAt{p0.I, p0.J, p0.qi + 8 * (2 * h + k), p0.qj}, sh);
                    v[k] = in ? v[k] : 0.0f;
                }
                w[h] = f2_pack(v[0], v[1]);
            }
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            sw[h] = f2_add(sw[h], w[h]);
            sz[h] = f2_fma(w[h], dzm[h], sz[h]);
        }
    };
    // The images entirely inside the cut are consecutive; their loop is unrolled
    // (n = 100,003, one loop for all / this: 7 images 11.5 / 11.2 ms, 31 images
    // 43.7 / 40.6; unrolled 2, 3 or 6 times up to 3 % slower).
    int m = m0;
    float fm = (float)(m0 - 64);
#pragma unroll 1
    while (m <= m1) {
        if (m >= i0 && m <= i1) {
#pragma unroll 4
            for (; m <= i1; m++, fm += 1.0f) image(fm, false);
        } else {
            image(fm, true);
            m++;
            fm += 1.0f;
        }
    }
}

// Far kernel vectors k (force on i per unit m_j, on j per unit -m_i) of two
// pairs with FP32 separations d. p0: the first pair; the second has qi + 8.
template <int K>
__device__ __forceinline__ void far_pairs(const BoxArgs &a, unsigned flags, PairAt p0, f2 dx, f2 dy, f2 dz, f2 &kx,
                                          f2 &ky, f2 &kz)
{
    float x[2], y[2], z[2], n[2][3], v[2][3];
    f2_unpack(dx, x[0], x[1]);
    f2_unpack(dy, y[0], y[1]);
    f2_unpack(dz, z[0], z[1]);
#pragma unroll
    for (int k = 0; k < 2; k++) {
        n[k][0] = x[k];
        n[k][1] = y[k];
        n[k][2] = z[k];
        if (flags & F_WRAP) {  // warp-uniform
            const PairAt p{p0.I, p0.J, p0.qi + 8 * k, p0.qj};
            if (is_t3(K) && (flags & 1u)) n[k][0] = wrap_far<K>(a, x[k], 0, p);
            if (is_t3(K) && (flags & 2u)) n[k][1] = wrap_far<K>(a, y[k], 1, p);
            if (flags & 4u) n[k][2] = wrap_far<K>(a, z[k], 2, p);
        }
        const float rho2 = fmaf(n[k][0], n[k][0], n[k][1] * n[k][1]);
        const float ri = rsqrt_mufu(fmaf(n[k][2], n[k][2], rho2));
        const float w = ri * ri * ri;
        float Dx, Dy, Dz;
        correction<K>(a, flags, x[k], y[k], is_t3(K) ? z[k] : n[k][2], rho2, Dx, Dy, Dz);
        v[k][0] = fmaf(w, n[k][0], -Dx);
        v[k][1] = fmaf(w, n[k][1], -Dy);
        v[k][2] = fmaf(w, n[k][2], -Dz);
    }
    kx = f2_pack(v[0][0], v[1][0]);
    ky = f2_pack(v[0][1], v[1][1]);
    kz = f2_pack(v[0][2], v[1][2]);
}

// Kernel vector of one near pair: double-float separation, spline, every
// decision exact.
template <int K>
__device__ __forceinline__ void near_pair(const BoxArgs &a, unsigned flags, const float *ph, const float *pl, float4 q,
                                          float4 ql, float b, bool self, float *k)
{
    const float qh[3] = {q.x, q.y, q.z}, qt[3] = {ql.x, ql.y, ql.z};
    float d[3], n[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        d[c] = self ? 0.0f : (qh[c] - ph[c]) + (qt[c] - pl[c]);
        n[c] = d[c];
        if (K != B_S1_IMG && (is_t3(K) || c == 2) && (flags >> c & 1u) && !self)
            n[c] = nearest_image(d[c], qh[c], ph[c], qt[c], pl[c], a.t.L, a.t.halfL, a.t.halfL_lo, a.t.wrap_tol);
    }
    const float rho2 = fmaf(n[0], n[0], n[1] * n[1]), b2 = b * b;
    if (K == B_S1_IMG) {
        float sw = 0.0f, sz = 0.0f;
        const int m1 = (int)(flags >> 7 & 127u) - 64;
        // the other images are outside the cut (all 2 emax + 1 in turn: n = 20,000
        // 0.79 ms, n = 100,003 11.4; this 0.73 and 11.1; not unrolled, 31 images
        // 2.63 instead of 2.41 ms at n = 20,000)
#pragma unroll 2
        for (int m = (int)(flags & 127u) - 64; m <= m1; m++) {
            const float sh = (float)m * a.t.L, dzm = d[2] + sh;
            const float r2 = fmaf(dzm, dzm, rho2);
            const float ri = rsqrt_mufu(r2);
            float w = ri * ri * ri;
            if (r2 < b2) w = spline_inner_f32(r2, b);
            bool in = fabsf(dzm) <= a.t.cutL;
            if (!self && fabsf(fabsf(dzm) - a.t.cutL) < a.t.cut_tol)
                in = cut_in_exact(qh[2], qt[2], ph[2], pl[2], sh, a.t.cutL);
            if (!in) w = 0.0f;
            sw += w;
            sz = fmaf(w, dzm, sz);
        }
        k[0] = sw * d[0];
        k[1] = sw * d[1];
        k[2] = sz;
        return;
    }
    const float r2 = fmaf(n[2], n[2], rho2);
    const float ri = rsqrt_mufu(r2);
    float w = ri * ri * ri;
    if (r2 < b2) w = spline_inner_f32(r2, b);
    float Dx, Dy, Dz;
    correction<K>(a, flags, d[0], d[1], is_t3(K) ? d[2] : n[2], rho2, Dx, Dy, Dz);
    k[0] = fmaf(w, n[0], -Dx);
    k[1] = fmaf(w, n[1], -Dy);
    k[2] = fmaf(w, n[2], -Dz);
}

// Sum over the 8 lanes of equal b.
__device__ __forceinline__ float sum_a(float v)
{
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    return v + __shfl_xor_sync(0xffffffffu, v, 16);
}

// Sums of v0 (even a) and v1 (odd a) over the 8 lanes of equal b.
__device__ __forceinline__ float sum_a2(float v0, float v1, bool odd)
{
    float v = (odd ? v1 : v0) + __shfl_xor_sync(0xffffffffu, odd ? v0 : v1, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    return v + __shfl_xor_sync(0xffffffffu, v, 16);
}

// 4-lane transpose-reduce over b: lane b ends with the sum of v[b].
__device__ __forceinline__ float sum_b(const float *v, int b)
{
    const bool hi = (b & 2) != 0, odd = (b & 1) != 0;
    const float h0 = (hi ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[2], 2);
    const float h1 = (hi ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, hi ? v[1] : v[3], 2);
    return (odd ? h1 : h0) + __shfl_xor_sync(0xffffffffu, odd ? h0 : h1, 1);
}

// Blocks per SM asked of the register allocator: the 8 records in flight of the
// wide stencils want registers, the others warps (n = 100,001, 3 / 4 / 5 / 6
// blocks: trilinear 36.7 / 35.8 / 36.8 / 38.8 ms, tricubic 254 / 269 / 275 /
// 278, CIC 24.6 / 21.3 / 19.8 / 19.2, TSC 42.7 / 45.4 / 47.0 / 48.8, images
// 11.6 with 4, 11.2 with 5, 11.5 with 6; T^3 nearest image 7.8 / 7.1 / 6.7).
constexpr int box_blocks(int K)
{
    return K == B_T3_CUB || K == B_S1_TSC ? 3 : K == B_T3_LIN ? 4 : K == B_S1_IMG || K == B_S1_NEAR ? 5 : 6;
}

template <int K>
__global__ void __launch_bounds__(SYM_THREADS, box_blocks(K)) k_sym_box(BoxArgs a)
{
    __shared__ __align__(16) float4 shq[SYM_WARPS][SYM_T];
    // j particles whose sums go over the lanes together: 9 shuffles for 8 pairs
    // instead of 4. The T^3 stencils are slower for it (n = 100,001: trilinear
    // 36.2 -> 40.5 ms, tricubic 254 -> 303, in registers and code size).
    constexpr int U = K == B_T3_LIN || K == B_T3_CUB ? 1 : 2;
    const int lane = threadIdx.x & 31, la = lane >> 2, lb = lane & 3;
    float4 *sq = shq[threadIdx.x >> 5];
    const size_t npad = a.s.npad;

    for (;;) {
        int item = 0;
        if (lane == 0) item = (int)atomicAdd(a.s.counter, 1u);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= a.s.nitems) return;
        const int A = item / a.s.C, ch = item - A * a.s.C;
        const int b0 = A * a.s.G, b1 = min(a.s.nrows, b0 + a.s.G);  // the group's i blocks
        const int I0 = b0 >> 2, tiles = a.s.njt - I0;
        const int J0 = I0 + (int)((long long)tiles * ch / a.s.C);
        const int J1 = I0 + (int)((long long)tiles * (ch + 1) / a.s.C);
        if (!check_item(A, div_up(a.s.nrows, a.s.G), ch, a.s.C, 32LL * b0, 32LL * b1, (long long)J0 * SYM_T,
                        (long long)J1 * SYM_T, a.s.step, a.s.tri, npad, (long long)a.s.njt * SYM_T))
            continue;
        const size_t jlo = a.s.tri ? (size_t)I0 * SYM_T : 0, jlen = npad - jlo;
        double *pj = a.s.pj + 3 * sym_slab(A, a.s.step, a.s.tri, npad);
        double *pi = a.s.pi + (size_t)ch * 3 * npad;

        for (int I = I0; 4 * I < b1; I++) {
            const int ib0 = max(0, b0 - 4 * I), ib1 = min(4, b1 - 4 * I);
            const int Ja = max(J0, I);
            if (Ja >= J1) {
                for (int k = ib0; k < ib1; k++)
#pragma unroll
                    for (int c = 0; c < 3; c++) pi[c * npad + (size_t)I * SYM_T + 32 * k + lane] = 0.0;
                continue;
            }
            for (int J = Ja; J < J1; ++J) {
                __syncwarp();
#pragma unroll
                for (int g = 0; g < 4; g++) sq[g * 32 + lane] = __ldg(a.s.pack + (size_t)J * SYM_T + g * 32 + lane);
                const unsigned myflags = classify<K>(a, I, J, lane >> 2 & 3, lane & 3);
                __syncwarp();
                const bool firsti = J == Ja;
#pragma unroll 1
                for (int ib = ib0; ib < ib1; ib++) {
                    const size_t qi = (size_t)I * SYM_T + ib * 32 + la;  // + 8 A
                    f2 PX[2], PY[2], PZ[2], PM[2], AX[2], AY[2], AZ[2];
                    {
                        float dO[3], eO[3];
                        box_frame<K>(a, I, J, dO, eO);
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            float v[2][4];
#pragma unroll
                            for (int k = 0; k < 2; k++) {
                                const float4 p = __ldg(a.s.pack + qi + 8 * (2 * h + k)),
                                             l = __ldg(a.s.resid + qi + 8 * (2 * h + k));
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
                    }
#pragma unroll 1
                    for (int g = J > I ? 0 : ib; g < 4; g++) {  // earlier blocks met this one already
                        const unsigned flags = __shfl_sync(0xffffffffu, myflags, ib * 4 + g);
                        const size_t qj0 = (size_t)J * SYM_T + g * 32;
                        float sx = 0.0f, sy = 0.0f, sz = 0.0f;  // j sums of particle qj0 + lane
                        if (!(flags & F_NEAR)) {
#pragma unroll 1
                            for (int B2 = 0; B2 < 8; B2 += U) {
                                float t[U][3];  // j sums of this lane for B2 (and B2 + 1)
#pragma unroll
                                for (int u = 0; u < U; u++) {
                                    const int B = B2 + u;
                                    const float4 q = sq[g * 32 + 4 * B + lb];
                                    const f2 qx = f2_bcast(q.x), qy = f2_bcast(q.y), qz = f2_bcast(q.z), qm = f2_bcast(q.w);
                                    f2 JX = 0ull, JY = 0ull, JZ = 0ull;
                                    f2 dx[2], dy[2], dz[2], kx[2], ky[2], kz[2];
#pragma unroll
                                    for (int h = 0; h < 2; h++) {
                                        dx[h] = f2_sub(qx, PX[h]);
                                        dy[h] = f2_sub(qy, PY[h]);
                                        dz[h] = f2_sub(qz, PZ[h]);
                                    }
                                    const PairAt p0{I, J, qi, qj0 + 4 * B + lb};
                                    if constexpr (K == B_S1_IMG) {
                                        f2 sw[2];
                                        far_images(a, flags, p0, dx, dy, dz, sw, kz);
#pragma unroll
                                        for (int h = 0; h < 2; h++) {
                                            kx[h] = f2_mul(sw[h], dx[h]);
                                            ky[h] = f2_mul(sw[h], dy[h]);
                                        }
                                    } else {
#pragma unroll
                                        for (int h = 0; h < 2; h++)
                                            far_pairs<K>(a, flags, PairAt{I, J, qi + 16 * h, p0.qj}, dx[h], dy[h], dz[h],
                                                         kx[h], ky[h], kz[h]);
                                    }
#pragma unroll
                                    for (int h = 0; h < 2; h++) {
                                        AX[h] = f2_fma(qm, kx[h], AX[h]);
                                        AY[h] = f2_fma(qm, ky[h], AY[h]);
                                        AZ[h] = f2_fma(qm, kz[h], AZ[h]);
                                        JX = f2_fma(PM[h], kx[h], JX);
                                        JY = f2_fma(PM[h], ky[h], JY);
                                        JZ = f2_fma(PM[h], kz[h], JZ);
                                    }
                                    float lo, hi;
                                    f2_unpack(JX, lo, hi);
                                    t[u][0] = lo + hi;
                                    f2_unpack(JY, lo, hi);
                                    t[u][1] = lo + hi;
                                    f2_unpack(JZ, lo, hi);
                                    t[u][2] = lo + hi;
                                }
#pragma unroll
                                for (int c = 0; c < 3; c++)
                                    t[0][c] = U == 2 ? sum_a2(t[0][c], t[U - 1][c], la & 1) : sum_a(t[0][c]);
                                if (la / U == B2 / U) {
                                    sx = t[0][0];
                                    sy = t[0][1];
                                    sz = t[0][2];
                                }
                            }
                        } else {
#pragma unroll 1
                            for (int A4 = 0; A4 < 4; A4++) {
                                float dO[3], eO[3], ph[3], pl[3], f[3] = {0.0f, 0.0f, 0.0f};
                                box_frame<K>(a, I, J, dO, eO);
                                const float4 p = __ldg(a.s.pack + qi + 8 * A4), l = __ldg(a.s.resid + qi + 8 * A4);
                                const float ei = __ldg(a.s.eps + qi + 8 * A4);
                                const uint32_t ii = __ldg(a.s.idx + qi + 8 * A4);
                                frame_split(p.x, l.x, dO[0], eO[0], ph[0], pl[0]);
                                frame_split(p.y, l.y, dO[1], eO[1], ph[1], pl[1]);
                                frame_split(p.z, l.z, dO[2], eO[2], ph[2], pl[2]);
#pragma unroll 1
                                for (int B = 0; B < 8; B++) {
                                    const size_t qj = qj0 + 4 * B + lb;
                                    const float4 q = sq[g * 32 + 4 * B + lb], ql = __ldg(a.s.resid + qj);
                                    const uint32_t jj = __ldg(a.s.idx + qj);
                                    float k[3];
                                    near_pair<K>(a, flags, ph, pl, q, ql, ei + __ldg(a.s.eps + qj), jj == ii, k);
                                    if (jj == PAD_J || ii == PAD_J) k[0] = k[1] = k[2] = 0.0f;  // padding
                                    f[0] = fmaf(q.w, k[0], f[0]);
                                    f[1] = fmaf(q.w, k[1], f[1]);
                                    f[2] = fmaf(q.w, k[2], f[2]);
                                    const float tx = sum_a(p.w * k[0]), ty = sum_a(p.w * k[1]), tz = sum_a(p.w * k[2]);
                                    if (la == B) {
                                        sx += tx;
                                        sy += ty;
                                        sz += tz;
                                    }
                                }
#pragma unroll
                                for (int h = 0; h < 2; h++) {
                                    const bool lo = A4 == 2 * h, hi = A4 == 2 * h + 1;
                                    AX[h] = f2_add(AX[h], f2_pack(lo ? f[0] : 0.0f, hi ? f[0] : 0.0f));
                                    AY[h] = f2_add(AY[h], f2_pack(lo ? f[1] : 0.0f, hi ? f[1] : 0.0f));
                                    AZ[h] = f2_add(AZ[h], f2_pack(lo ? f[2] : 0.0f, hi ? f[2] : 0.0f));
                                }
                            }
                        }
                        if (J > I || g > ib) {  // a block against itself is one-sided
                            double *o = pj + (qj0 + lane - jlo);
                            const bool first = 4 * I + ib == b0;
                            add_slab(o, (double)sx, first);
                            add_slab(o + jlen, (double)sy, first);
                            add_slab(o + 2 * jlen, (double)sz, first);
                        }
                    }
                    float v[4];
                    double *o = pi + (size_t)I * SYM_T + ib * 32 + 8 * lb + la;
                    f2_unpack(AX[0], v[0], v[1]);
                    f2_unpack(AX[1], v[2], v[3]);
                    add_slab(o, (double)sum_b(v, lb), firsti);
                    f2_unpack(AY[0], v[0], v[1]);
                    f2_unpack(AY[1], v[2], v[3]);
                    add_slab(o + npad, (double)sum_b(v, lb), firsti);
                    f2_unpack(AZ[0], v[0], v[1]);
                    f2_unpack(AZ[1], v[2], v[3]);
                    add_slab(o + 2 * npad, (double)sum_b(v, lb), firsti);
                }
            }
        }
    }
}

}  // namespace

// Largest |T(c) + T(mirror of c)| and |T(c)| of the T^3 table, or for the
// (rho, z) table of D_rho(z) - D_rho(-z) and D_z(z) + D_z(-z). Bit patterns of
// magnitudes order as integers, NaN above all. A thread takes a cell and its
// mirror at a time and a block ends with one atomic per word: the first call
// after an upload waits for this kernel, and with two atomics per cell on the
// same two words it took 2.6 ms at Ng = 127 and 21 ms at 255 (with the copy and
// the wait; now 0.04 and 0.22).
constexpr int PARITY_THREADS = 256;
__device__ __forceinline__ unsigned long long magnitude_bits(double v)
{
    return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffULL;
}

__global__ void __launch_bounds__(PARITY_THREADS) k_table_parity(const double *__restrict__ t, long long ncell, int nz,
                                                                unsigned long long *out)
{
    unsigned long long odd = 0, big = 0;
    const int half = nz ? (nz + 1) / 2 : 0;
    const long long npair = nz ? ncell / nz * half : (ncell + 1) / 2;
    for (long long q = (long long)blockIdx.x * PARITY_THREADS + threadIdx.x; q < npair;
         q += (long long)gridDim.x * PARITY_THREADS) {
        if (nz == 0) {
            const double *a = t + 3 * q, *b = t + 3 * (ncell - 1 - q);
#pragma unroll
            for (int k = 0; k < 3; k++) {
                odd = max(odd, magnitude_bits(a[k] + b[k]));
                big = max(big, max(magnitude_bits(a[k]), magnitude_bits(b[k])));
            }
        } else {
            const long long row = q / half * nz;
            const int z = (int)(q % half);
            const double *a = t + 2 * (row + z), *b = t + 2 * (row + nz - 1 - z);
            odd = max(odd, max(magnitude_bits(a[0] - b[0]), magnitude_bits(a[1] + b[1])));
#pragma unroll
            for (int k = 0; k < 2; k++) big = max(big, max(magnitude_bits(a[k]), magnitude_bits(b[k])));
        }
    }
    __shared__ unsigned long long red[2][PARITY_THREADS / 32];
    for (int o = 16; o > 0; o >>= 1) {
        odd = max(odd, __shfl_xor_sync(0xffffffffu, odd, o));
        big = max(big, __shfl_xor_sync(0xffffffffu, big, o));
    }
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = odd;
        red[1][threadIdx.x >> 5] = big;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        unsigned long long m = 0;
        for (int w = 0; w < PARITY_THREADS / 32; w++) m = max(m, red[threadIdx.x][w]);
        atomicMax(&out[threadIdx.x], m);
    }
}

// Largest asymmetry of a table over its largest entry (NaN: not comparable).
static double asymmetry(const double *t, long long ncell, int nz)
{
    Ctx &c = ctx();
    unsigned long long *d = c.bbox.ensure<unsigned long long>(8), h[2];
    STEPS_CUDA(cudaMemsetAsync(d, 0, 2 * sizeof *d, c.stream));
    const long long blocks = std::min((ncell + PARITY_THREADS - 1) / PARITY_THREADS, 8LL * c.nsm);
    k_table_parity<<<(unsigned)blocks, PARITY_THREADS, 0, c.stream>>>(t, ncell, nz, d);
    note_launch("k_table_parity");
    STEPS_CUDA(cudaMemcpyAsync(h, d, sizeof h, cudaMemcpyDeviceToHost, c.stream));
    STEPS_CUDA(cudaStreamSynchronize(c.stream));
    double v[2];
    memcpy(v, h, sizeof v);
    return v[0] == 0.0 ? v[0] * v[1] : v[0] / v[1];
}

// The correction table of a call is odd in the separation to tol of its largest
// entry. Looked at once per table.
static bool table_odd(const KParams &kp, const Tables &tb, double tol)
{
    Ctx &c = ctx();
    if (kp.topology == STEPS_T3) {
        if (c.t3_odd_version != c.t3_version) {
            c.t3_odd = asymmetry(tb.t3, (long long)tb.t3_ng * tb.t3_ng * tb.t3_ng, 0);
            c.t3_odd_version = c.t3_version;
        }
        return c.t3_odd <= tol;
    }
    if (c.s1_odd_version != c.s1r2_version) {
        c.s1_odd = asymmetry(tb.s1r2, (long long)tb.nrho * tb.nz, tb.nz);
        c.s1_odd_version = c.s1r2_version;
    }
    return c.s1_odd <= tol;
}

static int box_kind(const KParams &kp)
{
    if (kp.topology == STEPS_T3) return kp.is_periodic < 2 ? B_T3_NEAR : kp.order == 4 ? B_T3_CUB : B_T3_LIN;
    if (kp.is_periodic < 2) return B_S1_NEAR;
    if (kp.s1r2_images) return B_S1_IMG;
    return kp.order == 2 ? B_S1_CIC : kp.order == 4 ? B_S1_TSC : -1;
}

bool box_supported(const KParams &kp, const Tables &tb)
{
    Ctx &c = ctx();
    const int kind = box_kind(kp);
    // NGP picks a cell by a floor, which two particles on opposite sides of a
    // face decide differently: it stays one-sided.
    if (kind < 0) return false;
    if (kind == B_S1_IMG) return kp.emax < 64;  // 7 bits per image number
    if (kind == B_S1_NEAR) return kp.L < 1e11 && kp.rsim < 1e11;  // r^-3 stays a normal FP32 number
    if ((kind == B_T3_LIN || kind == B_T3_CUB) && c.shape.t3_cells > 0)
        return false;  // the caller asked for the shared-memory window
    // Odd to 1e-9 of the largest entry: 1/60 of the FP32 rounding of the entries
    // that the mixed kernels read. The builders' tables are odd exactly or to
    // rounding; any other table takes the one-sided kernels.
    return kind == B_T3_NEAR || table_odd(kp, tb, 1e-9);
}

bool fp64_odd(const KParams &kp, const Tables &tb)
{
    const int kind = kp.topology == STEPS_R3 ? B_S1_NEAR : box_kind(kp);
    return kind >= 0 && (kind == B_S1_NEAR || kind == B_S1_IMG || kind == B_T3_NEAR || table_odd(kp, tb, 1e-16));
}

// Granules are the 32-particle i blocks: groups of one or two of them for sets
// whose tiles are too few to fill the GPU, of whole tiles otherwise.
bool box_plan(int n, SymPlan &p)
{
    p.NP = 0;
    p.ntiles = div_up(n, SYM_T);
    p.npad = (size_t)p.ntiles * SYM_T;
    p.gran = 32;
    p.nrows = div_up(n, 32);
    const bool ok = sym_split(p);
    if (!p.tri && p.G > 2) {  // whole tiles
        p.G = div_up(p.G, 4) * 4;
        p.tri = 1;
        p.step = p.gran * p.G;
        p.groups = div_up(p.nrows, p.G);
        p.doubles = 3 * ((size_t)p.C * p.npad + sym_slab(p.groups, p.step, p.tri, p.npad));
    }
    return ok;
}

template <int K>
static void launch(const BoxArgs &a)
{
    Ctx &c = ctx();
    int occ = 0;
    STEPS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_sym_box<K>, SYM_THREADS, 0));
    const int grid = std::min(div_up(a.s.nitems, SYM_WARPS), c.nsm * std::max(occ, 1));
    k_sym_box<K><<<grid, SYM_THREADS, 0, c.stream>>>(a);
    note_launch("k_sym_box");
}

void box_launch(const KParams &kp, const Tables &tb, const SymArgs &s)
{
    Ctx &c = ctx();
    BoxArgs a{};
    a.s = s;
    period_args(a.t, kp);
    if (kp.topology == STEPS_T3) t3_args(a.t, kp, tb, c.stream);
    else if (kp.is_periodic >= 2 && !kp.s1r2_images) s1tab_args(a.t, kp, tb, c.stream);
    switch (box_kind(kp)) {
    case B_T3_NEAR: launch<B_T3_NEAR>(a); break;
    case B_T3_LIN: launch<B_T3_LIN>(a); break;
    case B_T3_CUB: launch<B_T3_CUB>(a); break;
    case B_S1_NEAR: launch<B_S1_NEAR>(a); break;
    case B_S1_CIC: launch<B_S1_CIC>(a); break;
    case B_S1_TSC: launch<B_S1_TSC>(a); break;
    default: launch<B_S1_IMG>(a); break;
    }
}

}  // namespace steps
