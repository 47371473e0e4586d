// Interpolation of the FP32 correction tables in the mixed-precision kernels:
// the T^3 Ewald table (trilinear, Catmull-Rom tricubic) and the S1xR2
// (rho, z) table (NGP, CIC, TSC).
#pragma once

#include "common.cuh"
#include "mixed.cuh"

namespace steps {
namespace mixed {

__device__ __forceinline__ int pmod(int i, int n)
{
    int r = i % n;
    return r < 0 ? r + n : r;
}

// i mod n for i in [-2n, 3n), without a division; any other i (positions
// outside the box, NaN) is clamped into [0, n) so the read stays in the table.
__device__ __forceinline__ int wrap_index(int i, int n)
{
    i += i < 0 ? n : 0;
    i += i < 0 ? n : 0;
    i -= i >= n ? n : 0;
    i -= i >= n ? n : 0;
    return min(max(i, 0), n - 1);
}

template <int ORDER>
__device__ __forceinline__ void weights(float t, float *w)
{
    if (ORDER == 4) {  // Catmull-Rom, StePS/src/ewald_space.cc:440-449
        const float t2 = t * t, t3 = t2 * t;
        w[0] = -0.5f * t3 + t2 - 0.5f * t;
        w[1] = 1.5f * t3 - 2.5f * t2 + 1.0f;
        w[2] = -1.5f * t3 + 2.0f * t2 + 0.5f * t;
        w[3] = 0.5f * t3 - 0.5f * t2;
    } else {  // 2-point Lagrange (trilinear)
        w[0] = 1.0f - t;
        w[1] = t;
    }
}

// T^3 stencil records, one float4 per component, in two arrays of the same
// record index: the x and y components as one 32-byte record (a.t3r, read with
// one 256-bit load) and the z component as one 16-byte record (a.t3rz): two
// L1 requests per record instead of three, in the same 48 bytes per cell.
// (Records padded to 64 bytes for the same purpose were 13-17 % slower: the
// larger table loses L1 hits.)
//
// Index of the record of cell (x, y, z) of the haloed table of extent E. The L1
// path, which bounds the table kernels, takes one cycle per 128-byte line that a
// group of 4 (256-bit) or 8 (128-bit) lanes touches, and the lanes' cells spread
// over all three axes. Trilinear: bricks of 2 x 2 x 2 cells (40,961 particles,
// pairwise kernel, against rows along z: 6.59 / 6.93 ms at ng = 63, 10.97 / 11.80
// ms at ng = 127; one-sided 17.34 / 17.58 and 23.96 / 24.46). Tricubic: rows along
// z, since its 16 records need 8 indices instead of one (pairwise 52.8 ms, bricks
// 52.1; one-sided 124.4 ms, bricks 138.4).
template <int ORDER>
__host__ __device__ __forceinline__ int t3_record(int x, int y, int z, int E)
{
    if (ORDER == 4) return (x * E + y) * E + z;
    const int H = (E + 1) >> 1;
    return ((((x >> 1) * H + (y >> 1)) * H + (z >> 1)) << 3) + ((x & 1) << 2) + ((y & 1) << 1) + (z & 1);
}

// Room for the records of either order: an even extent holds whole bricks.
__host__ __device__ __forceinline__ size_t t3_records(int E)
{
    const size_t e = ((size_t)E + 1) / 2 * 2;
    return e * e * e;
}

// Two float4 of a 32-byte aligned record in one 256-bit load (sm_100+):
// the L1 data path, which bounds the table kernels, sees one request per
// record instead of two. The S1xR2 CIC and TSC records are 32 bytes: CIC
// 2.71e11 -> 3.53e11 and TSC 1.06e11 -> 1.31e11 pairs/s at N = 2^20.
__device__ __forceinline__ void ldg_v8(const float4 *p, float4 &a, float4 &b)
{
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}

// w . v for the 4 z taps of a z-row record.
__device__ __forceinline__ float dot4(const float *w, float4 v)
{
    return fmaf(w[3], v.w, fmaf(w[2], v.z, fmaf(w[1], v.y, w[0] * v.x)));
}

// Sum of the NT^3 stencil taps fetch(a, b, c) weighted by wx[a] wy[b] wz[c].
// Trilinear: 8 products of the three weights (36 FP ops). Tricubic: nested,
// sum_a wx_a sum_b wy_b sum_c wz_c T_abc (252 FP ops instead of 272).
template <int ORDER, class Fetch>
__device__ __forceinline__ void stencil(const float *wx, const float *wy, const float *wz, Fetch fetch, float &Dx,
                                        float &Dy, float &Dz)
{
    constexpr int NT = ORDER;
    if constexpr (ORDER == 4) {
#pragma unroll
        for (int aa = 0; aa < NT; aa++) {
            float rx = 0.0f, ry = 0.0f, rz = 0.0f;
#pragma unroll
            for (int bb = 0; bb < NT; bb++) {
                float sx = 0.0f, sy = 0.0f, sz = 0.0f;
#pragma unroll
                for (int cc = 0; cc < NT; cc++) {
                    const float4 v = fetch(aa, bb, cc);
                    sx = fmaf(wz[cc], v.x, sx);
                    sy = fmaf(wz[cc], v.y, sy);
                    sz = fmaf(wz[cc], v.z, sz);
                }
                rx = fmaf(wy[bb], sx, rx);
                ry = fmaf(wy[bb], sy, ry);
                rz = fmaf(wy[bb], sz, rz);
            }
            Dx = fmaf(wx[aa], rx, Dx);
            Dy = fmaf(wx[aa], ry, Dy);
            Dz = fmaf(wx[aa], rz, Dz);
        }
    } else {
#pragma unroll
        for (int aa = 0; aa < NT; aa++)
#pragma unroll
            for (int bb = 0; bb < NT; bb++) {
                const float wxy = wx[aa] * wy[bb];
#pragma unroll
                for (int cc = 0; cc < NT; cc++) {
                    const float4 v = fetch(aa, bb, cc);
                    const float ww = wxy * wz[cc];
                    Dx = fmaf(ww, v.x, Dx);
                    Dy = fmaf(ww, v.y, Dy);
                    Dz = fmaf(ww, v.z, Dz);
                }
            }
    }
}

// Cell index of a nearest-image z in [-L/2, L/2]: floor(uz) lies in [-1, nz]
// up to rounding, so one conditional shift wraps it; anything else
// (non-finite input) is clamped into [0, nz).
__device__ __forceinline__ int wrap_near(float f, int nz)
{
    int i = (int)f;
    i += i < 0 ? nz : 0;
    i -= i >= nz ? nz : 0;
    return min(max(i, 0), nz - 1);
}

// (rho, z) table interpolation in FP32 from the float2 copy of the S1xR2
// table: NGP / CIC / TSC exactly as StePS/src/ewald_space.cc:803-1000
// (rho clamped to [0, rho_max], z index periodic).
// CIC reads whole-stencil records (k_table2_cic): 2 loads from one 32-byte
// sector per pair. TSC reads z-triplet records (k_table2_zrec): record
// (ir, iz) = cells (ir, iz-1), (ir, iz), (ir, iz+1), z periodic, as (Dr, Dz)
// pairs in 2 float4, so one rho row of its stencil is 2 loads instead of 3.
// (Whole TSC stencils in 128-byte records -- 5 loads from one line -- were
// 20 % slower: the table grows 4x and falls out of L1.)
template <int ORDER>
__device__ __forceinline__ void s1r2_interp_f32(const float2 *__restrict__ T, const float4 *__restrict__ R, int nrho,
                                                int nz, float irho, float rho_max, float iz, float halfL, float rho,
                                                float z, float &Dr, float &Dz)
{
    const float rr = fminf(fmaxf(rho, 0.0f), rho_max);
    const float ur = rr * irho;
    const float uz = (z + halfL) * iz - 0.5f;
    Dr = 0.0f;
    Dz = 0.0f;
    if (ORDER == 0) {
        int ir = (int)floorf(ur + 0.5f);
        ir = ir < 0 ? 0 : (ir > nrho - 1 ? nrho - 1 : ir);
        int izc = wrap_near(floorf(uz + 0.5f), nz);
        STEPS_CHECK_IDX(ir, nrho, CK_S1_CELL);
        STEPS_CHECK_IDX(izc, nz, CK_S1_CELL);
        const float2 v = __ldg(T + (size_t)ir * nz + izc);
        Dr = v.x;
        Dz = v.y;
    } else if (ORDER == 2) {
        int ir0 = (int)floorf(ur);
        float fr = ur - (float)ir0;
        if (ir0 < 0) { ir0 = 0; fr = 0.0f; }
        if (ir0 > nrho - 2) { ir0 = nrho - 2 > 0 ? nrho - 2 : 0; fr = 1.0f; }
        const float iz0r = floorf(uz);
        const float fz = uz - iz0r;
        int iz0 = wrap_near(iz0r, nz);
        int ra = ir0;
        STEPS_CHECK_IDX(ra, nrho - 1, CK_S1_CELL);
        STEPS_CHECK_IDX(iz0, nz, CK_S1_CELL);
        // record (ir0, iz0): rows ir0, ir0 + 1 x cells iz0, iz0 + 1 (periodic)
        float4 r0, r1;
        ldg_v8(R + 2 * ((size_t)ra * nz + iz0), r0, r1);  // 32-byte records, 256-byte aligned base
        const float w00 = (1.0f - fr) * (1.0f - fz), w10 = fr * (1.0f - fz), w01 = (1.0f - fr) * fz, w11 = fr * fz;
        Dr = w00 * r0.x + w10 * r1.x + w01 * r0.z + w11 * r1.z;
        Dz = w00 * r0.y + w10 * r1.y + w01 * r0.w + w11 * r1.w;
    } else {
        const int jr = (int)floorf(ur + 0.5f), jz = (int)floorf(uz + 0.5f);
        const float sr = ur - (float)jr, sz = uz - (float)jz;
        const float wr[3] = {0.5f * (0.5f - sr) * (0.5f - sr), 0.75f - sr * sr, 0.5f * (0.5f + sr) * (0.5f + sr)};
        const float wz[3] = {0.5f * (0.5f - sz) * (0.5f - sz), 0.75f - sz * sz, 0.5f * (0.5f + sz) * (0.5f + sz)};
        int ir[3] = {jr - 1, jr, jr + 1};
        if (ir[0] < 0) ir[0] = 0;
        if (ir[1] < 0) ir[1] = 0;
        if (ir[1] > nrho - 1) ir[1] = nrho - 1;
        if (ir[2] > nrho - 1) ir[2] = nrho - 1;
        int iz1 = wrap_near((float)jz, nz);
        STEPS_CHECK_IDX(iz1, nz, CK_S1_CELL);
#pragma unroll
        for (int r = 0; r < 3; r++) STEPS_CHECK_IDX(ir[r], nrho, CK_S1_CELL);
#pragma unroll
        for (int r = 0; r < 3; r++) {  // record (ir, iz1): cells iz1 - 1, iz1, iz1 + 1
            float4 v01, v2;
            ldg_v8(R + 2 * ((size_t)ir[r] * nz + iz1), v01, v2);  // 32-byte records
            const float sr_ = fmaf(wz[2], v2.x, fmaf(wz[1], v01.z, wz[0] * v01.x));
            const float sz_ = fmaf(wz[2], v2.y, fmaf(wz[1], v01.w, wz[0] * v01.y));
            Dr = fmaf(wr[r], sr_, Dr);
            Dz = fmaf(wr[r], sz_, Dz);
        }
    }
}

// Ewald correction D(d) of one pair from the FP32 table (not the window):
// stencil records of the haloed copy when the tile pair's stencils stay in
// the halo, else taps of the haloed copy at indices wrapped once per axis.
template <int ORDER>
__device__ __forceinline__ void t3_correction(const MixedArgs &a, bool halo, float dx, float dy, float dz, float &Dx,
                                              float &Dy, float &Dz)
{
    constexpr int NT = ORDER;
    constexpr int OFF = ORDER == 4 ? 1 : 0;
    float wx[4], wy[4], wz[4];
    Dx = Dy = Dz = 0.0f;
    if (halo) {
        const float uh = a.u0 + (float)a.halo;
        const float ux = fmaf(dx, a.ih, uh), uy = fmaf(dy, a.ih, uh), uz = fmaf(dz, a.ih, uh);
        const float fxl = floorf(ux), fyl = floorf(uy), fzl = floorf(uz);
        weights<ORDER>(ux - fxl, wx);
        weights<ORDER>(uy - fyl, wy);
        weights<ORDER>(uz - fzl, wz);
        const int E = a.ext;
        int bx = min(max((int)fxl - OFF, 0), E - NT);
        int by = min(max((int)fyl - OFF, 0), E - NT);
        int bz = min(max((int)fzl - OFF, 0), E - NT);
#ifdef STEPS_CHECK
        const long long hfirst = ((long long)bx * E + by) * E + bz;
        if (!check_span(hfirst, hfirst + (long long)(NT - 1) * ((long long)E * E + E + 1), (long long)E * E * E,
                        CK_T3_CELL))
            bx = by = bz = 0;
#endif
        if (ORDER == 4) {  // z-row records
#pragma unroll
            for (int aa = 0; aa < 4; aa++) {
                float rx = 0.0f, ry = 0.0f, rz = 0.0f;
#pragma unroll
                for (int bb = 0; bb < 4; bb++) {
                    int cr = t3_record<4>(bx + aa, by + bb, bz, E);
                    STEPS_CHECK_IDX(cr, t3_records(E), CK_T3_CELL);
                    float4 vx, vy;
                    ldg_v8(a.t3r + 2 * (size_t)cr, vx, vy);
                    const float4 vz = __ldg(a.t3rz + cr);
                    rx = fmaf(wy[bb], dot4(wz, vx), rx);
                    ry = fmaf(wy[bb], dot4(wz, vy), ry);
                    rz = fmaf(wy[bb], dot4(wz, vz), rz);
                }
                Dx = fmaf(wx[aa], rx, Dx);
                Dy = fmaf(wx[aa], ry, Dy);
                Dz = fmaf(wx[aa], rz, Dz);
            }
        } else {  // (y, z) quad records
            const float q00 = wy[0] * wz[0], q01 = wy[0] * wz[1], q10 = wy[1] * wz[0], q11 = wy[1] * wz[1];
#pragma unroll
            for (int aa = 0; aa < 2; aa++) {
                int cr = t3_record<2>(bx + aa, by, bz, E);
                STEPS_CHECK_IDX(cr, t3_records(E), CK_T3_CELL);
                float4 vx, vy;
                ldg_v8(a.t3r + 2 * (size_t)cr, vx, vy);
                const float4 vz = __ldg(a.t3rz + cr);
                Dx = fmaf(wx[aa], fmaf(q11, vx.w, fmaf(q10, vx.z, fmaf(q01, vx.y, q00 * vx.x))), Dx);
                Dy = fmaf(wx[aa], fmaf(q11, vy.w, fmaf(q10, vy.z, fmaf(q01, vy.y, q00 * vy.x))), Dy);
                Dz = fmaf(wx[aa], fmaf(q11, vz.w, fmaf(q10, vz.z, fmaf(q01, vz.y, q00 * vz.x))), Dz);
            }
        }
    } else {
        const float ux = fmaf(dx, a.ih, a.u0), uy = fmaf(dy, a.ih, a.u0), uz = fmaf(dz, a.ih, a.u0);
        const float fxl = floorf(ux), fyl = floorf(uy), fzl = floorf(uz);
        weights<ORDER>(ux - fxl, wx);
        weights<ORDER>(uy - fyl, wy);
        weights<ORDER>(uz - fzl, wz);
        const int bx = (int)fxl - OFF, by = (int)fyl - OFF, bz = (int)fzl - OFF;
        int gx[NT], gy[NT], gz[NT];
#pragma unroll
        for (int t = 0; t < NT; t++) {
            gx[t] = wrap_index(bx + t, a.ng) + a.halo;
            gy[t] = wrap_index(by + t, a.ng) + a.halo;
            gz[t] = wrap_index(bz + t, a.ng) + a.halo;
            STEPS_CHECK_IDX(gx[t], a.ext, CK_T3_CELL);
            STEPS_CHECK_IDX(gy[t], a.ext, CK_T3_CELL);
            STEPS_CHECK_IDX(gz[t], a.ext, CK_T3_CELL);
        }
        stencil<ORDER>(wx, wy, wz,
                       [&](int aa, int bb, int cc) { return __ldg(a.t3f + (gx[aa] * a.ext + gy[bb]) * a.ext + gz[cc]); },
                       Dx, Dy, Dz);
    }
}

}  // namespace mixed
}  // namespace steps
