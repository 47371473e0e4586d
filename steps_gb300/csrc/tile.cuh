// The tile builder of the ordering pass (order.cu). The persistent ensemble
// kernel (ensemble.cu) rebuilds its tiles with the same arithmetic, one warp to
// a tile.
#pragma once

#include "common.cuh"

namespace steps {

__device__ __forceinline__ unsigned long long warp_min(unsigned long long v)
{
    for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Builds tile `tile` (the T particles of sorted positions [sbase, sbase + cnt),
// padded to T) with a block of NT threads: FP32-exact centre, half extents and
// largest softening (meta), FP32 offsets (pack, soa), their FP32 residuals
// (lo), softening (epsf), original indices (idx) and the sub-tile boxes (sub).
// perm holds original indices below nx (checked in bounds-checked builds).
template <int NT>
__device__ __forceinline__ void build_tile(int tile, int sbase, int cnt, const double *__restrict__ x,
                                           const double *__restrict__ m, const double *__restrict__ eps,
                                           const uint32_t *__restrict__ perm, long long nx, int T,
                                           float4 *__restrict__ pack,
                                           float *__restrict__ epsf, float4 *__restrict__ meta,
                                           uint32_t *__restrict__ idx, uint32_t pad_id, float4 *__restrict__ lo,
                                           float *__restrict__ soa, float4 *__restrict__ sub)
{
    // The box is taken on ordered integer images: FP64 comparisons, 41 a warp at
    // 16 cycles each, were most of the kernel's time (n = 200,003: 40 us, now 17).
    __shared__ unsigned long long red[7][NT / 32];
    __shared__ float s_c[3];
    int t = threadIdx.x, lane = t & 31, w = t >> 5;
    unsigned long long mm[7] = {~0ull, ~0ull, ~0ull, ~0ull, ~0ull, ~0ull, ~0ull};  // min, ~max; ~max of eps
    for (int e = t; e < T; e += NT) {
        if (e < cnt) {
            uint32_t o = perm[sbase + e];
            STEPS_CHECK_IDX(o, nx, CK_PERM);
            for (int k = 0; k < 3; k++) extend_box(x[3 * (size_t)o + k], mm[k], mm[3 + k]);
            const double ev = eps[o];
            if (!is_nan_bits(ev)) mm[6] = min(mm[6], ~ordered_bits(ev));
        }
    }
#pragma unroll
    for (int k = 0; k < 7; k++) {
        mm[k] = warp_min(mm[k]);
        if (lane == 0) red[k][w] = mm[k];
    }
    __syncthreads();
    if (t < 3) {  // axis t; softening lengths count from 0 up
        unsigned long long a0 = ~0ull, a1 = ~0ull, a2 = ~ordered_bits(0.0);
        for (int v = 0; v < NT / 32; v++) {
            a0 = min(a0, red[t][v]);
            a1 = min(a1, red[3 + t][v]);
            a2 = min(a2, red[6][v]);
        }
        double lo_t = 0.0, hi_t = 0.0;  // an empty tile
        if (a0 <= ~a1) {
            lo_t = from_ordered_bits(a0);
            hi_t = from_ordered_bits(~a1);
        }
        const float c = __double2float_rn(0.5 * (lo_t + hi_t));
        const double ext = fmax(hi_t - (double)c, (double)c - lo_t);
        s_c[t] = c;
        float *mt = reinterpret_cast<float *>(meta + 2 * tile);
        mt[t] = c;
        // Round up so the FP32 half extent bounds every FP32 offset.
        mt[4 + t] = __double2float_ru(ext * (1.0 + 1e-6)) + 1e-30f;
        if (t == 0) {
            mt[3] = __double2float_ru(from_ordered_bits(~a2));
            mt[7] = 0.0f;
        }
    }
    __syncthreads();
    double cx = s_c[0], cy = s_c[1], cz = s_c[2];
    for (int e = t; e < T; e += NT) {
        const int q = tile * T + e;
        if (e < cnt) {
            uint32_t o = perm[sbase + e];
            STEPS_CHECK_IDX(o, nx, CK_PERM);
            const double ox = x[3 * (size_t)o] - cx, oy = x[3 * (size_t)o + 1] - cy, oz = x[3 * (size_t)o + 2] - cz;
            const float hx = __double2float_rn(ox), hy = __double2float_rn(oy), hz = __double2float_rn(oz);
            pack[q] = make_float4(hx, hy, hz, __double2float_rn(m[o]));
            if (soa) {  // tile-blocked SoA copy: X[T], Y[T], Z[T], M[T] per tile
                float *b = soa + (size_t)tile * 4 * T;
                b[e] = hx;
                b[T + e] = hy;
                b[2 * T + e] = hz;
                b[3 * T + e] = __double2float_rn(m[o]);
            }
            // What FP32 dropped from the offset: i particles carry it so that
            // their position in another tile's frame keeps full precision.
            if (lo)
                lo[q] = make_float4(__double2float_rn(ox - hx), __double2float_rn(oy - hy), __double2float_rn(oz - hz),
                                    0.f);
            epsf[q] = __double2float_rn(eps[o]);
            if (idx) idx[q] = o;
        } else {
            pack[q] = make_float4(0.f, 0.f, 0.f, 0.f);  // massless padding at the tile centre
            if (soa) {
                float *b = soa + (size_t)tile * 4 * T;
                b[e] = b[T + e] = b[2 * T + e] = b[3 * T + e] = 0.f;
            }
            if (lo) lo[q] = make_float4(0.f, 0.f, 0.f, 0.f);
            epsf[q] = 0.f;
            if (idx) idx[q] = pad_id;
        }
        if (sub) {
            // Sub-tile boxes: the SUBTILE consecutive particles of a half warp
            // (padding included, at the tile centre), in the tile's FP32 offset
            // frame, widened by 1e-6 relative so they hold the exact positions.
            const float4 pq = pack[q];
            float l3[3] = {pq.x, pq.y, pq.z}, h3[3] = {pq.x, pq.y, pq.z};
            float se = epsf[q];
#pragma unroll
            for (int o = SUBTILE / 2; o > 0; o >>= 1) {
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    l3[k] = fminf(l3[k], __shfl_xor_sync(0xffffffffu, l3[k], o));
                    h3[k] = fmaxf(h3[k], __shfl_xor_sync(0xffffffffu, h3[k], o));
                }
                se = fmaxf(se, __shfl_xor_sync(0xffffffffu, se, o));
            }
            if ((e & (SUBTILE - 1)) == 0) {
                float c3[3], w3[3];
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    c3[k] = 0.5f * (l3[k] + h3[k]);
                    const float w = fmaxf(h3[k] - c3[k], c3[k] - l3[k]);
                    w3[k] = w * 1.000001f + 1e-6f * (fabsf(c3[k]) + w) + 1e-30f;
                }
                float4 *d = sub + 2 * ((size_t)tile * (T / SUBTILE) + e / SUBTILE);
                d[0] = make_float4(c3[0], c3[1], c3[2], se);
                d[1] = make_float4(w3[0], w3[1], w3[2], 0.0f);
            }
        }
    }
}


}  // namespace steps
