// Plain FP64 direct-summation kernels (all topologies): the GPU-side
// correctness reference, FP64 end to end.
//
// One thread per i particle, i in registers; j particles staged 128 at a time
// in shared memory as (x, y, z, m) double4 plus their softening, and visited
// in ascending j order, so each i's sum is taken in the order of the
// reference's sequential j loop (StePS/src/forces.cc:538). The j range may be
// split into chunks (blockIdx.y) whose FP64 partial sums are added in chunk
// order by the reduction, which also applies the background term.
//
// Calls for all particles evaluate each pair once and add it to both
// (k_sym_fp64): 18 FP64 instructions a pair in R^3 instead of 2 x 14.
#include <algorithm>

#include "common.cuh"
#include "context.cuh"
#include "sym.cuh"

namespace steps {

namespace {

constexpr int FP64_THREADS = 128;

enum Fp64Mode { M_R3 = 0, M_T3_EWALD, M_NEAREST3, M_S1_IMAGES, M_S1_NEAREST, M_S1_TABLE };

__device__ __forceinline__ int pos_mod(int i, int n)
{
    int r = i % n;
    return r < 0 ? r + n : r;
}

// Tensor-product T^3 table interpolation (StePS/src/ewald_space.cc:452-523,
// StePS/src/forces_cuda.cu:113-167): ORDER 2 = trilinear (2-point Lagrange),
// ORDER 4 = Catmull-Rom tricubic, on cell centres (i + 1/2) h - L/2.
template <int ORDER>
__device__ __forceinline__ void t3_interp_fp64(const double *__restrict__ tab, int ng, double L, double ih, double dx,
                                               double dy, double dz, double &Dx, double &Dy, double &Dz)
{
    double d[3] = {dx, dy, dz};
    int i0[3];
    double w[3][4];
    for (int k = 0; k < 3; k++) {
        double u = (d[k] + 0.5 * L) * ih - 0.5;
        double uf = floor(u);
        i0[k] = pos_mod((int)uf, ng);
        double t = u - uf;
        if (ORDER == 4) {
            double t2 = t * t, t3 = t2 * t;
            w[k][0] = -0.5 * t3 + t2 - 0.5 * t;
            w[k][1] = 1.5 * t3 - 2.5 * t2 + 1.0;
            w[k][2] = -1.5 * t3 + 2.0 * t2 + 0.5 * t;
            w[k][3] = 0.5 * t3 - 0.5 * t2;
        } else {
            w[k][0] = 1.0 - t;
            w[k][1] = t;
        }
    }
    constexpr int OFF = ORDER == 4 ? -1 : 0;
    double s0 = 0, s1 = 0, s2 = 0;
    if constexpr (ORDER == 4) {
        // nested: 252 FP64 instructions instead of 272
        int iy[4], iz[4];
#pragma unroll
        for (int b = 0; b < 4; b++) {
            iy[b] = pos_mod(i0[1] + OFF + b, ng);
            iz[b] = pos_mod(i0[2] + OFF + b, ng);
            STEPS_CHECK_IDX(iy[b], ng, CK_T3_FP64);
            STEPS_CHECK_IDX(iz[b], ng, CK_T3_FP64);
        }
#pragma unroll
        for (int a = 0; a < 4; a++) {
            int ix = pos_mod(i0[0] + OFF + a, ng);
            STEPS_CHECK_IDX(ix, ng, CK_T3_FP64);
            double p[3];
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const double *row = tab + (size_t)(ix * ng + iy[b]) * ng * 3;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    double z = w[2][0] * __ldg(row + 3 * iz[0] + c);
                    z = fma(w[2][1], __ldg(row + 3 * iz[1] + c), z);
                    z = fma(w[2][2], __ldg(row + 3 * iz[2] + c), z);
                    z = fma(w[2][3], __ldg(row + 3 * iz[3] + c), z);
                    p[c] = b == 0 ? w[1][0] * z : fma(w[1][b], z, p[c]);
                }
            }
            s0 = fma(w[0][a], p[0], s0);
            s1 = fma(w[0][a], p[1], s1);
            s2 = fma(w[0][a], p[2], s2);
        }
        Dx = s0;
        Dy = s1;
        Dz = s2;
        return;
    }
#pragma unroll
    for (int a = 0; a < ORDER; a++) {
        int ix = pos_mod(i0[0] + OFF + a, ng);
        STEPS_CHECK_IDX(ix, ng, CK_T3_FP64);
#pragma unroll
        for (int b = 0; b < ORDER; b++) {
            int iy = pos_mod(i0[1] + OFF + b, ng);
            STEPS_CHECK_IDX(iy, ng, CK_T3_FP64);
            double wxy = w[0][a] * w[1][b];
            const double *row = tab + (size_t)(ix * ng + iy) * ng * 3;
#pragma unroll
            for (int c = 0; c < ORDER; c++) {
                int iz = pos_mod(i0[2] + OFF + c, ng);
                STEPS_CHECK_IDX(iz, ng, CK_T3_FP64);
                double ww = wxy * w[2][c];
                s0 += ww * __ldg(row + 3 * iz);
                s1 += ww * __ldg(row + 3 * iz + 1);
                s2 += ww * __ldg(row + 3 * iz + 2);
            }
        }
    }
    Dx = s0;
    Dy = s1;
    Dz = s2;
}

// (rho, z) table interpolation, NGP / CIC / TSC (StePS/src/ewald_space.cc:803-1048,
// StePS/src/forces_cuda.cu:188-455), then D_rho mapped to (x, y).
template <int ORDER>
__device__ __forceinline__ void s1r2_interp_fp64(const double *__restrict__ T, int nrho, int nz, double rho_max,
                                                 double lz, double dx, double dy, double dz, double &Dx, double &Dy,
                                                 double &Dz)
{
    double rho = sqrt(dx * dx + dy * dy);
    double half = 0.5 * lz;
    double drho = rho_max / (double)(nrho - 1 > 1 ? nrho - 1 : 1);
    double dzc = lz / (double)nz;
    double rr = rho < 0 ? 0 : (rho > rho_max ? rho_max : rho);
    double ur = drho > 0 ? rr / drho : 0.0;
    double uz = (dz + half) / dzc - 0.5;
    double Dr = 0, Dzz = 0;
    auto at = [&](int ir, int iz, int c) {
        STEPS_CHECK_IDX(ir, nrho, CK_S1_CELL);
        STEPS_CHECK_IDX(iz, nz, CK_S1_CELL);
        return __ldg(T + ((size_t)ir * nz + iz) * 2 + c);
    };
    if (ORDER == 0) {
        int ir = (int)floor(ur + 0.5);
        int iz = (int)floor(uz + 0.5);
        ir = ir < 0 ? 0 : (ir > nrho - 1 ? nrho - 1 : ir);
        iz = pos_mod(iz, nz);
        Dr = at(ir, iz, 0);
        Dzz = at(ir, iz, 1);
    } else if (ORDER == 2) {
        int ir0 = (int)floor(ur);
        double fr = ur - (double)ir0;
        if (ir0 < 0) { ir0 = 0; fr = 0; }
        if (ir0 > nrho - 2) { ir0 = nrho - 2 > 0 ? nrho - 2 : 0; fr = 1.0; }
        int ir1 = ir0 + 1;
        int iz0 = (int)floor(uz);
        double fz = uz - (double)iz0;
        iz0 = pos_mod(iz0, nz);
        int iz1 = pos_mod(iz0 + 1, nz);
        double w00 = (1.0 - fr) * (1.0 - fz), w10 = fr * (1.0 - fz), w01 = (1.0 - fr) * fz, w11 = fr * fz;
        Dr = w00 * at(ir0, iz0, 0) + w10 * at(ir1, iz0, 0) + w01 * at(ir0, iz1, 0) + w11 * at(ir1, iz1, 0);
        Dzz = w00 * at(ir0, iz0, 1) + w10 * at(ir1, iz0, 1) + w01 * at(ir0, iz1, 1) + w11 * at(ir1, iz1, 1);
    } else {
        int jr = (int)floor(ur + 0.5);
        int jz = (int)floor(uz + 0.5);
        double sr = ur - (double)jr, sz = uz - (double)jz;
        double wr[3] = {0.5 * (0.5 - sr) * (0.5 - sr), 0.75 - sr * sr, 0.5 * (0.5 + sr) * (0.5 + sr)};
        double wz[3] = {0.5 * (0.5 - sz) * (0.5 - sz), 0.75 - sz * sz, 0.5 * (0.5 + sz) * (0.5 + sz)};
        // a NaN separation converts to the lowest int: clamped before it is used
        const int jc = min(max(jr, 0), nrho - 1), zc = pos_mod(jz, nz);
        const int ir[3] = {max(jc - 1, 0), jc, min(jc + 1, nrho - 1)};
        const int izs[3] = {zc > 0 ? zc - 1 : nz - 1, zc, zc < nz - 1 ? zc + 1 : 0};
#pragma unroll
        for (int zr = 0; zr < 3; zr++) {
            double w0 = wr[0] * wz[zr], w1 = wr[1] * wz[zr], w2 = wr[2] * wz[zr];
            Dr += w0 * at(ir[0], izs[zr], 0) + w1 * at(ir[1], izs[zr], 0) + w2 * at(ir[2], izs[zr], 0);
            Dzz += w0 * at(ir[0], izs[zr], 1) + w1 * at(ir[1], izs[zr], 1) + w2 * at(ir[2], izs[zr], 1);
        }
    }
    double ex = rho > 0 ? dx / rho : 0.0;
    double ey = rho > 0 ? dy / rho : 0.0;
    Dx = Dr * ex;
    Dy = Dr * ey;
    Dz = Dzz;
}

__device__ __forceinline__ double nearest(double d, double L, double halfL)
{
    // Subtract L sign(d) once when |d| > L/2 (StePS/src/forces.cc:812-817).
    // Non-negative doubles compare as their bits: no FP64 instruction (NaN
    // compares above and stays NaN).
    return (__double_as_longlong(d) & 0x7fffffffffffffffLL) > __double_as_longlong(halfL) ? d - copysign(L, d) : d;
}

constexpr int MAX_EMAX = 64;  // derive_params refuses more images

// m L for the images of the S1xR2 image sum, once per block.
template <int MODE>
__device__ __forceinline__ void image_shifts(const KParams &kp, double *smL)
{
    if (MODE != M_S1_IMAGES) return;
    for (int m = threadIdx.x; m <= 2 * kp.emax; m += blockDim.x) smL[m] = (double)(m - kp.emax) * kp.L;
    __syncthreads();
}

// Kernel vector k of one pair: the force on i is m_j k, on j -m_i k.
template <int MODE, int ORDER, class Beta>
__device__ __forceinline__ void pair_fp64(const KParams &kp, const Tables &tb, double ih, const double *smL, double dx,
                                          double dy, double dz, float b2, Beta beta, double *k)
{
    const double L = kp.L, halfL = kp.halfL;
    if (MODE == M_T3_EWALD || MODE == M_NEAREST3) {
        dx = nearest(dx, L, halfL);
        dy = nearest(dy, L, halfL);
    }
    if (MODE != M_S1_IMAGES && MODE != M_R3) dz = nearest(dz, L, halfL);
    if (MODE == M_S1_IMAGES) {
        // Images m in [-emax, emax] along z inside the cut
        // (StePS/src/forces.cc:1250-1290).
        const double rho2 = dx * dx + dy * dy;
        double sw = 0, sz = 0;
        for (int m = 0; m <= 2 * kp.emax; ++m) {
            const double dzm = dz + smL[m];
            // |dzm| <= cutL on the bits, as in nearest()
            if ((__double_as_longlong(dzm) & 0x7fffffffffffffffLL) <= __double_as_longlong(kp.cutL)) {
                const double w = weight_fp64(rho2 + dzm * dzm, b2, beta);
                sw += w;
                sz = fma(w, dzm, sz);
            }
        }
        k[0] = sw * dx;
        k[1] = sw * dy;
        k[2] = sz;
        return;
    }
    const double w = weight_fp64(dx * dx + dy * dy + dz * dz, b2, beta);
    if (MODE == M_T3_EWALD || MODE == M_S1_TABLE) {
        double Dx, Dy, Dz;
        if constexpr (MODE == M_T3_EWALD) t3_interp_fp64<ORDER>(tb.t3, tb.t3_ng, L, ih, dx, dy, dz, Dx, Dy, Dz);
        else s1r2_interp_fp64<ORDER>(tb.s1r2, tb.nrho, tb.nz, tb.rho_max, L, dx, dy, dz, Dx, Dy, Dz);
        k[0] = fma(w, dx, -Dx);
        k[1] = fma(w, dy, -Dy);
        k[2] = fma(w, dz, -Dz);
    } else {
        k[0] = w * dx;
        k[1] = w * dy;
        k[2] = w * dz;
    }
}

template <int MODE, int ORDER>
__global__ void __launch_bounds__(FP64_THREADS)
    k_pair_fp64(const double4_16a *__restrict__ pj, const double *__restrict__ ej, const float *__restrict__ ejf, int n,
                int id_min, int ni, int jchunk, KParams kp, Tables tb, double *__restrict__ part)
{
    __shared__ double4_16a sp[FP64_THREADS];
    __shared__ float se[FP64_THREADS];
    __shared__ double smL[2 * MAX_EMAX + 1];
    int t = threadIdx.x;
    int li = blockIdx.x * FP64_THREADS + t;
    bool active = li < ni;
    double4_16a pi = active ? pj[id_min + li] : make_double4_16a(0, 0, 0, 0);
    const size_t ii = active ? id_min + li : 0;
    const float ei = ejf[ii];
    image_shifts<MODE>(kp, smL);
    int j0 = blockIdx.y * jchunk;
    int j1 = min(n, j0 + jchunk);
    double ax = 0, ay = 0, az = 0;
    const double ih = MODE == M_T3_EWALD ? (double)tb.t3_ng / kp.L : 0.0;
    for (int jb = j0; jb < j1; jb += FP64_THREADS) {
        int cnt = min(FP64_THREADS, j1 - jb);
        __syncthreads();
        if (t < cnt) {
            sp[t] = pj[jb + t];
            se[t] = ejf[jb + t];
        }
        __syncthreads();
        for (int jj = 0; jj < cnt; ++jj) {
            double4_16a q = sp[jj];
            const double dx = q.x - pi.x, dy = q.y - pi.y, dz = q.z - pi.z;
            const auto beta = [&] { return ej[ii] + ej[jb + jj]; };
            if (MODE == M_R3) {
                const double w = q.w * weight_fp64(dx * dx + dy * dy + dz * dz, support2_fp32(ei, se[jj]), beta);
                ax = fma(w, dx, ax);
                ay = fma(w, dy, ay);
                az = fma(w, dz, az);
            } else {
                double k[3];
                pair_fp64<MODE, ORDER>(kp, tb, ih, smL, dx, dy, dz, support2_fp32(ei, se[jj]), beta, k);
                ax = fma(q.w, k[0], ax);
                ay = fma(q.w, k[1], ay);
                az = fma(q.w, k[2], az);
            }
        }
    }
    if (active) {
        double *o = part + ((size_t)blockIdx.y * ni + li) * 3;
        o[0] = ax;
        o[1] = ay;
        o[2] = az;
    }
}

// The j stream (x, y, z, m) and the softening lengths rounded up to FP32.
__global__ void k_pack64(const double *__restrict__ x, const double *__restrict__ m, const double *__restrict__ eps, int n,
                         double4_16a *__restrict__ out, float *__restrict__ epsf)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = make_double4_16a(x[3 * (size_t)i], x[3 * (size_t)i + 1], x[3 * (size_t)i + 2], m[i]);
    epsf[i] = __double2float_ru(eps[i]);
}

// All particles, each pair once (Newton's third law). The kernel is bound by
// the FP64 pipe, which retires one warp instruction in 16 cycles per SM, so
// everything that runs beside it is free: a lane holds one i particle of a row
// of 32 and meets j particle (lane + s) mod 32 of a group of 32 in step s; the
// j sums move one lane on after each step (6 shuffles) and are added to the
// group's slab in the memory system. Items, slabs and reduction as in
// pair_sym.cu, in the caller's order. A row meets itself one-sided.
struct SymFp64Args {
    const double4_16a *p;
    const double *eps;
    const float *epsf;
    int n, nrows, G, C, nitems, step, tri;
    unsigned *counter;
    double *pi, *pj;
    size_t npad;
};

template <int MODE, int ORDER>
__global__ void __launch_bounds__(FP64_THREADS) k_sym_fp64(SymFp64Args a, KParams kp, Tables tb)
{
    __shared__ double smL[2 * MAX_EMAX + 1];
    image_shifts<MODE>(kp, smL);
    const int lane = threadIdx.x & 31, nxt = (lane + 1) & 31;
    const double ih = MODE == M_T3_EWALD ? (double)tb.t3_ng / kp.L : 0.0;
    for (;;) {
        int item = 0;
        if (lane == 0) item = (int)atomicAdd(a.counter, 1u);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= a.nitems) return;
        const int A = item / a.C, ch = item - A * a.C;
        const int r0 = A * a.G, r1 = min(a.nrows, r0 + a.G);
        const int J0 = r0 + (int)((long long)(a.nrows - r0) * ch / a.C);
        const int J1 = r0 + (int)((long long)(a.nrows - r0) * (ch + 1) / a.C);
        if (!check_item(A, div_up(a.nrows, a.G), ch, a.C, 32LL * r0, 32LL * r1, 32LL * J0, 32LL * J1, a.step, a.tri, a.npad,
                        (long long)a.npad))
            continue;
        const size_t jlo = a.tri ? (size_t)r0 * 32 : 0, jlen = a.npad - jlo;
        double *pj = a.pj + 3 * sym_slab(A, a.step, a.tri, a.npad);
        for (int r = r0; r < r1; r++) {
            const size_t i = (size_t)r * 32 + lane;
            const bool ivalid = i < (size_t)a.n;
            const size_t ic = ivalid ? i : 0;
            const double4_16a pi = a.p[ic];
            const float ei = a.epsf[ic];
            double f[3] = {0, 0, 0};
            for (int J = max(J0, r); J < J1; J++) {
                double g[3] = {0, 0, 0};
#pragma unroll 1
                for (int s = 0; s < 32; s++) {
                    const size_t j = (size_t)J * 32 + ((lane + s) & 31);
                    const bool valid = ivalid && j < (size_t)a.n;
                    const size_t jc = valid ? j : ic;
                    const double4_16a q = a.p[jc];
                    const double dx = q.x - pi.x, dy = q.y - pi.y, dz = q.z - pi.z;
                    const float b2 = support2_fp32(ei, a.epsf[jc]);
                    const auto beta = [&] { return a.eps[ic] + a.eps[jc]; };
                    const double mj = valid ? q.w : 0.0, mi = valid ? pi.w : 0.0;
                    if (MODE == M_R3) {
                        const double w = weight_fp64(dx * dx + dy * dy + dz * dz, b2, beta);
                        const double wi = mj * w, wj = mi * w;
                        f[0] = fma(wi, dx, f[0]);
                        f[1] = fma(wi, dy, f[1]);
                        f[2] = fma(wi, dz, f[2]);
                        g[0] = fma(wj, dx, g[0]);
                        g[1] = fma(wj, dy, g[1]);
                        g[2] = fma(wj, dz, g[2]);
                    } else {
                        double k[3];
                        pair_fp64<MODE, ORDER>(kp, tb, ih, smL, dx, dy, dz, b2, beta, k);
#pragma unroll
                        for (int c = 0; c < 3; c++) {
                            f[c] = fma(mj, k[c], f[c]);
                            g[c] = fma(mi, k[c], g[c]);
                        }
                    }
#pragma unroll
                    for (int c = 0; c < 3; c++) g[c] = __shfl_sync(0xffffffffu, g[c], nxt);
                }
                if (J > r) {
                    double *o = pj + ((size_t)J * 32 + lane - jlo);
#pragma unroll
                    for (int c = 0; c < 3; c++) add_slab(o + c * jlen, g[c], r == r0);
                }
            }
#pragma unroll
            for (int c = 0; c < 3; c++) a.pi[((size_t)ch * 3 + c) * a.npad + i] = f[c];
        }
    }
}

}  // namespace

namespace {

__global__ void k_reduce_fp64(const double *__restrict__ part, int S, int ni, int id_min, const double *__restrict__ x,
                              Background bg, double *__restrict__ F)
{
    int li = blockIdx.x * blockDim.x + threadIdx.x;
    if (li >= ni) return;
    double f[3] = {0, 0, 0};
    for (int s = 0; s < S; s++)
        for (int k = 0; k < 3; k++) f[k] += part[((size_t)s * ni + li) * 3 + k];
    add_background(bg, x + 3 * (size_t)(id_min + li), f);
    for (int k = 0; k < 3; k++) F[3 * (size_t)li + k] = f[k];
}

template <int MODE, int ORDER>
void launch_fp64(dim3 grid, int n, int id_min, int ni, int jchunk, const KParams &kp, const Tables &tb, double *part,
                 cudaStream_t st, const SymPlan *sym)
{
    Ctx &c = ctx();
    if (sym) {
        SymFp64Args a{};
        a.p = c.pack64.as<double4_16a>();
        a.eps = c.eps64.as<double>();
        a.epsf = c.epsf64.as<float>();
        a.n = n;
        a.nrows = sym->nrows;
        a.G = sym->G;
        a.C = sym->C;
        a.nitems = sym->groups * sym->C;
        a.step = sym->step;
        a.tri = sym->tri;
        a.counter = c.counter.as<unsigned>();
        a.npad = sym->npad;
        a.pi = part;
        a.pj = part + 3 * (size_t)sym->C * sym->npad;
        int occ = 0;
        STEPS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_sym_fp64<MODE, ORDER>, FP64_THREADS, 0));
        const int blocks = std::min(div_up(a.nitems, FP64_THREADS / 32), c.nsm * std::max(occ, 1));
        k_sym_fp64<MODE, ORDER><<<blocks, FP64_THREADS, 0, st>>>(a, kp, tb);
        note_launch("k_sym_fp64");
        return;
    }
    k_pair_fp64<MODE, ORDER><<<grid, FP64_THREADS, 0, st>>>(c.pack64.as<double4_16a>(), c.eps64.as<double>(),
                                                            c.epsf64.as<float>(), n, id_min, ni, jchunk, kp, tb, part);
    note_launch("k_pair_fp64");
}

}  // namespace

Background background_of(const KParams &kp, const Tables &tb)
{
    Background bg{0, 0.0, kp.rsim, tb.radial, tb.radial_size};
    if (kp.comoving_bg == 0) return bg;
    if (kp.topology == STEPS_R3) {
        bg.mode = 1;
        bg.coef = kp.bg_coef;
    } else if (kp.topology == STEPS_S1R2) {
        bool table_mode = kp.is_periodic >= 2 && !kp.s1r2_images;
        if (kp.comoving_bg == 1 && !table_mode) {
            if (!tb.radial || tb.radial_size < 2) fail(STEPS_E_STATE, "S1R2 comoving run needs the radial force table");
            bg.mode = 3;
        } else {
            bg.mode = 2;
        }
        bg.coef = kp.bg_coef;
    }
    return bg;
}

// Rows of 32 particles in the caller's order.
static bool fp64_plan(int n, SymPlan &p)
{
    p.NP = 0;
    p.nrows = p.ntiles = div_up(n, 32);
    p.npad = (size_t)p.nrows * 32;
    p.gran = 32;
    const bool ok = sym_split(p, 32);
    return ok;
}

void forces_fp64(const KParams &kp, const Tables &tb, const double *x, int n, int id_min, int ni, double *F)
{
    Ctx &c = ctx();
    cudaStream_t st = c.stream;
    c.pack64.ensure<double4_16a>(n);
    STEPS_CUDA(cudaEventRecord(c.phase[0], st));
    k_pack64<<<div_up(n, 256), 256, 0, st>>>(x, c.m64.as<double>(), c.eps64.as<double>(), n, c.pack64.as<double4_16a>(),
                                            c.epsf64.ensure<float>(n));
    note_launch("k_pack64");
    STEPS_CUDA(cudaEventRecord(c.phase[1], st));

    // Enough blocks for several waves of the GPU: split the j range.
    int bx = div_up(ni, FP64_THREADS);
    int target = c.nsm * 16;
    int S = div_up(target, bx);
    int maxS = div_up(n, FP64_THREADS);
    if (S > maxS) S = maxS;
    if (S < 1) S = 1;
    int jchunk = div_up(div_up(n, S), FP64_THREADS) * FP64_THREADS;
    S = div_up(n, jchunk);
    SymPlan plan, *sym = nullptr;
    if (id_min == 0 && ni == n && n >= SYM_FP64_MIN_N && fp64_odd(kp, tb) && fp64_plan(n, plan) &&
        c.partial.fits(plan.doubles * sizeof(double))) {
        try {
            c.partial.ensure<double>(plan.doubles);
            c.counter.ensure<unsigned>(4);
            STEPS_CUDA(cudaMemsetAsync(c.counter.p, 0, sizeof(unsigned), st));
            sym = &plan;
        } catch (const Error &e) {
            if (e.code != STEPS_E_NOMEM) throw;  // the one-sided kernel needs less
        }
    }
    double *part = sym ? c.partial.as<double>() : c.partial.ensure<double>((size_t)S * ni * 3);
    dim3 grid(bx, S);

    if (kp.topology == STEPS_R3) {
        launch_fp64<M_R3, 0>(grid, n, id_min, ni, jchunk, kp, tb, part, st, sym);
    } else if (kp.topology == STEPS_T3) {
        if (kp.is_periodic >= 2) {
            if (kp.order == 4) launch_fp64<M_T3_EWALD, 4>(grid, n, id_min, ni, jchunk, kp, tb, part, st, sym);
            else launch_fp64<M_T3_EWALD, 2>(grid, n, id_min, ni, jchunk, kp, tb, part, st, sym);
        } else {
            launch_fp64<M_NEAREST3, 0>(grid, n, id_min, ni, jchunk, kp, tb, part, st, sym);
        }
    } else {
        if (kp.is_periodic < 2) launch_fp64<M_S1_NEAREST, 0>(grid, n, id_min, ni, jchunk, kp, tb, part, st, sym);
        else if (kp.s1r2_images) launch_fp64<M_S1_IMAGES, 0>(grid, n, id_min, ni, jchunk, kp, tb, part, st, sym);
        else if (kp.order == 0) launch_fp64<M_S1_TABLE, 0>(grid, n, id_min, ni, jchunk, kp, tb, part, st, sym);
        else if (kp.order == 2) launch_fp64<M_S1_TABLE, 2>(grid, n, id_min, ni, jchunk, kp, tb, part, st, sym);
        else launch_fp64<M_S1_TABLE, 4>(grid, n, id_min, ni, jchunk, kp, tb, part, st, sym);
    }
    STEPS_CUDA(cudaEventRecord(c.phase[2], st));
    if (sym) {
        sym_reduce(plan, part, nullptr, n, x, background_of(kp, tb), F);
    } else {
        k_reduce_fp64<<<div_up(ni, 256), 256, 0, st>>>(part, S, ni, id_min, x, background_of(kp, tb), F);
        note_launch("k_reduce_fp64");
    }
    STEPS_CUDA(cudaEventRecord(c.phase[3], st));
    c.phase_valid = true;
    c.last_pairs = (double)ni * (double)n;
}

}  // namespace steps
