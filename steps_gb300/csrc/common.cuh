// Shared declarations of libsteps_gb300: the persistent device context,
// error handling, kernel parameter blocks and device math helpers.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "steps_gb300.h"

namespace steps {

// ---------------------------------------------------------------- errors --

struct Error {
    int code;
    std::string msg;
};

[[noreturn]] void fail(int code, const std::string &msg);
void check_cuda(cudaError_t e, const char *what, const char *file, int line);
#define STEPS_CUDA(expr) ::steps::check_cuda((expr), #expr, __FILE__, __LINE__)

// ------------------------------------------------------------ device buf --

// A growable device allocation owned by the context. Grows (free + malloc)
// only when a request exceeds its capacity; never shrinks until shutdown.
struct DevBuf {
    void *p = nullptr;
    size_t bytes = 0;
    template <class T>
    T *as() const { return static_cast<T *>(p); }
    template <class T>
    T *ensure(size_t count) { grow(count * sizeof(T)); return static_cast<T *>(p); }
    void grow(size_t want);
    // Whether the buffer holds `want` bytes, or could if it were released and
    // allocated again: a call that has a way to do with less asks first, since a
    // grow() that fails has released the old buffer.
    bool fits(size_t want) const;
    void release();
};

// ------------------------------------------------- kernel parameter blocks --

// Physics parameters as the kernels read them (derived once per call).
struct KParams {
    int topology;
    int is_periodic;
    int comoving_bg;   // 0 none, 1 mass_in_unit_sphere * x, 2 H0^2 Omega_L * x
    int s1r2_images;   // S1R2 with is_periodic >= 2: explicit images (1) or table (0)
    int emax;          // S1R2 image range [-emax, emax] (ewald_max = IS_PERIODIC + 1)
    int order;         // interpolation order of the active table
    double L, halfL, cutL;  // cutL = (emax - 0.4) * L
    double bg_coef;
    double rsim;
};

// Tables resident on the device (FP64 as StePS builds them).
struct Tables {
    const double *t3;  // ngrid^3 * 3
    int t3_ng;
    const double *s1r2;  // nrho * nz * 2
    int nrho, nz;
    double rho_max;
    const double *radial;  // cylindrical background multiplier
    int radial_size;
};

// A set of particles ordered along a Morton curve and cut into tiles of T.
// pack[q] = (x - c, y - c, z - c, m) of the q-th particle in curve order,
// relative to its tile's centre c (exactly representable in FP32);
// meta[2t] = (c.x, c.y, c.z, eps_max), meta[2t+1] = (half extents, 0).
struct TileSet {
    int lo = 0, count = 0;  // original index range [lo, lo + count)
    int T = 0, ntiles = 0;
    DevBuf keys[2], vals[2], hist;
    DevBuf pack, eps, meta;
    DevBuf idx;  // idx[q] = original index of curve position q; padding holds pad_id
    DevBuf resid;  // resid[q] = (x - c) - pack[q].xyz, the FP32 residual of the offset
    DevBuf soa;    // tile-blocked SoA copy of pack: X[T], Y[T], Z[T], M[T] per tile
    DevBuf sub;    // per SUBTILE particles: (box centre offset, eps_max), (half extents, 0)
    int perm_sel = 0;  // vals[perm_sel] holds curve position -> original index
    bool ordered = false;
    const uint32_t *perm() const { return vals[perm_sel].as<uint32_t>(); }
};

// Mixed-kernel launch shape (one-sided kernels; auto_shape where the caller set none).
struct Shape {
    int threads = 128;
    int ipt = 2;
    int jsplit = 0;
    int variant = 0;  // R^3: 0 scalar FP32 pair loop; 1, 2, 3 packed FP32x2 (0, 768, 1024 threads/SM
                      // asked); 4 packed with the bulk-copy (TMA) + mbarrier pipeline
    bool sym = true;  // full-range calls may evaluate each pair once (pair_sym.cu); off once the caller chose a shape or pair loop
    float guard = 30.0f;  // tile-pair scale / gap above which the double-float path runs
    int t3_cells = 0;  // T^3: shared-memory table window capacity in cells (0 = haloed table via L1/L2)
};

// ------------------------------------------------------------- utilities --

inline __host__ __device__ int div_up(int a, int b) { return (a + b - 1) / b; }

// Particles per j sub-tile: the near/far decision of the packed R^3 kernel is
// taken per (warp, sub-tile) from the sub-tile boxes the tile build writes.
constexpr int SUBTILE = 16;

// Kernel-launch bookkeeping: counts launches and surfaces launch errors.
void note_launch(const char *name);
// Adds kernels launched by other means (the kernel nodes of a graph launch).
void add_launches(long long k);

// ------------------------------------------------- debug bounds checks --
//
// Compiled with -DSTEPS_CHECK (libsteps_gb300_check.so), STEPS_CHECK_IDX(v,
// bound, site) compares the index variable v with [0, bound). The first index
// out of range in this translation unit is recorded (site, index, bound), v
// is set to 0 so that the access it guards stays inside its buffer, and the
// C-ABI call that launched the kernel returns STEPS_E_BOUNDS with the record
// in its message. In the normal build the macro is empty.
enum CheckSite {
    CK_NONE = 0,
    CK_I_TILE,      // i tile of a work item
    CK_J_TILE,      // j tile range of a work item
    CK_CHUNK,       // j chunk (partial slab) of a work item
    CK_SLOT,        // partial slot of a work-list item or of an i tile
    CK_OUTPUT,      // caller-order output row (curve position -> original index - id_min)
    CK_T3_CELL,     // cell of the FP32 T^3 table (haloed copy, window or wrapped read)
    CK_T3_FP64,     // cell of the FP64 T^3 table
    CK_S1_CELL,     // (rho, z) cell of the S1xR2 table or of its records
    CK_RADIAL,      // entry of the cylindrical radial-force table
    CK_PERM,        // original particle index read from the ordering
    CK_SCATTER,     // destination of a radix-sort scatter
    CK_SELFTEST,    // steps_gpu_test_bounds_check
    CK_NSITES
};

struct CheckRecord {
    int code;  // 0, or STEPS_E_BOUNDS once an index failed
    int site;
    long long index, bound;
};

#ifdef STEPS_CHECK
static __device__ CheckRecord g_check_record;

static __device__ __noinline__ void check_failed(long long index, long long bound, int site)
{
    if (atomicCAS(&g_check_record.code, 0, STEPS_E_BOUNDS) == 0) {
        g_check_record.site = site;
        g_check_record.index = index;
        g_check_record.bound = bound;
        __threadfence();
    }
}

#define STEPS_CHECK_IDX(v, bound, site)                                                          \
    do {                                                                                         \
        if ((unsigned long long)(long long)(v) >= (unsigned long long)(long long)(bound)) {     \
            ::steps::check_failed((long long)(v), (long long)(bound), (site));                   \
            (v) = 0;                                                                             \
        }                                                                                        \
    } while (0)

// True when the cells [first, last] lie in [0, bound); otherwise records the
// offending end and returns false (the caller then moves the access to 0).
static __device__ __forceinline__ bool check_span(long long first, long long last, long long bound, int site)
{
    if (first >= 0 && last < bound) return true;
    check_failed(first < 0 ? first : last, bound, site);
    return false;
}

// Each translation unit registers where its record lives; the C-ABI reads
// every record after each call.
int register_check_record(void *(*where)());
static void *check_record_address()
{
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, g_check_record) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return p;
}
static const int g_check_registered = register_check_record(&check_record_address);
#else
#define STEPS_CHECK_IDX(v, bound, site) ((void)0)
#endif

// ---------------------------------------------------- device math helpers --

// Order-preserving integer image of a double (atomic min/max of bounding boxes).
__device__ __forceinline__ unsigned long long ordered_bits(double d)
{
    unsigned long long b = (unsigned long long)__double_as_longlong(d);
    return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}

__device__ __forceinline__ double from_ordered_bits(unsigned long long u)
{
    unsigned long long b = (u & 0x8000000000000000ull) ? (u & 0x7fffffffffffffffull) : ~u;
    return __longlong_as_double((long long)b);
}

__device__ __forceinline__ bool is_nan_bits(double v)
{
    return (__double_as_longlong(v) & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL;
}

// Extends lo = min and nhi = ~max of ordered images by v; NaN is left out.
__device__ __forceinline__ void extend_box(double v, unsigned long long &lo, unsigned long long &nhi)
{
    const unsigned long long u = ordered_bits(v);
    if (is_nan_bits(v)) return;
    lo = min(lo, u);
    nhi = min(nhi, ~u);
}

__device__ __forceinline__ unsigned long long spread3(unsigned long long v)
{
    // Spread the low 21 bits of v to every third bit.
    v &= 0x1fffffull;
    v = (v | (v << 32)) & 0x1f00000000ffffull;
    v = (v | (v << 16)) & 0x1f0000ff0000ffull;
    v = (v | (v << 8)) & 0x100f00f00f00f00full;
    v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
    v = (v | (v << 2)) & 0x1249249249249249ull;
    return v;
}



// MUFU reciprocal square root, approximate (relative error < 2^-22), FTZ.
__device__ __forceinline__ float rsqrt_mufu(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float sqrt_mufu(float x)
{
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float rcp_mufu(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// r^-3 of a pair known to be outside its softening support, from r^2, on as few
// FP64 instructions as it takes (4). The FP64 pipe, 1/64 of the FP32 rate,
// bounds the FP64 kernels, so what other pipes can do exactly or accurately
// enough is moved there. With the MUFU seed y ~ r^-1 and e = 1 - r^2 y^2,
//   r^-3 = y^3 (1 + 3 e / 2 + 15 e^2 / 8 + O(e^3)),  |e| < 2^-20.9:
//   * r^2 and y change format by integer instructions (the conversions run on
//     the FP64 pipe);
//   * y^2 is exact in 48 bits, an integer product;
//   * 15 e^2 / 8 < 2^-40.8 is needed to 2^-13 of itself: FP32.
// b2: an FP32 upper bound of the squared support. False, with w untouched,
// where r^2 may lie inside it or outside the FP32 range: the caller then takes
// softening_fp64. Against a reciprocal root of 10 instructions with its
// conversions and cube, and 3 for the comparison: R^3 at n = 32,768, one-sided
// 43.7 -> 31.1 ms (with 6 instructions here).
__device__ __forceinline__ double widen_fp32(int bits)  // a normal, positive float
{
    return __hiloint2double((bits >> 3) + (896 << 20), bits << 29);
}

__device__ __forceinline__ bool far_r3_fp64(double r2, float b2, double &w)
{
    const int hi = __double2hiint(r2), lo = __double2loint(r2);
    const float f = __int_as_float((int)__funnelshift_l((unsigned)lo, (unsigned)hi - (896u << 20), 3));  // truncated
    if (!((unsigned)hi - (897u << 20) < (253u << 20) && f > b2)) return false;
    const int yb = __float_as_int(rsqrt_mufu(f));
    const double y = widen_fp32(yb);
    // y^2 = M^2 2^(2 E) with a 24-bit M: M^2 has 47 or 48 bits
    const unsigned m = ((unsigned)yb & 0x7fffffu) | 0x800000u;
    const unsigned long long mm = (unsigned long long)m * m;
    const int top = (int)(mm >> 47);
    const long long ex = 2 * ((yb >> 23) - 127) + top + 1022;
    const double q = __longlong_as_double((long long)(mm << (6 - top)) + (ex << 52));
    const double e = fma(-r2, q, 1.0), y3 = q * y;
    const int eh = max(__double2hiint(e) & 0x7fffffff, 897 << 20);
    const float ef = __int_as_float((eh - (896 << 20)) << 3);
    const double s2 = widen_fp32(__float_as_int(1.875f * ef * ef));  // 2^-127 where it underflows
    w = fma(y3, fma(1.5, e, s2), y3);
    return true;
}

// FP32 bound for far_r3_fp64 of the support (ei + ej)^2, from softening lengths
// rounded up to FP32 (1e-5 covers the FP32 sum and square and f's truncation).
__device__ __forceinline__ float support2_fp32(float ei, float ej)
{
    const float b = ei + ej;
    return b * b * 1.00001f;
}

// Cubic-spline softened force coefficient w(r, beta) for r < beta (the
// r >= beta branch is 1/r^3). StePS/src/forces.cc:52-87,
// StePS/src/forces_cuda.cu:466-519, written in u = r / beta:
//   u <= 1/2 : (32 u^3 - 38.4 u^2 + 32/3) / beta^3
//   u >  1/2 : (-32/3 u^3 + 38.4 u^2 - 48 u + 64/3) / beta^3 - (1/15) / r^3
__device__ __forceinline__ double spline_inner_fp64(double r, double beta)
{
    double ib = 1.0 / beta;
    double u = r * ib;
    double ib3 = ib * ib * ib;
    if (u <= 0.5) return ib3 * (u * u * (32.0 * u - 38.4) + 32.0 / 3.0);
    double r3 = r * r * r;
    return ib3 * (u * (u * (-32.0 / 3.0 * u + 38.4) - 48.0) + 64.0 / 3.0) - (1.0 / 15.0) / r3;
}

// Any r^2: few pairs come here (far_r3_fp64), those whose r^2 is outside the
// FP32 range among them.
__device__ __forceinline__ double softening_fp64(double r2, double beta)
{
    if (r2 >= beta * beta) {
        const double y = 1.0 / sqrt(r2);
        return y * y * y;
    }
    return spline_inner_fp64(sqrt(r2), beta);
}

// Softened weight w(r^2) of a pair; beta() gives its softening support, read
// only where it matters.
template <class Beta>
__device__ __forceinline__ double weight_fp64(double r2, float b2, Beta beta)
{
    double w;
    if (!far_r3_fp64(r2, b2, w)) w = softening_fp64(r2, beta());
    return w;
}

__device__ __forceinline__ float spline_inner_f32(float r2, float beta)
{
    float r = sqrt_mufu(r2);
    float ib = rcp_mufu(beta);
    float u = r * ib;
    float ib3 = ib * ib * ib;
    if (u <= 0.5f) return ib3 * (u * u * (32.0f * u - 38.4f) + (32.0f / 3.0f));
    float ir = rcp_mufu(r);
    return ib3 * (u * (u * (-32.0f / 3.0f * u + 38.4f) - 48.0f) + (64.0f / 3.0f)) -
           (1.0f / 15.0f) * ir * ir * ir;
}

}  // namespace steps
