// Spatial ordering of a particle set for the mixed-precision kernels:
//   1. bounding box (FP64, atomic min/max on order-preserving integer images),
//   2. 63-bit Morton keys (21 bits per axis) of the positions in the box,
//   3. a stable least-significant-digit radix sort of (key, index) pairs,
//   4. tiles of T consecutive particles along the curve: each tile gets an
//      FP32-exact centre c, FP32 offsets x - c computed in FP64, half extents
//      and its largest softening length.
// The order only sets locality (tile size, hence FP32 offset magnitude and
// the near/far split); the forces do not depend on it beyond rounding.
//
// Sets of at most 32,768 particles are ordered by one kernel, a thread-block
// cluster that holds all of them in shared memory (k_order_cluster).
#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"
#include "context.cuh"
#include "tile.cuh"

namespace steps {

namespace {

constexpr int SORT_THREADS = 256;
constexpr int SORT_ITEMS = 8;  // elements per thread per block
constexpr int SORT_TILE = SORT_THREADS * SORT_ITEMS;
constexpr int RADIX_BITS = 8;
constexpr int RADIX = 1 << RADIX_BITS;

__global__ void k_bbox_init(unsigned long long *bb)
{
    int t = threadIdx.x;
    if (t < 3) bb[t] = ~0ull;        // min
    else if (t < 6) bb[t] = 0ull;    // max
}

// Minima of the 6 values over a block, in threads 0 to 5 (the values of other
// threads are not changed). Integer: FP64 instructions take 16 cycles each.
template <int THREADS>
__device__ __forceinline__ unsigned long long block_min6(unsigned long long *mm,
                                                         unsigned long long (*red)[THREADS / 32])
{
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
#pragma unroll
    for (int k = 0; k < 6; k++) {
        mm[k] = warp_min(mm[k]);
        if (lane == 0) red[k][w] = mm[k];
    }
    __syncthreads();
    unsigned long long v = ~0ull;
    if (t < 6)
        for (int k = 0; k < THREADS / 32; k++) v = min(v, red[t][k]);
    return v;
}

// Bounding box on the ordered images of the coordinates, NaN left out: bb[0..2]
// the minima, bb[3..5] the maxima. Two blocks per SM, since every block ends
// with atomics on the same 6 words (n = 200,003, FP64 comparisons and 782
// blocks with 8 times the atomics: 33 us, now 5).
__global__ void __launch_bounds__(SORT_THREADS) k_bbox(const double *__restrict__ x, int lo, int count,
                                                      unsigned long long *bb)
{
    __shared__ unsigned long long red[6][SORT_THREADS / 32];
    unsigned long long mm[6] = {~0ull, ~0ull, ~0ull, ~0ull, ~0ull, ~0ull};  // min, and ~max
    for (int q = blockIdx.x * SORT_THREADS + threadIdx.x; q < count; q += gridDim.x * SORT_THREADS)
#pragma unroll
        for (int k = 0; k < 3; k++) extend_box(x[3 * (size_t)(lo + q) + k], mm[k], mm[3 + k]);
    const unsigned long long v = block_min6<SORT_THREADS>(mm, red);
    if (threadIdx.x < 3) atomicMin(&bb[threadIdx.x], v);
    else if (threadIdx.x < 6) atomicMax(&bb[threadIdx.x], ~v);
}

// 63-bit keys of particles lo..lo+count-1. The three divisions by the box's
// extents are made once per block (a division per coordinate: 19 us at
// n = 200,003, now 8).
__global__ void __launch_bounds__(SORT_THREADS) k_keys(const double *__restrict__ x, int lo, int count,
                                                      const unsigned long long *bb, unsigned long long *keys,
                                                      uint32_t *vals)
{
    constexpr int CELLS = 1 << 21;
    __shared__ double s_lo[3], s_scale[3];
    if (threadIdx.x < 3) {
        const double l = from_ordered_bits(bb[threadIdx.x]), span = from_ordered_bits(bb[3 + threadIdx.x]) - l;
        s_lo[threadIdx.x] = l;
        s_scale[threadIdx.x] = span > 0 ? (double)CELLS / span : 0.0;
    }
    __syncthreads();
    const int q = blockIdx.x * SORT_THREADS + threadIdx.x;
    if (q >= count) return;
    const double *p = x + 3 * (size_t)(lo + q);
    unsigned long long key = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        // conversions saturate, and NaN (0 times an infinite scale) gives 0
        const int c = min(max(__double2int_rz((p[k] - s_lo[k]) * s_scale[k]), 0), CELLS - 1);
        key |= spread3((unsigned long long)c) << k;
    }
    keys[q] = key;
    vals[q] = (uint32_t)(lo + q);
}

// Per-block digit histograms, stored digit-major: hist[d * nblk + b], and the
// sums over the blocks in total[d].
__global__ void __launch_bounds__(SORT_THREADS) k_hist(const unsigned long long *__restrict__ keys, int n, int shift,
                                                      uint32_t *hist, uint32_t *total)
{
    __shared__ uint32_t h[RADIX];
    h[threadIdx.x] = 0;
    __syncthreads();
    int base = blockIdx.x * SORT_TILE;
    for (int r = 0; r < SORT_ITEMS; r++) {
        int q = base + r * SORT_THREADS + threadIdx.x;
        if (q < n) atomicAdd(&h[(keys[q] >> shift) & (RADIX - 1)], 1u);
    }
    __syncthreads();
    const uint32_t c = h[threadIdx.x];
    hist[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = c;
    if (c) atomicAdd(&total[threadIdx.x], c);
}

// Exclusive scan of hist, a warp per digit: it starts from the totals of the
// lower digits and goes through the digit's blocks 32 at a time (one block of
// 1,024 threads over the whole array: 19 us at n = 200,003, now 4).
__global__ void __launch_bounds__(SORT_THREADS) k_scan(uint32_t *hist, const uint32_t *__restrict__ total, int nblk)
{
    const int lane = threadIdx.x & 31, d = blockIdx.x * (SORT_THREADS / 32) + (threadIdx.x >> 5);  // < RADIX
    uint32_t run = 0;
    for (int k = lane; k < d; k += 32) run += total[k];
    run = __reduce_add_sync(0xffffffffu, run);
    for (int b0 = 0; b0 < nblk; b0 += 32) {
        const int b = b0 + lane;
        const uint32_t c = b < nblk ? hist[(size_t)d * nblk + b] : 0u;
        uint32_t inc = c;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        if (b < nblk) hist[(size_t)d * nblk + b] = run + inc - c;
        run += __shfl_sync(0xffffffffu, inc, 31);
    }
}

// Stable scatter: element order inside a block is (round, warp, lane), which is
// the input order, and ranks among equal digits follow that order.
__global__ void __launch_bounds__(SORT_THREADS) k_scatter(const unsigned long long *__restrict__ kin,
                                                         const uint32_t *__restrict__ vin, int n, int shift,
                                                         const uint32_t *__restrict__ hist,
                                                         unsigned long long *__restrict__ kout,
                                                         uint32_t *__restrict__ vout)
{
    constexpr int WARPS = SORT_THREADS / 32;
    __shared__ uint32_t wc[WARPS][RADIX];
    int t = threadIdx.x, lane = t & 31, w = t >> 5;
    uint32_t run = hist[(size_t)t * gridDim.x + blockIdx.x];  // thread t owns digit t
    unsigned lt = (1u << lane) - 1u;
    int base = blockIdx.x * SORT_TILE;
    for (int r = 0; r < SORT_ITEMS; r++) {
        for (int k = 0; k < WARPS; k++) wc[k][t] = 0;
        __syncthreads();
        int q = base + r * SORT_THREADS + t;
        bool valid = q < n;
        unsigned long long key = valid ? kin[q] : 0ull;
        uint32_t val = valid ? vin[q] : 0u;
        int d = valid ? (int)((key >> shift) & (RADIX - 1)) : RADIX;  // invalid lanes form their own group
        unsigned peers = __match_any_sync(0xffffffffu, d);
        int rank = __popc(peers & lt);
        int leader = __ffs(peers) - 1;
        if (valid && lane == leader) wc[w][d] = __popc(peers);
        __syncthreads();
        // Per digit: exclusive prefix over warps, continuing from earlier rounds.
        for (int k = 0; k < WARPS; k++) {
            uint32_t c = wc[k][t];
            wc[k][t] = run;
            run += c;
        }
        __syncthreads();
        if (valid) {
            uint32_t pos = wc[w][d] + rank;
            STEPS_CHECK_IDX(pos, n, CK_SCATTER);
            kout[pos] = key;
            vout[pos] = val;
        }
        __syncthreads();
    }
}

// Steps 1 to 3 for small sets in one launch: a cluster of up to 8 blocks keeps
// (key, index) elements in shared memory through all passes; digit counts and
// scattered elements travel by distributed shared memory. With a launch per
// step the chain of 15 small kernels, not their work, was the time (whole
// preparation, tiles included: 3,001 particles 93 -> 27 us, 8,192 99 -> 29,
// 32,768 113 -> 57).
// Block b of the cluster holds positions [b CAP, (b + 1) CAP), CAP = 512 E;
// warp w of it the next 32 E, in rounds of 32, so (warp, round, lane) is the
// order of the positions.
constexpr int OC_THREADS = 512, OC_WARPS = OC_THREADS / 32, OC_MAX_E = 8, OC_MAX_CLUSTER = 8;
constexpr int OC_MAX_N = OC_THREADS * OC_MAX_E * OC_MAX_CLUSTER;

struct OrderShared {
    uint32_t cnt[OC_WARPS][RADIX];  // digit counts of each warp, then offsets within the block
    uint32_t hist[RADIX];           // digit counts of the block, read by the cluster
    uint32_t base[RADIX];           // first position of the block's elements of each digit
    unsigned long long box[6];      // box of the block, read by the cluster
    unsigned long long red[6][OC_WARPS];
    unsigned long long all[6];
    unsigned long long e[2][1];     // element buffers, CAP each (dynamic)
};

// |v| 2^-(ex >> 20) truncated to FP32 (0 below its normal range, NaN included),
// for results below 2^127.
__device__ __forceinline__ float scaled_fp32(double v, int ex)
{
    const int hi = (__double2hiint(v) & 0x7fffffff) - ex;
    if (hi < (897 << 20) || is_nan_bits(v)) return 0.0f;
    return __int_as_float((int)__funnelshift_l((unsigned)__double2loint(v), (unsigned)hi - (896u << 20), 3));
}

template <int E>
__global__ void __launch_bounds__(OC_THREADS) k_order_cluster(const double *__restrict__ x, int lo, int count, int bits,
                                                             uint32_t *__restrict__ vals)
{
    namespace cg = cooperative_groups;
    constexpr int CAP = OC_THREADS * E;
    extern __shared__ __align__(16) unsigned char oc_smem[];
    OrderShared &sh = *reinterpret_cast<OrderShared *>(oc_smem);
    unsigned long long *buf0 = &sh.e[0][0], *buf1 = buf0 + CAP;
    cg::cluster_group cl = cg::this_cluster();
    const int nb = (int)cl.num_blocks(), b = (int)cl.block_rank();
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int first = b * CAP + w * 32 * E + lane;  // position of round 0

    // Bounding box on the ordered images of the coordinates: few SMs work here,
    // and FP64 instructions (16 cycles each) would be most of the time.
    unsigned long long mm[6] = {~0ull, ~0ull, ~0ull, ~0ull, ~0ull, ~0ull};  // min, and ~max
#pragma unroll
    for (int r = 0; r < E; r++) {
        const int q = first + 32 * r;
        if (q < count)
            for (int k = 0; k < 3; k++) extend_box(x[3 * (size_t)(lo + q) + k], mm[k], mm[3 + k]);
    }
    const unsigned long long least = block_min6<OC_THREADS>(mm, sh.red);
    if (t < 6) sh.box[t] = least;
    cl.sync();
    if (t < 6) {
        unsigned long long v = ~0ull;
        for (int k = 0; k < nb; k++) v = min(v, *cl.map_shared_rank(&sh.box[t], k));
        sh.all[t] = v;
    }
    __syncthreads();

    // Elements: Morton key of `bits` bits per axis above the index. The offset
    // from the box's corner is taken in FP64, scaled by a power of two so that
    // the box is 1 to 2 wide, and truncated to FP32 on its bits.
    const int cells = 1 << bits;
    double lo3[3];
    float inv[3];
    int ex[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        lo3[k] = from_ordered_bits(sh.all[k]);
        const double span = from_ordered_bits(~sh.all[3 + k]) - lo3[k];
        const int hi = __double2hiint(span);
        ex[k] = (hi & 0x7ff00000) - (1023 << 20);
        const bool ok = span > 0 && span < 1e300;
        inv[k] = ok ? (float)cells / scaled_fp32(span, ex[k]) : 0.0f;
    }
    unsigned long long el[E];
#pragma unroll
    for (int r = 0; r < E; r++) {
        const int q = first + 32 * r;
        unsigned long long key = 0;
        if (q < count)
            for (int k = 0; k < 3; k++) {
                const float u = scaled_fp32(x[3 * (size_t)(lo + q) + k] - lo3[k], ex[k]) * inv[k];
                const int c = min((int)u, cells - 1);  // u >= 0
                key |= spread3((unsigned long long)c) << k;
            }
        el[r] = key << 32 | (unsigned)(lo + q);
    }

    const unsigned lt = (1u << lane) - 1u;
    for (int shift = 0; shift < 3 * bits; shift += RADIX_BITS) {
        unsigned long long *out = (shift / RADIX_BITS) & 1 ? buf1 : buf0;
        for (int d = lane; d < RADIX; d += 32) sh.cnt[w][d] = 0;
        __syncwarp();
        uint32_t rank[E];
#pragma unroll
        for (int r = 0; r < E; r++) {
            const bool valid = first + 32 * r < count;
            const int d = valid ? (int)(el[r] >> (32 + shift) & (RADIX - 1)) : RADIX;
            const unsigned peers = __match_any_sync(0xffffffffu, d);
            const uint32_t before = valid ? sh.cnt[w][d] : 0u;
            rank[r] = before + __popc(peers & lt);
            __syncwarp();
            if (valid && lane == __ffs(peers) - 1) sh.cnt[w][d] = before + __popc(peers);
            __syncwarp();
        }
        __syncthreads();
        if (t < RADIX) {
            uint32_t run = 0;
            for (int k = 0; k < OC_WARPS; k++) {
                const uint32_t c = sh.cnt[k][t];
                sh.cnt[k][t] = run;
                run += c;
            }
            sh.hist[t] = run;
        }
        cl.sync();
        if (t < RADIX) {
            uint32_t before = 0, total = 0;
            for (int k = 0; k < nb; k++) {
                const uint32_t c = *cl.map_shared_rank(&sh.hist[t], k);
                before += k < b ? c : 0u;
                total += c;
            }
            // exclusive scan of the totals over the digits
            uint32_t inc = total;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += v;
            }
            if (lane == 31) sh.red[0][w] = inc;
            sh.base[t] = before + inc - total;
        }
        __syncthreads();
        if (t < RADIX) {
            uint32_t add = 0;
            for (int k = 0; k < w; k++) add += (uint32_t)sh.red[0][k];
            sh.base[t] += add;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < E; r++)
            if (first + 32 * r < count) {
                const int d = (int)(el[r] >> (32 + shift) & (RADIX - 1));
                uint32_t pos = sh.base[d] + sh.cnt[w][d] + rank[r];
                STEPS_CHECK_IDX(pos, count, CK_SCATTER);
                *cl.map_shared_rank(out + pos % CAP, pos / CAP) = el[r];
            }
        cl.sync();
#pragma unroll
        for (int r = 0; r < E; r++)
            if (first + 32 * r < count) el[r] = out[w * 32 * E + 32 * r + lane];
    }
#pragma unroll
    for (int r = 0; r < E; r++)
        if (first + 32 * r < count) vals[first + 32 * r] = (uint32_t)el[r];
}

template <int E>
void launch_order(const double *x, int lo, int count, int bits, uint32_t *vals, int blocks, cudaStream_t st)
{
    const size_t smem = sizeof(OrderShared) + 2 * sizeof(unsigned long long) * OC_THREADS * E;
    STEPS_CUDA(cudaFuncSetAttribute(k_order_cluster<E>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(OC_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = blocks;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    STEPS_CUDA(cudaLaunchKernelEx(&cfg, k_order_cluster<E>, x, lo, count, bits, vals));
    note_launch("k_order_cluster");
}

// Orders a small set: about 1,024 particles a block (2 a thread), more from
// 8,192 on, where the cluster is full.
void order_small(const double *x, int lo, int count, int bits, uint32_t *vals, cudaStream_t st)
{
    int blocks = 1;
    while (blocks < OC_MAX_CLUSTER && blocks * OC_THREADS * 2 < count) blocks *= 2;
    const int e = div_up(count, blocks * OC_THREADS);
    if (e <= 2) launch_order<2>(x, lo, count, bits, vals, blocks, st);
    else if (e <= 4) launch_order<4>(x, lo, count, bits, vals, blocks, st);
    else launch_order<8>(x, lo, count, bits, vals, blocks, st);
}

constexpr int TB_THREADS = 256;

// One block per tile of T particles in curve order. Without descriptors the
// tiles cut one sorted set; with them (batches) every tile names its own
// start and count.
__global__ void __launch_bounds__(TB_THREADS) k_tile_build(const double *__restrict__ x, const double *__restrict__ m,
                                                          const double *__restrict__ eps,
                                                          const uint32_t *__restrict__ perm, long long nx,
                                                          int count, int T,
                                                          float4 *__restrict__ pack, float *__restrict__ epsf,
                                                          float4 *__restrict__ meta, uint32_t *__restrict__ idx,
                                                          uint32_t pad_id, float4 *__restrict__ lo,
                                                          float *__restrict__ soa, const int2 *__restrict__ tdesc,
                                                          float4 *__restrict__ sub)
{
    const int tile = blockIdx.x;
    const int sbase = tdesc ? tdesc[tile].x : tile * T;
    int cnt = tdesc ? tdesc[tile].y : min(T, count - tile * T);
#ifdef STEPS_CHECK
    if (!check_span(sbase, (long long)sbase + cnt - 1, count, CK_PERM)) cnt = 0;
#endif
    build_tile<TB_THREADS>(tile, sbase, cnt, x, m, eps, perm, nx, T, pack, epsf, meta, idx, pad_id, lo, soa,
                                  sub);
}

}  // namespace

// Leading Morton bits that order a set of n particles into compact tiles:
// 2^(bits/3) cells per axis, at least 2^5 times the mean particle spacing,
// so clustered sets still see about one particle per cell in dense regions.
// Bits below are left in input order (the sort is stable).
int morton_sort_bits(int n)
{
    int lg = 0;
    while ((1LL << lg) < (long long)n) lg++;
    const int bits = 3 * ((lg + 2) / 3 + 5);
    return bits < 63 ? bits : 63;
}

// Sorts by key bits lo_bit to hi_bit - 1.
void sort_pairs(TileSet &ts, int n, cudaStream_t st, int lo_bit, int hi_bit)
{
    const int nblk = std::max(div_up(n, SORT_TILE), 1), passes = div_up(hi_bit - lo_bit, RADIX_BITS);
    uint32_t *hist = ts.hist.ensure<uint32_t>((size_t)RADIX * (nblk + passes));
    uint32_t *total = hist + (size_t)RADIX * nblk;
    STEPS_CUDA(cudaMemsetAsync(total, 0, sizeof(uint32_t) * RADIX * passes, st));
    int cur = 0;
    for (int pass = 0; pass < passes; pass++, total += RADIX) {
        const int shift = lo_bit + pass * RADIX_BITS;
        k_hist<<<nblk, SORT_THREADS, 0, st>>>(ts.keys[cur].as<unsigned long long>(), n, shift, hist, total);
        note_launch("k_hist");
        k_scan<<<RADIX * 32 / SORT_THREADS, SORT_THREADS, 0, st>>>(hist, total, nblk);
        note_launch("k_scan");
        k_scatter<<<nblk, SORT_THREADS, 0, st>>>(ts.keys[cur].as<unsigned long long>(), ts.vals[cur].as<uint32_t>(), n,
                                                 shift, hist, ts.keys[cur ^ 1].as<unsigned long long>(),
                                                 ts.vals[cur ^ 1].as<uint32_t>());
        note_launch("k_scatter");
        cur ^= 1;
    }
    ts.perm_sel = cur;
}

// Orders particles [lo, lo+count) of the AoS FP64 array x along a Morton curve
// (unless reuse is set and an order already exists) and (re)builds the tiles.
void build_tiles(TileSet &ts, const double *x, const double *m64, const double *eps64, int lo, int count, int T,
                 bool reuse, cudaStream_t st, unsigned long long *bbox_scratch, uint32_t pad_id, int round_tiles)
{
    if (count <= 0) fail(STEPS_E_ARG, "empty particle set");
    bool same = ts.ordered && ts.lo == lo && ts.count == count;
    ts.T = T;
    ts.ntiles = div_up(count, T);
    const int nbuilt = div_up(ts.ntiles, round_tiles) * round_tiles;  // the rest are empty (all padding)
    size_t padded = (size_t)nbuilt * T;
    if (!(reuse && same)) {
        const int sort_bits = morton_sort_bits(count);
        if (count <= OC_MAX_N && sort_bits <= 30) {
            order_small(x, lo, count, sort_bits / 3, ts.vals[0].ensure<uint32_t>(count), st);
            ts.perm_sel = 0;
        } else {
            for (int b = 0; b < 2; b++) {
                ts.keys[b].ensure<unsigned long long>(count);
                ts.vals[b].ensure<uint32_t>(count);
            }
            k_bbox_init<<<1, 32, 0, st>>>(bbox_scratch);
            note_launch("k_bbox_init");
            const int g = div_up(count, SORT_THREADS);
            k_bbox<<<std::min(g, 2 * ctx().nsm), SORT_THREADS, 0, st>>>(x, lo, count, bbox_scratch);
            note_launch("k_bbox");
            k_keys<<<g, SORT_THREADS, 0, st>>>(x, lo, count, bbox_scratch, ts.keys[0].as<unsigned long long>(),
                                               ts.vals[0].as<uint32_t>());
            note_launch("k_keys");
            // whole digits; one bit too many for them is left out (33 bits, up
            // to 2^18 particles: 4 passes instead of 5)
            sort_pairs(ts, count, st, 63 - RADIX_BITS * div_up(sort_bits - 1, RADIX_BITS), 63);
        }
        ts.lo = lo;
        ts.count = count;
        ts.ordered = true;
    }
    ts.pack.ensure<float4>(padded);
    ts.eps.ensure<float>(padded);
    ts.meta.ensure<float4>(2 * (size_t)nbuilt);
    ts.idx.ensure<uint32_t>(padded);
    ts.resid.ensure<float4>(padded);
    ts.soa.ensure<float4>(padded);
    ts.sub.ensure<float4>(2 * (padded / SUBTILE));
    k_tile_build<<<nbuilt, TB_THREADS, 0, st>>>(x, m64, eps64, ts.perm(), (long long)lo + count, count, T,
                                                   ts.pack.as<float4>(),
                                                   ts.eps.as<float>(), ts.meta.as<float4>(), ts.idx.as<uint32_t>(),
                                                   pad_id, ts.resid.as<float4>(), ts.soa.as<float>(), nullptr,
                                                   ts.sub.as<float4>());
    note_launch("k_tile_build");
}

void tile_build_range(const double *x, const double *m64, const double *eps64, const uint32_t *perm, int count, int T,
                      float4 *pack, float *epsf, float4 *meta, uint32_t *idx, uint32_t pad_id, float4 *lo, float *soa,
                      const int2 *tdesc, int ntiles, cudaStream_t st, float4 *sub)
{
    int nt = tdesc ? ntiles : div_up(count, T);
    k_tile_build<<<nt, TB_THREADS, 0, st>>>(x, m64, eps64, perm, count, count, T, pack, epsf, meta, idx, pad_id, lo,
                                            soa, tdesc, sub);
    note_launch("k_tile_build");
}

}  // namespace steps
