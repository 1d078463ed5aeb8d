// Encode, bounding box, tree topology and aggregation kernels.
//
// Reference stages replaced here (Astro/Renderer.swift:505-533,714-755):
//   generateMortonCodes + fillIndices (MortonCode.metal:26-52, Octree.metal:39-51)
//   countUniqueMortonCodes per layer: markUniques, the scan, scatterUniques,
//     copyLastScanToParentCount (Octree.metal:282-334)
//   aggregateLeafNodes / aggregateNodes (Octree.metal:53-202)
// The reference finds the runs of every layer with one sort + scan + scatter
// per layer over all N entries. Here a single pass over the sorted keys finds
// the node starts of all layers at once (topology_kernel); the large layers
// are aggregated one launch each and the small top layers in one launch of a
// thread-block cluster (aggregate_top_kernel).
#include <algorithm>
#include <mutex>
#include <type_traits>

#include <cooperative_groups.h>

#include "build_kernels.cuh"
#include "common.cuh"
#include "internal.h"

namespace cg = cooperative_groups;

namespace astro {

// ------------------------------------------------------------- encode ----

// Zeroes what the next build and traversal count in. One memset for each of
// these small buffers cost a step seven launches of 1 us and their gaps.
__device__ __forceinline__ void clear_scratch(const ClearArgs& c) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, threads = gridDim.x * blockDim.x;
    for (uint32_t k = i; k < c.lookback_words; k += threads) c.lookback[k] = 0u;
    for (uint32_t k = i; k < kCounterWords; k += threads)
        if (k < kClearedWords || k >= kWorkCounts) c.counters[k] = 0u;
    for (uint32_t k = i; k < c.num_stats; k += threads) c.stats[k] = 0ull;
}

// generateMortonCodes with the reference quantiser (u32)(p + 1e6): the
// float-to-uint conversion saturates and rounds toward zero.
__global__ void encode_ref_kernel(const float4* __restrict__ pos, uint64_t* __restrict__ codes,
                                  uint32_t n_tree, uint32_t unused_bits, float offset, ClearArgs clear) {
    clear_scratch(clear);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_tree) return;
    const float4 q = pos[i];
    const uint32_t x = __float2uint_rz(__fadd_rn(q.x, offset));
    const uint32_t y = __float2uint_rz(__fadd_rn(q.y, offset));
    const uint32_t z = __float2uint_rz(__fadd_rn(q.z, offset));
    codes[i] = interleave3(x, y, z) >> unused_bits;
}

__device__ __forceinline__ uint32_t quantise(float x, float lo, float scale) {
    return min(__float2uint_rz(__fmul_rn(__fsub_rn(x, lo), scale)), kQuantMax);
}

// Bounding-box quantiser of the PHYSICAL preset, one block per chunk. In the
// precision form the FP32 frame relative to the system origin is written
// to pos here (x64 is the master copy).
template <bool kPrec>
__global__ __launch_bounds__(256) void encode_phys_kernel(const Chunk* __restrict__ chunks,
                                                          const SysInfo* sys,
                                                          float4* pos,
                                                          const double* __restrict__ x64,
                                                          uint64_t* codes, uint32_t n,
                                                          uint32_t lbits) {
    after_previous();
    const Chunk c = chunks[blockIdx.x];
    const SysInfo& s = sys[c.sys];
    const float lox = s.lo[0], loy = s.lo[1], loz = s.lo[2], scale = s.scale;
    const uint32_t unused_bits = 63u - 3u * lbits;
    const uint64_t sys_bits = (uint64_t)c.sys << (3u * lbits);
    double ox = 0, oy = 0, oz = 0;
    if (kPrec) {
        ox = s.origin[0];
        oy = s.origin[1];
        oz = s.origin[2];
    }
    for (uint32_t i = c.begin + threadIdx.x; i < c.end; i += blockDim.x) {
        float4 q = pos[i];
        if (kPrec) {
            q.x = __double2float_rn(__dsub_rn(x64[i], ox));
            q.y = __double2float_rn(__dsub_rn(x64[(size_t)n + i], oy));
            q.z = __double2float_rn(__dsub_rn(x64[2 * (size_t)n + i], oz));
            pos[i] = q;
        }
        const uint32_t qx = quantise(q.x, lox, scale);
        const uint32_t qy = quantise(q.y, loy, scale);
        const uint32_t qz = quantise(q.z, loz, scale);
        codes[i] = sys_bits | (interleave3(qx, qy, qz) >> unused_bits);
    }
}

// ------------------------------------------------------- bounding box ----

template <typename T>
__device__ __forceinline__ T warp_min(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(kFullMask, v, o));
    return v;
}
template <typename T>
__device__ __forceinline__ T warp_max(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(kFullMask, v, o));
    return v;
}

// Block-level min/max of six ordered keys followed by one atomic per value.
template <typename U>
__device__ __forceinline__ void block_bbox_commit(U lo[3], U hi[3], U* acc) {
    __shared__ U s_red[8][6];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = warp_min(lo[a]);
        hi[a] = warp_max(hi[a]);
    }
    if (lane == 0)
        for (int a = 0; a < 3; ++a) {
            s_red[warp][a] = lo[a];
            s_red[warp][3 + a] = hi[a];
        }
    __syncthreads();
    if (threadIdx.x < 6) {
        const uint32_t nw = blockDim.x >> 5;
        U v = s_red[0][threadIdx.x];
        for (uint32_t w = 1; w < nw; ++w)
            v = threadIdx.x < 3 ? min(v, s_red[w][threadIdx.x]) : max(v, s_red[w][threadIdx.x]);
        if (threadIdx.x < 3) atomicMin(acc + threadIdx.x, v);
        else atomicMax(acc + threadIdx.x, v);
    }
}

// Bounding box of the current positions, one block per chunk, accumulated
// per system with one atomic per block and value.
template <bool kPrec>
__global__ __launch_bounds__(256) void bbox_kernel(const Chunk* __restrict__ chunks,
                                                   const float4* __restrict__ pos,
                                                   const double* __restrict__ x64, uint32_t n,
                                                   uint32_t* __restrict__ bb32,
                                                   unsigned long long* __restrict__ bb64) {
    after_previous();
    const Chunk c = chunks[blockIdx.x];
    if (kPrec) {
        unsigned long long lo[3] = {~0ull, ~0ull, ~0ull}, hi[3] = {0, 0, 0};
        for (uint32_t i = c.begin + threadIdx.x; i < c.end; i += blockDim.x)
            for (int a = 0; a < 3; ++a) {
                unsigned long long o = f64_to_ordered(x64[(size_t)a * n + i]);
                lo[a] = min(lo[a], o);
                hi[a] = max(hi[a], o);
            }
        block_bbox_commit(lo, hi, bb64 + 6ull * c.sys);
    } else {
        uint32_t lo[3] = {~0u, ~0u, ~0u}, hi[3] = {0, 0, 0};
        for (uint32_t i = c.begin + threadIdx.x; i < c.end; i += blockDim.x) {
            const float4 q = pos[i];
            const float v[3] = {q.x, q.y, q.z};
            for (int a = 0; a < 3; ++a) {
                uint32_t o = f32_to_ordered(v[a]);
                lo[a] = min(lo[a], o);
                hi[a] = max(hi[a], o);
            }
        }
        block_bbox_commit(lo, hi, bb32 + 6ull * c.sys);
    }
}

// Per-system quantiser and opening thresholds from the box accumulators,
// which are then reset for the next accumulation.
template <bool kPrec>
__global__ void setup_kernel(SysInfo* __restrict__ sys, uint32_t nsys,
                             uint32_t* __restrict__ bb32, unsigned long long* __restrict__ bb64,
                             uint32_t lbits, float theta, uint32_t root_offset) {
    after_previous();
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nsys) return;
    SysInfo& info = sys[s];
    float lo[3], hi[3];
    if (kPrec) {
        for (int a = 0; a < 3; ++a) {
            const double l = ordered_to_f64(bb64[6ull * s + a]);
            const double h = ordered_to_f64(bb64[6ull * s + 3 + a]);
            const double o = __dmul_rn(__dadd_rn(l, h), 0.5);
            info.origin[a] = o;
            lo[a] = __double2float_rn(__dsub_rn(l, o));
            hi[a] = __double2float_rn(__dsub_rn(h, o));
            bb64[6ull * s + a] = ~0ull;
            bb64[6ull * s + 3 + a] = 0ull;
        }
    } else {
        for (int a = 0; a < 3; ++a) {
            lo[a] = ordered_to_f32(bb32[6ull * s + a]);
            hi[a] = ordered_to_f32(bb32[6ull * s + 3 + a]);
            info.origin[a] = 0.0;
            bb32[6ull * s + a] = ~0u;
            bb32[6ull * s + 3 + a] = 0u;
        }
    }
    float ext = 0.0f;
    for (int a = 0; a < 3; ++a) {
        info.lo[a] = lo[a];
        ext = fmaxf(ext, __fsub_rn(hi[a], lo[a]));
    }
    if (!(ext > 0.0f) || !isfinite(ext)) ext = 1.0f;
    info.ext = ext;
    info.scale = __fdiv_rn(kQuantCells, ext);
    info.root = root_offset + s;
    for (uint32_t l = 0; l <= lbits; ++l) {
        const float c = __fdiv_rn(__fmul_rn(ext, exp2_exact((int)l - (int)lbits)), theta);
        info.crit2[l] = __fmul_rn(c, c);
    }
}

// ------------------------------------------------------------ reorder ----

// Permute the PHYSICAL state into the new Morton order (B <- A[perm]).
template <bool kPrec>
__global__ void reorder_kernel(const uint32_t* perm, const float4* __restrict__ pos_a,
                               const float4* __restrict__ vel_a, const uint32_t* __restrict__ id_a,
                               const double* __restrict__ x_a, float4* __restrict__ pos_b,
                               float4* __restrict__ vel_b, uint32_t* __restrict__ id_b,
                               double* __restrict__ x_b, uint32_t n, ClearArgs clear) {
    after_previous();
    clear_scratch(clear);
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const uint32_t s = perm[j];
    pos_b[j] = pos_a[s];
    vel_b[j] = vel_a[s];
    id_b[j] = id_a[s];
    if (kPrec) {
        x_b[j] = x_a[s];
        x_b[(size_t)n + j] = x_a[(size_t)n + s];
        x_b[2 * (size_t)n + j] = x_a[2 * (size_t)n + s];
    }
}

// ----------------------------------------------------------- topology ----

constexpr int kTopoThreads = 256;
constexpr int kTopoWarps = kTopoThreads / 32;

// Keys per thread: few where the array is small, so that the tiles spread over
// the chip and the serial loops over keys and layers are short (16,384 bodies,
// two keys: 6.6 us, eight keys: 15.4; 524,288 bodies, four keys: 18 us, eight:
// 24); eight where the look-back over many tiles would cost more.
constexpr uint32_t kTopoSmall = 1u << 17, kTopoMedium = 1u << 20;
constexpr uint32_t topo_items(uint32_t n) { return n <= kTopoSmall ? 2u : (n <= kTopoMedium ? 4u : 8u); }

// One pass over the sorted keys finds the nodes of every layer. Position i
// starts a node at layer l when its key differs from key i-1 above bit 3l,
// i.e. for l <= lev(i) = floor(msb(k[i] ^ k[i-1]) / 3) (capped at lbits;
// lev(0) = lbits). The index of that node inside its layer is the number of
// starts before i, found per layer with warp ballots and a decoupled
// look-back across tiles. Each start writes the node's first particle and,
// above layer 0, its first child (the node starting at i one layer down).
// This yields the runs of markUniques/scatterUniques (Octree.metal:282-318)
// for all layers without re-sorting or re-scanning per layer. Each node
// below the top layer also gets its parent: the node one layer up that
// holds its first particle (the bottom-up aggregation climbs these links).
template <int kTopoItems>
__global__ __launch_bounds__(kTopoThreads) void topology_kernel(TopoArgs a) {
    after_previous();
    constexpr int kTopoTile = kTopoThreads * kTopoItems;
    __shared__ uint32_t s_tile;
    __shared__ uint32_t s_off[ASTRO_MAX_LAYERS];
    __shared__ uint32_t s_wcnt[kTopoWarps][32];
    __shared__ uint32_t s_prefix[32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int lbits = (int)a.lbits;
    if (tid == 0) s_tile = atomicAdd(a.tile_counter, 1u);
    if (tid < ASTRO_MAX_LAYERS) s_off[tid] = a.offset[tid];
    if (tid < 32)
        for (int w = 0; w < kTopoWarps; ++w) s_wcnt[w][tid] = 0;
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint64_t base = (uint64_t)tile * kTopoTile;
    if (base >= a.n) return;
    const uint64_t warp_base = base + (uint64_t)warp * 32 * kTopoItems;
    const uint32_t lt = lanemask_lt();

    uint64_t key[kTopoItems];
    int lev[kTopoItems];
    uint64_t carry = (warp_base > 0 && warp_base <= a.n) ? a.keys[warp_base - 1] : 0ull;
#pragma unroll
    for (int k = 0; k < kTopoItems; ++k) {
        const uint64_t i = warp_base + 32ull * k + lane;
        const bool valid = i < a.n;
        key[k] = valid ? a.keys[i] : 0ull;
        uint64_t prev = __shfl_up_sync(kFullMask, key[k], 1);
        if (lane == 0) prev = carry;
        carry = __shfl_sync(kFullMask, key[k], 31);
        int lv = -1;
        if (valid) {
            if (i == 0) lv = lbits;
            else if (key[k] != prev) lv = min(lbits, (63 - __clzll((long long)(key[k] ^ prev))) / 3);
        }
        lev[k] = lv;
    }
    // Starts per layer within this warp (lane l keeps layer l).
    uint32_t my_cnt = 0;
#pragma unroll
    for (int k = 0; k < kTopoItems; ++k)
        for (int l = 0; l <= lbits; ++l) {
            const uint32_t b = __ballot_sync(kFullMask, lev[k] >= l);
            if (b == 0) break;
            if ((int)lane == l) my_cnt += __popc(b);
        }
    if ((int)lane <= lbits) s_wcnt[warp][lane] = my_cnt;
    __syncthreads();
    if ((int)tid <= lbits) {
        uint32_t run = 0;
        for (int w = 0; w < kTopoWarps; ++w) {
            const uint32_t c = s_wcnt[w][tid];
            s_wcnt[w][tid] = run;
            run += c;
        }
        uint32_t* word = a.lookback + (size_t)tile * 32 + tid;
        st_relaxed_u32(word, (tile == 0 ? kLbInclusive : kLbAggregate) | run);
        uint32_t prefix = 0;
        if (tile > 0) {
            prefix = lookback_window(a.lookback, tile, tid, a.err, 32);
            st_relaxed_u32(word, kLbInclusive | (prefix + run));
        }
        s_prefix[tid] = prefix;
        if (tile == a.ntiles - 1) a.layer_count[tid] = prefix + run;
    }
    __syncthreads();
    uint32_t running = (int)lane <= lbits ? s_prefix[lane] + s_wcnt[warp][lane] : 0u;
#pragma unroll
    for (int k = 0; k < kTopoItems; ++k) {
        const uint32_t i = (uint32_t)(warp_base + 32ull * k + lane);
        uint32_t idx_below = 0;
        uint32_t pending = kNoParent;  // this lane's node one layer down, parent not yet written
        for (int l = 0; l <= lbits; ++l) {
            const uint32_t b = __ballot_sync(kFullMask, lev[k] >= l);
            const uint32_t base_l = __shfl_sync(kFullMask, running, l);
            // Starts of layer l before particle i.
            const uint32_t rank = base_l + __popc(b & lt);
            if (pending != kNoParent) {
                // The parent holds i: the layer-l node starting at i, else the
                // last one starting before it.
                a.parent[pending] = s_off[l] + (lev[k] >= l ? rank : rank - 1u);
                pending = kNoParent;
            }
            if (b == 0) break;
            if (lev[k] >= l) {
                const uint32_t node = s_off[l] + rank;
                a.pbeg[node] = i;
                a.node_key[node] = key[k] >> (3u * l);
                if (l > 0) a.cbeg[node] = s_off[l - 1] + idx_below;
                idx_below = rank;
                if (l < lbits) pending = node;
                else a.parent[node] = kNoParent;
            }
            if ((int)lane == l) running += __popc(b);
        }
    }
}

// -------------------------------------------------------- aggregation ----

// Traceless quadrupole accumulation of mass m at offset d from the centre of
// mass: Q += m (3 d d^T - |d|^2 I), components Qxx, Qyy, Qxy, Qxz, Qyz, each
// product and sum rounded separately.
__device__ __forceinline__ void quad_add(float q[5], float m, float dx, float dy, float dz) {
    const float r2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
    const float tx = __fmul_rn(3.0f, dx), ty = __fmul_rn(3.0f, dy);
    q[0] = __fadd_rn(q[0], __fmul_rn(m, __fsub_rn(__fmul_rn(tx, dx), r2)));
    q[1] = __fadd_rn(q[1], __fmul_rn(m, __fsub_rn(__fmul_rn(ty, dy), r2)));
    q[2] = __fadd_rn(q[2], __fmul_rn(m, __fmul_rn(tx, dy)));
    q[3] = __fadd_rn(q[3], __fmul_rn(m, __fmul_rn(tx, dz)));
    q[4] = __fadd_rn(q[4], __fmul_rn(m, __fmul_rn(ty, dz)));
}

// Opening radius^2 of a node: (size / theta + w |com - cell centre|)^2, the
// cell found from the node's key prefix in its system's box.
// Geometric centre (x, y, z) and edge (w) of the layer-l cell of a node;
// node_key = first key >> 3l: the system above bit 3 (lbits - l), the
// cell's code below it (3 (lbits - l) <= 63).
__device__ __forceinline__ float4 cell_box(const AggArgs& a, uint64_t node_key, uint32_t l) {
    const uint32_t below = 3u * (a.lbits - l);
    const uint32_t s = (uint32_t)(node_key >> below);
    const SysInfo& si = a.sys[s];
    const uint64_t code = node_key & ((1ull << below) - 1ull);
    const float size = __fmul_rn(si.ext, exp2_exact((int)l - (int)a.lbits));
    const float half = __fmul_rn(0.5f, size);
    return make_float4(__fadd_rn(si.lo[0], __fmul_rn((float)(2u * compact3_21(code) + 1u), half)),
                       __fadd_rn(si.lo[1], __fmul_rn((float)(2u * compact3_21(code >> 1) + 1u), half)),
                       __fadd_rn(si.lo[2], __fmul_rn((float)(2u * compact3_21(code >> 2) + 1u), half)),
                       size);
}

__device__ __forceinline__ float node_crit2(const AggArgs& a, uint64_t node_key, uint32_t l, float4 cm) {
    const float4 box = cell_box(a, node_key, l);
    const float size = box.w, cx = box.x, cy = box.y, cz = box.z;
    const float dx = __fsub_rn(cm.x, cx), dy = __fsub_rn(cm.y, cy), dz = __fsub_rn(cm.z, cz);
    const float dd = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
    const float crit = __fadd_rn(__fdiv_rn(size, a.theta), __fmul_rn(a.delta_weight, __fsqrt_rn(dd)));
    return __fmul_rn(crit, crit);
}

// PHYSICAL centre of mass (and mass) from the raw sums: one reciprocal of
// the mass and three products; zero for a massless node. FP32: a correctly
// rounded reciprocal. Precision form: the FP32 reciprocal refined by one
// FP64 Newton step, r = r0 + r0 (1 - m r0) (about 46 bits, two FMAs instead
// of an FP64 division), then FP64 products rounded to FP32.
__device__ __forceinline__ float4 com_from_sums(float sx, float sy, float sz, float m) {
    if (!(m > 0.f)) return make_float4(0.f, 0.f, 0.f, m);
    const float inv = __fdiv_rn(1.0f, m);
    return make_float4(__fmul_rn(sx, inv), __fmul_rn(sy, inv), __fmul_rn(sz, inv), m);
}
__device__ __forceinline__ float4 com_from_sums(double sx, double sy, double sz, double m) {
    if (!(m > 0.0)) return make_float4(0.f, 0.f, 0.f, __double2float_rn(m));
    const double r0 = (double)__fdiv_rn(1.0f, __double2float_rn(m));
    const double inv = __fma_rn(r0, __fma_rn(-m, r0, 1.0), r0);
    return make_float4(__double2float_rn(__dmul_rn(sx, inv)), __double2float_rn(__dmul_rn(sy, inv)),
                       __double2float_rn(__dmul_rn(sz, inv)), __double2float_rn(m));
}

// Slots for c groups of this thread: the warp's lanes (all of them call) add
// their counts and one lane claims the slots with a single atomic (instead of
// one per group on the shared counter); lanes take their runs in lane order.
// Most calls have nothing to claim.
__device__ __forceinline__ uint32_t reserve_groups(uint32_t* counter, uint32_t c) {
    if (__ballot_sync(kFullMask, c != 0u) == 0u) return 0u;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    uint32_t base = 0;
    if (lane == 31u) base = atomicAdd(counter, incl);
    return __shfl_sync(kFullMask, base, 31) + incl - c;
}

// Visits the particles [pb, pe) in order (the sums stay in particle order),
// kBatch at a time with the next batch loaded ahead. One thread sums a leaf, so
// a crowded leaf is a serial chain: with the next batch not loaded ahead the leaf
// pass of a 524,288-body disk (leaves of up to about 70) took 47 us; 35 us in
// batches of four, 28 us of eight (two or three batches ahead: 34 us). The
// precision form, bound by the FP64 pipe, runs best at four (174 us against 217
// for 4,194,304 bodies).
template <uint32_t kBatch, typename F>
__device__ __forceinline__ void for_particles(const float4* __restrict__ pos, uint32_t pb,
                                              uint32_t pe, F&& f) {
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 next[kBatch];
#pragma unroll
    for (uint32_t u = 0; u < kBatch; ++u) next[u] = pb + u < pe ? __ldg(&pos[pb + u]) : zero;
    for (uint32_t i = pb; i < pe; i += kBatch) {
        float4 q[kBatch];
#pragma unroll
        for (uint32_t u = 0; u < kBatch; ++u) {
            q[u] = next[u];
            next[u] = i + kBatch + u < pe ? __ldg(&pos[i + kBatch + u]) : zero;
        }
#pragma unroll
        for (uint32_t u = 0; u < kBatch; ++u)
            if (i + u < pe) f(q[u]);
    }
}

// Mass moments of a leaf's particles about a point c (the cell's centre):
// first moments D = sum m d and second moments S = sum m d d^T, d = x - c,
// in FP32, each product and sum rounded separately. quadrupole() shifts them
// to the centre of mass e + c (e = com - c): P = S - e D^T - D e^T + M e e^T,
// Q = 3 P - tr(P) I (traceless), components Qxx, Qyy, Qxy, Qxz, Qyz. The
// particles lie inside the cell, so |d| is at most its half diagonal and
// the shift loses little; one read of the particles then gives the sums and
// the quadrupole together (a second pass about the centre of mass re-read
// them from DRAM once the position array had streamed through L2).
struct CellMoments {
    float dx = 0.f, dy = 0.f, dz = 0.f;
    float sxx = 0.f, syy = 0.f, szz = 0.f, sxy = 0.f, sxz = 0.f, syz = 0.f;
    __device__ __forceinline__ void add(float4 q, float4 c) {
        const float ux = __fsub_rn(q.x, c.x), uy = __fsub_rn(q.y, c.y), uz = __fsub_rn(q.z, c.z);
        const float tx = __fmul_rn(q.w, ux), ty = __fmul_rn(q.w, uy), tz = __fmul_rn(q.w, uz);
        dx = __fadd_rn(dx, tx);
        dy = __fadd_rn(dy, ty);
        dz = __fadd_rn(dz, tz);
        sxx = __fadd_rn(sxx, __fmul_rn(tx, ux));
        syy = __fadd_rn(syy, __fmul_rn(ty, uy));
        szz = __fadd_rn(szz, __fmul_rn(tz, uz));
        sxy = __fadd_rn(sxy, __fmul_rn(tx, uy));
        sxz = __fadd_rn(sxz, __fmul_rn(tx, uz));
        syz = __fadd_rn(syz, __fmul_rn(ty, uz));
    }
    // P_ab = ((S_ab - e_a D_b) - e_b D_a) + e_a (M e_b)
    __device__ __forceinline__ static float shifted(float s, float ea, float eb, float da, float db,
                                                    float m) {
        return __fadd_rn(__fsub_rn(__fsub_rn(s, __fmul_rn(ea, db)), __fmul_rn(eb, da)),
                         __fmul_rn(ea, __fmul_rn(m, eb)));
    }
    __device__ __forceinline__ void quadrupole(float4 cm, float4 c, float q[5]) const {
        const float ex = __fsub_rn(cm.x, c.x), ey = __fsub_rn(cm.y, c.y), ez = __fsub_rn(cm.z, c.z);
        const float m = cm.w;
        const float pxx = shifted(sxx, ex, ex, dx, dx, m);
        const float pyy = shifted(syy, ey, ey, dy, dy, m);
        const float pzz = shifted(szz, ez, ez, dz, dz, m);
        const float pxy = shifted(sxy, ex, ey, dx, dy, m);
        const float pxz = shifted(sxz, ex, ez, dx, dz, m);
        const float pyz = shifted(syz, ey, ez, dy, dz, m);
        const float tr = __fadd_rn(__fadd_rn(pxx, pyy), pzz);
        q[0] = __fsub_rn(__fmul_rn(3.0f, pxx), tr);
        q[1] = __fsub_rn(__fmul_rn(3.0f, pyy), tr);
        q[2] = __fmul_rn(3.0f, pxy);
        q[3] = __fmul_rn(3.0f, pxz);
        q[4] = __fmul_rn(3.0f, pyz);
    }
};

// REFERENCE: aggregateLeafNodes (Octree.metal:53-117), one thread per leaf.
// State in upload order, gathered through perm; FP32 sums of m and x*m in
// sorted order; the last leaf sums [start, numUnique) as the reference does
// (Octree.metal:71).
__device__ __forceinline__ void aggregate_ref_leaf(const AggArgs& a, uint32_t j, uint32_t u0) {
    const uint32_t pb = a.pbeg[j];
    const uint32_t pe = (j + 1 < u0) ? a.pbeg[j + 1] : a.n;
    const uint32_t sum_end = (j + 1 < u0) ? pe : u0;
    float4 cm = make_float4(0.f, 0.f, 0.f, 0.f);
    float m = 0.f, sx = 0.f, sy = 0.f, sz = 0.f;
    // Stars (type 0): colours summed, positions averaged (Octree.metal:85-99).
    float4 ec = make_float4(0.f, 0.f, 0.f, 0.f), en = ec;
    uint32_t suns = 0;
    for (uint32_t i = pb; i < sum_end; ++i) {
        const uint32_t pi = a.perm[i];
        const float4 q = a.pos[pi];
        m = __fadd_rn(m, q.w);
        sx = __fadd_rn(sx, __fmul_rn(q.x, q.w));
        sy = __fadd_rn(sy, __fmul_rn(q.y, q.w));
        sz = __fadd_rn(sz, __fmul_rn(q.z, q.w));
        if (a.node_ecol && a.types[pi] == 0u) {
            const float4 c = a.colors[pi];
            ec = make_float4(__fadd_rn(ec.x, c.x), __fadd_rn(ec.y, c.y), __fadd_rn(ec.z, c.z),
                             __fadd_rn(ec.w, c.w));
            en = make_float4(__fadd_rn(en.x, q.x), __fadd_rn(en.y, q.y), __fadd_rn(en.z, q.z), 0.f);
            ++suns;
        }
    }
    if (m > 0.f) cm = make_float4(__fdiv_rn(sx, m), __fdiv_rn(sy, m), __fdiv_rn(sz, m), m);
    else cm.w = m;
    if (a.node_ecol) {
        const float ns = fmaxf((float)suns, 1e-9f);
        a.node_ecol[j] = ec;
        a.node_ecen[j] = make_float4(__fdiv_rn(en.x, ns), __fdiv_rn(en.y, ns), __fdiv_rn(en.z, ns), 0.f);
    }
    a.node_cm[j] = cm;
    a.node_rng[j] = make_uint4(0u, 0u, pb, pe);
}

// Children are read through L2 (ld.global.cg): the cluster kernels below
// read records that other blocks wrote in the same launch.
__device__ __forceinline__ float4 ld_l2(const float4* p) { return __ldcg(p); }
__device__ __forceinline__ float ld_l2(const float* p) { return __ldcg(p); }
__device__ __forceinline__ uint4 ld_l2(const uint4* p) { return __ldcg(p); }
__device__ __forceinline__ double4 ld_l2(const double4* p) {
    const double2 lo = __ldcg(reinterpret_cast<const double2*>(p));
    const double2 hi = __ldcg(reinterpret_cast<const double2*>(p) + 1);
    return make_double4(lo.x, lo.y, hi.x, hi.y);
}

// REFERENCE: aggregateNodes (Octree.metal:120-202) for node j of layer l (one
// thread): child centre of mass times child mass, summed in child order.
// Children are the contiguous run of layer l-1 nodes sharing code >> 3 (at
// most 8); their records are loaded together.
__device__ __forceinline__ void aggregate_ref_internal(const AggArgs& a, uint32_t l, uint32_t j,
                                                       uint32_t u) {
    const uint32_t off = a.offset[l], off_below = a.offset[l - 1];
    const uint32_t node = off + j;
    const uint32_t cb = a.node_cbeg[node];
    const uint32_t ce = (j + 1 < u) ? a.node_cbeg[node + 1] : off_below + a.layer_count[l - 1];
    const uint32_t pb = a.pbeg[node];
    const uint32_t pe = (j + 1 < u) ? a.pbeg[node + 1] : a.n;
    if (ce - cb > 8u) atomicOr(a.err, kErrBadLayer);
    const uint32_t nch = min(ce - cb, 8u);
    float4 cm = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 ccm[8];
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k)
        ccm[k] = k < nch ? ld_l2(a.node_cm + cb + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    float m = 0.f, sx = 0.f, sy = 0.f, sz = 0.f;
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
        if (k < nch) {
            const float4 q = ccm[k];
            m = __fadd_rn(m, q.w);
            sx = __fadd_rn(sx, __fmul_rn(q.x, q.w));
            sy = __fadd_rn(sy, __fmul_rn(q.y, q.w));
            sz = __fadd_rn(sz, __fmul_rn(q.z, q.w));
        }
    }
    if (m > 0.f) cm = make_float4(__fdiv_rn(sx, m), __fdiv_rn(sy, m), __fdiv_rn(sz, m), m);
    else cm.w = m;
    if (a.node_ecol) {
        // Children whose emitted colour has alpha > 0: colours summed,
        // centres averaged over those children (Octree.metal:155-178).
        float4 ec = make_float4(0.f, 0.f, 0.f, 0.f), en = ec;
        uint32_t suns = 0;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            if (k < nch) {
                const float4 c = ld_l2(a.node_ecol + cb + k);
                if (c.w > 0.f) {
                    const float4 e = ld_l2(a.node_ecen + cb + k);
                    ec = make_float4(__fadd_rn(ec.x, c.x), __fadd_rn(ec.y, c.y),
                                     __fadd_rn(ec.z, c.z), __fadd_rn(ec.w, c.w));
                    en = make_float4(__fadd_rn(en.x, e.x), __fadd_rn(en.y, e.y),
                                     __fadd_rn(en.z, e.z), 0.f);
                    ++suns;
                }
            }
        }
        if (suns > 0) {
            const float ns = (float)suns;
            en = make_float4(__fdiv_rn(en.x, ns), __fdiv_rn(en.y, ns), __fdiv_rn(en.z, ns), 0.f);
        }
        a.node_ecol[node] = ec;
        a.node_ecen[node] = en;
    }
    a.node_cm[node] = cm;
    a.node_rng[node] = make_uint4(cb, ce, pb, pe);
}

// ---- PHYSICAL ----

// A node's record as the thread that makes it holds it: raw sums (FP32 in the
// plain form, FP64 in the precision form), centre of mass and mass,
// quadrupole, particles and key.
template <bool kPrec>
struct NodeRec {
    using Sum = typename std::conditional<kPrec, double4, float4>::type;
    Sum sum;
    float4 cm;
    float q[5];
    uint32_t pb, pe;
    uint64_t key;
};

// Writes node's record but for its sums.
template <bool kPrec, bool kQuad>
__device__ __forceinline__ void store_node(const AggArgs& a, uint32_t node, uint32_t l, uint32_t cb,
                                           uint32_t ce, const NodeRec<kPrec>& r) {
    a.node_cm[node] = r.cm;
    a.node_rng[node] = make_uint4(cb, ce, r.pb, r.pe);
    if (kQuad) {
        a.node_q[node] = make_float4(r.q[0], r.q[1], r.q[2], r.q[3]);
        a.node_qyz[node] = r.q[4];
    }
    if (a.want_delta) a.node_crit2[node] = node_crit2(a, r.key, l, r.cm);
}

// aggregateLeafNodes (Octree.metal:53-117), state already in sorted order.
// Plain: raw FP32 sums of m and m*x. Precision: FP64 sums over the FP32
// positions relative to the system origin. The quadrupole comes from the same
// read: moments about the cell's centre, shifted to the centre of mass after.
template <bool kPrec, bool kQuad>
__device__ __forceinline__ NodeRec<kPrec> aggregate_leaf(const AggArgs& a, uint32_t j, uint32_t u0) {
    NodeRec<kPrec> r;
    r.pb = a.pbeg[j];
    r.pe = (j + 1 < u0) ? a.pbeg[j + 1] : a.n;
    r.key = a.node_key[j];
    const float4 box = kQuad ? cell_box(a, r.key, 0) : make_float4(0.f, 0.f, 0.f, 0.f);
    CellMoments mom;
    if constexpr (!kPrec) {
        float m = 0.f, sx = 0.f, sy = 0.f, sz = 0.f;
        for_particles<8>(a.pos, r.pb, r.pe, [&](const float4 q) {
            m = __fadd_rn(m, q.w);
            sx = __fadd_rn(sx, __fmul_rn(q.w, q.x));
            sy = __fadd_rn(sy, __fmul_rn(q.w, q.y));
            sz = __fadd_rn(sz, __fmul_rn(q.w, q.z));
            if (kQuad) mom.add(q, box);
        });
        r.sum = make_float4(sx, sy, sz, m);
        r.cm = com_from_sums(sx, sy, sz, m);
    } else {
        // The product of two floats is exact in FP64, so each FMA rounds
        // once, exactly as a multiply-then-add would.
        double m = 0, sx = 0, sy = 0, sz = 0;
        for_particles<4>(a.pos, r.pb, r.pe, [&](const float4 q) {
            const double mi = (double)q.w;
            m = __dadd_rn(m, mi);
            sx = __fma_rn(mi, (double)q.x, sx);
            sy = __fma_rn(mi, (double)q.y, sy);
            sz = __fma_rn(mi, (double)q.z, sz);
            if (kQuad) mom.add(q, box);
        });
        r.sum = make_double4(sx, sy, sz, m);
        if (r.pe - r.pb == 1 && m >= 1.17549435e-38) {
            // One particle of normal FP32 mass: the sums are m*x exactly and
            // the reciprocal is within 2^-47 of 1/m, so the FP32 centre of
            // mass is x itself (+0 for -0, as the sums give).
            const float4 q = a.pos[r.pb];
            r.cm = make_float4(__fadd_rn(q.x, 0.f), __fadd_rn(q.y, 0.f), __fadd_rn(q.z, 0.f), q.w);
        } else {
            r.cm = com_from_sums(sx, sy, sz, m);
        }
    }
    if (kQuad) mom.quadrupole(r.cm, box, r.q);
    store_node<kPrec, kQuad>(a, j, 0, 0u, 0u, r);
    return r;
}

// A leaf holding more than one group is cut into group-sized chunks (all lanes
// of the warp call; those without a leaf pass pe = pb).
__device__ __forceinline__ void emit_chunks(const AggArgs& a, uint32_t pb, uint32_t pe) {
    const uint32_t gs = a.group_size;
    const uint32_t c = pe - pb > gs ? (pe - pb + gs - 1u) / gs : 0u;
    const uint32_t slot = reserve_groups(a.group_count, c);
    for (uint32_t i = 0; i < c; ++i)
        a.groups[slot + i] = make_uint4(pb + i * gs, min(pb + (i + 1u) * gs, pe), pe, i);
}

// Groups of a node with several children that holds more particles than a
// group: runs of consecutive small children (greedy, in child order). The
// packing runs twice: to count the groups, then to write them into the slots
// reserved for this node. All lanes of the warp call; those without such a node
// pass ce = cb, and `root` marks a group [pb, pe) of its own.
__device__ __forceinline__ void emit_groups(const AggArgs& a, uint32_t cb, uint32_t ce, bool root, uint32_t pb,
                                            uint32_t pe) {
    const uint32_t gs = a.group_size, nch = min(ce - cb, 8u);
    // The children's particles follow each other from pb to pe; where each begins
    // the topology pass has written.
    uint2 cr[8];
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) cr[k].x = k == 0 ? pb : (k < nch ? a.pbeg[cb + k] : pe);
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) cr[k].y = k < 7 ? cr[(k + 1) % 8].x : pe;
    auto pack = [&](auto&& emit) {
        uint32_t gb = 0, ge = 0;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            if (k >= nch) break;
            const uint32_t cc = cr[k].y - cr[k].x;
            if (cc <= gs) {
                if (ge == gb) {
                    gb = cr[k].x;
                    ge = cr[k].y;
                } else if ((ge - gb) + cc <= gs) {
                    ge = cr[k].y;
                } else {
                    emit(gb, ge);
                    gb = cr[k].x;
                    ge = cr[k].y;
                }
            } else if (ge != gb) {
                emit(gb, ge);
                gb = ge = 0;
            }
        }
        if (ge != gb) emit(gb, ge);
        if (root) emit(pb, pe);
    };
    uint32_t c = 0;
    pack([&](uint32_t, uint32_t) { ++c; });
    uint32_t slot = reserve_groups(a.group_count, c);
    pack([&](uint32_t b, uint32_t e) { a.groups[slot++] = make_uint4(b, e, e, 0u); });
}

// aggregateNodes (Octree.metal:120-202) for a node with several children (at
// most 8): their records loaded together, sums and quadrupoles added in child
// order with the roundings of a sequential loop.
template <bool kPrec, bool kQuad>
__device__ __forceinline__ void aggregate_internal(const AggArgs& a, uint32_t l, uint32_t node,
                                                   uint32_t cb, uint32_t ce, NodeRec<kPrec>& r) {
    using Sum = typename NodeRec<kPrec>::Sum;
    if (ce - cb > 8u) atomicOr(a.err, kErrBadLayer);
    const uint32_t nch = min(ce - cb, 8u);
    const Sum* sum = reinterpret_cast<const Sum*>(a.node_sum);
    {
        Sum cs[8];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) cs[k] = k < nch ? ld_l2(sum + cb + k) : Sum{};
        Sum t{};
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            if (k < nch) {
                if constexpr (kPrec) {
                    t.x = __dadd_rn(t.x, cs[k].x);
                    t.y = __dadd_rn(t.y, cs[k].y);
                    t.z = __dadd_rn(t.z, cs[k].z);
                    t.w = __dadd_rn(t.w, cs[k].w);
                } else {
                    t.x = __fadd_rn(t.x, cs[k].x);
                    t.y = __fadd_rn(t.y, cs[k].y);
                    t.z = __fadd_rn(t.z, cs[k].z);
                    t.w = __fadd_rn(t.w, cs[k].w);
                }
            }
        }
        r.sum = t;
        r.cm = com_from_sums(t.x, t.y, t.z, t.w);
    }
    if constexpr (kQuad) {
        float4 ccm[8], qc[8];
        float qyz[8];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            ccm[k] = k < nch ? ld_l2(a.node_cm + cb + k) : make_float4(0.f, 0.f, 0.f, 0.f);
            qc[k] = k < nch ? ld_l2(a.node_q + cb + k) : make_float4(0.f, 0.f, 0.f, 0.f);
            qyz[k] = k < nch ? ld_l2(a.node_qyz + cb + k) : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 5; ++i) r.q[i] = 0.f;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            if (k < nch) {
                const float4 cc = ccm[k];
                quad_add(r.q, cc.w, __fsub_rn(cc.x, r.cm.x), __fsub_rn(cc.y, r.cm.y),
                         __fsub_rn(cc.z, r.cm.z));
                r.q[0] = __fadd_rn(r.q[0], qc[k].x);
                r.q[1] = __fadd_rn(r.q[1], qc[k].y);
                r.q[2] = __fadd_rn(r.q[2], qc[k].z);
                r.q[3] = __fadd_rn(r.q[3], qc[k].w);
                r.q[4] = __fadd_rn(r.q[4], qyz[k]);
            }
        }
    }
    store_node<kPrec, kQuad>(a, node, l, cb, ce, r);
}

// The bottom-up aggregation. Layers of at least kLayerMinNodes nodes (capacity)
// run one launch each, a thread per node with coalesced records; the rest of
// the tree runs in one launch (aggregate_top_kernel).
//
// A parent with one child takes the child's sums, centre of mass and
// quadrupole as they are (each sum is 0 + the child's, and no sum is -0), so
// the thread that made the child writes the parent from its registers, and so
// on up the single-child chain; a layer's own launch only takes the nodes with
// several children: from a work list in layers of at least kWorkMinNodes nodes
// (capacity), by looking at every node in smaller ones, where the list's
// atomics and indirection cost more than the idle threads.
//
// What bounds it: the record stores (56 bytes a node of a chain), the latency of
// the leaves' dependent loads, and in small trees the launches. (Not the FP64
// pipe: conversions done with integers instead left the leaf pass of 4,194,304
// bodies in the precision form at 175 us.) Aggregation before and after
// (one launch a layer, each re-reading its children): 6,000,007-body cube at 21
// bits 4.55 -> 1.83 ms, two Plummer spheres of 4,194,304 in the precision form
// 481 -> 342 us, 256 systems 590 -> 424 us, 524,288-body disk 146 -> 105 us.
// Work lists in every layer: disk 14 us more; in none: merger 64 us, 21 bits
// 0.7 ms more; the whole tree in one climbing launch: merger 594 us, disk 124 us.
// Layers of 16,384 to 24,575 nodes by launches / in the cluster, us a step: cubes of
// 20,000 bodies at 21 bits 198 / 255, of 24,000 at 8 bits 132 / 145 (but a sphere of
// 16,384 at 8 bits 149 / 138, 256 systems with 16,384 nodes in a layer 8,050 / 7,864).
// The top layer, too, is a launch of its own where there are that many systems
// (24,000 of 16 bodies 244 / 260).
constexpr uint32_t kLayerMinNodes = 18432;
constexpr uint32_t kWorkMinNodes = 1u << 20;
static_assert(kWorkMinNodes > ASTRO_MAX_SYSTEMS, "all nodes of the top layer are looked at, for the groups");

// The children [cb, ce) of node jp of layer l (u nodes there, `below` nodes
// one layer down).
struct Children {
    uint32_t cb, ce;
};
__device__ __forceinline__ Children children_of(const AggArgs& a, uint32_t p, uint32_t jp, uint32_t u,
                                                uint32_t l, uint32_t below) {
    return {a.node_cbeg[p], (jp + 1 < u) ? a.node_cbeg[p + 1] : a.offset[l - 1] + below};
}

// Writes the single-child chain above node (of layer l) in the layers below
// `top`, then the sums of the chain's last node, which its parent adds. A
// parent with several children in a layer below `work_top` goes to its layer's
// work list, once: by the thread that ends the chain of its first child.
template <bool kPrec, bool kQuad>
__device__ __forceinline__ void climb_chain(const AggArgs& a, uint32_t l, uint32_t node, uint32_t top,
                                            uint32_t work_top, NodeRec<kPrec>& r) {
    uint32_t work = kNoParent, k = l + 1;
    for (; k < top; ++k) {
        const uint32_t p = a.parent[node];
        const uint32_t u = a.layer_count[k], jp = p - a.offset[k];
        if (jp >= u) {
            atomicOr(a.err, kErrBadLayer);
            return;
        }
        const Children c = children_of(a, p, jp, u, k, a.layer_count[k - 1]);
        if (c.ce - c.cb != 1u) {
            if (c.cb == node && k < work_top) work = p;
            break;
        }
        r.key >>= 3;
        store_node<kPrec, kQuad>(a, p, k, c.cb, c.ce, r);
        node = p;
    }
    reinterpret_cast<typename NodeRec<kPrec>::Sum*>(a.node_sum)[node] = r.sum;
    // One atomic per layer and warp for the slots of the list.
    const uint32_t mask = __activemask();
    const uint32_t peers = __match_any_sync(mask, work != kNoParent ? k : 0xFFFFu);
    if (work == kNoParent) return;
    const uint32_t lane = threadIdx.x & 31u, leader = (uint32_t)__ffs(peers) - 1u;
    uint32_t slot = 0;
    if (lane == leader) slot = atomicAdd(&a.work_count[k], (uint32_t)__popc(peers));
    slot = __shfl_sync(peers, slot, leader) + __popc(peers & lanemask_lt());
    a.work[a.offset[k] + slot] = work;
}

template <bool kPrec, bool kQuad>
__global__ __launch_bounds__(128) void aggregate_leaf_kernel(AggArgs a, uint32_t top, uint32_t work_top) {
    after_previous();
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t u0 = a.layer_count[0];
    NodeRec<kPrec> r;
    r.pb = r.pe = 0;
    if (j < u0) r = aggregate_leaf<kPrec, kQuad>(a, j, u0);
    emit_chunks(a, r.pb, r.pe);
    if (j < u0) climb_chain<kPrec, kQuad>(a, 0, j, top, work_top, r);
}

// The nodes of layer l with several children: the layer's work list (kWork;
// the blocks stride over it), or all nodes, the others left out.
template <bool kPrec, bool kQuad, bool kWork>
__global__ __launch_bounds__(128) void aggregate_internal_kernel(AggArgs a, uint32_t l, uint32_t top,
                                                                 uint32_t work_top) {
    after_previous();
    const uint32_t u = a.layer_count[l], count = kWork ? a.work_count[l] : u;
    for (uint32_t i0 = blockIdx.x * blockDim.x; i0 < count; i0 += gridDim.x * blockDim.x) {
        const uint32_t i = i0 + threadIdx.x;
        uint32_t node = 0;
        Children c{0u, 0u};
        NodeRec<kPrec> r;
        r.pb = r.pe = 0;
        bool several = false, root = false;
        if (i < count) {
            node = kWork ? a.work[a.offset[l] + i] : a.offset[l] + i;
            const uint32_t j = node - a.offset[l];
            c = children_of(a, node, j, u, l, a.layer_count[l - 1]);
            several = kWork || c.ce - c.cb != 1u;
            if (several || l == a.lbits) {
                r.pb = a.pbeg[node];
                r.pe = (j + 1 < u) ? a.pbeg[node + 1] : a.n;
            }
            // The root of a system no larger than a group is a group by itself.
            root = l == a.lbits && r.pe - r.pb <= a.group_size;
            if (several) {
                r.key = a.node_key[node];
                aggregate_internal<kPrec, kQuad>(a, l, node, c.cb, c.ce, r);
            }
        }
        const bool large = several && r.pe - r.pb > a.group_size;
        if (__any_sync(kFullMask, large || root)) emit_groups(a, c.cb, large ? c.ce : c.cb, root, r.pb, r.pe);
        if (several) climb_chain<kPrec, kQuad>(a, l, node, top, work_top, r);
    }
}

// A node's links from the topology pass.
struct Links {
    uint32_t cb, ce, pb, pe;
    uint64_t key;
};
__device__ __forceinline__ Links load_links(const AggArgs& a, uint32_t l, uint32_t j, uint32_t u,
                                            uint32_t below) {
    Links k{0u, 0u, 0u, 0u, 0ull};
    if (j >= u) return k;
    const uint32_t node = a.offset[l] + j;
    const Children c = children_of(a, node, j, u, l, below);
    k.cb = c.cb;
    k.ce = c.ce;
    k.pb = a.pbeg[node];
    k.pe = (j + 1 < u) ? a.pbeg[node + 1] : a.n;
    k.key = a.node_key[node];
    return k;
}

// A node by eight lanes (all lanes of the warp call; `live`: the lane's group
// has a node): every record of its children loaded at once, then lane c adds
// component c of the sums and of the quadrupole, in child order. The same
// roundings as aggregate_internal, an eighth of its serial work.
template <bool kPrec, bool kQuad>
__device__ __forceinline__ void aggregate_wide(const AggArgs& a, uint32_t l, uint32_t node, bool live,
                                               const Links& k) {
    using Comp = typename std::conditional<kPrec, double, float>::type;
    const uint32_t c = threadIdx.x & 7u;
    if (live && k.ce - k.cb > 8u) atomicOr(a.err, kErrBadLayer);
    const uint32_t nch = live ? min(k.ce - k.cb, 8u) : 0u;
    Comp* const sums = reinterpret_cast<Comp*>(a.node_sum);
    float* const quads = reinterpret_cast<float*>(a.node_q);
    Comp sv[8];
    float qv[8];
    float4 ccm[8];
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        sv[i] = c < 4u && i < nch ? __ldcg(sums + 4ull * (k.cb + i) + c) : Comp(0);
        ccm[i] = i < nch ? ld_l2(a.node_cm + k.cb + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        qv[i] = 0.f;
        if (kQuad && i < nch && c < 5u)
            qv[i] = __ldcg(c < 4u ? quads + 4ull * (k.cb + i) + c : a.node_qyz + k.cb + i);
    }
    Comp sum = Comp(0);
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i)
        if (i < nch) {
            if constexpr (kPrec) sum = __dadd_rn(sum, sv[i]);
            else sum = __fadd_rn(sum, sv[i]);
        }
    const Comp m = __shfl_sync(kFullMask, sum, 3, 8);
    const float4 com = com_from_sums(sum, sum, sum, m);  // this lane's component in x
    float4 cm = make_float4(__shfl_sync(kFullMask, com.x, 0, 8), __shfl_sync(kFullMask, com.x, 1, 8),
                            __shfl_sync(kFullMask, com.x, 2, 8), com.w);
    float q = 0.f;
    if (nch == 1u) {
        cm = ccm[0];
        q = qv[0];
    } else if (kQuad) {
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i)
            if (i < nch) {
                const float dx = __fsub_rn(ccm[i].x, cm.x), dy = __fsub_rn(ccm[i].y, cm.y),
                            dz = __fsub_rn(ccm[i].z, cm.z);
                const float r2 =
                    __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
                // xx: tx dx - r2, yy: ty dy - r2, xy: tx dy, xz: tx dz, yz: ty dz.
                const float t = __fmul_rn(3.0f, c == 1u || c == 4u ? dy : dx);
                float v = __fmul_rn(t, c == 0u ? dx : (c < 3u ? dy : dz));
                if (c < 2u) v = __fsub_rn(v, r2);
                q = __fadd_rn(__fadd_rn(q, __fmul_rn(ccm[i].w, v)), qv[i]);
            }
    }
    if (!live) return;
    if (c < 4u) sums[4ull * node + c] = sum;
    if (kQuad && c < 5u) *(c < 4u ? quads + 4ull * node + c : a.node_qyz + node) = q;
    if (c == 5u) a.node_cm[node] = cm;
    if (c == 6u) a.node_rng[node] = make_uint4(k.cb, k.ce, k.pb, k.pe);
    if (c == 7u && a.want_delta) a.node_crit2[node] = node_crit2(a, k.key, l, cm);
}

// Layers l0 and up in one launch of one thread-block cluster: a layer's nodes
// are spread over its blocks, and the cluster barrier (which makes the blocks'
// records visible to each other) ends the layer. The next layer's links, which
// the topology pass wrote, are loaded while the barrier completes; the groups
// are written after the shared layers. Layers of few nodes give a node eight lanes.
// What bounds it: the chain up the layers, each a barrier (about 1,000 cycles
// until the stores have landed), the children's records and the arithmetic. A
// tree of 9 layers: 26 us with 1,024 bodies, 34 us with 16,384. Climbing with an
// arrival count per parent (fences, an atomic, one thread a node): 36 and 44 us;
// this kernel with one thread a node and the groups written layer by layer: 37
// and 49 us (3,500 to 4,600 cycles a node, 4,400 to 5,800 a layer of groups).
// With the last layers left to one block, while the others write the groups from
// the topology's ranges, a 1,024-body frame takes 130 us instead of 135, a step of
// 16,384 bodies 138 instead of 142.
constexpr uint32_t kTopThreads = 512;
template <bool kPrec, bool kQuad>
__global__ __launch_bounds__(kTopThreads, 1) void aggregate_top_kernel(AggArgs a, uint32_t l0) {
    after_previous();
    using Sum = typename NodeRec<kPrec>::Sum;
    cg::cluster_group cluster = cg::this_cluster();
    // Consecutive warps of nodes go to different blocks.
    const uint32_t first = ((threadIdx.x >> 5) * cluster.num_blocks() + cluster.block_rank()) * 32u +
                           (threadIdx.x & 31u);
    const uint32_t stride = cluster.num_blocks() * kTopThreads;
    Sum* const sums = reinterpret_cast<Sum*>(a.node_sum);
    uint32_t u = a.layer_count[l0], below = l0 > 0 ? a.layer_count[l0 - 1] : 0u;
    // Layers of few nodes give each node eight lanes.
    const auto wide = [&](uint32_t l, uint32_t nodes) { return l > 0 && nodes <= stride / 4u; };
    Links links{0u, 0u, 0u, 0u, 0ull};
    // The last layers, of nodes that one block's lanes can hold, are the first
    // block's alone: they need only its own barrier, and the other blocks go on to
    // the groups.
    const auto alone = [&](uint32_t l, uint32_t nodes) { return wide(l, nodes) && nodes <= kTopThreads / 8u; };
    const auto place = [&](uint32_t l, uint32_t nodes) {
        return alone(l, nodes) ? threadIdx.x / 8u : (wide(l, nodes) ? first / 8u : first);
    };
    if (l0 > 0) links = load_links(a, l0, place(l0, u), u, below);
    for (uint32_t l = l0; l <= a.lbits; ++l) {
        const bool by_eight = wide(l, u), by_one = alone(l, u);
        if (by_one && cluster.block_rank() != 0u) break;
        // Of the warp's first eight lanes.
        const uint32_t warp_node = (by_one ? threadIdx.x : first) / 32u * 4u;
        for (uint32_t j0 = by_eight ? warp_node : u; j0 < u; j0 += stride / 8u) {
            const uint32_t j = j0 + (threadIdx.x & 31u) / 8u;
            const Links k = j0 == warp_node ? links : load_links(a, l, j, u, below);
            aggregate_wide<kPrec, kQuad>(a, l, a.offset[l] + j, j < u, k);
        }
        for (uint32_t j = by_eight ? u : first; j < u; j += stride) {
            const uint32_t node = a.offset[l] + j;
            if (l == 0) {
                const NodeRec<kPrec> r = aggregate_leaf<kPrec, kQuad>(a, j, u);
                sums[node] = r.sum;
                continue;
            }
            const Links k = j == first ? links : load_links(a, l, j, u, below);
            NodeRec<kPrec> r;
            r.pb = k.pb;
            r.pe = k.pe;
            r.key = k.key;
            if (k.ce - k.cb == 1u) {
                r.sum = ld_l2(sums + k.cb);
                r.cm = ld_l2(a.node_cm + k.cb);
                if (kQuad) {
                    const float4 q = ld_l2(a.node_q + k.cb);
                    r.q[0] = q.x, r.q[1] = q.y, r.q[2] = q.z, r.q[3] = q.w;
                    r.q[4] = ld_l2(a.node_qyz + k.cb);
                }
                store_node<kPrec, kQuad>(a, node, l, k.cb, k.ce, r);
            } else {
                aggregate_internal<kPrec, kQuad>(a, l, node, k.cb, k.ce, r);
            }
            sums[node] = r.sum;
        }
        if (!by_one) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        const uint32_t above = l < a.lbits ? a.layer_count[l + 1] : 0u;
        if (l < a.lbits) links = load_links(a, l + 1u, place(l + 1u, above), above, u);
        if (by_one) __syncthreads();
        else asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        below = u;
        u = above;
    }
    // The groups of all these layers together (nothing above waits for them), by
    // the other blocks if there are any.
    const uint32_t helpers = cluster.num_blocks() - 1u;
    if (helpers > 0u && cluster.block_rank() == 0u) return;
    const uint32_t g_first =
        helpers > 0u ? ((threadIdx.x >> 5) * helpers + cluster.block_rank() - 1u) * 32u : threadIdx.x & ~31u;
    const uint32_t g_stride = max(helpers, 1u) * kTopThreads;
    uint32_t total = 0;
    for (uint32_t l = l0; l <= a.lbits; ++l) total += a.layer_count[l];
    for (uint32_t t0 = g_first; t0 < total; t0 += g_stride) {
        uint32_t j = t0 + (threadIdx.x & 31u), l = l0;
        const bool some = j < total;
        while (some && j >= a.layer_count[l]) j -= a.layer_count[l++];
        Links k{0u, 0u, 0u, 0u, 0ull};
        if (some && l > 0) k = load_links(a, l, j, a.layer_count[l], a.layer_count[l - 1]);
        if (some && l == 0) {
            k.pb = a.pbeg[j];
            k.pe = j + 1 < a.layer_count[0] ? a.pbeg[j + 1] : a.n;
        }
        const bool large = k.pe - k.pb > a.group_size;
        if (l0 == 0) emit_chunks(a, k.pb, some && l == 0 ? k.pe : k.pb);
        // The root of a system no larger than a group is a group by itself.
        const bool root = some && l == a.lbits && !large;
        if (__any_sync(kFullMask, root || (large && l > 0)))
            emit_groups(a, k.cb, large && k.ce - k.cb > 1u ? k.ce : k.cb, root, k.pb, k.pe);
    }
}

// ---- REFERENCE ----

// One launch per large layer, the rest of the tree in one cluster.
__global__ __launch_bounds__(128) void aggregate_ref_leaf_kernel(AggArgs a) {
    after_previous();
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t u0 = a.layer_count[0];
    if (j < u0) aggregate_ref_leaf(a, j, u0);
}

__global__ __launch_bounds__(128) void aggregate_ref_internal_kernel(AggArgs a, uint32_t l) {
    after_previous();
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t u = a.layer_count[l];
    if (j < u) aggregate_ref_internal(a, l, j, u);
}

// Layers l0 and up in one launch of one cluster, as above.
__global__ __launch_bounds__(kTopThreads, 1) void aggregate_ref_top_kernel(AggArgs a, uint32_t l0) {
    after_previous();
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t first = ((threadIdx.x >> 5) * cluster.num_blocks() + cluster.block_rank()) * 32u +
                           (threadIdx.x & 31u);
    const uint32_t stride = cluster.num_blocks() * kTopThreads;
    for (uint32_t l = l0; l <= a.lbits; ++l) {
        const uint32_t u = a.layer_count[l];
        for (uint32_t j = first; j < u; j += stride) {
            if (l == 0) aggregate_ref_leaf(a, j, u);
            else aggregate_ref_internal(a, l, j, u);
        }
        cluster.sync();
    }
}

// ---------------------------------------------------------- integrate ----

// updateSpheres (BarnesHut.metal:169-196): a = F * scale[type];
// v = v * damping + a * dt; x += v * dt.
__global__ void integrate_ref_kernel(float4* __restrict__ pos, float4* __restrict__ vel,
                                     const float4* __restrict__ acc,
                                     const uint32_t* __restrict__ types, uint32_t n, float dt,
                                     float damping, float s0, float s1, float s2) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 a = acc[i];
    const uint32_t t = types[i];
    if (t <= 2u) {
        const float s = t == 0 ? s0 : (t == 1 ? s1 : s2);
        a.x = __fmul_rn(a.x, s);
        a.y = __fmul_rn(a.y, s);
        a.z = __fmul_rn(a.z, s);
    }
    float4 v = vel[i];
    v.x = __fadd_rn(__fmul_rn(v.x, damping), __fmul_rn(a.x, dt));
    v.y = __fadd_rn(__fmul_rn(v.y, damping), __fmul_rn(a.y, dt));
    v.z = __fadd_rn(__fmul_rn(v.z, damping), __fmul_rn(a.z, dt));
    vel[i] = v;
    float4 p = pos[i];
    p.x = __fadd_rn(p.x, __fmul_rn(v.x, dt));
    p.y = __fadd_rn(p.y, __fmul_rn(v.y, dt));
    p.z = __fadd_rn(p.z, __fmul_rn(v.z, dt));
    pos[i] = p;
}

// ------------------------------------------------- upload / download -----

template <bool kPrec>
__global__ void upload_convert_kernel(const PositionMass* __restrict__ pm,
                                      const VelocityRadius* __restrict__ vr,
                                      const ColorType* __restrict__ ct, float4* __restrict__ pos,
                                      float4* __restrict__ vel, uint32_t* __restrict__ ids,
                                      uint32_t* __restrict__ types, double* __restrict__ x64,
                                      uint32_t n, uint32_t n_tree) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p0 = *reinterpret_cast<const float4*>(&pm[i].position[0]);
    const float m = pm[i].mass;
    const float4 v0 = *reinterpret_cast<const float4*>(&vr[i].velocity[0]);
    pos[i] = make_float4(p0.x, p0.y, p0.z, m);
    vel[i] = make_float4(v0.x, v0.y, v0.z, vr[i].radius);
    if (ids) ids[i] = i;
    if (types) types[i] = ct ? ct[i].type : (i < n_tree ? 1u : 2u);
    if (kPrec) {
        x64[i] = (double)p0.x;
        x64[(size_t)n + i] = (double)p0.y;
        x64[2 * (size_t)n + i] = (double)p0.z;
    }
}

template <bool kPrec>
__global__ void download_convert_kernel(const float4* __restrict__ pos, const float4* __restrict__ vel,
                                        const uint32_t* __restrict__ ids,
                                        const double* __restrict__ x64, PositionMass* __restrict__ pm,
                                        VelocityRadius* __restrict__ vr, uint32_t n) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const uint32_t i = ids ? ids[j] : j;
    const float4 p = pos[j], v = vel[j];
    float4 out_p = make_float4(p.x, p.y, p.z, 0.f);
    if (kPrec)
        out_p = make_float4(__double2float_rn(x64[j]), __double2float_rn(x64[(size_t)n + j]),
                            __double2float_rn(x64[2 * (size_t)n + j]), 0.f);
    *reinterpret_cast<float4*>(&pm[i].position[0]) = out_p;
    *reinterpret_cast<float4*>(&pm[i].mass) = make_float4(p.w, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4*>(&vr[i].velocity[0]) = make_float4(v.x, v.y, v.z, 0.f);
    *reinterpret_cast<float4*>(&vr[i].radius) = make_float4(v.w, 0.f, 0.f, 0.f);
}

// The same conversion as a gather: output slot o (upload order) reads state
// slot inv[o] (inv = the inverse of ids), so the 64 bytes written per
// particle are contiguous across a warp and only the reads are scattered.
template <bool kPrec>
__global__ void download_gather_kernel(const float4* __restrict__ pos, const float4* __restrict__ vel,
                                       const uint32_t* __restrict__ inv,
                                       const double* __restrict__ x64, PositionMass* __restrict__ pm,
                                       VelocityRadius* __restrict__ vr, uint32_t n) {
    const uint32_t o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= n) return;
    const uint32_t j = inv ? __ldg(&inv[o]) : o;
    const float4 p = __ldg(&pos[j]), v = __ldg(&vel[j]);
    float4 out_p = make_float4(p.x, p.y, p.z, 0.f);
    if (kPrec)
        out_p = make_float4(__double2float_rn(x64[j]), __double2float_rn(x64[(size_t)n + j]),
                            __double2float_rn(x64[2 * (size_t)n + j]), 0.f);
    *reinterpret_cast<float4*>(&pm[o].position[0]) = out_p;
    *reinterpret_cast<float4*>(&pm[o].mass) = make_float4(p.w, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4*>(&vr[o].velocity[0]) = make_float4(v.x, v.y, v.z, 0.f);
    *reinterpret_cast<float4*>(&vr[o].radius) = make_float4(v.w, 0.f, 0.f, 0.f);
}

// Scatter a per-state-slot array back to upload order through ids.
template <typename T>
__global__ void scatter_by_id_kernel(const T* __restrict__ src, const uint32_t* __restrict__ ids,
                                     T* __restrict__ dst, uint32_t n) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    dst[ids ? ids[j] : j] = src[j];
}

// AoS OctreeNode (bridge.h:47-65) for the slots [first, first+count) of
// layer l; slots past the live count read as the cleared node
// (clearOctreeNodeBuffer, Octree.metal:253-269).
__global__ void readback_nodes_kernel(const float4* __restrict__ node_cm,
                                      const uint4* __restrict__ node_rng,
                                      const uint64_t* __restrict__ node_key,
                                      const float4* __restrict__ node_ecol,
                                      const float4* __restrict__ node_ecen,
                                      const uint32_t* __restrict__ layer_count, uint32_t l,
                                      uint32_t layer_offset, uint32_t first_in_layer,
                                      uint32_t count, OctreeNode* __restrict__ out) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const uint32_t j = first_in_layer + k;
    OctreeNode o;
    uint32_t* w = reinterpret_cast<uint32_t*>(&o);
    for (int q = 0; q < 32; ++q) w[q] = 0;
    o.mortonCode = ASTRO_INVALID_MORTON_CODE;
    for (int c = 0; c < 8; ++c) o.children[c] = ASTRO_INVALID_CHILD;
    if (j < layer_count[l]) {
        const uint32_t node = layer_offset + j;
        const float4 cm = node_cm[node];
        o.mortonCode = node_key[node];
        o.centerOfMass[0] = cm.x;
        o.centerOfMass[1] = cm.y;
        o.centerOfMass[2] = cm.z;
        o.totalMass = cm.w;
        o.layer = l;
        if (node_ecol) {
            const float4 ec = node_ecol[node], en = node_ecen[node];
            o.emittedColor[0] = ec.x;
            o.emittedColor[1] = ec.y;
            o.emittedColor[2] = ec.z;
            o.emittedColor[3] = ec.w;
            o.emittedColorCenter[0] = en.x;
            o.emittedColorCenter[1] = en.y;
            o.emittedColorCenter[2] = en.z;
        }
        if (l > 0) {
            const uint4 r = node_rng[node];
            for (uint32_t c = 0; c < 8 && r.x + c < r.y; ++c) o.children[c] = r.x + c;
        }
    }
    out[k] = o;
}

// ------------------------------------------------ FP64 direct sum --------

constexpr int kDirectSamples = 8;

// Softened FP64 direct sum for sampled particles (error reference). Each
// block takes kDirectSamples samples and one slice of their particles
// (threads stride over it) and adds its partial sums to the output.
__global__ __launch_bounds__(256) void direct_sum_f64_kernel(DirectArgs a) {
    __shared__ double s_red[8][kDirectSamples][3];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t first = blockIdx.x * kDirectSamples;
    double xi[kDirectSamples][3], acc[kDirectSamples][3];
    uint32_t self[kDirectSamples], lo[kDirectSamples], hi[kDirectSamples];
    uint32_t glo = 0xFFFFFFFFu, ghi = 0;
    for (int s = 0; s < kDirectSamples; ++s) {
        const uint32_t k = first + s;
        const bool ok = k < a.n_sample;
        const uint32_t slot = ok ? a.slot[k] : 0u;
        self[s] = ok ? slot : 0xFFFFFFFFu;
        lo[s] = ok ? a.sys_begin[k] : 1u;
        hi[s] = ok ? a.sys_end[k] : 0u;
        if (ok) {
            glo = min(glo, lo[s]);
            ghi = max(ghi, hi[s]);
        }
        for (int c = 0; c < 3; ++c) {
            xi[s][c] = ok ? (a.x64 ? a.x64[(size_t)c * a.n + slot]
                                   : (double)(&a.pos[slot].x)[c])
                          : 0.0;
            acc[s][c] = 0.0;
        }
    }
    // blockIdx.y takes one of gridDim.y slices of the samples' particle range.
    const uint32_t span = ghi > glo ? ghi - glo : 0u;
    const uint32_t per = (span + gridDim.y - 1) / gridDim.y;
    const uint32_t jb = glo + blockIdx.y * per, je = min(ghi, jb + per);
    for (uint32_t j = jb + tid; j < je; j += blockDim.x) {
        const float4 q = a.pos[j];
        double xj[3];
        for (int c = 0; c < 3; ++c)
            xj[c] = a.x64 ? a.x64[(size_t)c * a.n + j] : (double)(&q.x)[c];
        const double gm = a.g * (double)q.w;
        for (int s = 0; s < kDirectSamples; ++s) {
            if (j < lo[s] || j >= hi[s] || j == self[s]) continue;
            const double dx = xj[0] - xi[s][0], dy = xj[1] - xi[s][1], dz = xj[2] - xi[s][2];
            const double r2 = dx * dx + dy * dy + dz * dz + a.eps2;
            const double inv = 1.0 / sqrt(r2);
            const double w = gm * inv * inv * inv;
            acc[s][0] += w * dx;
            acc[s][1] += w * dy;
            acc[s][2] += w * dz;
        }
    }
    for (int s = 0; s < kDirectSamples; ++s)
        for (int c = 0; c < 3; ++c) {
            double v = acc[s][c];
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFullMask, v, o);
            if (lane == 0) s_red[warp][s][c] = v;
        }
    __syncthreads();
    if (tid < kDirectSamples * 3) {
        const int s = tid / 3, c = tid % 3;
        double v = 0;
        for (uint32_t w = 0; w < (blockDim.x >> 5); ++w) v += s_red[w][s][c];
        if (first + s < a.n_sample) atomicAdd(&a.out[3ull * (first + s) + c], v);
    }
}

__global__ void gather_u32_kernel(const uint32_t* __restrict__ src, const uint32_t* __restrict__ idx,
                                  uint32_t* __restrict__ dst, uint32_t n) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) dst[k] = src[idx[k]];
}

__global__ void types_from_colors_kernel(const ColorType* __restrict__ ct, uint32_t* __restrict__ types,
                                         float4* __restrict__ colors, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    types[i] = ct[i].type;
    if (colors) colors[i] = *reinterpret_cast<const float4*>(&ct[i].color[0]);
}

// lightingPass (BarnesHut.metal:103-167) for the particles in upload order:
// the lights' positions and colours (lights[0..nl) and lights[kMaxLights..])
// were copied before the pass, so no light reads a colour written here.
constexpr uint32_t kMaxLights = 5;
constexpr float kLightAttenuation = 4e5f;  // LIGHT_ATTENUATION_DISTANCE, bridge.h:98

__global__ void lights_snapshot_kernel(const float4* __restrict__ pos,
                                       const float4* __restrict__ colors, float4* __restrict__ lights,
                                       uint32_t nl) {
    const uint32_t s = threadIdx.x;
    if (s < nl) {
        lights[s] = pos[s];
        lights[kMaxLights + s] = colors[s];
    }
}

__global__ void lighting_kernel(const float4* __restrict__ pos, const uint32_t* __restrict__ types,
                                const float4* __restrict__ lights, float4* __restrict__ colors,
                                uint32_t n, uint32_t nl) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t type = types[i];
    if (type != 1u && type != 2u) return;
    const float4 p = pos[i];
    float lr = 0.f, lg = 0.f, lb = 0.f;
    for (uint32_t s = 0; s < nl; ++s) {
        const float4 q = lights[s], c = lights[kMaxLights + s];
        const float dx = __fsub_rn(q.x, p.x), dy = __fsub_rn(q.y, p.y), dz = __fsub_rn(q.z, p.z);
        const float dist =
            __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)));
        const float dn = fmaxf(__fdiv_rn(dist, kLightAttenuation), 1e-9f);
        const float att = __fdiv_rn(1.0f, __fmul_rn(dn, dn));
        lr = __fadd_rn(lr, __fmul_rn(c.x, att));
        lg = __fadd_rn(lg, __fmul_rn(c.y, att));
        lb = __fadd_rn(lb, __fmul_rn(c.z, att));
    }
    const float a = type == 2u ? fminf(fmaxf(lr, fmaxf(lg, lb)), 0.25f) : 1.0f;
    colors[i] = make_float4(lr, lg, lb, a);
}

// ColorType in upload order from colours and types.
__global__ void colors_out_kernel(const float4* __restrict__ colors, const uint32_t* __restrict__ types,
                                  ColorType* __restrict__ out, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    *reinterpret_cast<float4*>(&out[i].color[0]) = colors[i];
    *reinterpret_cast<uint4*>(&out[i].type) = make_uint4(types[i], 0u, 0u, 0u);
}

// Stand-alone PHYSICAL kick-drift (the same arithmetic as the traversal
// epilogue): v += a dt, x += v dt, x in FP64 in the precision form.
template <bool kPrec>
__global__ void kick_drift_kernel(float4* __restrict__ pos, float4* __restrict__ vel,
                                  double* __restrict__ x64, const float4* __restrict__ acc,
                                  uint32_t n, float dt) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 a = acc[i];
    float4 v = vel[i];
    v.x = __fadd_rn(v.x, __fmul_rn(a.x, dt));
    v.y = __fadd_rn(v.y, __fmul_rn(a.y, dt));
    v.z = __fadd_rn(v.z, __fmul_rn(a.z, dt));
    vel[i] = v;
    if (kPrec) {
        const double ddt = (double)dt;
        x64[i] = __dadd_rn(x64[i], __dmul_rn((double)v.x, ddt));
        x64[(size_t)n + i] = __dadd_rn(x64[(size_t)n + i], __dmul_rn((double)v.y, ddt));
        x64[2 * (size_t)n + i] = __dadd_rn(x64[2 * (size_t)n + i], __dmul_rn((double)v.z, ddt));
    } else {
        float4 p = pos[i];
        p.x = __fadd_rn(p.x, __fmul_rn(v.x, dt));
        p.y = __fadd_rn(p.y, __fmul_rn(v.y, dt));
        p.z = __fadd_rn(p.z, __fmul_rn(v.z, dt));
        pos[i] = p;
    }
}

__global__ void inverse_ids_kernel(const uint32_t* __restrict__ ids, uint32_t* __restrict__ inv,
                                   uint32_t n) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < n) inv[ids[j]] = j;
}

// ------------------------------------------------------------ launchers --

namespace {
inline uint32_t blocks_for(uint64_t n, uint32_t t) { return (uint32_t)((n + t - 1) / t); }
}  // namespace

cudaError_t launch_encode_ref(const float4* pos, uint64_t* codes, uint32_t n_tree, uint32_t lbits,
                              float offset, const ClearArgs& clear, cudaStream_t st) {
    if (n_tree == 0) return cudaSuccess;
    encode_ref_kernel<<<blocks_for(n_tree, 256), 256, 0, st>>>(pos, codes, n_tree, 63u - 3u * lbits,
                                                               offset, clear);
    return cudaGetLastError();
}

cudaError_t launch_encode_phys(bool prec, const Chunk* chunks, uint32_t nchunks, const SysInfo* sys,
                               float4* pos, const double* x64, uint64_t* codes, uint32_t n,
                               uint32_t lbits, cudaStream_t st) {
    return launch_after(prec ? encode_phys_kernel<true> : encode_phys_kernel<false>, nchunks, 256, 0, st, chunks, sys,
                        pos, x64, codes, n, lbits);
}

cudaError_t launch_bbox(bool prec, const Chunk* chunks, uint32_t nchunks, const float4* pos,
                        const double* x64, uint32_t n, uint32_t* bb32, unsigned long long* bb64,
                        cudaStream_t st) {
    if (prec) bbox_kernel<true><<<nchunks, 256, 0, st>>>(chunks, pos, x64, n, bb32, bb64);
    else bbox_kernel<false><<<nchunks, 256, 0, st>>>(chunks, pos, x64, n, bb32, bb64);
    return cudaGetLastError();
}

cudaError_t launch_setup(bool prec, SysInfo* sys, uint32_t nsys, uint32_t* bb32,
                         unsigned long long* bb64, uint32_t lbits, float theta, uint32_t root_offset,
                         cudaStream_t st) {
    return launch_after(prec ? setup_kernel<true> : setup_kernel<false>, blocks_for(nsys, 128), 128, 0, st, sys, nsys,
                        bb32, bb64, lbits, theta, root_offset);
}

cudaError_t launch_reorder(bool prec, const uint32_t* perm, const float4* pos_a, const float4* vel_a,
                           const uint32_t* id_a, const double* x_a, float4* pos_b, float4* vel_b,
                           uint32_t* id_b, double* x_b, uint32_t n, const ClearArgs& clear,
                           cudaStream_t st) {
    return launch_after(prec ? reorder_kernel<true> : reorder_kernel<false>, blocks_for(n, 256), 256, 0, st, perm, pos_a,
                        vel_a, id_a, x_a, pos_b, vel_b, id_b, x_b, n, clear);
}

uint32_t topology_tiles(uint32_t n) { return blocks_for(n, kTopoThreads * topo_items(n)); }
// Of any count up to max_n (the tiles grow with the count).
uint32_t topology_tiles_max(uint32_t max_n) {
    return std::max(topology_tiles(max_n),
                    std::max(topology_tiles(std::min(max_n, kTopoSmall)), topology_tiles(std::min(max_n, kTopoMedium))));
}

cudaError_t launch_topology(const TopoArgs& a, cudaStream_t st) {
    if (a.n == 0) return cudaSuccess;
    switch (topo_items(a.n)) {
        case 2: return launch_after(topology_kernel<2>, a.ntiles, kTopoThreads, 0, st, a);
        case 4: return launch_after(topology_kernel<4>, a.ntiles, kTopoThreads, 0, st, a);
        default: return launch_after(topology_kernel<8>, a.ntiles, kTopoThreads, 0, st, a);
    }
}

namespace {
uint32_t top_first_layer(const LayerTable& t) {
    uint32_t l0 = 0;
    while (l0 < t.n_layers && t.size[l0] >= kLayerMinNodes) ++l0;
    return l0;
}

// Blocks of the cluster that a device runs (0: not asked yet), for every
// cluster kernel.
constexpr int kMaxDevices = 64;
uint32_t g_top_blocks[kMaxDevices] = {};
std::mutex g_top_mutex;
using TopKernel = void (*)(AggArgs, uint32_t);
const TopKernel kTopKernels[] = {aggregate_top_kernel<false, false>, aggregate_top_kernel<false, true>,
                                 aggregate_top_kernel<true, false>, aggregate_top_kernel<true, true>,
                                 aggregate_ref_top_kernel};

void cluster_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, uint32_t blocks, cudaStream_t st) {
    *cfg = cudaLaunchConfig_t{};
    cfg->gridDim = dim3(blocks);
    cfg->blockDim = dim3(kTopThreads);
    cfg->stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = blocks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // as launch_after does
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg->attrs = attr;
    cfg->numAttrs = 2;
}

cudaError_t launch_cluster(TopKernel kernel, const AggArgs& a, uint32_t l0, cudaStream_t st) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    uint32_t blocks = 0;
    {
        std::lock_guard<std::mutex> lock(g_top_mutex);
        if (dev >= 0 && dev < kMaxDevices) blocks = g_top_blocks[dev];
    }
    if (blocks == 0) return cudaErrorInvalidDevice;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    cluster_config(&cfg, attr, blocks, st);
    return cudaLaunchKernelEx(&cfg, kernel, a, l0);
}

constexpr uint32_t kWorkBlocks = 152 * 16;  // several waves at any register count

template <bool kPrec, bool kQuad>
cudaError_t launch_physical(const AggArgs& a, const LayerTable& t, cudaStream_t st) {
    const uint32_t t0 = 128, l0 = top_first_layer(t);
    uint32_t lw = 0;  // layers below lw have work lists (sizes fall with the layer; not the top one's)
    while (lw < l0 && t.size[lw] >= kWorkMinNodes) ++lw;
    for (uint32_t l = 0; l < l0; ++l) {
        const uint32_t g = blocks_for(t.size[l], t0);
        cudaError_t e;
        if (l == 0) e = launch_after(aggregate_leaf_kernel<kPrec, kQuad>, g, t0, 0, st, a, l0, lw);
        else if (l < lw)
            e = launch_after(aggregate_internal_kernel<kPrec, kQuad, true>, std::min(g, kWorkBlocks), t0, 0, st, a, l,
                             l0, lw);
        else e = launch_after(aggregate_internal_kernel<kPrec, kQuad, false>, g, t0, 0, st, a, l, l0, lw);
        if (e != cudaSuccess) return e;
    }
    return l0 < t.n_layers ? launch_cluster(aggregate_top_kernel<kPrec, kQuad>, a, l0, st) : cudaSuccess;
}
}  // namespace

// Cluster kernels: their attributes and the largest cluster, once per device;
// called before any stream capture.
cudaError_t build_init() {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_top_mutex);
    if (g_top_blocks[dev]) return cudaSuccess;
    uint32_t blocks = 16;
    for (TopKernel k : kTopKernels) {
        e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return e;
        for (; blocks > 1; blocks /= 2) {
            cudaLaunchConfig_t cfg;
            cudaLaunchAttribute attr[2];
            cluster_config(&cfg, attr, blocks, nullptr);
            cfg.numAttrs = 1;
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, k, &cfg) == cudaSuccess && clusters > 0) break;
            (void)cudaGetLastError();
        }
    }
    g_top_blocks[dev] = blocks;
    return cudaSuccess;
}

cudaError_t launch_aggregate(int mode, const AggArgs& a, const LayerTable& t, cudaStream_t st) {
    const uint32_t t0 = 128;
    if (mode == 1) return a.want_quad ? launch_physical<false, true>(a, t, st) : launch_physical<false, false>(a, t, st);
    if (mode == 2) return a.want_quad ? launch_physical<true, true>(a, t, st) : launch_physical<true, false>(a, t, st);
    const uint32_t l0 = top_first_layer(t);
    for (uint32_t l = 0; l < l0; ++l) {
        const uint32_t g = blocks_for(t.size[l], t0);
        const cudaError_t e = l == 0 ? launch_after(aggregate_ref_leaf_kernel, g, t0, 0, st, a)
                                     : launch_after(aggregate_ref_internal_kernel, g, t0, 0, st, a, l);
        if (e != cudaSuccess) return e;
    }
    return launch_cluster(aggregate_ref_top_kernel, a, l0, st);
}

cudaError_t launch_integrate_ref(float4* pos, float4* vel, const float4* acc, const uint32_t* types,
                                 uint32_t n, float dt, const astro_params& p, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    integrate_ref_kernel<<<blocks_for(n, 256), 256, 0, st>>>(
        pos, vel, acc, types, n, dt, p.damping, p.type_accel_scale[0], p.type_accel_scale[1],
        p.type_accel_scale[2]);
    return cudaGetLastError();
}

cudaError_t launch_upload_convert(bool prec, const PositionMass* pm, const VelocityRadius* vr,
                                  const ColorType* ct, float4* pos, float4* vel, uint32_t* ids,
                                  uint32_t* types, double* x64, uint32_t n, uint32_t n_tree,
                                  cudaStream_t st) {
    if (prec)
        upload_convert_kernel<true><<<blocks_for(n, 256), 256, 0, st>>>(pm, vr, ct, pos, vel, ids,
                                                                        types, x64, n, n_tree);
    else
        upload_convert_kernel<false><<<blocks_for(n, 256), 256, 0, st>>>(pm, vr, ct, pos, vel, ids,
                                                                         types, x64, n, n_tree);
    return cudaGetLastError();
}

cudaError_t launch_download_convert(bool prec, const float4* pos, const float4* vel,
                                    const uint32_t* ids, const double* x64, PositionMass* pm,
                                    VelocityRadius* vr, uint32_t n, cudaStream_t st,
                                    uint32_t* inv_scratch) {
    if (inv_scratch || !ids) {
        // The inverse permutation (a 4-byte scatter), then a gather with
        // contiguous 64-byte writes.
        if (ids) inverse_ids_kernel<<<blocks_for(n, 256), 256, 0, st>>>(ids, inv_scratch, n);
        const uint32_t* inv = ids ? inv_scratch : nullptr;
        if (prec)
            download_gather_kernel<true><<<blocks_for(n, 256), 256, 0, st>>>(pos, vel, inv, x64, pm,
                                                                             vr, n);
        else
            download_gather_kernel<false><<<blocks_for(n, 256), 256, 0, st>>>(pos, vel, inv, x64, pm,
                                                                              vr, n);
        return cudaGetLastError();
    }
    if (prec)
        download_convert_kernel<true><<<blocks_for(n, 256), 256, 0, st>>>(pos, vel, ids, x64, pm,
                                                                          vr, n);
    else
        download_convert_kernel<false><<<blocks_for(n, 256), 256, 0, st>>>(pos, vel, ids, x64, pm,
                                                                           vr, n);
    return cudaGetLastError();
}

cudaError_t launch_scatter_u64(const uint64_t* src, const uint32_t* ids, uint64_t* dst, uint32_t n,
                               cudaStream_t st) {
    scatter_by_id_kernel<uint64_t><<<blocks_for(n, 256), 256, 0, st>>>(src, ids, dst, n);
    return cudaGetLastError();
}
cudaError_t launch_scatter_f4(const float4* src, const uint32_t* ids, float4* dst, uint32_t n,
                              cudaStream_t st) {
    scatter_by_id_kernel<float4><<<blocks_for(n, 256), 256, 0, st>>>(src, ids, dst, n);
    return cudaGetLastError();
}

cudaError_t launch_readback_nodes(const float4* cm, const uint4* rng, const uint64_t* key,
                                  const float4* ecol, const float4* ecen,
                                  const uint32_t* layer_count, uint32_t l, uint32_t layer_offset,
                                  uint32_t first_in_layer, uint32_t count, OctreeNode* out,
                                  cudaStream_t st) {
    if (count == 0) return cudaSuccess;
    readback_nodes_kernel<<<blocks_for(count, 128), 128, 0, st>>>(
        cm, rng, key, ecol, ecen, layer_count, l, layer_offset, first_in_layer, count, out);
    return cudaGetLastError();
}

cudaError_t launch_direct_sum(const DirectArgs& a, cudaStream_t st) {
    if (a.n_sample == 0) return cudaSuccess;
    // Sample blocks times slices of the particle range (each slice adds its
    // partial sums), about 1,024 blocks in all, slices of at least 8,192.
    const uint32_t xb = blocks_for(a.n_sample, kDirectSamples);
    const uint32_t ys = std::max(1u, std::min((1024u + xb - 1) / xb, (a.n + 8191u) / 8192u));
    cudaError_t e = cudaMemsetAsync(a.out, 0, 24ull * a.n_sample, st);
    if (e != cudaSuccess) return e;
    direct_sum_f64_kernel<<<dim3(xb, ys), 256, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_inverse_ids(const uint32_t* ids, uint32_t* inv, uint32_t n, cudaStream_t st) {
    inverse_ids_kernel<<<blocks_for(n, 256), 256, 0, st>>>(ids, inv, n);
    return cudaGetLastError();
}

cudaError_t launch_gather_u32(const uint32_t* src, const uint32_t* idx, uint32_t* dst, uint32_t n,
                              cudaStream_t st) {
    gather_u32_kernel<<<blocks_for(n, 256), 256, 0, st>>>(src, idx, dst, n);
    return cudaGetLastError();
}

cudaError_t launch_types_from_colors(const ColorType* ct, uint32_t* types, float4* colors, uint32_t n,
                                     cudaStream_t st) {
    types_from_colors_kernel<<<blocks_for(n, 256), 256, 0, st>>>(ct, types, colors, n);
    return cudaGetLastError();
}

cudaError_t launch_lighting(const float4* pos, const uint32_t* types, float4* colors, float4* lights,
                            uint32_t n, uint32_t num_stars, cudaStream_t st) {
    const uint32_t nl = std::min(std::min(num_stars, kMaxLights), n);
    if (n == 0) return cudaSuccess;
    if (nl > 0) lights_snapshot_kernel<<<1, 32, 0, st>>>(pos, colors, lights, nl);
    lighting_kernel<<<blocks_for(n, 256), 256, 0, st>>>(pos, types, lights, colors, n, nl);
    return cudaGetLastError();
}

cudaError_t launch_colors_out(const float4* colors, const uint32_t* types, ColorType* out, uint32_t n,
                              cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    colors_out_kernel<<<blocks_for(n, 256), 256, 0, st>>>(colors, types, out, n);
    return cudaGetLastError();
}

cudaError_t launch_kick_drift(bool prec, float4* pos, float4* vel, double* x64, const float4* acc,
                              uint32_t n, float dt, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    if (prec) kick_drift_kernel<true><<<blocks_for(n, 256), 256, 0, st>>>(pos, vel, x64, acc, n, dt);
    else kick_drift_kernel<false><<<blocks_for(n, 256), 256, 0, st>>>(pos, vel, x64, acc, n, dt);
    return cudaGetLastError();
}

}  // namespace astro
