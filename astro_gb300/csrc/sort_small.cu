// The radix sort of few pairs in one launch: one thread-block cluster makes
// every pass.
//
// The onesweep passes of sort.cu take a launch, a round of HBM latency and a
// look-back each, whatever the count: 60,001 pairs of 64-bit keys took a
// histogram of 11 us and eight passes of 8 us with the gaps between them. Here
// each block of a cluster of up to 16 holds a slice of the array (at most 8,192
// pairs); a pass loads the slice from L2, ranks it (warp peer masks, per-warp
// digit counts), sends the block's digit counts to every block through
// distributed shared memory, stages the pairs in digit order meanwhile, and
// after the cluster barrier stores each digit's run to its place in the other
// buffer. A digit that all keys share is not moved. The passes are stable, so
// the result is the one of sort.cu.
//
// What bounds it: the chain of latencies of a pass (two cluster barriers, the
// loads, shared-memory scatter): 9 us a pass at 60,001 pairs, 4 us at 16,384.
// Sort of 60,001 64-bit keys 76 us and nine launches -> 73 us and one; 16,384
// 18-bit keys 28 us and four launches -> 16 us. Tried first: pairs kept in shared
// memory and scattered through distributed shared memory; remote stores move
// about 6 bytes a cycle and block (10 us a pass of 60,001 pairs). Peer masks by
// match instead of votes: 89 us. From kClusterPairs on the onesweep passes are
// as fast (100,003 42-bit keys: 66 us there, 67 us here).
//
// At most kBlockPairs pairs are sorted by one block in shared memory: by radix
// passes (sort_block_kernel), or, at most kTinyPairs pairs of more than
// kTinyBits bits, by a bitonic network on (key, position). Radix / bitonic, us:
// 300 pairs of 24 bits 4.3 / 7.2, of 63 bits 9.7 / 7.2; 1,024 of 24 bits 7.6 /
// 12.0, of 63 bits 17.9 / 12.0; 2,048 of 63 bits 23.8 / 24.9; 4,096 of 24 bits
// 14.5 / 51.7, of 63 bits 35.7 / 51.6.
#include <algorithm>
#include <mutex>

#include <cooperative_groups.h>

#include "common.cuh"
#include "internal.h"

namespace cg = cooperative_groups;

namespace astro {
namespace {

constexpr uint32_t kRadix = 256;
constexpr uint32_t kBlockPairs = 4096;     // one block
constexpr uint32_t kTinyPairs = 1024, kTinyBits = 40;
constexpr uint32_t kClusterPairs = 65536;  // a cluster, radix passes
constexpr uint32_t kMaxSlice = 8192;  // pairs per block
constexpr uint32_t kMaxThreads = 1024;
constexpr uint32_t kMaxBlocks = 16;   // of the cluster
constexpr uint32_t kMaxItems = kMaxSlice / kMaxThreads;
constexpr uint32_t kMaxDevices = 64;

__host__ __device__ constexpr size_t small_smem(uint32_t slice, uint32_t threads) {
    return (size_t)slice * 12u + (size_t)(threads / 32u) * kRadix * 2u + 4u * kRadix * (kMaxBlocks + 2u) +
           4u * 32u;
}

// Threads of a block that holds `slice` pairs: four pairs a thread, then eight.
inline uint32_t small_threads(uint32_t slice) {
    return std::min(kMaxThreads, std::max(kRadix, (slice / 4u + 31u) / 32u * 32u));
}

// The two halves of the cluster barrier (release, acquire).
__device__ __forceinline__ void cluster_arrive() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

__device__ __forceinline__ uint32_t warp_scan(uint32_t v, uint32_t lane) {  // inclusive
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFullMask, v, o);
        if (lane >= (uint32_t)o) v += y;
    }
    return v;
}
// Sum of the totals of the digit warps (8) before this one.
__device__ __forceinline__ uint32_t warps_before(const uint32_t* tmp, uint32_t warp, uint32_t lane) {
    return __reduce_add_sync(kFullMask, lane < warp ? tmp[lane] : 0u);
}

__global__ __launch_bounds__(kMaxThreads, 1) void sort_small_kernel(
    const uint64_t* keys_in, const uint32_t* vals_in, uint64_t* keys_out,
    uint32_t* vals_out, uint64_t* keys_tmp, uint32_t* vals_tmp, const uint32_t* d_count,
    uint32_t n_est, uint32_t key_bits, uint32_t slice, uint32_t* __restrict__ clear_err) {
    after_previous();
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, warps = blockDim.x >> 5;
    const uint32_t rank = cluster.block_rank(), blocks = cluster.num_blocks();
    uint64_t* const keys = reinterpret_cast<uint64_t*>(smem_raw);  // the slice in digit order
    uint32_t* const vals = reinterpret_cast<uint32_t*>(keys + slice);
    uint32_t* const table = vals + slice;  // [kMaxBlocks][kRadix]: every block's digit counts
    uint32_t* const base = table + kMaxBlocks * kRadix;
    uint32_t* const start = base + kRadix;  // first staged slot of each digit
    uint32_t* const scan_tmp = start + kRadix;
    uint16_t* const warp_hist = reinterpret_cast<uint16_t*>(scan_tmp + 32u);  // [warps][kRadix]
    uint16_t* const my_hist = warp_hist + warp * kRadix;

    const uint32_t n = d_count ? min(*d_count, n_est) : n_est;
    if (clear_err && rank == 0 && tid == 0) *clear_err = 0u;
    if (n == 0) return;  // every block of the cluster
    const uint32_t first = rank * slice;
    const uint32_t mine = first < n ? min(slice, n - first) : 0u;  // pairs in this block
    // Warp w ranks a contiguous part of the slice, 32 pairs at a time in order.
    const uint32_t items = (slice + blockDim.x - 1u) / blockDim.x;
    const uint32_t warp_first = warp * 32u * items;
    const uint32_t lt = lanemask_lt();
    const uint32_t passes = key_bits == 0 ? 1u : (key_bits + 7u) / 8u;
    const uint64_t* ksrc = keys_in;
    const uint32_t* vsrc = vals_in;
    // The two other buffers alternate; the last pass writes the output, if none
    // is left out.
    bool to_out = passes % 2u != 0u;
    // All blocks are running before any remote access.
    cluster.sync();
    for (uint32_t p = 0; p < passes; ++p) {
        const uint32_t shift = 8u * p;
        const uint32_t bits = min(8u, key_bits - min(shift, key_bits));
        const uint32_t dmask = (1u << bits) - 1u;
        reinterpret_cast<uint4*>(my_hist)[lane] = make_uint4(0u, 0u, 0u, 0u);
        uint64_t key[kMaxItems];
        uint32_t val[kMaxItems], pos[kMaxItems];
#pragma unroll
        for (uint32_t k = 0; k < kMaxItems; ++k) {
            if (k >= items) break;
            const uint32_t i = warp_first + 32u * k + lane;
            const bool valid = i < mine;
            // Through L2: other blocks wrote the buffer in this launch.
            key[k] = valid ? __ldcg(ksrc + first + i) : 0ull;
            val[k] = valid ? (vsrc ? __ldcg(vsrc + first + i) : first + i) : 0u;
        }
        __syncwarp();
#pragma unroll
        for (uint32_t k = 0; k < kMaxItems; ++k) {
            if (k >= items) break;
            const bool valid = warp_first + 32u * k + lane < mine;
            const uint32_t digit = (uint32_t)(key[k] >> shift) & dmask;
            uint32_t peers = __ballot_sync(kFullMask, valid);
#pragma unroll
            for (uint32_t t = 0; t < 8u; ++t) {
                const bool bit = (digit >> t) & 1u;
                const uint32_t m = __ballot_sync(kFullMask, bit);
                peers &= bit ? m : ~m;
            }
            const uint32_t lower = __popc(peers & lt), cnt = __popc(peers);
            uint32_t old = 0;
            if (valid) old = my_hist[digit];
            __syncwarp();
            if (valid && lower + 1u == cnt) my_hist[digit] = (uint16_t)(old + cnt);
            __syncwarp();
            pos[k] = old + lower;
        }
        __syncthreads();
        // The warps' exclusive offsets of every digit and the block's count, four
        // lanes a digit with a quarter of the warps each, 1,024 or 256 threads.
        for (uint32_t d0 = 0; d0 < kRadix; d0 += blockDim.x / 4u) {
            const uint32_t d = d0 + tid / 4u, q = tid % 4u;
            uint32_t c[kMaxThreads / 128u], sum = 0;
#pragma unroll
            for (uint32_t t = 0; t < kMaxThreads / 128u; ++t) {
                const uint32_t w = q * (kMaxThreads / 128u) + t;
                c[t] = w < warps && d < kRadix ? (uint32_t)warp_hist[w * kRadix + d] : 0u;
                sum += c[t];
            }
            uint32_t run = sum;
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFullMask, run, o, 4);
                if (q >= (uint32_t)o) run += y;
            }
            const uint32_t count = __shfl_sync(kFullMask, run, 3, 4);
            run -= sum;
#pragma unroll
            for (uint32_t t = 0; t < kMaxThreads / 128u; ++t) {
                const uint32_t w = q * (kMaxThreads / 128u) + t;
                if (w < warps && d < kRadix) warp_hist[w * kRadix + d] = (uint16_t)run;
                run += c[t];
            }
            // The count goes to every block of the cluster.
            if (d < kRadix) {
                if (q == 0u) start[d] = count;
                for (uint32_t r = q; r < blocks; r += 4u)
                    *cluster.map_shared_rank(table + rank * kRadix + d, r) = count;
            }
        }
        cluster_arrive();
        // Meanwhile the block's pairs are staged in digit order.
        __syncthreads();
        uint32_t local = 0, incl = 0, count = 0;
        if (tid < kRadix) {
            count = start[tid];
            incl = warp_scan(count, lane);
            if (lane == 31u) scan_tmp[warp] = incl;
        }
        __syncthreads();
        if (tid < kRadix) {
            local = incl - count + warps_before(scan_tmp, warp, lane);
            start[tid] = local;
        }
        __syncthreads();
#pragma unroll
        for (uint32_t k = 0; k < kMaxItems; ++k) {
            if (k >= items) break;
            if (warp_first + 32u * k + lane >= mine) continue;
            const uint32_t digit = (uint32_t)(key[k] >> shift) & dmask;
            const uint32_t at = start[digit] + my_hist[digit] + pos[k];
            keys[at] = key[k];
            vals[at] = val[k];
        }
        cluster_wait();
        // Digit totals, and the keys of the digit in earlier blocks.
        uint32_t total = 0, before = 0;
        if (tid < kRadix) {
#pragma unroll
            for (uint32_t r = 0; r < kMaxBlocks; ++r) {
                const uint32_t c = r < blocks ? table[r * kRadix + tid] : 0u;
                total += c;
                before += r < rank ? c : 0u;
            }
            incl = warp_scan(total, lane);
            if (lane == 31u) scan_tmp[8u + warp] = incl;
        }
        // One digit: nothing moves (every block finds the same).
        if (!__syncthreads_or(tid < kRadix && total == n)) {
            uint64_t* const kdst = to_out ? keys_out : keys_tmp;
            uint32_t* const vdst = to_out ? vals_out : vals_tmp;
            if (tid < kRadix)
                base[tid] = incl - total + warps_before(scan_tmp + 8, warp, lane) + before - local;
            __syncthreads();
            // A digit's pairs lie in a run here and go to consecutive places.
            for (uint32_t i = tid; i < mine; i += blockDim.x) {
                const uint64_t k = keys[i];
                const uint32_t o = base[(uint32_t)(k >> shift) & dmask] + i;
                kdst[o] = k;
                vdst[o] = vals[i];
            }
            ksrc = kdst;
            vsrc = vdst;
            to_out = !to_out;
        }
        // Also: no block sends counts for the next pass, or leaves, while
        // another reads the ones of this pass.
        cluster.sync();
    }
    if (ksrc != keys_out)
        for (uint32_t i = tid; i < mine; i += blockDim.x) {
            keys_out[first + i] = __ldcg(ksrc + first + i);
            vals_out[first + i] = vsrc ? __ldcg(vsrc + first + i) : first + i;
        }
}

// Radix passes of one block over pairs that stay in shared memory between them:
// kItems pairs a thread, ranked as in sort_small_kernel.
__host__ __device__ constexpr size_t block_smem(uint32_t pairs, uint32_t threads) {
    return (size_t)pairs * 12u + (size_t)(threads / 32u) * kRadix * 2u + 4u * kRadix + 4u * 8u;
}
template <int kItems>
__global__ __launch_bounds__(kMaxThreads, 1) void sort_block_kernel(
    const uint64_t* keys_in, const uint32_t* vals_in, uint64_t* __restrict__ keys_out,
    uint32_t* __restrict__ vals_out, const uint32_t* d_count, uint32_t n_est, uint32_t key_bits,
    uint32_t* __restrict__ clear_err) {
    after_previous();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, warps = blockDim.x >> 5;
    const uint32_t room = kItems * blockDim.x;
    uint64_t* const keys = reinterpret_cast<uint64_t*>(smem_raw);
    uint32_t* const vals = reinterpret_cast<uint32_t*>(keys + room);
    uint16_t* const warp_hist = reinterpret_cast<uint16_t*>(vals + room);  // [warps][kRadix]
    uint32_t* const start = reinterpret_cast<uint32_t*>(warp_hist + warps * kRadix);
    uint32_t* const scan_tmp = start + kRadix;
    uint16_t* const my_hist = warp_hist + warp * kRadix;
    const uint32_t n = d_count ? min(*d_count, n_est) : n_est;
    if (clear_err && tid == 0) *clear_err = 0u;
    const uint32_t warp_first = warp * 32u * kItems + lane;
    const uint32_t lt = lanemask_lt();
    uint64_t key[kItems];
    uint32_t val[kItems], pos[kItems];
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const uint32_t i = warp_first + 32u * k;
        key[k] = i < n ? keys_in[i] : 0ull;
        val[k] = i < n ? (vals_in ? vals_in[i] : i) : 0u;
    }
    const uint32_t passes = key_bits == 0 ? 1u : (key_bits + 7u) / 8u;
#pragma unroll 1
    for (uint32_t p = 0; p < passes; ++p) {
        const uint32_t shift = 8u * p;
        const uint32_t dmask = (1u << min(8u, key_bits - min(shift, key_bits))) - 1u;
        reinterpret_cast<uint4*>(my_hist)[lane] = make_uint4(0u, 0u, 0u, 0u);
        if (p > 0) {
#pragma unroll
            for (int k = 0; k < kItems; ++k) {
                key[k] = keys[warp_first + 32u * k];
                val[k] = vals[warp_first + 32u * k];
            }
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            const bool valid = warp_first + 32u * k < n;
            const uint32_t digit = (uint32_t)(key[k] >> shift) & dmask;
            uint32_t peers = __ballot_sync(kFullMask, valid);
#pragma unroll
            for (uint32_t t = 0; t < 8u; ++t) {
                const bool bit = (digit >> t) & 1u;
                const uint32_t m = __ballot_sync(kFullMask, bit);
                peers &= bit ? m : ~m;
            }
            pos[k] = __popc(peers & lt);
            if (valid) pos[k] += my_hist[digit];
            __syncwarp();
            if (valid && (peers & ~lt) == (1u << lane)) my_hist[digit] = (uint16_t)(pos[k] + 1u);
            __syncwarp();
        }
        __syncthreads();
        // The warps' exclusive offsets of every digit and its count, four lanes a
        // digit with a quarter of the warps each.
        for (uint32_t d0 = 0; d0 < kRadix; d0 += blockDim.x / 4u) {
            const uint32_t d = d0 + tid / 4u, q = tid % 4u;
            uint32_t c[kMaxThreads / 128u], sum = 0;
#pragma unroll
            for (uint32_t t = 0; t < kMaxThreads / 128u; ++t) {
                const uint32_t w = q * (kMaxThreads / 128u) + t;
                c[t] = w < warps && d < kRadix ? (uint32_t)warp_hist[w * kRadix + d] : 0u;
                sum += c[t];
            }
            uint32_t run = sum;
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFullMask, run, o, 4);
                if (q >= (uint32_t)o) run += y;
            }
            if (q == 3u && d < kRadix) start[d] = run;
            run -= sum;
#pragma unroll
            for (uint32_t t = 0; t < kMaxThreads / 128u; ++t) {
                const uint32_t w = q * (kMaxThreads / 128u) + t;
                if (w < warps && d < kRadix) warp_hist[w * kRadix + d] = (uint16_t)run;
                run += c[t];
            }
        }
        __syncthreads();
        uint32_t incl = 0, count = 0;
        if (tid < kRadix) {
            count = start[tid];
            incl = warp_scan(count, lane);
            if (lane == 31u) scan_tmp[warp] = incl;
        }
        __syncthreads();
        if (tid < kRadix) start[tid] = incl - count + warps_before(scan_tmp, warp, lane);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            if (warp_first + 32u * k >= n) continue;
            const uint32_t digit = (uint32_t)(key[k] >> shift) & dmask;
            const uint32_t at = start[digit] + my_hist[digit] + pos[k];
            keys[at] = key[k];
            vals[at] = val[k];
        }
        __syncthreads();
    }
    for (uint32_t i = tid; i < n; i += blockDim.x) {
        keys_out[i] = keys[i];
        vals_out[i] = vals[i];
    }
}

// Bitonic sort of at most kTinyPairs pairs in shared memory, a compare-exchange a
// thread and stage. Strides of up to 32 stay inside a warp's 64
// elements, so those stages only need the warp.
constexpr uint32_t kTinyThreads = 1024;
__global__ __launch_bounds__(kTinyThreads, 1) void sort_tiny_kernel(
    const uint64_t* keys_in, const uint32_t* vals_in,
    uint64_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out,
    const uint32_t* d_count, uint32_t n_est, uint64_t mask, uint32_t size,
    uint32_t* __restrict__ clear_err) {
    after_previous();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* const keys = reinterpret_cast<uint64_t*>(smem_raw);
    uint32_t* const at = reinterpret_cast<uint32_t*>(keys + size);
    const uint32_t tid = threadIdx.x;
    const uint32_t n = d_count ? min(*d_count, n_est) : n_est;
    if (clear_err && tid == 0) *clear_err = 0u;
    // Padding sorts behind every pair: the largest key, later positions.
    for (uint32_t i = tid; i < size; i += blockDim.x) {
        keys[i] = i < n ? keys_in[i] : ~0ull;
        at[i] = i;
    }
    __syncthreads();
    for (uint32_t k = 2; k <= size; k *= 2u) {
        for (uint32_t j = k / 2u; j > 0u; j /= 2u) {
            for (uint32_t t = tid; t < size / 2u; t += blockDim.x) {
                const uint32_t i = 2u * t - (t & (j - 1u)), o = i + j;
                const uint64_t a = keys[i], b = keys[o];
                const uint32_t pa = at[i], pb = at[o];
                const uint64_t ma = a & mask, mb = b & mask;
                const bool greater = ma > mb || (ma == mb && pa > pb);
                if (greater == ((i & k) == 0u)) {
                    keys[i] = b, keys[o] = a;
                    at[i] = pb, at[o] = pa;
                }
            }
            // The next stage's stride is j / 2, or k when this merge is done.
            if ((j > 1u ? j / 2u : k) <= 32u && j <= 32u) __syncwarp();
            else __syncthreads();
        }
    }
    for (uint32_t i = tid; i < n; i += blockDim.x) {
        keys_out[i] = keys[i];
        vals_out[i] = vals_in ? vals_in[at[i]] : at[i];
    }
}

uint32_t g_cluster[kMaxDevices] = {};  // largest cluster the device runs; 0: not asked yet
std::mutex g_small_mutex;

void launch_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, uint32_t blocks,
                   uint32_t threads, uint32_t slice, cudaStream_t st) {
    *cfg = cudaLaunchConfig_t{};
    cfg->gridDim = dim3(blocks);
    cfg->blockDim = dim3(threads);
    cfg->dynamicSmemBytes = small_smem(slice, threads);
    cfg->stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = blocks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // as launch_after does
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg->attrs = attr;
    cfg->numAttrs = 2;
}

}  // namespace

// Kernel attributes and the largest cluster, once per device.
cudaError_t sort_small_init(int dev) {
    if (dev < 0 || dev >= (int)kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_small_mutex);
    if (g_cluster[dev]) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(sort_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)small_smem(kMaxSlice, kMaxThreads));
    if (e != cudaSuccess) return e;
    for (auto k : {sort_block_kernel<1>, sort_block_kernel<2>, sort_block_kernel<4>}) {
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)block_smem(kBlockPairs, kMaxThreads));
        if (e != cudaSuccess) return e;
    }
    e = cudaFuncSetAttribute(sort_tiny_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(kTinyPairs * 12u));
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(sort_small_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    uint32_t size = 16;
    for (; size > 1; size /= 2) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[2];
        launch_config(&cfg, attr, size, kMaxThreads, kMaxSlice, nullptr);
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, sort_small_kernel, &cfg) == cudaSuccess && clusters > 0)
            break;
        (void)cudaGetLastError();
    }
    g_cluster[dev] = size;
    return cudaSuccess;
}

uint32_t sort_small_max(int dev) {
    std::lock_guard<std::mutex> lock(g_small_mutex);
    return dev >= 0 && dev < (int)kMaxDevices && g_cluster[dev] > 0
               ? std::max(kBlockPairs, std::min(kClusterPairs, g_cluster[dev] * kMaxSlice))
               : 0u;
}

cudaError_t sort_small(const uint64_t* keys_in, const uint32_t* vals_in, uint64_t* keys_out,
                       uint32_t* vals_out, uint64_t* keys_tmp, uint32_t* vals_tmp, uint32_t n_est,
                       const uint32_t* d_count, uint32_t key_bits, int dev, cudaStream_t st,
                       uint32_t* clear_err) {
    uint32_t cap;
    {
        std::lock_guard<std::mutex> lock(g_small_mutex);
        cap = g_cluster[dev];
    }
    if (n_est <= kBlockPairs && (n_est > kTinyPairs || key_bits <= kTinyBits)) {
        const uint32_t items = n_est <= 1024u ? 1u : (n_est <= 2048u ? 2u : 4u);
        const uint32_t threads = std::max(kRadix, ((n_est + items - 1u) / items + 31u) / 32u * 32u);
        auto kernel = items == 1u ? sort_block_kernel<1> : (items == 2u ? sort_block_kernel<2> : sort_block_kernel<4>);
        return launch_after(kernel, 1, threads, block_smem(items * threads, threads), st, keys_in, vals_in, keys_out,
                            vals_out, d_count, n_est, key_bits, clear_err);
    }
    if (n_est <= kTinyPairs) {
        uint32_t size = 64;
        while (size < n_est) size *= 2u;
        const uint64_t mask = key_bits >= 64u ? ~0ull : (1ull << key_bits) - 1ull;
        return launch_after(sort_tiny_kernel, 1, std::min(kTinyThreads, size / 2u), size * 12u, st, keys_in, vals_in,
                            keys_out, vals_out, d_count, n_est, mask, size, clear_err);
    }
    // About a thousand pairs a block, then more per block once the cluster is
    // full, in equal slices (a multiple of 32 pairs).
    uint32_t blocks = 1;
    while (blocks < cap && blocks * 1024u < n_est) blocks *= 2u;
    const uint32_t slice = std::max(256u, ((n_est + blocks - 1u) / blocks + 31u) / 32u * 32u);
    if (slice > kMaxSlice) return cudaErrorInvalidValue;
    const uint32_t threads = small_threads(slice);
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    launch_config(&cfg, attr, blocks, threads, slice, st);
    return cudaLaunchKernelEx(&cfg, sort_small_kernel, keys_in, vals_in, keys_out, vals_out, keys_tmp,
                              vals_tmp, d_count, n_est, key_bits, slice, clear_err);
}

}  // namespace astro
