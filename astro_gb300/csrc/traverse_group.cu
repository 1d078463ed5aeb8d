// Group walk of the PHYSICAL preset: barnesHut (Astro/BarnesHut.metal:22-101)
// with the opening decisions made once per group of consecutive
// Morton-sorted particles: the walk and the far-node sums here, the
// evaluation in group_eval.cu.
//
// group_walk_kernel — one warp per group of at most 64 particles (a tree
//   cell or a pack of sibling cells, emitted with the tree); the chunks a
//   leaf larger than a group is cut into share one walk against the whole
//   leaf's box (its particles are in no spatial order inside the leaf, so
//   each chunk's box is nearly the leaf's anyway). The warp walks
//   the tree breadth first from the system's root, testing 32 frontier nodes
//   at a time against the walk's bounding box: an accepted node goes to the
//   cell list, or to the far list when its centre of mass lies further than
//   r_g / far_ratio from the box centre (r_g the box's half diagonal); an
//   opened leaf or bucket goes to the leaf list; any other opened node puts
//   its children in the next frontier. Each list is a chain of 64-word
//   blocks of a shared pool (the warp takes blocks from the pool in batches);
//   a per-walk record holds the chains and the box centre.
// group_far_kernel — the far nodes' second-order field expansion about the
//   walk's box centre, once per walk: lane l expands far nodes l, l + 32, ...
//   into its partial of the 19 coefficients, the partials are combined by an
//   xor butterfly (16 .. 1) and the sums go into the walk's record.
//
// The walk needs few registers and many resident warps (it waits on node
// loads); the evaluation needs registers for its sums. Split, each runs at
// its own occupancy.
#include <algorithm>
#include <mutex>

#include "build_kernels.cuh"
#include "common.cuh"
#include "group_lists.cuh"
#include "traverse_terms.cuh"

namespace astro {
namespace {

// Walk kernel: warps per block and the resident warps per SM it is sized for.
constexpr int kWalkWarps = 4;
constexpr int kWalkWarpsPerSm = 32;
constexpr uint32_t kNoBlock = 0xFFFFFFFFu;

// The tail of one list of the group being walked: its first and current
// blocks, the items in the current block and in the list.
struct ListTail {
    uint32_t first, blk, fill, count;
};

// Blocks of the pool a walk warp holds for its lists: [next, end), taken
// from the pool kBlockBatch at a time (one atomic per batch).
constexpr uint32_t kBlockBatch = 16;
struct BlockCache {
    uint32_t next, end;
};

// Appends the items of the lanes in `mask` (in lane order) to list L, whose
// items are kWords words each (this lane's words w0, w1). A full block is
// chained to a new one. Blocks numbered past the pool's end are not
// written: the walk goes on counting them (the pool counter ends at the
// demand), `failed` marks the group and the error bit makes the evaluation
// skip, so the host can grow the pool and run the traversal again.
// `mask` is warp-uniform.
template <uint32_t kWords>
__device__ __forceinline__ void list_append(const TraverseArgs& a, ListTail& L, BlockCache& bc,
                                            uint32_t mask, uint32_t lane, uint32_t lt, uint32_t w0,
                                            uint32_t w1, bool& failed) {
    constexpr uint32_t kCap = kListBlockWords / kWords;
    const uint32_t cnt = __popc(mask);
    const uint32_t rank = __popc(mask & lt);
    auto alloc = [&]() {
        if (bc.next == bc.end) {
            uint32_t b = 0;
            if (lane == 0) b = atomicAdd(a.lists_used, kBlockBatch);
            b = __shfl_sync(kFullMask, b, 0);
            bc.next = b;
            bc.end = b + kBlockBatch;
        }
        const uint32_t blk = bc.next++;
        if (blk >= a.lists_blocks && !failed) {
            if (lane == 0) atomicOr(a.err, kErrFrontier);
            failed = true;
        }
        return blk;
    };
    if (L.blk == kNoBlock) {
        L.blk = L.first = alloc();
        L.fill = 0;
    }
    uint32_t b = L.blk, slot = L.fill + rank;
    const uint32_t room = kCap - L.fill;
    if (cnt > room) {
        const uint32_t nb = alloc();
        if (lane == 0 && L.blk < a.lists_blocks && nb < a.lists_blocks) a.list_next[L.blk] = nb;
        if (rank >= room) {
            b = nb;
            slot = rank - room;
        }
        L.blk = nb;
        L.fill = cnt - room;
    } else {
        L.fill += cnt;
    }
    L.count += cnt;
    if (((mask >> lane) & 1u) && b < a.lists_blocks) {
        uint32_t* dst = a.lists + (size_t)b * kListBlockWords + slot * kWords;
        if constexpr (kWords == 2) *reinterpret_cast<uint2*>(dst) = make_uint2(w0, w1);
        else *dst = w0;
    }
}

}  // namespace

// ------------------------------------------------------------------ walk --

__global__ __launch_bounds__(kWalkWarps * 32, kWalkWarpsPerSm / kWalkWarps) void group_walk_kernel(
    TraverseArgs a) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt = lanemask_lt();
    const uint32_t gw = blockIdx.x * kWalkWarps + warp;
    uint32_t* const buf0 = a.frontier + (size_t)gw * 2 * a.frontier_cap;
    uint32_t* const buf1 = buf0 + a.frontier_cap;
    const uint32_t ngroups = *a.group_count;
    const bool far_on = a.far2 > 0.f;
    unsigned long long visits = 0, far_nodes = 0;
    BlockCache bcache{0u, 0u};

    while (true) {
        uint32_t gi = 0;
        if (lane == 0) gi = atomicAdd(a.queue, 1u);
        gi = __shfl_sync(kFullMask, gi, 0);
        if (gi >= ngroups) break;
        gi = group_of_ticket(gi, ngroups, a.group_chunk);
        const uint4 gr = a.groups[gi];
        // Later chunks of a leaf use the walk of its first chunk.
        if (gr.w != 0u) continue;
        // The walk's box: the group, or the whole leaf a first chunk stands
        // for (any number of particles, 64 at a time).
        const uint32_t wcount = gr.z - gr.x;
        float lo_x = INFINITY, lo_y = INFINITY, lo_z = INFINITY;
        float hi_x = -INFINITY, hi_y = -INFINITY, hi_z = -INFINITY;
        for (uint32_t b = 0; b < wcount; b += 64u) {
            const bool v0 = b + lane < wcount, v1 = b + 32u + lane < wcount;
            if (v0) {
                const float4 p0 = a.pos[gr.x + b + lane];
                lo_x = fminf(lo_x, p0.x), lo_y = fminf(lo_y, p0.y), lo_z = fminf(lo_z, p0.z);
                hi_x = fmaxf(hi_x, p0.x), hi_y = fmaxf(hi_y, p0.y), hi_z = fmaxf(hi_z, p0.z);
            }
            if (v1) {
                const float4 p1 = a.pos[gr.x + b + 32u + lane];
                lo_x = fminf(lo_x, p1.x), lo_y = fminf(lo_y, p1.y), lo_z = fminf(lo_z, p1.z);
                hi_x = fmaxf(hi_x, p1.x), hi_y = fmaxf(hi_y, p1.y), hi_z = fmaxf(hi_z, p1.z);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo_x = fminf(lo_x, __shfl_xor_sync(kFullMask, lo_x, o));
            lo_y = fminf(lo_y, __shfl_xor_sync(kFullMask, lo_y, o));
            lo_z = fminf(lo_z, __shfl_xor_sync(kFullMask, lo_z, o));
            hi_x = fmaxf(hi_x, __shfl_xor_sync(kFullMask, hi_x, o));
            hi_y = fmaxf(hi_y, __shfl_xor_sync(kFullMask, hi_y, o));
            hi_z = fmaxf(hi_z, __shfl_xor_sync(kFullMask, hi_z, o));
        }
        const float gcx = __fmul_rn(__fadd_rn(lo_x, hi_x), 0.5f);
        const float gcy = __fmul_rn(__fadd_rn(lo_y, hi_y), 0.5f);
        const float gcz = __fmul_rn(__fadd_rn(lo_z, hi_z), 0.5f);
        const float hrx = __fmul_rn(__fsub_rn(hi_x, lo_x), 0.5f);
        const float hry = __fmul_rn(__fsub_rn(hi_y, lo_y), 0.5f);
        const float hrz = __fmul_rn(__fsub_rn(hi_z, lo_z), 0.5f);
        const float rg2 =
            __fadd_rn(__fmul_rn(hrx, hrx), __fadd_rn(__fmul_rn(hry, hry), __fmul_rn(hrz, hrz)));
        const uint32_t sys = a.nsys > 1 ? (uint32_t)(a.sorted_keys[gr.x] >> (3u * a.lbits)) : 0u;
        const float* crit_layer = a.sys[sys].crit2;
        ListTail cells{kNoBlock, kNoBlock, 0u, 0u}, leaves = cells, fars = cells;
        bool failed = false;
        uint32_t tested = 0;

        // One frontier chunk: node nd (when `has`) at `layer`. Appends the
        // accepted, far and opened-leaf nodes to the lists in frontier order
        // and returns the opened node's child range (empty otherwise).
        auto test_nodes = [&](bool has, uint32_t nd, int layer) -> uint2 {
            float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
            uint4 r = make_uint4(0u, 0u, 0u, 0u);
            float crit = 0.f;
            if (has) {
                c = __ldg(&a.node_cm[nd]);
                r = __ldg(&a.node_rng[nd]);
                crit = a.delta ? __ldg(&a.node_crit2[nd]) : __ldg(&crit_layer[layer]);
            }
            const float bx = fmaxf(fmaxf(__fsub_rn(lo_x, c.x), __fsub_rn(c.x, hi_x)), 0.f);
            const float by = fmaxf(fmaxf(__fsub_rn(lo_y, c.y), __fsub_rn(c.y, hi_y)), 0.f);
            const float bz = fmaxf(fmaxf(__fsub_rn(lo_z, c.z), __fsub_rn(c.z, hi_z)), 0.f);
            const float dist2 =
                __fadd_rn(__fadd_rn(__fmul_rn(bx, bx), __fmul_rn(by, by)), __fmul_rn(bz, bz));
            const bool accepted = has && dist2 > crit;
            const bool leaf = has && !accepted && (layer == 0 || r.w - r.z <= a.bucket);
            const bool opn = has && !accepted && !leaf;
            bool far = false;
            if (far_on && accepted) {
                const float Dx = __fsub_rn(c.x, gcx), Dy = __fsub_rn(c.y, gcy), Dz = __fsub_rn(c.z, gcz);
                const float D2 =
                    __fadd_rn(__fmul_rn(Dx, Dx), __fadd_rn(__fmul_rn(Dy, Dy), __fmul_rn(Dz, Dz)));
                far = __fmul_rn(a.far2, D2) > rg2;
            }
            const bool acc = accepted && !far;
            tested += __popc(__ballot_sync(kFullMask, has));
            const uint32_t bfar = __ballot_sync(kFullMask, far);
            if (bfar) list_append<1>(a, fars, bcache, bfar, lane, lt, nd, 0u, failed);
            const uint32_t bacc = __ballot_sync(kFullMask, acc);
            if (bacc) list_append<1>(a, cells, bcache, bacc, lane, lt, nd, 0u, failed);
            const uint32_t bleaf = __ballot_sync(kFullMask, leaf);
            if (bleaf) list_append<2>(a, leaves, bcache, bleaf, lane, lt, r.z, r.w, failed);
            return opn ? make_uint2(r.x, r.y) : make_uint2(0u, 0u);
        };

        if (a.walk_runs) {
            // The frontier holds runs of consecutive node indices (first,
            // count) in walk order: an opened node's children are consecutive,
            // so it adds one run, and a chunk of 32 nodes is found by a shuffle
            // search over 32 runs loaded at once.
            uint2* cur = reinterpret_cast<uint2*>(buf0);
            uint2* nxt = reinterpret_cast<uint2*>(buf1);
            const uint32_t run_cap = a.frontier_cap / 2u;
            if (lane == 0) cur[0] = make_uint2(a.sys[sys].root, 1u);
            uint32_t ncur = 1;
            int layer = (int)a.lbits;
            __syncwarp();
            while (ncur > 0) {
                uint32_t nnext = 0;
                for (uint32_t rb = 0; rb < ncur; rb += 32u) {
                    const uint32_t nrun = min(32u, ncur - rb);
                    const uint2 run = lane < nrun ? cur[rb + lane] : make_uint2(0u, 0u);
                    uint32_t rincl = run.y;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t y = __shfl_up_sync(kFullMask, rincl, o);
                        if (lane >= (uint32_t)o) rincl += y;
                    }
                    const uint32_t rpre = rincl - run.y;
                    const uint32_t rtotal = __shfl_sync(kFullMask, rincl, 31);
                    for (uint32_t t0 = 0; t0 < rtotal; t0 += 32u) {
                        const uint32_t pos = t0 + lane;
                        uint32_t e = 0;
#pragma unroll
                        for (uint32_t step = 16; step > 0; step >>= 1) {
                            const uint32_t cand = e + step;
                            const uint32_t pc = __shfl_sync(kFullMask, rpre, cand & 31u);
                            if (cand < nrun && pc <= pos) e = cand;
                        }
                        const uint32_t first = __shfl_sync(kFullMask, run.x, e);
                        const uint32_t estart = __shfl_sync(kFullMask, rpre, e);
                        const bool has = pos < rtotal;
                        const uint2 ch = test_nodes(has, has ? first + (pos - estart) : 0u, layer);
                        const bool opn = ch.y > ch.x;
                        const uint32_t bopen = __ballot_sync(kFullMask, opn);
                        if (bopen) {
                            if (nnext + __popc(bopen) <= run_cap) {
                                if (opn) nxt[nnext + __popc(bopen & lt)] = make_uint2(ch.x, ch.y - ch.x);
                                nnext += __popc(bopen);
                            } else if (lane == 0) {
                                atomicOr(a.err, kErrFrontier);
                                atomicMax(a.frontier_need, 2u * (nnext + __popc(bopen)));
                            }
                        }
                    }
                }
                __syncwarp();
                uint2* t = cur;
                cur = nxt;
                nxt = t;
                ncur = nnext;
                --layer;
            }
        } else {
            // The frontier holds node indices, each opened node adding its
            // children one by one.
            uint32_t* cur = buf0;
            uint32_t* nxt = buf1;
            if (lane == 0) cur[0] = a.sys[sys].root;
            uint32_t ncur = 1;
            int layer = (int)a.lbits;
            __syncwarp();
            while (ncur > 0) {
                uint32_t nnext = 0;
                for (uint32_t base = 0; base < ncur; base += 32u) {
                    const uint32_t k = base + lane;
                    const bool has = k < ncur;
                    const uint2 ch = test_nodes(has, has ? cur[k] : 0u, layer);
                    const uint32_t cnt = ch.y - ch.x;
                    uint32_t incl = cnt;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
                        if (lane >= (uint32_t)o) incl += y;
                    }
                    const uint32_t total = __shfl_sync(kFullMask, incl, 31);
                    if (nnext + total <= a.frontier_cap) {
                        const uint32_t o0 = nnext + incl - cnt;
                        for (uint32_t j = 0; j < cnt; ++j) nxt[o0 + j] = ch.x + j;
                        nnext += total;
                    } else if (lane == 0) {
                        atomicOr(a.err, kErrFrontier);
                        atomicMax(a.frontier_need, nnext + total);
                    }
                }
                __syncwarp();
                uint32_t* t = cur;
                cur = nxt;
                nxt = t;
                ncur = nnext;
                --layer;
            }
        }

        // The group's descriptor (empty lists if the pool ran out).
        if (failed) leaves.count = cells.count = fars.count = 0;
        if (lane < 12) {
            const uint32_t w[12] = {leaves.first, leaves.count, cells.first, cells.count,
                                    fars.first, fars.count, __float_as_uint(gcx), __float_as_uint(gcy),
                                    __float_as_uint(gcz), 0u, 0u, 0u};
            uint32_t v = w[0];
#pragma unroll
            for (int k = 1; k < 12; ++k)
                if (lane == (uint32_t)k) v = w[k];
            reinterpret_cast<uint32_t*>(a.desc + gi)[lane] = v;
        }
        // Per particle of the walk; one expansion per walk and far node.
        visits += (unsigned long long)wcount * tested;
        far_nodes += fars.count;
    }
    if (lane == 0) {
        atomicAdd(&a.stats[1], visits);
        if (far_nodes) atomicAdd(&a.stats[3], far_nodes);
    }
}

// ------------------------------------------------------------ far nodes --

namespace {

// Blocks of four warps per SM (64 registers): the record loaded ahead takes
// 9 of them. 524,288-body disk 168 us, 4,194,304-body merger 749 us, 256
// systems 757 us; at 9 blocks (56 registers) 195, 873 and 843 us; 7 blocks
// the same as 8.
constexpr int kFarBlocks = 8;

// v[0 .. 2 kHalf) of lane and of lane ^ kBit added; the lane with kBit clear
// keeps the first half of the sums, the other the second, in v[0 .. kHalf).
template <int kHalf, int kBit>
__device__ __forceinline__ void fold_halves(float* v, uint32_t lane) {
    const bool up = (lane & kBit) != 0;
#pragma unroll
    for (int k = 0; k < kHalf; ++k) {
        const float keep = up ? v[k + kHalf] : v[k], give = up ? v[k] : v[k + kHalf];
        v[k] = keep + __shfl_xor_sync(kFullMask, give, kBit);
    }
}

}  // namespace

// The far-node expansion of every walk, once: lane l sums the coefficients
// of far nodes l, l + 32, ... in walk order, the lanes' partials are combined,
// and the sums go into the walk's record, where the evaluation of each group
// sharing the walk reads them (the exact form: pairwise, lane l + lane l^o,
// o = 16 .. 1; the fast form's sums are finished by far_finish there). One
// warp per record, records in order.
//
// What bounds it: FMA work behind gathered node records. With about 115
// operations a node instead of 170 (far_coefs_fast) and the next record
// loaded while the current one is expanded: disk 213 -> 168 us, merger
// 910 -> 749 us, 16,777,216-body cube 1182 -> 981 us.
template <bool kExact, bool kQuad>
__global__ __launch_bounds__(128, kExact ? 1 : kFarBlocks) void group_far_kernel(TraverseArgs a) {
    const uint32_t lane = threadIdx.x & 31;
    // A walk that ran out of room left incomplete lists: nothing to expand.
    if (*reinterpret_cast<volatile const uint32_t*>(a.err) & kErrFrontier) return;
    const uint32_t ngroups = *a.group_count;
    const uint32_t nwarps = gridDim.x * (blockDim.x / 32u);
    const float eps2 = a.eps2;
    for (uint32_t gi = blockIdx.x * (blockDim.x / 32u) + (threadIdx.x >> 5); gi < ngroups;
         gi += nwarps) {
        if (a.groups[gi].w != 0u) continue;  // a later chunk: no walk of its own
        GroupDesc* const dp = a.desc + gi;
        const uint32_t n_far = dp->n_far;
        if (n_far == 0u) continue;
        const float gcx = dp->gcx, gcy = dp->gcy, gcz = dp->gcz;
        float fc[kFarCoefs];
#pragma unroll
        for (int k = 0; k < kFarCoefs; ++k) fc[k] = 0.f;
        // Far node f sits at position f mod 64 of block f / 64 of the chain.
        // Each lane loads node f + 32's record and reads node f + 64's id
        // before it expands node f; the expansions stay in walk order.
        struct Record {
            float4 c, q;
            float qyz;
        };
        auto load = [&](uint32_t nd) {
            Record r{__ldg(&a.node_cm[nd]), make_float4(0.f, 0.f, 0.f, 0.f), 0.f};
            if constexpr (kQuad) {
                r.q = __ldg(&a.node_q[nd]);
                r.qyz = __ldg(&a.node_qyz[nd]);
            }
            return r;
        };
        ChainCursor cur{dp->far_first};
        // Id of node f, f growing by 32 from call to call.
        auto id = [&](uint32_t f) -> uint32_t {
            if (f >= n_far) return 0u;
            if (f >= kListBlockWords && (f % kListBlockWords) < 32u) cur.advance(a);
            return __ldg(cur.words(a) + f % kListBlockWords);
        };
        Record next = load(id(lane));
        uint32_t nd = id(lane + 32u);
        for (uint32_t f = lane; f < n_far; f += 32u) {
            const Record r = next;
            next = load(nd);
            nd = id(f + 64u);
            if constexpr (kExact)
                far_coefs_exact<kQuad>(r.c, r.q, r.qyz, -(r.q.x + r.q.y), gcx, gcy, gcz, eps2, fc);
            else
                far_coefs_fast<kQuad>(r.c, r.q, r.qyz, gcx, gcy, gcz, eps2, fc);
        }
        if constexpr (kExact) {
#pragma unroll
            for (int k = 0; k < kFarCoefs; ++k) {
                float v = fc[k];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(kFullMask, v, o));
                fc[k] = v;
            }
            float v = fc[0];
#pragma unroll
            for (int k = 1; k < kFarCoefs; ++k)
                if (lane == (uint32_t)k) v = fc[k];
            if (lane < (uint32_t)kFarCoefs) dp->far_co[lane] = v;
        } else {
            // Each step a lane gives half of its sums to its partner and keeps
            // the other half: 21 shuffles instead of 95, one sum a lane at the end.
            float v[20];
#pragma unroll
            for (int k = 0; k < kFarCoefs; ++k) v[k] = fc[k];
            v[19] = 0.f;
            fold_halves<10, 16>(v, lane);
            fold_halves<5, 8>(v, lane);
            v[5] = 0.f;
            fold_halves<3, 4>(v, lane);
            v[3] = 0.f;
            fold_halves<2, 2>(v, lane);
            fold_halves<1, 1>(v, lane);
            const uint32_t k3 = 2u * ((lane >> 1) & 1u) + (lane & 1u);
            const uint32_t k5 = 3u * ((lane >> 2) & 1u) + k3;
            if (k3 < 3u && k5 < 5u) dp->far_co[10u * (lane >> 4) + 5u * ((lane >> 3) & 1u) + k5] = v[0];
        }
    }
}

// ------------------------------------------------------------- launches --

namespace {

constexpr int kMaxDevices = 64;
int g_sms[kMaxDevices] = {};
int g_walk_per_sm[kMaxDevices] = {};
std::mutex g_mutex;

int device_index() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
    return dev;
}

int sm_count() {
    const int dev = device_index();
    std::lock_guard<std::mutex> lock(g_mutex);
    if (g_sms[dev] == 0) {
        int n = 0;
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        g_sms[dev] = n > 0 ? n : 1;
    }
    return g_sms[dev];
}

uint32_t walk_blocks() {
    const int dev = device_index();
    int per_sm = 0;
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        per_sm = g_walk_per_sm[dev];
    }
    if (per_sm == 0) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, group_walk_kernel, kWalkWarps * 32, 0);
        per_sm = std::max(1, per_sm);
        std::lock_guard<std::mutex> lock(g_mutex);
        g_walk_per_sm[dev] = per_sm;
    }
    return (uint32_t)per_sm * (uint32_t)sm_count();
}

}  // namespace

uint32_t group_walk_warps() { return walk_blocks() * (uint32_t)kWalkWarps; }

size_t group_list_blocks(uint32_t n, uint32_t group_size) {
    // Measured lists run to about 1,800 words per group (a 524,288-body disk
    // with far nodes at ratio 0.15, groups of at most 32), with at most three
    // partly filled blocks per group; groups average at least half the group
    // size. 2,048 words per group of half the group size, plus the batches of
    // blocks the walk warps hold, leaves room.
    const size_t groups = (size_t)n / std::max(1u, group_size / 2u) + 1;
    const size_t words = std::max<size_t>(groups * 2048, (size_t)1 << 22);
    const size_t blocks = words / kListBlockWords + (size_t)group_walk_warps() * kBlockBatch;
    return std::min<size_t>(blocks, 0xFFFFFF00ull);
}

cudaError_t launch_traverse_groups(const TraverseArgs& a, const TraverseConfig& c, cudaStream_t st,
                                   cudaEvent_t* ev) {
    if (a.n == 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(a.queue, 0, sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    // Evaluation queue and list pool counter (adjacent words).
    e = cudaMemsetAsync(a.eval_queue, 0, 2 * sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    if (ev && (e = cudaEventRecord(ev[0], st)) != cudaSuccess) return e;
    group_walk_kernel<<<walk_blocks(), kWalkWarps * 32, 0, st>>>(a);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (ev && (e = cudaEventRecord(ev[1], st)) != cudaSuccess) return e;
    if (a.far2 > 0.f) {
        const uint32_t blocks = (uint32_t)sm_count() * kFarBlocks;
        if (c.exact)
            c.quad ? group_far_kernel<true, true><<<blocks, 128, 0, st>>>(a)
                   : group_far_kernel<true, false><<<blocks, 128, 0, st>>>(a);
        else
            c.quad ? group_far_kernel<false, true><<<blocks, 128, 0, st>>>(a)
                   : group_far_kernel<false, false><<<blocks, 128, 0, st>>>(a);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    if ((e = launch_group_eval(a, c, st)) != cudaSuccess) return e;
    return ev ? cudaEventRecord(ev[2], st) : cudaSuccess;
}

}  // namespace astro
