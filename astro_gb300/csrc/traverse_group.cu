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

// Walk kernel: warps per block; the resident warps per SM its registers are
// sized for (80; it uses up to 72) and the ones launched, which then fit.
// Sized for 28 or 32 (72 and 64 registers) the compiler computes the distances
// twice, 178 instead of 144 instructions for 32 nodes: 524,288-body disk 248
// and 245 us against 207; 24 launched: 217 us.
constexpr int kWalkWarps = 4;
constexpr int kWalkWarpsSized = 24;
constexpr int kWalkWarpsPerSm = 28;
constexpr uint32_t kNoBlock = 0xFFFFFFFFu;

// A list of the group being walked: its first and last written blocks of the
// pool and the items in them.
struct ListOut {
    uint32_t first, last, done;
};

// Blocks of the pool a walk warp holds for its lists: [next, end), taken
// from the pool kBlockBatch at a time (one atomic per batch).
constexpr uint32_t kBlockBatch = 16;
struct BlockCache {
    uint32_t next, end;
    bool failed;  // a list of this group ran past the pool's end
};

// A warp's buffers, one after the other in slots of two words: the far and
// cell lists (one block and one chunk's 32 items each), the leaf list (ranges)
// and the next frontier (runs). A tested node becomes one item of one of them.
constexpr uint32_t kFarSlot = 0u, kCellSlot = kFarSlot + kListBlockWords + 32u;
constexpr uint32_t kLeafSlot = kCellSlot + kListBlockWords + 32u, kRunSlot = kLeafSlot + 64u;
constexpr uint32_t kWalkSlots = kRunSlot + 64u;

// Takes the next block for list L and chains it to the list's last one; n of
// its items are in it. Blocks numbered past the pool's end are not written:
// the walk goes on counting them (the pool counter ends at the demand),
// `failed` marks the group and the error bit makes the evaluation skip, so
// the host can grow the pool and run the traversal again.
__device__ __forceinline__ uint32_t next_block(const TraverseArgs& a, ListOut& L, BlockCache& bc,
                                               uint32_t lane, uint32_t n) {
    if (bc.next == bc.end) {
        uint32_t b = 0;
        if (lane == 0) b = atomicAdd(a.lists_used, kBlockBatch);
        b = __shfl_sync(kFullMask, b, 0);
        bc.next = b;
        bc.end = b + kBlockBatch;
    }
    const uint32_t blk = bc.next++;
    if (blk >= a.lists_blocks) {
        if (lane == 0 && !bc.failed) atomicOr(a.err, kErrFrontier);
        bc.failed = true;
    } else if (lane == 0 && L.last < a.lists_blocks) {
        a.list_next[L.last] = blk;
    }
    if (L.last == kNoBlock) L.first = blk;
    L.last = blk;
    L.done += n;
    return blk;
}

// Writes the first n items (at most a block) of a list's buffer to the pool
// and moves what lies behind the block to the buffer's front: node ids (first
// words), 64 a block, or ranges, 32 a block. All lanes move a word, also where
// nothing is left: the warp waits before it returns, since other lanes put the
// next items into the same words and only a barrier orders the two stores.
__device__ __forceinline__ void write_ids(const TraverseArgs& a, ListOut& L, BlockCache& bc,
                                          uint2* buf, uint32_t lane, uint32_t n) {
    const uint32_t blk = next_block(a, L, bc, lane, n);
    __syncwarp();
    if (blk < a.lists_blocks) {
        uint32_t* dst = a.lists + (size_t)blk * kListBlockWords;
        dst[lane] = buf[lane].x;
        dst[lane + 32u] = buf[lane + 32u].x;
    }
    const uint2 rest = buf[kListBlockWords + lane];
    __syncwarp();
    buf[lane] = rest;
    __syncwarp();
}
__device__ __forceinline__ void write_ranges(const TraverseArgs& a, ListOut& L, BlockCache& bc,
                                             uint2* buf, uint32_t lane, uint32_t n) {
    const uint32_t blk = next_block(a, L, bc, lane, n);
    __syncwarp();
    if (blk < a.lists_blocks)
        reinterpret_cast<uint2*>(a.lists + (size_t)blk * kListBlockWords)[lane] = buf[lane];
    const uint2 rest = buf[32u + lane];
    __syncwarp();
    buf[lane] = rest;
    __syncwarp();
}
// The same for n <= 32 runs of the next frontier, at position `at` of nxt; a
// frontier buffer that is too small records what it wanted and drops them.
__device__ __forceinline__ uint32_t write_runs(const TraverseArgs& a, uint2* nxt, uint32_t at,
                                               uint2* buf, uint32_t lane, uint32_t n) {
    __syncwarp();
    const bool fits = at + n <= a.frontier_cap / 2u;
    if (fits) {
        if (lane < n) nxt[at + lane] = buf[lane];
    } else if (lane == 0) {
        atomicOr(a.err, kErrFrontier);
        atomicMax(a.frontier_need, 2u * (at + n));
    }
    const uint2 rest = buf[32u + lane];
    __syncwarp();
    buf[lane] = rest;
    __syncwarp();
    return fits ? at + n : at;
}

// A left shift that gives 0 for counts of 32 and more.
__device__ __forceinline__ uint32_t shl_clamped(uint32_t v, uint32_t n) {
    uint32_t r;
    asm("shl.b32 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(n));
    return r;
}

}  // namespace

// ------------------------------------------------------------------ walk --

// What bounds it: instruction issue (72% of the cycles with 24 warps), then the
// latency of the node records. So the work for 32 nodes is kept short: a
// node's run comes from one reduction and a population count; three votes
// give the four classes (far, near, leaf, opened), and each lane stores its
// one item into its class's shared buffer without a branch; blocks of the
// lists and the frontier go to memory when a buffer is full. 182 -> 144
// instructions for 32 nodes. Walks of a 524,288-body disk 333 -> 207 us, two
// Plummer spheres of 4,194,304 1180 -> 733 us, 256 systems 1740 -> 1090 us,
// 16,777,216-body cube 1262 -> 842 us, 16,384-body sphere 41 -> 25 us.
template <bool kDelta, bool kFar>
__global__ __launch_bounds__(kWalkWarps * 32, kWalkWarpsSized / kWalkWarps) void group_walk_kernel(
    TraverseArgs a) {
    __shared__ uint2 s_walk[kWalkWarps][kWalkSlots];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint2* const buf = s_walk[warp];
    const uint32_t lt = lanemask_lt(), le = lt | (1u << lane);
    const uint32_t gw = blockIdx.x * kWalkWarps + warp;
    uint32_t* const words = a.frontier + (size_t)gw * 2 * a.frontier_cap;
    uint2* const buf0 = reinterpret_cast<uint2*>(words);
    uint2* const buf1 = reinterpret_cast<uint2*>(words + a.frontier_cap);
    const uint32_t ngroups = *a.group_count;
    unsigned long long visits = 0, far_nodes = 0;
    BlockCache bcache{0u, 0u, false};

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
        lo_x = warp_min_f32(lo_x), lo_y = warp_min_f32(lo_y), lo_z = warp_min_f32(lo_z);
        hi_x = warp_max_f32(hi_x), hi_y = warp_max_f32(hi_y), hi_z = warp_max_f32(hi_z);
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
        ListOut cells{kNoBlock, kNoBlock, 0u}, leaves = cells, fars = cells;
        uint32_t far_n = 0, cell_n = 0, leaf_n = 0;  // items in the buffers
        bcache.failed = false;
        uint32_t tested = 0;

        // The frontier holds runs of consecutive node indices (first, count)
        // in walk order: an opened node's children are consecutive, so it
        // adds one run. 32 runs are taken at once and their nodes tested 32
        // at a time: the runs starting in a window of 32 nodes set a bit, and
        // a node's run is the count of starts up to it. A frontier of at most
        // 32 runs stays in registers and shared memory.
        uint2* cur = buf0;
        uint2* nxt = buf1;
        const uint32_t root = a.sys[sys].root;
        uint2 first_runs = lane == 0 ? make_uint2(root, 1u) : make_uint2(0u, 0u);
        bool stored = false;  // the frontier is in cur (else in first_runs)
        uint32_t ncur = 1;
        int layer = (int)a.lbits;
        while (ncur > 0) {
            uint32_t nnext = 0, run_n = 0;
            float crit_l = 0.f;
            if constexpr (!kDelta) crit_l = __ldg(&crit_layer[layer]);
            for (uint32_t rb = 0; rb < ncur; rb += 32u) {
                const bool is_run = rb + lane < ncur;
                uint2 run = first_runs;
                if (stored) run = is_run ? cur[rb + lane] : make_uint2(0u, 0u);
                uint32_t incl = run.y;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
                    if (lane >= (uint32_t)o) incl += y;
                }
                const uint32_t total = __shfl_sync(kFullMask, incl, 31);
                // First node of this lane's run; lanes without one never start.
                const uint32_t pre = is_run ? incl - run.y : 0x80000000u;
                const uint32_t base = run.x - (incl - run.y);
                uint32_t before = ~0u;  // runs started in earlier windows, less one
                tested += total;
                for (uint32_t t0 = 0; t0 < total; t0 += 32u) {
                    const uint32_t starts = __reduce_or_sync(kFullMask, shl_clamped(1u, pre - t0));
                    const uint32_t e = before + __popc(starts & le);
                    before += __popc(starts);
                    // Lanes past the last node load the root, and drop it.
                    const uint32_t present = min(32u, total - t0);
                    const bool has = lane < present;
                    const uint32_t at = __shfl_sync(kFullMask, base, e & 31u) + t0 + lane;
                    const uint32_t nd = has ? at : root;
                    const float4 c = __ldg(&a.node_cm[nd]);
                    const uint4 r = __ldg(&a.node_rng[nd]);
                    const float crit = kDelta ? __ldg(&a.node_crit2[nd]) : crit_l;
                    const float bx = fmaxf(fmaxf(__fsub_rn(lo_x, c.x), __fsub_rn(c.x, hi_x)), 0.f);
                    const float by = fmaxf(fmaxf(__fsub_rn(lo_y, c.y), __fsub_rn(c.y, hi_y)), 0.f);
                    const float bz = fmaxf(fmaxf(__fsub_rn(lo_z, c.z), __fsub_rn(c.z, hi_z)), 0.f);
                    const float dist2 =
                        __fadd_rn(__fadd_rn(__fmul_rn(bx, bx), __fmul_rn(by, by)), __fmul_rn(bz, bz));
                    const bool accepted = dist2 > crit;
                    const uint32_t mpresent = ~0u >> (32u - present);
                    const uint32_t macc = __ballot_sync(kFullMask, accepted) & mpresent;
                    uint32_t mfar = 0;
                    bool far = false;
                    if constexpr (kFar) {
                        const float Dx = __fsub_rn(c.x, gcx), Dy = __fsub_rn(c.y, gcy),
                                    Dz = __fsub_rn(c.z, gcz);
                        const float D2 = __fadd_rn(__fmul_rn(Dx, Dx),
                                                   __fadd_rn(__fmul_rn(Dy, Dy), __fmul_rn(Dz, Dz)));
                        far = __fmul_rn(a.far2, D2) > rg2;
                        mfar = __ballot_sync(kFullMask, far) & macc;
                    }
                    const bool leaf = layer == 0 || r.w - r.z <= a.bucket;
                    const uint32_t mleaf = __ballot_sync(kFullMask, leaf) & (mpresent & ~macc);
                    // This lane's class: the lanes in it, its buffer's next
                    // slot, and the item's words.
                    const uint32_t mnear = macc & ~mfar, mopen = mpresent & ~macc & ~mleaf;
                    const uint32_t mine = accepted ? (far ? mfar : mnear) : (leaf ? mleaf : mopen);
                    const uint32_t slot = accepted ? (far ? kFarSlot + far_n : kCellSlot + cell_n)
                                                   : (leaf ? kLeafSlot + leaf_n : kRunSlot + run_n);
                    const uint2 item = make_uint2(accepted ? nd : (leaf ? r.z : r.x),
                                                  leaf ? r.w : r.y - r.x);
                    if (has) buf[slot + __popc(mine & lt)] = item;
                    const uint32_t nacc = __popc(macc), nfar = __popc(mfar), nleaf = __popc(mleaf);
                    far_n += nfar;
                    cell_n += nacc - nfar;
                    leaf_n += nleaf;
                    run_n += present - nacc - nleaf;
                    if (max(max(far_n, cell_n), 2u * max(leaf_n, run_n)) >= kListBlockWords) {
                        if (kFar && far_n >= kListBlockWords) {
                            write_ids(a, fars, bcache, buf + kFarSlot, lane, kListBlockWords);
                            far_n -= kListBlockWords;
                        }
                        if (cell_n >= kListBlockWords) {
                            write_ids(a, cells, bcache, buf + kCellSlot, lane, kListBlockWords);
                            cell_n -= kListBlockWords;
                        }
                        if (leaf_n >= 32u) {
                            write_ranges(a, leaves, bcache, buf + kLeafSlot, lane, 32u);
                            leaf_n -= 32u;
                        }
                        if (run_n >= 32u) {
                            nnext = write_runs(a, nxt, nnext, buf + kRunSlot, lane, 32u);
                            run_n -= 32u;
                        }
                    }
                }
            }
            stored = nnext > 0;
            if (stored) {
                if (run_n > 0) nnext = write_runs(a, nxt, nnext, buf + kRunSlot, lane, run_n);
                ncur = nnext;
                uint2* t = cur;
                cur = nxt;
                nxt = t;
            } else {
                ncur = run_n;
            }
            __syncwarp();
            first_runs = lane < ncur ? buf[kRunSlot + lane] : make_uint2(0u, 0u);
            __syncwarp();
            --layer;
        }
        if (far_n) write_ids(a, fars, bcache, buf + kFarSlot, lane, far_n);
        if (cell_n) write_ids(a, cells, bcache, buf + kCellSlot, lane, cell_n);
        if (leaf_n) write_ranges(a, leaves, bcache, buf + kLeafSlot, lane, leaf_n);

        // The group's descriptor (empty lists if the pool ran out).
        if (bcache.failed) leaves.done = cells.done = fars.done = 0;
        if (lane < 12) {
            const uint32_t w[12] = {leaves.first, leaves.done, cells.first, cells.done,
                                    fars.first, fars.done, __float_as_uint(gcx), __float_as_uint(gcy),
                                    __float_as_uint(gcz), 0u, 0u, 0u};
            uint32_t v = w[0];
#pragma unroll
            for (int k = 1; k < 12; ++k)
                if (lane == (uint32_t)k) v = w[k];
            reinterpret_cast<uint32_t*>(a.desc + gi)[lane] = v;
        }
        // Per particle of the walk; one expansion per walk and far node.
        visits += (unsigned long long)wcount * tested;
        far_nodes += fars.done;
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

uint32_t walk_blocks() { return (uint32_t)sm_count() * (kWalkWarpsPerSm / kWalkWarps); }

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

cudaError_t launch_traverse_groups(const TraverseArgs& a, const TraverseConfig& c, bool clean,
                                   cudaStream_t st, cudaEvent_t* ev) {
    if (a.n == 0) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    if (!clean) {
        if ((e = cudaMemsetAsync(a.queue, 0, sizeof(uint32_t), st)) != cudaSuccess) return e;
        // Evaluation queue and list pool counter (adjacent words).
        if ((e = cudaMemsetAsync(a.eval_queue, 0, 2 * sizeof(uint32_t), st)) != cudaSuccess) return e;
    }
    if (ev && (e = cudaEventRecord(ev[0], st)) != cudaSuccess) return e;
    auto walk = a.delta ? (a.far2 > 0.f ? group_walk_kernel<true, true> : group_walk_kernel<true, false>)
                        : (a.far2 > 0.f ? group_walk_kernel<false, true> : group_walk_kernel<false, false>);
    walk<<<walk_blocks(), kWalkWarps * 32, 0, st>>>(a);
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
