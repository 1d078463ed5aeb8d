// Barnes-Hut force traversal: barnesHut (Astro/BarnesHut.metal:22-101).
//
// traverse_ref_kernel — the REFERENCE preset: one thread per particle in
//   upload order, a private stack, node size 2^(21+layer), monopole leaves
//   with the self-leaf skip and the r^2 > leaf_min cut, softening added to
//   r^2, clamp; correctly rounded FP32 operations in the reference's order.
// traverse_ref_small_kernel — the same where the whole tree fits in shared
//   memory, laid out in visiting order (no stacks).
//
// traverse_phys_kernel — the PHYSICAL preset: one warp per 32 consecutive
//   Morton-ordered particles. The warp walks the tree once for all its
//   lanes with a shared stack of child ranges {begin, end, layer, lane mask};
//   a lane only evaluates nodes whose mask holds its bit, and a node is
//   opened for the lanes that reject it, so every lane makes exactly the
//   decisions of its own depth-first walk, in the same order (children are
//   taken last first, as the reference's LIFO stack pops them). Node
//   records (SoA float4 centre of mass/mass + uint4 ranges) are read through
//   the read-only path as warp-broadcast loads. Opened leaves and buckets are
//   staged 32 particles at a time in shared memory and summed particle by
//   particle. The epilogue clamps, stores the acceleration and performs the
//   kick-drift (v += a dt, x += v dt).
#include <algorithm>

#include "build_kernels.cuh"
#include "common.cuh"
#include "traverse_terms.cuh"

namespace astro {

constexpr int kRefStack = 160;   // >= 7 * 21 + 1 entries (8 children per opened node)
constexpr int kPhysStack = 64;   // >= 32 roots + 22 layers of ranges

__global__ __launch_bounds__(128) void traverse_ref_kernel(TraverseArgs a) {
    const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= a.n) return;
    uint32_t st_node[kRefStack];
    uint8_t st_layer[kRefStack];
    uint32_t sp = 0;
    st_node[sp] = a.root;
    st_layer[sp] = (uint8_t)a.lbits;
    ++sp;
    const float4 me = a.pos[gid];
    const uint32_t type = a.types[gid];
    const uint64_t my_code =
        (type != 2u && gid < a.n_tree) ? a.codes[gid] : ASTRO_INVALID_MORTON_CODE;
    float fx = 0.f, fy = 0.f, fz = 0.f;
    uint32_t inter = 0, visits = 0;
    while (sp > 0) {
        --sp;
        const uint32_t nd = st_node[sp];
        const uint32_t layer = st_layer[sp];
        ++visits;
        const float4 c = __ldg(&a.node_cm[nd]);
        const float dx = __fsub_rn(c.x, me.x), dy = __fsub_rn(c.y, me.y), dz = __fsub_rn(c.z, me.z);
        float dist_sqr = __fadd_rn(
            __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)), a.eps2);
        dist_sqr = fmaxf(dist_sqr, 1e-6f);
        float dist = __fsqrt_rn(dist_sqr);
        dist = fmaxf(dist, 1e-6f);
        const bool is_leaf = layer == 0;
        bool add = false;
        if (is_leaf) {
            const bool is_self = type != 2u && my_code == __ldg(&a.node_key[nd]);
            add = !is_self && dist_sqr > a.leaf_min_dist2;
        } else if (__fdiv_rn(exp2_exact(21 + (int)layer), dist) < a.theta) {
            add = true;
        } else {
            const uint4 r = __ldg(&a.node_rng[nd]);
            for (uint32_t ch = r.x; ch < r.y; ++ch) {
                if (sp < kRefStack) {
                    st_node[sp] = ch;
                    st_layer[sp] = (uint8_t)(layer - 1);
                    ++sp;
                } else {
                    atomicOr(a.err, kErrStackOverflow);
                }
            }
        }
        if (add) {
            const float gm = __fmul_rn(a.g, c.w), den = __fmul_rn(dist_sqr, dist);
            fx = __fadd_rn(fx, __fdiv_rn(__fmul_rn(gm, dx), den));
            fy = __fadd_rn(fy, __fdiv_rn(__fmul_rn(gm, dy), den));
            fz = __fadd_rn(fz, __fdiv_rn(__fmul_rn(gm, dz), den));
            ++inter;
        }
    }
    const float cl = a.clampv;
    a.acc[gid] = make_float4(fminf(fmaxf(fx, -cl), cl), fminf(fmaxf(fy, -cl), cl),
                             fminf(fmaxf(fz, -cl), cl), 0.f);
    atomicAdd(&a.stats[0], (unsigned long long)inter);
    atomicAdd(&a.stats[1], (unsigned long long)visits);
    atomicAdd(&a.stats[2], (unsigned long long)inter);
}

// The same walk where the tree is small (the reference's scene: 205 bodies,
// some 900 nodes, and 500,000 particles that feel them). Each block lays the
// tree out in shared memory in the order the stack visits it (a node, then its
// children's subtrees, last child first), each node with the position behind
// its subtree, so a particle's walk is one index: the next node when this one
// is opened, the position behind the subtree when it is accepted. The warp
// takes the smallest index of its lanes, so lanes that part meet again and a
// node is visited once per warp. The opening test size / dist < theta is a
// comparison of dist^2 with a bound per layer: correctly rounded square root
// and division are monotone, so the bound is the smallest float that passes
// (found by bisection over the floats), and the decisions are the same. A
// layer whose bound lies beyond the largest distance between the warp's
// particles and the tree is opened by all of them: its nodes are counted and
// stepped over (`next`, one table per layer).
//
// What bounds it: instruction issue (about 25 instructions an opened node, 90
// a leaf with its square root and three divisions). 500,205 particles: 1548 us
// with the stack kernel (per-thread stacks in local memory, a square root and a
// division per opened node, three atomics per particle on the same words),
// 577 us with every node tested, 393 us here.
constexpr uint32_t kRefThreads = 512;  // 393 us; 256: 428, 384: 416 (shared memory limits the blocks)
constexpr uint32_t kRefNodes = 2048;  // capacity of the shared layout (57 bytes a node)
constexpr uint32_t kRefSkips = 8;     // tables: none left out, layers >= 1, ..., >= 7

struct RefSmem {
    float4* node;    // centre of mass, G m
    float2* bound;   // dist^2 from which the node is accepted; position behind its subtree (as bits)
    uint64_t* key;   // leaf key (internal: no key)
    uint32_t* size;  // subtree sizes, by compact index (layer by layer)
    uint32_t* pos;   // position in visiting order, by compact index
    uint16_t* next;  // [kRefSkips][capacity + 1]: first position from here on whose
                     // layer is below the table's (table 0: here)
    uint8_t* layer;  // by position
};
// Bytes of RefSmem's arrays for a tree of at most `capacity` nodes.
__host__ __device__ constexpr size_t ref_smem(uint32_t capacity) {
    return (size_t)capacity * 41u + 2u * kRefSkips * ((size_t)capacity + 1u);
}

// Smallest float d2 >= 1e-6 with size / max(sqrt(d2), 1e-6) < theta.
__device__ __forceinline__ float accept_from(float size, float theta) {
    uint32_t lo = __float_as_uint(1e-6f), hi = 0x7F800000u;  // the bound lies in [lo, hi]
    while (lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2u;
        const float dist = fmaxf(__fsqrt_rn(__uint_as_float(mid)), 1e-6f);
        if (__fdiv_rn(size, dist) < theta) hi = mid;
        else lo = mid + 1u;
    }
    return __uint_as_float(lo);
}

__global__ __launch_bounds__(kRefThreads) void traverse_ref_small_kernel(TraverseArgs a, RefTree t) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint32_t s_start[ASTRO_MAX_LAYERS + 1];
    __shared__ float s_bound[ASTRO_MAX_LAYERS];
    __shared__ unsigned long long s_stats[2];
    const uint32_t tid = threadIdx.x, lane = tid & 31u;
    RefSmem sm;
    sm.node = reinterpret_cast<float4*>(smem_raw);
    sm.bound = reinterpret_cast<float2*>(sm.node + t.capacity);
    sm.key = reinterpret_cast<uint64_t*>(sm.bound + t.capacity);
    sm.size = reinterpret_cast<uint32_t*>(sm.key + t.capacity);
    sm.pos = sm.size + t.capacity;
    sm.next = reinterpret_cast<uint16_t*>(sm.pos + t.capacity);
    sm.layer = reinterpret_cast<uint8_t*>(sm.next + kRefSkips * (t.capacity + 1u));
    const uint32_t row = t.capacity + 1u;
    if (tid == 0) {
        uint32_t run = 0;
        for (uint32_t l = 0; l <= a.lbits; ++l) {
            s_start[l] = run;
            run += min(t.layer_count[l], t.capacity - run);
        }
        s_start[a.lbits + 1] = run;
        s_stats[0] = s_stats[1] = 0;
    }
    if (tid >= 32u && tid - 32u <= a.lbits) {
        const uint32_t l = tid - 32u;
        // Leaves: dist^2 > leaf_min, as a bound from which on they count.
        s_bound[l] = l > 0 ? accept_from(exp2_exact(21 + (int)l), a.theta)
                           : (a.leaf_min_dist2 < INFINITY ? nextafterf(a.leaf_min_dist2, INFINITY)
                                                          : __uint_as_float(0x7FFFFFFFu));
    }
    __syncthreads();
    const uint32_t total = s_start[a.lbits + 1];
    // Subtree sizes bottom up, positions top down.
    auto child_range = [&](uint32_t l, uint32_t c, uint32_t& first, uint32_t& count) {
        const uint4 r = __ldg(&a.node_rng[t.offset[l] + (c - s_start[l])]);
        const uint32_t below = s_start[l] - s_start[l - 1];
        first = s_start[l - 1] + min(r.x - t.offset[l - 1], below);
        count = min(r.y - r.x, s_start[l] - first);
    };
    for (uint32_t l = 0; l <= a.lbits; ++l) {
        for (uint32_t c = s_start[l] + tid; c < s_start[l + 1]; c += kRefThreads) {
            uint32_t size = 1;
            if (l > 0) {
                uint32_t first, count;
                child_range(l, c, first, count);
                for (uint32_t k = 0; k < count; ++k) size += sm.size[first + k];
            }
            sm.size[c] = size;
            if (l == a.lbits) sm.pos[c] = 0;
        }
        __syncthreads();
    }
    for (uint32_t l = a.lbits; l <= a.lbits; --l) {  // down to 0, then wraps
        for (uint32_t c = s_start[l] + tid; c < s_start[l + 1]; c += kRefThreads) {
            const uint32_t nd = t.offset[l] + (c - s_start[l]);
            const uint32_t at = min(sm.pos[c], total - 1u);
            const float4 cm = __ldg(&a.node_cm[nd]);
            sm.node[at] = make_float4(cm.x, cm.y, cm.z, __fmul_rn(a.g, cm.w));
            sm.bound[at] = make_float2(s_bound[l], __uint_as_float(at + sm.size[c]));
            sm.key[at] = l == 0 ? __ldg(&a.node_key[nd]) : ASTRO_INVALID_MORTON_CODE;
            sm.layer[at] = (uint8_t)l;
            if (l > 0) {
                uint32_t first, count;
                child_range(l, c, first, count);
                uint32_t run = at + 1u;
                for (uint32_t k = count; k-- > 0;) {
                    sm.pos[first + k] = run;
                    run += sm.size[first + k];
                }
            }
        }
        __syncthreads();
    }

    for (uint32_t i = tid; i <= total; i += kRefThreads)
        for (uint32_t s = 0; s < kRefSkips; ++s) {
            uint32_t k = i;
            while (s > 0 && k < total && sm.layer[k] >= s) ++k;
            sm.next[s * row + i] = (uint16_t)k;
        }
    float nlo[3] = {INFINITY, INFINITY, INFINITY}, nhi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (uint32_t i = lane; i < total; i += 32u) {
        const float4 c = sm.node[i];
        const float v[3] = {c.x, c.y, c.z};
#pragma unroll
        for (int k = 0; k < 3; ++k) nlo[k] = fminf(nlo[k], v[k]), nhi[k] = fmaxf(nhi[k], v[k]);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) nlo[k] = warp_min_f32(nlo[k]), nhi[k] = warp_max_f32(nhi[k]);
    __syncthreads();

    uint32_t inter = 0, visits = 0;
    for (uint32_t base = blockIdx.x * kRefThreads; base < a.n; base += gridDim.x * kRefThreads) {
        const uint32_t gid = base + tid;
        const bool valid = gid < a.n;
        const float4 me = valid ? a.pos[gid] : make_float4(0.f, 0.f, 0.f, 0.f);
        // Only a tree particle that is not dust can meet its own leaf.
        const uint64_t my_code = valid && gid < a.n_tree && a.types[gid] != 2u
                                     ? a.codes[gid]
                                     : ASTRO_INVALID_MORTON_CODE;
        // The largest dist^2 a lane can meet (rounding is monotone, and the
        // operations are those of the test below).
        float far2 = 0.f;
        {
            const float v[3] = {me.x, me.y, me.z};
            float m[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const float lo = warp_min_f32(valid ? v[k] : INFINITY);
                const float hi = warp_max_f32(valid ? v[k] : -INFINITY);
                m[k] = fmaxf(fabsf(__fsub_rn(nhi[k], lo)), fabsf(__fsub_rn(nlo[k], hi)));
            }
            far2 = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m[0], m[0]), __fmul_rn(m[1], m[1])),
                                       __fmul_rn(m[2], m[2])),
                             a.eps2);
            far2 = fmaxf(far2, 1e-6f);
        }
        uint32_t skip = 0;  // layers >= skip are opened by every lane (0: none known)
        for (uint32_t l = min(a.lbits, kRefSkips - 1u); l >= 1u && s_bound[l] > far2; --l) skip = l;
        // NaN positions leave the box but never accept there either.
        const uint16_t* next = sm.next + skip * row;
        if (skip > 0u && valid) visits += total - s_start[skip];
        float fx = 0.f, fy = 0.f, fz = 0.f;
        uint32_t i = valid ? next[0] : total;  // this lane's next node
        while (true) {
            const uint32_t at = __reduce_min_sync(kFullMask, i);
            if (at >= total) break;
            const bool active = i == at;
            const float4 c = sm.node[at];
            const float2 b = sm.bound[at];
            const float dx = __fsub_rn(c.x, me.x), dy = __fsub_rn(c.y, me.y), dz = __fsub_rn(c.z, me.z);
            float dist_sqr = __fadd_rn(
                __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)), a.eps2);
            dist_sqr = fmaxf(dist_sqr, 1e-6f);
            const bool accept = active && dist_sqr >= b.x;
            if (accept && (my_code == ASTRO_INVALID_MORTON_CODE || my_code != sm.key[at])) {
                const float dist = fmaxf(__fsqrt_rn(dist_sqr), 1e-6f);
                const float den = __fmul_rn(dist_sqr, dist);
                fx = __fadd_rn(fx, __fdiv_rn(__fmul_rn(c.w, dx), den));
                fy = __fadd_rn(fy, __fdiv_rn(__fmul_rn(c.w, dy), den));
                fz = __fadd_rn(fz, __fdiv_rn(__fmul_rn(c.w, dz), den));
                ++inter;
            }
            visits += active ? 1u : 0u;
            if (active) i = next[accept ? __float_as_uint(b.y) : at + 1u];
        }
        if (valid) {
            const float cl = a.clampv;
            a.acc[gid] = make_float4(fminf(fmaxf(fx, -cl), cl), fminf(fmaxf(fy, -cl), cl),
                                     fminf(fmaxf(fz, -cl), cl), 0.f);
        }
    }
    const uint32_t wi = __reduce_add_sync(kFullMask, inter), wv = __reduce_add_sync(kFullMask, visits);
    if (lane == 0) {
        atomicAdd(&s_stats[0], (unsigned long long)wi);
        atomicAdd(&s_stats[1], (unsigned long long)wv);
    }
    __syncthreads();
    if (tid == 0) {
        atomicAdd(&a.stats[0], s_stats[0]);
        atomicAdd(&a.stats[1], s_stats[1]);
        atomicAdd(&a.stats[2], s_stats[0]);
    }
}

template <bool kExact, bool kPrec, bool kBatched, bool kPersistent, int kWarps>
__global__ __launch_bounds__(kWarps * 32) void traverse_phys_kernel(TraverseArgs a) {
    __shared__ uint4 s_stack[kWarps][kPhysStack];
    __shared__ float4 s_tile[kWarps][32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt = lanemask_lt();
    const uint32_t nchunks = (a.n + 31u) / 32u;
    const float g = a.g, eps2 = a.eps2;
    uint32_t inter = 0, visits = 0, cell_inter = 0;
    uint32_t chunk = blockIdx.x * kWarps + warp;
    while (true) {
        if (kPersistent) {
            uint32_t c = 0;
            if (lane == 0) c = atomicAdd(a.queue, 1u);
            chunk = __shfl_sync(kFullMask, c, 0);
        }
        if (chunk >= nchunks) break;
        const uint32_t ip = chunk * 32u + lane;
        const bool valid = ip < a.n;
        const float4 me = valid ? a.pos[ip] : make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t sys = 0;
        if (kBatched) sys = valid ? (uint32_t)(a.sorted_keys[ip] >> (3u * a.lbits)) : 0u;
        const float* crit2 = a.sys[sys].crit2;
        const uint32_t valid_mask = __ballot_sync(kFullMask, valid);

        // The current range lives in registers (the same in every lane); the
        // ranges below it wait in the warp's shared-memory stack.
        uint32_t sp = 0;
        uint4 cur;
        if (kBatched) {
            // One root range per system present in the warp.
            uint32_t rem = valid_mask;
            bool first = true;
            while (rem) {
                const uint32_t leader = __ffs(rem) - 1;
                const uint32_t s = __shfl_sync(kFullMask, sys, leader);
                const uint32_t grp = __ballot_sync(kFullMask, valid && sys == s);
                const uint32_t root = a.sys[s].root;
                const uint4 e = make_uint4(root, root + 1, a.lbits, grp);
                if (first) {
                    cur = e;
                    first = false;
                } else {
                    if (lane == 0) s_stack[warp][sp] = e;
                    ++sp;
                }
                rem &= ~grp;
            }
        } else {
            cur = make_uint4(a.root, a.root + 1, a.lbits, valid_mask);
        }
        __syncwarp();

        Accum<kExact, kPrec> acc;
        bool more = valid_mask != 0;
        while (more) {
            const uint32_t nd = cur.y - 1;
            cur.y = nd;
            const bool exhausted = cur.y == cur.x;
            const uint32_t layer = cur.z;
            const bool active = (cur.w >> lane) & 1u;
            const float4 c = __ldg(&a.node_cm[nd]);
            const float dx = __fsub_rn(c.x, me.x), dy = __fsub_rn(c.y, me.y),
                        dz = __fsub_rn(c.z, me.z);
            const float r2t =
                __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
            const float crit = a.delta ? __ldg(&a.node_crit2[nd]) : __ldg(&crit2[layer]);
            const bool accept = active && r2t > crit;
            if (accept) {
                float tx, ty, tz;
                float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                float qyz = 0.f;
                if (a.quad) {
                    q = __ldg(&a.node_q[nd]);
                    qyz = __ldg(&a.node_qyz[nd]);
                }
                cell_term<kExact>(dx, dy, dz, r2t, c.w, a.quad != 0, q, qyz, g, eps2, tx, ty, tz);
                acc.add(tx, ty, tz);
                ++inter;
                ++cell_inter;
            }
            visits += active ? 1u : 0u;
            const uint32_t open_mask = __ballot_sync(kFullMask, active && !accept);
            if (open_mask != 0) {
                const uint4 r = __ldg(&a.node_rng[nd]);
                if (layer != 0 && r.w - r.z > a.bucket) {
                    // Open: descend into the children, keep the rest of this range.
                    if (!exhausted) {
                        if (sp < (uint32_t)kPhysStack) {
                            if (lane == 0) s_stack[warp][sp] = cur;
                            ++sp;
                        } else if (lane == 0) {
                            atomicOr(a.err, kErrStackOverflow);
                        }
                    }
                    cur = make_uint4(r.x, r.y, layer - 1, open_mask);
                    continue;
                }
                // Leaf or bucket: particle-particle sums over 32-particle tiles.
                const bool open = (open_mask >> lane) & 1u;
                for (uint32_t t = r.z; t < r.w; t += 32u) {
                    const uint32_t j = t + lane;
                    if (j < r.w) s_tile[warp][lane] = __ldg(&a.pos[j]);
                    __syncwarp();
                    const uint32_t cnt = min(32u, r.w - t);
                    if (open) {
                        for (uint32_t q = 0; q < cnt; ++q) {
                            const float4 p = s_tile[warp][q];
                            if (t + q != ip) {
                                float tx, ty, tz;
                                particle_term<kExact>(__fsub_rn(p.x, me.x), __fsub_rn(p.y, me.y),
                                                      __fsub_rn(p.z, me.z), p.w, g, eps2, tx, ty, tz);
                                acc.add(tx, ty, tz);
                            }
                        }
                        inter += cnt - ((ip - t) < cnt ? 1u : 0u);
                    }
                    __syncwarp();
                }
            }
            if (exhausted) {
                if (sp == 0) {
                    more = false;
                } else {
                    __syncwarp();
                    cur = s_stack[warp][--sp];
                }
            }
        }

        if (valid) {
            const float cl = a.clampv, dt = a.dt;
            const float ax = fminf(fmaxf(acc.ax, -cl), cl);
            const float ay = fminf(fmaxf(acc.ay, -cl), cl);
            const float az = fminf(fmaxf(acc.az, -cl), cl);
            a.acc[ip] = make_float4(ax, ay, az, 0.f);
            // Kick-drift: updateSpheres' v += a dt, x += v dt (no damping).
            float4 v = a.vel_in[ip];
            v.x = __fadd_rn(v.x, __fmul_rn(ax, dt));
            v.y = __fadd_rn(v.y, __fmul_rn(ay, dt));
            v.z = __fadd_rn(v.z, __fmul_rn(az, dt));
            a.vel_out[ip] = v;
            a.id_out[ip] = a.id_in[ip];
            if (kPrec) {
                const size_t n = a.n;
                const double ddt = (double)dt;
                a.x64_out[ip] = __dadd_rn(a.x64_in[ip], __dmul_rn((double)v.x, ddt));
                a.x64_out[n + ip] = __dadd_rn(a.x64_in[n + ip], __dmul_rn((double)v.y, ddt));
                a.x64_out[2 * n + ip] = __dadd_rn(a.x64_in[2 * n + ip], __dmul_rn((double)v.z, ddt));
                a.pos_out[ip] = me;
            } else {
                a.pos_out[ip] = make_float4(__fadd_rn(me.x, __fmul_rn(v.x, dt)),
                                            __fadd_rn(me.y, __fmul_rn(v.y, dt)),
                                            __fadd_rn(me.z, __fmul_rn(v.z, dt)), me.w);
            }
        }
        if (!kPersistent) break;
    }
    // Statistics: one atomic per warp.
    unsigned long long i64 = inter, v64 = visits, c64 = cell_inter;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        i64 += __shfl_xor_sync(kFullMask, i64, o);
        v64 += __shfl_xor_sync(kFullMask, v64, o);
        c64 += __shfl_xor_sync(kFullMask, c64, o);
    }
    if (lane == 0) {
        atomicAdd(&a.stats[0], i64);
        atomicAdd(&a.stats[1], v64);
        atomicAdd(&a.stats[2], c64);
    }
    (void)lt;
}


namespace {

int sm_count() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 1;
    }
    return n;
}

template <bool kExact, bool kPrec, bool kBatched, bool kPersistent, int kWarps>
cudaError_t launch_phys_t(const TraverseArgs& a, cudaStream_t st) {
    auto kernel = traverse_phys_kernel<kExact, kPrec, kBatched, kPersistent, kWarps>;
    const uint32_t chunks = (a.n + 31u) / 32u;
    uint32_t blocks;
    if (kPersistent) {
        int per_sm = 0;
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kWarps * 32, 0);
        if (e != cudaSuccess) return e;
        blocks = (uint32_t)std::max(1, per_sm) * (uint32_t)sm_count();
        blocks = std::min<uint32_t>(blocks, (chunks + kWarps - 1) / kWarps);
        cudaMemsetAsync(a.queue, 0, sizeof(uint32_t), st);
    } else {
        blocks = (chunks + kWarps - 1) / kWarps;
    }
    if (blocks == 0) return cudaSuccess;
    kernel<<<blocks, kWarps * 32, 0, st>>>(a);
    return cudaGetLastError();
}

template <bool kExact, bool kPrec, bool kBatched, bool kPersistent>
cudaError_t launch_phys_w(const TraverseArgs& a, int warps, cudaStream_t st) {
    switch (warps) {
        case 2: return launch_phys_t<kExact, kPrec, kBatched, kPersistent, 2>(a, st);
        case 8: return launch_phys_t<kExact, kPrec, kBatched, kPersistent, 8>(a, st);
        default: return launch_phys_t<kExact, kPrec, kBatched, kPersistent, 4>(a, st);
    }
}

template <bool kExact, bool kPrec, bool kBatched>
cudaError_t launch_phys_p(const TraverseArgs& a, const TraverseConfig& c, cudaStream_t st) {
    return c.persistent ? launch_phys_w<kExact, kPrec, kBatched, true>(a, c.warps, st)
                        : launch_phys_w<kExact, kPrec, kBatched, false>(a, c.warps, st);
}

template <bool kExact, bool kPrec>
cudaError_t launch_phys_b(const TraverseArgs& a, const TraverseConfig& c, cudaStream_t st) {
    return c.batched ? launch_phys_p<kExact, kPrec, true>(a, c, st)
                     : launch_phys_p<kExact, kPrec, false>(a, c, st);
}

}  // namespace

// Kernel attributes of the reference walk, set once per device; called before
// any stream capture.
cudaError_t traverse_init() {
    return cudaFuncSetAttribute(traverse_ref_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)ref_smem(kRefNodes));
}

cudaError_t launch_traverse_ref(const TraverseArgs& a, const RefTree& t, cudaStream_t st) {
    if (a.n == 0) return cudaSuccess;
    if (t.capacity > kRefNodes) {
        traverse_ref_kernel<<<(a.n + 127) / 128, 128, 0, st>>>(a);
        return cudaGetLastError();
    }
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, traverse_ref_small_kernel, kRefThreads,
                                                          ref_smem(t.capacity));
    if (e != cudaSuccess) return e;
    const uint32_t blocks = std::min<uint32_t>((a.n + kRefThreads - 1) / kRefThreads,
                                               (uint32_t)(std::max(1, per_sm) * std::max(1, sms)));
    traverse_ref_small_kernel<<<blocks, kRefThreads, ref_smem(t.capacity), st>>>(a, t);
    return cudaGetLastError();
}

cudaError_t launch_traverse_phys(const TraverseArgs& a, const TraverseConfig& c, cudaStream_t st) {
    if (a.n == 0) return cudaSuccess;
    if (c.exact)
        return c.precision ? launch_phys_b<true, true>(a, c, st) : launch_phys_b<true, false>(a, c, st);
    return c.precision ? launch_phys_b<false, true>(a, c, st) : launch_phys_b<false, false>(a, c, st);
}

}  // namespace astro
