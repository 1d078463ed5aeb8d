// Evaluation of the group walk's interaction lists (PHYSICAL preset): the
// forces of every group's particles and the fused kick-drift.
//
// One warp per group, groups taken from a queue in the walk's order. Each
// particle evaluates the walk's far-node expansion at its offset from the
// box centre; listed cells are gathered into shared memory and summed; the
// listed leaves' particles are staged in tiles and summed. The epilogue
// clamps, stores the acceleration and performs the kick-drift (v += a dt,
// x += v dt).
//
// group_eval_fast_kernel — the fast form: a lane holds up to eight of the
//   group's particles as packed FP32 pairs, and the warp's lanes split each
//   list into four or eight parts.
// group_eval_general_kernel — the exact form (every operation rounded as the
//   CPU restatement rounds it, in its order), and the fast form where eps^2
//   is no normal float (a particle's own entry is skipped).
#include <algorithm>
#include <mutex>

#include "build_kernels.cuh"
#include "common.cuh"
#include "group_lists.cuh"
#include "traverse_terms.cuh"

namespace astro {
namespace {

// The packed loops need no self test and may sum massless particles as padding:
// a source at distance zero adds its factor m / eps^3 times a zero offset, and
// eps^2 >= 2^-80 keeps 1 / eps^3 at most 2^120 (the factor is finite for masses
// below 2^128 eps^3, 256 at the bound). Every r^2 is then a normal float, so
// rsqrt_ftz applies. Below the bound, down to the smallest normal eps^2, the loops
// multiply the offset by 1/r three times and the mass last (kTiny), which stays
// finite: three more products a pair, a step of a 50,000-body disk at eps 5e-13 in
// groups of 32 483 us against 1,416 in the general kernel. A quadrupole's factor
// 1 / r^5 is finite from 2e-8 only, so cells are padded with a massless one where a
// listed cell lies, not at the origin.
constexpr float kPackedMinEps2 = 8.2718061e-25f;  // 2^-80

// Clamp, acceleration and kick-drift of particle i (updateSpheres' v += a dt,
// x += v dt without damping).
template <bool kPrec>
__device__ __forceinline__ void store_particle(const TraverseArgs& a, uint32_t i, float4 me, float sx,
                                               float sy, float sz) {
    const float cl = a.clampv, dt = a.dt;
    const float ax = fminf(fmaxf(sx, -cl), cl);
    const float ay = fminf(fmaxf(sy, -cl), cl);
    const float az = fminf(fmaxf(sz, -cl), cl);
    a.acc[i] = make_float4(ax, ay, az, 0.f);
    float4 v = a.vel_in[i];
    v.x = __fadd_rn(v.x, __fmul_rn(ax, dt));
    v.y = __fadd_rn(v.y, __fmul_rn(ay, dt));
    v.z = __fadd_rn(v.z, __fmul_rn(az, dt));
    a.vel_out[i] = v;
    a.id_out[i] = a.id_in[i];
    if (kPrec) {
        const size_t n = a.n;
        const double ddt = (double)dt;
        a.x64_out[i] = __dadd_rn(a.x64_in[i], __dmul_rn((double)v.x, ddt));
        a.x64_out[n + i] = __dadd_rn(a.x64_in[n + i], __dmul_rn((double)v.y, ddt));
        a.x64_out[2 * n + i] = __dadd_rn(a.x64_in[2 * n + i], __dmul_rn((double)v.z, ddt));
        a.pos_out[i] = me;
    } else {
        a.pos_out[i] = make_float4(__fadd_rn(me.x, __fmul_rn(v.x, dt)),
                                   __fadd_rn(me.y, __fmul_rn(v.y, dt)),
                                   __fadd_rn(me.z, __fmul_rn(v.z, dt)), me.w);
    }
}

// The walk's summed far-node coefficients (group_far_kernel).
template <bool kExact>
__device__ __forceinline__ void load_far(const float* far_co, float eps2, float (&fc)[kFarCoefs]) {
    float buf[kFarCoefs + 1];
#pragma unroll
    for (int k = 0; k < (kFarCoefs + 1) / 4; ++k) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(far_co) + k);
        buf[4 * k] = v.x, buf[4 * k + 1] = v.y, buf[4 * k + 2] = v.z, buf[4 * k + 3] = v.w;
    }
#pragma unroll
    for (int k = 0; k < kFarCoefs; ++k) fc[k] = buf[k];
    if constexpr (!kExact) far_finish(eps2, fc);
}

// One warp adds its counts (the same in every lane) to the statistics.
__device__ __forceinline__ void add_stats(const TraverseArgs& a, uint32_t lane,
                                          unsigned long long inter, unsigned long long cells,
                                          unsigned long long fars) {
    if (lane != 0) return;
    if (inter) atomicAdd(&a.stats[0], inter);
    if (cells) atomicAdd(&a.stats[2], cells);
    if (fars) atomicAdd(&a.stats[4], fars);
}

// ------------------------------------------------------------ fast form --
//
// What bounds it: the FMA pipe and the register file's read ports. A packed
// instruction takes one cycle per distinct 64-bit operand on this chip
// (measured, 4 warps per scheduler: FADD2 and FMUL2 2.0 cycles, FFMA2 2.0 with
// a repeated operand and 3.0 with three distinct ones; a scalar FFMA of three
// distinct registers 1.66), so a source against one pair of particles takes
// 29.4 cycles in the best of six mixes of packed and scalar forms tried in a
// loop of its own. What can be saved is idle lanes and everything around that loop:
// - Pairs are of two particles, not of two sources: a lane holds up to eight
//   particles and the warp's lanes split each list into 32 / width parts, so
//   a group of 5 <= g <= 32 costs ceil(g / 8) / 8 of a pass over the lists per lane
//   and one of g <= 64 ceil(g / 16) / 4 (one particle a lane: 1 for every g
//   from 17 to 32). Sums, positions and the source take half the registers
//   that source pairs took, and four independent pairs hide the latencies.
// - The tile's particles come by cp.async, one tile ahead, and a position's
//   range is found with one reduction and one ballot for 32 positions instead
//   of a five-step shuffle search.
// - The loops for 1 to 4 pairs share one staging code and are not unrolled
//   for 3 and 4: with the whole list code instantiated four times the
//   instruction cache missed (3.6 stall cycles per issue, disk 750 us).
// Evaluation with far sums, before and after: 100,003-body disk (no far
// nodes, groups of 32) 905 -> 645 us, 524,288-body disk 667 -> 635 us, two
// Plummer spheres of 4,194,304 in the precision form 3.12 -> 2.95 ms, 256
// systems 4.25 -> 4.07 ms, 16,777,216-body cube 14.80 -> 14.44 ms, 16,384-body
// sphere (groups of 8) 78 -> 59 us.

constexpr int kFastWarps = 4;                        // warps per block
constexpr int kTile = 128;                           // leaf particles per staged tile
constexpr int kCellWords = 20;                       // staged cell: 16 words, padded to 80 bytes
constexpr int kMaxPairs = 4;                         // particle pairs per lane

// Per warp: the staged cells of one list block or two leaf tiles, and each
// lane's running sums (the tiles' partial sums are added to them; in the
// precision form a Kahan correction beside each).
template <bool kPrec>
struct __align__(16) FastSmem {
    union {
        float cell[kListBlockWords * kCellWords];
        float4 tile[2][kTile];
    } u;
    float2 sum[kPrec ? 2 : 1][3][kMaxPairs][32];
};

__device__ __forceinline__ void copy_async16(void* dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(valid ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kLeft>
__device__ __forceinline__ void copy_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(kLeft) : "memory");
}

// Negated positions of a lane's particle pairs, and their sums of one tile.
struct PairSet {
    float2 nx[kMaxPairs], ny[kMaxPairs], nz[kMaxPairs];
    float2 sx[kMaxPairs], sy[kMaxPairs], sz[kMaxPairs];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int q = 0; q < kMaxPairs; ++q) sx[q] = sy[q] = sz[q] = make_float2(0.f, 0.f);
    }
};

// One source against the first kPairs pairs: m d / (r^2 + eps^2)^(3/2) without G.
template <int kPairs, bool kTiny>
__device__ __forceinline__ void add_source(PairSet& t, float4 p, float2 e2) {
#pragma unroll
    for (int q = 0; q < kPairs; ++q) {
        const float2 dx = make_float2(p.x + t.nx[q].x, p.x + t.nx[q].y);
        const float2 dy = make_float2(p.y + t.ny[q].x, p.y + t.ny[q].y);
        const float2 dz = make_float2(p.z + t.nz[q].x, p.z + t.nz[q].y);
        const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, e2)));
        const float2 inv = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
        if constexpr (kTiny) {
            const float2 u = __fmul2_rn(inv, inv), m = make_float2(p.w, p.w);
            t.sx[q] = __ffma2_rn(__fmul2_rn(__fmul2_rn(dx, inv), u), m, t.sx[q]);
            t.sy[q] = __ffma2_rn(__fmul2_rn(__fmul2_rn(dy, inv), u), m, t.sy[q]);
            t.sz[q] = __ffma2_rn(__fmul2_rn(__fmul2_rn(dz, inv), u), m, t.sz[q]);
        } else {
            const float2 inv3 = __fmul2_rn(__fmul2_rn(inv, inv), inv);
            const float2 sc = make_float2(p.w * inv3.x, p.w * inv3.y);
            t.sx[q] = __ffma2_rn(dx, sc, t.sx[q]);
            t.sy[q] = __ffma2_rn(dy, sc, t.sy[q]);
            t.sz[q] = __ffma2_rn(dz, sc, t.sz[q]);
        }
    }
}

// One cell with its quadrupole against the first kPairs pairs. Staged words: x, y, z, m,
// then -Qxx, -Qyy, -Qxy, -Qxz, -Qyz, -Qzz, each twice. The term is
// inv^3 (M + 5/2 u^2 d.Qd) d - inv^5 Qd with u = 1/r^2; with Q negated,
// qx.. = -(Qd) and dqd = -d.Qd.
template <int kPairs>
__device__ __forceinline__ void add_cell_quad(PairSet& t, const float* s, float2 e2) {
    const float4 c = *reinterpret_cast<const float4*>(s);
    const float4 qa = *reinterpret_cast<const float4*>(s + 4);
    const float4 qb = *reinterpret_cast<const float4*>(s + 8);
    const float4 qc = *reinterpret_cast<const float4*>(s + 12);
    const float2 nxx = make_float2(qa.x, qa.y), nyy = make_float2(qa.z, qa.w);
    const float2 nxy = make_float2(qb.x, qb.y), nxz = make_float2(qb.z, qb.w);
    const float2 nyz = make_float2(qc.x, qc.y), nzz = make_float2(qc.z, qc.w);
#pragma unroll
    for (int q = 0; q < kPairs; ++q) {
        const float2 dx = make_float2(c.x + t.nx[q].x, c.x + t.nx[q].y);
        const float2 dy = make_float2(c.y + t.ny[q].x, c.y + t.ny[q].y);
        const float2 dz = make_float2(c.z + t.nz[q].x, c.z + t.nz[q].y);
        const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, e2)));
        const float2 inv = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
        const float2 u = __fmul2_rn(inv, inv), inv3 = __fmul2_rn(u, inv);
        const float2 qx = __ffma2_rn(nxx, dx, __ffma2_rn(nxy, dy, __fmul2_rn(nxz, dz)));
        const float2 qy = __ffma2_rn(nxy, dx, __ffma2_rn(nyy, dy, __fmul2_rn(nyz, dz)));
        const float2 qz = __ffma2_rn(nxz, dx, __ffma2_rn(nyz, dy, __fmul2_rn(nzz, dz)));
        const float2 dqd = __ffma2_rn(dx, qx, __ffma2_rn(dy, qy, __fmul2_rn(dz, qz)));
        const float2 uu = __fmul2_rn(make_float2(-2.5f * u.x, -2.5f * u.y), u);
        const float2 sa =
            __fmul2_rn(inv3, make_float2(fmaf(uu.x, dqd.x, c.w), fmaf(uu.y, dqd.y, c.w)));
        const float2 sb = __fmul2_rn(inv3, u);
        t.sx[q] = __ffma2_rn(sb, qx, __ffma2_rn(sa, dx, t.sx[q]));
        t.sy[q] = __ffma2_rn(sb, qy, __ffma2_rn(sa, dy, t.sy[q]));
        t.sz[q] = __ffma2_rn(sb, qz, __ffma2_rn(sa, dz, t.sz[q]));
    }
}

// Adds a tile's sums to the lane's running sums and clears them.
template <bool kPrec>
__device__ __forceinline__ void flush(FastSmem<kPrec>& sm, PairSet& t, uint32_t lane, uint32_t pairs) {
#pragma unroll
    for (int q = 0; q < kMaxPairs; ++q) {
        if (q >= (int)pairs) break;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float2 v = c == 0 ? t.sx[q] : (c == 1 ? t.sy[q] : t.sz[q]);
            float2 s = sm.sum[0][c][q][lane];
            if constexpr (kPrec) {
                float2 k = sm.sum[kPrec ? 1 : 0][c][q][lane];
                const float2 y = make_float2(v.x - k.x, v.y - k.y);
                const float2 n = make_float2(s.x + y.x, s.y + y.y);
                k = make_float2((n.x - s.x) - y.x, (n.y - s.y) - y.y);
                s = n;
                sm.sum[kPrec ? 1 : 0][c][q][lane] = k;
            } else {
                s = __fadd2_rn(s, v);
            }
            sm.sum[0][c][q][lane] = s;
        }
    }
    t.clear();
}

// The staged cells (count padded to the copies) or particles of one copy.
template <bool kQuad, bool kTiny, int kPairs>
__device__ __forceinline__ void sum_cells(PairSet& t, const float* cell, uint32_t copies,
                                          uint32_t iters, float2 e2) {
    constexpr int kUnroll = kPairs == 1 ? 2 : 1;
#pragma unroll kUnroll
    for (uint32_t i = 0; i < iters; ++i) {
        if constexpr (kQuad) add_cell_quad<kPairs>(t, cell, e2);
        else add_source<kPairs, kTiny>(t, *reinterpret_cast<const float4*>(cell), e2);
        cell += copies * (kQuad ? kCellWords : 4);
    }
}
template <bool kTiny, int kPairs>
__device__ __forceinline__ void sum_tile(PairSet& t, const float4* src, uint32_t copies,
                                         uint32_t iters, float2 e2) {
    constexpr int kUnroll = kPairs == 1 ? 4 : (kPairs == 2 ? 2 : 1);
#pragma unroll kUnroll
    for (uint32_t i = 0; i < iters; ++i) {
        add_source<kPairs, kTiny>(t, *src, e2);
        src += copies;
    }
}

// The lists of one group: lane = copy * width + slot holds the particles
// slot + width * k, k = 0 .. 2 pairs - 1, and its copy takes every
// copies-th source (width 8: four copies; 4: eight; 2 and 1: 16 and 32). Returns
// the particles listed. width = 2^wbits, so that nothing is divided by it: divisions
// by a width of four values made the kernel 52 KB instead of 42 (precision form with
// quadrupoles), and its instruction cache misses cost 256 systems 190 us of 7,640,
// 300 of 3,000 bodies 71 of 920 and 60,000 of 16 bodies 9 of 435 a step.
template <bool kPrec, bool kQuad, bool kTiny>
__device__ __forceinline__ uint32_t sum_lists(const TraverseArgs& a, uint2 gr, const GroupDesc& d,
                                              FastSmem<kPrec>& sm, uint32_t lane, uint32_t wbits,
                                              uint32_t pairs) {
    const uint32_t gcount = gr.y - gr.x;
    const uint32_t width = 1u << wbits, copies = 32u >> wbits;
    const uint32_t copy = lane >> wbits, slot = lane & (width - 1u);
    const float2 e2 = make_float2(a.eps2, a.eps2);
    PairSet t;
#pragma unroll
    for (int q = 0; q < kMaxPairs; ++q) {
        const uint32_t t0 = slot + width * (2 * q), t1 = t0 + width;
        const float4 p0 = t0 < gcount ? __ldg(&a.pos[gr.x + t0]) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 p1 = t1 < gcount ? __ldg(&a.pos[gr.x + t1]) : make_float4(0.f, 0.f, 0.f, 0.f);
        t.nx[q] = make_float2(-p0.x, -p1.x);
        t.ny[q] = make_float2(-p0.y, -p1.y);
        t.nz[q] = make_float2(-p0.z, -p1.z);
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int k = 0; k < (kPrec ? 2 : 1); ++k) sm.sum[k][c][q][lane] = make_float2(0.f, 0.f);
    }
    t.clear();

    // Cells, one list block (64) at a time: gathered into shared memory, massless at
    // the first one's place past the list's end (loaded from there: with the place
    // passed on after the loads, groups of 1 and 4 of 50,000 bodies took 649 and 316 us
    // a step instead of 630 and 310). The next block's ids are loaded before the
    // current block is summed.
    if (d.n_cell > 0) {
        uint32_t blk = d.cell_first, left = d.n_cell;
        uint32_t id0, id1;
        auto load_ids = [&]() {
            const uint32_t* w = a.lists + (size_t)blk * kListBlockWords;
            id0 = lane < left ? __ldg(w + lane) : 0u;
            id1 = lane + 32u < left ? __ldg(w + lane + 32u) : 0u;
        };
        load_ids();
        while (true) {
            const uint32_t m = min(kListBlockWords, left);
            const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
            float4 cm[2], qd[2] = {zero, zero};
            float qyz[2] = {0.f, 0.f};
            const uint32_t first = __shfl_sync(kFullMask, id0, 0);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const bool listed = lane + 32u * h < m;
                const uint32_t nd = listed ? (h == 0 ? id0 : id1) : first;
                cm[h] = __ldg(&a.node_cm[nd]);
                if (!listed) {
                    cm[h].w = 0.f;
                } else if constexpr (kQuad) {
                    qd[h] = __ldg(&a.node_q[nd]);
                    qyz[h] = __ldg(&a.node_qyz[nd]);
                }
            }
            __syncwarp();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t j = lane + 32u * h;
                if constexpr (kQuad) {
                    float4* r = reinterpret_cast<float4*>(sm.u.cell + j * kCellWords);
                    const float zz = qd[h].x + qd[h].y;
                    r[0] = cm[h];
                    r[1] = make_float4(-qd[h].x, -qd[h].x, -qd[h].y, -qd[h].y);
                    r[2] = make_float4(-qd[h].z, -qd[h].z, -qd[h].w, -qd[h].w);
                    r[3] = make_float4(-qyz[h], -qyz[h], zz, zz);
                } else {
                    reinterpret_cast<float4*>(sm.u.cell)[j] = cm[h];
                }
            }
            __syncwarp();
            left -= m;
            if (left > 0) {
                blk = __ldg(&a.list_next[blk]);
                load_ids();
            }
            const uint32_t iters = (m + copies - 1u) >> (5u - wbits);
            const float* cell = sm.u.cell + copy * (kQuad ? kCellWords : 4);
            if (pairs == 4u) sum_cells<kQuad, kTiny, 4>(t, cell, copies, iters, e2);
            else if (pairs == 3u) sum_cells<kQuad, kTiny, 3>(t, cell, copies, iters, e2);
            else if (pairs == 2u) sum_cells<kQuad, kTiny, 2>(t, cell, copies, iters, e2);
            else sum_cells<kQuad, kTiny, 1>(t, cell, copies, iters, e2);
            flush(sm, t, lane, pairs);
            if (left == 0) break;
        }
        __syncwarp();
    }

    // Leaf particles: the ranges of one list block (32) are concatenated and
    // staged kTile particles at a time; the next tile's copies run while the
    // current tile is summed. A range's lane finds its first position by a
    // prefix sum; in each window of 32 positions the ranges starting there
    // set a bit, and a position's range is the count of starts up to it.
    uint32_t sources = 0, left = d.n_leaf;
    if (left == 0) return 0u;
    auto load_ranges = [&](uint32_t b, uint32_t rem) {
        const uint2* w = reinterpret_cast<const uint2*>(a.lists + (size_t)b * kListBlockWords);
        return lane < rem ? __ldg(w + lane) : make_uint2(0u, 0u);
    };
    uint2 next_rg = load_ranges(d.leaf_first, left);
    uint32_t next_blk = left > 32u ? __ldg(&a.list_next[d.leaf_first]) : 0u;
    uint32_t pre = 0, base = 0, total = 0, pos0 = 0;
    bool range = false;
    const uint32_t le = lanemask_lt() | (1u << lane);
    uint32_t cnt = 0;  // particles of the tile staged last
    for (int b = 0;; b ^= 1) {
        // Stage the next tile into buffer b.
        const uint32_t cur = cnt;
        if (pos0 >= total && left > 0) {
            const uint32_t rlen = next_rg.y - next_rg.x;
            range = rlen > 0u;
            uint32_t incl = rlen;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
                if (lane >= (uint32_t)o) incl += y;
            }
            pre = incl - rlen;
            base = next_rg.x - pre;
            total = __shfl_sync(kFullMask, incl, 31);
            pos0 = 0;
            sources += total;
            left -= min(32u, left);
            if (left > 0) {
                next_rg = load_ranges(next_blk, left);
                if (left > 32u) next_blk = __ldg(&a.list_next[next_blk]);
            }
        }
        cnt = min((uint32_t)kTile, total - pos0);
#pragma unroll 1
        for (uint32_t w0 = pos0; w0 < pos0 + cnt; w0 += 32u) {
            const uint32_t off = pre - w0;  // wraps for ranges that started before
            const uint32_t starts = __reduce_or_sync(kFullMask, range && off < 32u ? 1u << off : 0u);
            const uint32_t before = __popc(__ballot_sync(kFullMask, range && pre < w0));
            const uint32_t e = before + __popc(starts & le) - 1u;
            const uint32_t idx = __shfl_sync(kFullMask, base, e & 31u) + w0 + lane;
            const bool valid = w0 + lane < total;
            copy_async16(&sm.u.tile[b][w0 - pos0 + lane], a.pos + (valid ? idx : gr.x), valid);
        }
        pos0 += cnt;
        copy_commit();
        if (cur > 0) {
            copy_wait<1>();
            __syncwarp();
            const uint32_t iters = (cur + copies - 1u) >> (5u - wbits);
            const float4* src = sm.u.tile[b ^ 1] + copy;
            if (pairs == 4u) sum_tile<kTiny, 4>(t, src, copies, iters, e2);
            else if (pairs == 3u) sum_tile<kTiny, 3>(t, src, copies, iters, e2);
            else if (pairs == 2u) sum_tile<kTiny, 2>(t, src, copies, iters, e2);
            else sum_tile<kTiny, 1>(t, src, copies, iters, e2);
            flush(sm, t, lane, pairs);
            __syncwarp();
        }
        if (cnt == 0) break;
    }
    copy_wait<0>();
    return sources;
}

// Resident blocks per SM the register allocation is sized for: four (128
// registers, 8 bytes spilled). Walk's lists of a 524,288-body disk, evaluation
// and far sums together: 635 us, against 655 at three blocks (168 registers)
// and 637 at five (96); 16,777,216-body cube 14.44, 15.64 and 14.64 ms.
constexpr int kFastBlocks = 4;

template <bool kPrec, bool kQuad, bool kTiny>
__global__ __launch_bounds__(kFastWarps * 32, kFastBlocks) void group_eval_fast_kernel(
    TraverseArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    FastSmem<kPrec>& sm = reinterpret_cast<FastSmem<kPrec>*>(smem_raw)[warp];
    // A walk that ran out of frontier or list room left incomplete lists:
    // nothing is evaluated or integrated (the state stays as it was) and
    // the host runs the traversal again with larger buffers.
    if (*reinterpret_cast<volatile const uint32_t*>(a.err) & kErrFrontier) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(a.evals_done, 1u);
    const uint32_t ngroups = *a.group_count;
    unsigned long long inter = 0, cell_inter = 0, far_inter = 0;
    while (true) {
        uint32_t gi = 0;
        if (lane == 0) gi = atomicAdd(a.eval_queue, 1u);
        gi = __shfl_sync(kFullMask, gi, 0);
        if (gi >= ngroups) break;
        gi = group_of_ticket(gi, ngroups, a.group_chunk);
        const uint4 rec = a.groups[gi];
        const uint2 gr = make_uint2(rec.x, rec.y);
        const uint32_t gcount = gr.y - gr.x;
        // The walk of the leaf's first chunk.
        const GroupDesc* dp = a.desc + (gi - rec.w);
        const GroupDesc d = load_desc(dp);
        // Groups of one to four fill fewer slots, so more lanes split the lists
        // (a step of a 50,000-body sphere in groups of 1 / 2 / 4: four slots 876 / 557 /
        // 373 us, 630 / 420 / 310 so; one lane a particle and copy 821 / 600 / 474).
        const uint32_t wbits = gcount > 32u ? 3u : (gcount > 4u ? 2u : (gcount > 2u ? 1u : 0u));
        const uint32_t width = 1u << wbits, pairs = (gcount + 2u * width - 1u) >> (wbits + 1u);
        const uint32_t sources = sum_lists<kPrec, kQuad, kTiny>(a, gr, d, sm, lane, wbits, pairs);
        __syncwarp();
        // Each lane finishes up to two particles: the copies' sums, the
        // far-node expansion, G, and the kick-drift. A particle's own entry
        // in the leaf lists added exactly zero and is not counted.
        const uint64_t per = (uint64_t)d.n_far + d.n_cell + sources - 1u;
        inter += gcount * per;
        cell_inter += (uint64_t)gcount * (d.n_far + d.n_cell);
        far_inter += (uint64_t)gcount * d.n_far;
        float fc[kFarCoefs];
        if (d.n_far > 0) load_far<false>(dp->far_co, a.eps2, fc);
        for (uint32_t t = lane; t < gcount; t += 32u) {
            const uint32_t k = t >> wbits, q = k >> 1, slot = t & (width - 1u);
            float s[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float* p = reinterpret_cast<const float*>(&sm.sum[0][c][q][slot]) + (k & 1u);
                const float* pk = kPrec ? reinterpret_cast<const float*>(&sm.sum[kPrec ? 1 : 0][c][q][slot]) + (k & 1u)
                                        : p;
                float v = 0.f;
                for (uint32_t r = 0; r < 64u; r += 2u * width) v += kPrec ? p[r] - pk[r] : p[r];
                s[c] = v;
            }
            const uint32_t i = gr.x + t;
            const float4 me = a.pos[i];
            float fx = 0.f, fy = 0.f, fz = 0.f;
            if (d.n_far > 0) far_eval<false>(fc, me.x - d.gcx, me.y - d.gcy, me.z - d.gcz, fx, fy, fz);
            store_particle<kPrec>(a, i, me, (s[0] + fx) * a.g, (s[1] + fy) * a.g, (s[2] + fz) * a.g);
        }
        __syncwarp();
    }
    add_stats(a, lane, inter, cell_inter, far_inter);
}

// --------------------------------------------------------- general form --

constexpr int kGeneralWarps = 4;
constexpr int kGeneralCells = 2 * (int)kListBlockWords;  // cells staged per warp

// A staged accepted cell: centre of mass and mass, and with quadrupoles
// {Qxx, Qyy, Qxy, Qxz} and {Qyz, Qzz}.
template <bool kQuad>
struct CellSlot {
    float4 cm;
    float4 q;
    float4 q2;
};
template <>
struct CellSlot<false> {
    float4 cm;
};

// Evaluation of one group whose particles sit kPer per lane (kPer = 2:
// particles lane and lane + 32), sources in list order. In the fast form a group of
// at most 16 runs as 32 / gcount copies (lane = rep * gcount + particle), each
// of which takes every reps-th source of a staged part; a part's sum is added (in
// the precision form Kahan-added) once. Without softening, 50,000-body disk in
// groups of 16, lists and far sums: 563 us, one copy 1,223; of 32 555
// (1,178 with every term compensated by itself).
template <bool kExact, bool kPrec, bool kQuad, int kPer>
__device__ __forceinline__ void eval_group(const TraverseArgs& a, const uint2 gr, const GroupDesc& d,
                                           const float* __restrict__ far_co,
                                           CellSlot<kQuad>* s_cell, float4* s_tile, uint32_t* s_jdx,
                                           uint32_t lane, uint32_t& inter, uint32_t& cell_inter,
                                           uint32_t& far_inter) {
    const uint32_t gcount = gr.y - gr.x;
    const float g = a.g, eps2 = a.eps2;
    const uint32_t reps = kExact || kPer == 2 ? 1u : 32u / gcount;
    const uint32_t rep = kPer == 2 ? 0u : lane / gcount;
    uint32_t ip[kPer];
    bool valid[kPer];
    float4 me[kPer];
    uint32_t owned = 0;  // particles whose counts this lane keeps
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const uint32_t slot = kPer == 2 ? lane + 32u * k : lane - rep * gcount;
        valid[k] = kPer == 2 ? slot < gcount : rep < reps;
        ip[k] = gr.x + slot;
        me[k] = valid[k] ? a.pos[ip[k]] : make_float4(0.f, 0.f, 0.f, 0.f);
        owned += valid[k] && rep == 0u ? 1u : 0u;
    }

    float fx[kPer], fy[kPer], fz[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) fx[k] = fy[k] = fz[k] = 0.f;
    if (d.n_far > 0) {
        float fc[kFarCoefs];
        load_far<kExact>(far_co, eps2, fc);
#pragma unroll
        for (int k = 0; k < kPer; ++k)
            far_eval<kExact>(fc, xadd<kExact>(me[k].x, -d.gcx), xadd<kExact>(me[k].y, -d.gcy),
                             xadd<kExact>(me[k].z, -d.gcz), fx[k], fy[k], fz[k]);
        inter += owned * d.n_far;
        cell_inter += owned * d.n_far;
        far_inter += owned * d.n_far;
    }

    // G: in every term of the exact form, once at the end otherwise.
    Accum<kExact, kPrec> cells[kPer], leaves[kPer];
    ChainCursor ccur{d.cell_first};
    for (uint32_t c0 = 0; c0 < d.n_cell; c0 += (uint32_t)kGeneralCells) {
        const uint32_t m = min((uint32_t)kGeneralCells, d.n_cell - c0);
        if (c0 > 0) ccur.advance(a);
        const uint32_t* b0 = ccur.words(a);
        const uint32_t* b1 = b0;
        if (m > kListBlockWords) {
            ccur.advance(a);
            b1 = ccur.words(a);
        }
        __syncwarp();
#pragma unroll 4
        for (uint32_t j = lane; j < m; j += 32u) {
            const uint32_t nd = j < kListBlockWords ? b0[j] : b1[j - kListBlockWords];
            s_cell[j].cm = __ldg(&a.node_cm[nd]);
            if constexpr (kQuad) {
                const float4 q = __ldg(&a.node_q[nd]);
                s_cell[j].q = q;
                s_cell[j].q2 = make_float4(__ldg(&a.node_qyz[nd]), -(q.x + q.y), 0.f, 0.f);
            }
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            if (!valid[k]) continue;
            if constexpr (kExact) {
                for (uint32_t e = 0; e < m; ++e) {
                    const CellSlot<kQuad>& cs = s_cell[e];
                    const float4 c = cs.cm;
                    const float dx = __fsub_rn(c.x, me[k].x), dy = __fsub_rn(c.y, me[k].y),
                                dz = __fsub_rn(c.z, me[k].z);
                    const float r2t =
                        __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
                    float tx, ty, tz;
                    if constexpr (kQuad)
                        cell_term<true>(dx, dy, dz, r2t, c.w, true, cs.q, cs.q2.x, g, eps2, tx, ty, tz);
                    else
                        cell_term<true>(dx, dy, dz, r2t, c.w, false, make_float4(0.f, 0.f, 0.f, 0.f),
                                        0.f, g, eps2, tx, ty, tz);
                    cells[k].push(tx, ty, tz);
                    cells[k].step();
                }
            } else {
                float px = 0.f, py = 0.f, pz = 0.f;
#pragma unroll 2
                for (uint32_t e = rep; e < m; e += reps) {
                    const CellSlot<kQuad>& cs = s_cell[e];
                    const float4 c = cs.cm;
                    const float dx = c.x - me[k].x, dy = c.y - me[k].y, dz = c.z - me[k].z;
                    const float inv = rsqrtf(fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, eps2))));
                    const float u = inv * inv, inv3 = u * inv;
                    float sa = inv3 * c.w;
                    if constexpr (kQuad) {
                        // inv^3 (M + 5/2 u^2 d.Qd) d - inv^5 Qd, u = 1/r^2.
                        const float4 q = cs.q;
                        const float qyz = cs.q2.x, qzz = cs.q2.y;
                        const float qx = fmaf(q.x, dx, fmaf(q.z, dy, q.w * dz));
                        const float qy = fmaf(q.z, dx, fmaf(q.y, dy, qyz * dz));
                        const float qz = fmaf(q.w, dx, fmaf(qyz, dy, qzz * dz));
                        const float dqd = fmaf(dx, qx, fmaf(dy, qy, dz * qz));
                        sa = inv3 * fmaf(2.5f * u * u, dqd, c.w);
                        const float sb = -(inv3 * u);
                        px = fmaf(sb, qx, px);
                        py = fmaf(sb, qy, py);
                        pz = fmaf(sb, qz, pz);
                    }
                    px = fmaf(sa, dx, px);
                    py = fmaf(sa, dy, py);
                    pz = fmaf(sa, dz, pz);
                }
                cells[k].add(px, py, pz);
            }
        }
        inter += owned * m;
        cell_inter += owned * m;
    }

    // Leaf particles: the listed ranges, 32 at a time (one list block), are
    // concatenated and staged 32 particles at a time (a shuffle binary search
    // over the ranges' prefix sums finds each lane's particle), keeping the
    // walk order.
    ChainCursor lcur{d.leaf_first};
    for (uint32_t l0 = 0; l0 < d.n_leaf; l0 += 32u) {
        const uint32_t nl = min(32u, d.n_leaf - l0);
        if (l0 > 0) lcur.advance(a);
        uint32_t rb = 0, rlen = 0;
        if (lane < nl) {
            const uint2 rg = reinterpret_cast<const uint2*>(lcur.words(a))[lane];
            rb = rg.x;
            rlen = rg.y - rg.x;
        }
        uint32_t incl = rlen;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        const uint32_t pre = incl - rlen;
        const uint32_t total = __shfl_sync(kFullMask, incl, 31);
        for (uint32_t t0 = 0; t0 < total; t0 += 32u) {
            const uint32_t pos = t0 + lane;
            uint32_t e = 0;
#pragma unroll
            for (uint32_t step = 16; step > 0; step >>= 1) {
                const uint32_t cand = e + step;
                const uint32_t pc = __shfl_sync(kFullMask, pre, cand & 31u);
                if (cand < nl && pc <= pos) e = cand;
            }
            const uint32_t eb = __shfl_sync(kFullMask, rb, e);
            const uint32_t ep = __shfl_sync(kFullMask, pre, e);
            const uint32_t j = eb + (pos - ep);
            __syncwarp();
            if (pos < total) {
                s_tile[lane] = __ldg(&a.pos[j]);
                s_jdx[lane] = j;
            }
            __syncwarp();
            const uint32_t cnt = min(32u, total - t0);
#pragma unroll
            for (int k = 0; k < kPer; ++k) {
                if (!valid[k]) continue;
                if constexpr (kExact) {
                    for (uint32_t q = 0; q < cnt; ++q) {
                        if (s_jdx[q] != ip[k]) {
                            const float4 p = s_tile[q];
                            float tx, ty, tz;
                            particle_term<true>(__fsub_rn(p.x, me[k].x), __fsub_rn(p.y, me[k].y),
                                                __fsub_rn(p.z, me[k].z), p.w, g, eps2, tx, ty, tz);
                            leaves[k].push(tx, ty, tz);
                            ++inter;
                        }
                        leaves[k].step();
                    }
                } else {
                    float px = 0.f, py = 0.f, pz = 0.f;
#pragma unroll 4
                    for (uint32_t q = rep; q < cnt; q += reps) {
                        const float4 p = s_tile[q];
                        const float dx = p.x - me[k].x, dy = p.y - me[k].y, dz = p.z - me[k].z;
                        const float inv = rsqrtf(fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, eps2))));
                        const bool other = s_jdx[q] != ip[k];
                        const float sc = other ? p.w * (inv * inv * inv) : 0.f;
                        px = fmaf(dx, sc, px);
                        py = fmaf(dy, sc, py);
                        pz = fmaf(dz, sc, pz);
                        inter += other ? 1u : 0u;
                    }
                    leaves[k].add(px, py, pz);
                }
            }
            __syncwarp();
        }
    }

#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        cells[k].finish();
        leaves[k].finish();
        float sx, sy, sz;
        if (kExact) {
            sx = __fadd_rn(cells[k].ax, leaves[k].ax);
            sy = __fadd_rn(cells[k].ay, leaves[k].ay);
            sz = __fadd_rn(cells[k].az, leaves[k].az);
            if (d.n_far > 0) {
                sx = __fadd_rn(sx, __fmul_rn(g, fx[k]));
                sy = __fadd_rn(sy, __fmul_rn(g, fy[k]));
                sz = __fadd_rn(sz, __fmul_rn(g, fz[k]));
            }
        } else {
            // Compensated sums: the running sum minus its pending correction.
            sx = (cells[k].ax - cells[k].cx) + (leaves[k].ax - leaves[k].cx);
            sy = (cells[k].ay - cells[k].cy) + (leaves[k].ay - leaves[k].cy);
            sz = (cells[k].az - cells[k].cz) + (leaves[k].az - leaves[k].cz);
            if (reps > 1u) {  // the copies' sums, in the owner's lane
                __syncwarp();
                s_tile[lane] = make_float4(sx, sy, sz, 0.f);
                __syncwarp();
                if (rep == 0u)
                    for (uint32_t r = 1; r < reps; ++r) {
                        const float4 t = s_tile[lane + r * gcount];
                        sx += t.x;
                        sy += t.y;
                        sz += t.z;
                    }
                __syncwarp();
            }
            sx = (sx + fx[k]) * g;
            sy = (sy + fy[k]) * g;
            sz = (sz + fz[k]) * g;
        }
        if (valid[k] && rep == 0u) store_particle<kPrec>(a, ip[k], me[k], sx, sy, sz);
    }
}

template <bool kExact, bool kPrec, bool kQuad>
__global__ __launch_bounds__(kGeneralWarps * 32) void group_eval_general_kernel(TraverseArgs a) {
    __shared__ CellSlot<kQuad> s_cell[kGeneralWarps][kGeneralCells];
    __shared__ float4 s_tile[kGeneralWarps][32];
    __shared__ uint32_t s_jdx[kGeneralWarps][32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // As in the fast form: incomplete lists are not evaluated.
    if (*reinterpret_cast<volatile const uint32_t*>(a.err) & kErrFrontier) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(a.evals_done, 1u);
    const uint32_t ngroups = *a.group_count;
    uint32_t inter = 0, cell_inter = 0, far_inter = 0;
    while (true) {
        uint32_t gi = 0;
        if (lane == 0) gi = atomicAdd(a.eval_queue, 1u);
        gi = __shfl_sync(kFullMask, gi, 0);
        if (gi >= ngroups) break;
        gi = group_of_ticket(gi, ngroups, a.group_chunk);
        const uint4 rec = a.groups[gi];
        const uint2 gr = make_uint2(rec.x, rec.y);
        const GroupDesc* dp = a.desc + (gi - rec.w);
        const GroupDesc d = load_desc(dp);
        if (gr.y - gr.x > 32u)
            eval_group<kExact, kPrec, kQuad, 2>(a, gr, d, dp->far_co, s_cell[warp], s_tile[warp],
                                                s_jdx[warp], lane, inter, cell_inter, far_inter);
        else
            eval_group<kExact, kPrec, kQuad, 1>(a, gr, d, dp->far_co, s_cell[warp], s_tile[warp],
                                                s_jdx[warp], lane, inter, cell_inter, far_inter);
    }
    unsigned long long i64 = inter, c64 = cell_inter, f64 = far_inter;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        i64 += __shfl_xor_sync(kFullMask, i64, o);
        c64 += __shfl_xor_sync(kFullMask, c64, o);
        f64 += __shfl_xor_sync(kFullMask, f64, o);
    }
    add_stats(a, lane, i64, c64, f64);
}

// ------------------------------------------------------------- launches --

constexpr int kMaxDevices = 64;
std::mutex g_mutex;

// A persistent launch: as many blocks as the device holds at once. The
// block count (and the shared-memory attribute) is set once per device.
struct Persistent {
    uint32_t blocks[kMaxDevices] = {};
    cudaError_t get(const void* kernel, int threads, size_t smem, uint32_t* out) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
        std::lock_guard<std::mutex> lock(g_mutex);
        if (blocks[dev] == 0) {
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return e;
            int per_sm = 0, sms = 0;
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
            if (e != cudaSuccess) return e;
            e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            if (e != cudaSuccess) return e;
            blocks[dev] = (uint32_t)std::max(1, per_sm) * (uint32_t)std::max(1, sms);
        }
        *out = blocks[dev];
        return cudaSuccess;
    }
};

template <bool kPrec, bool kQuad, bool kTiny>
cudaError_t launch_fast(const TraverseArgs& a, cudaStream_t st) {
    static Persistent shape;
    auto kernel = group_eval_fast_kernel<kPrec, kQuad, kTiny>;
    const size_t smem = sizeof(FastSmem<kPrec>) * kFastWarps;
    uint32_t blocks = 0;
    const cudaError_t e = shape.get((const void*)kernel, kFastWarps * 32, smem, &blocks);
    if (e != cudaSuccess) return e;
    kernel<<<blocks, kFastWarps * 32, smem, st>>>(a);
    return cudaGetLastError();
}

template <bool kExact, bool kPrec, bool kQuad>
cudaError_t launch_general(const TraverseArgs& a, cudaStream_t st) {
    static Persistent shape;
    auto kernel = group_eval_general_kernel<kExact, kPrec, kQuad>;
    uint32_t blocks = 0;
    const cudaError_t e = shape.get((const void*)kernel, kGeneralWarps * 32, 0, &blocks);
    if (e != cudaSuccess) return e;
    kernel<<<blocks, kGeneralWarps * 32, 0, st>>>(a);
    return cudaGetLastError();
}

template <bool kPrec, bool kQuad>
cudaError_t launch_form(const TraverseArgs& a, bool exact, cudaStream_t st) {
    if (exact) return launch_general<true, kPrec, kQuad>(a, st);
    if (a.eps2 >= kPackedMinEps2) return launch_fast<kPrec, kQuad, false>(a, st);
    return a.eps2 >= kFltMin ? launch_fast<kPrec, kQuad, true>(a, st) : launch_general<false, kPrec, kQuad>(a, st);
}

}  // namespace

cudaError_t launch_group_eval(const TraverseArgs& a, const TraverseConfig& c, cudaStream_t st) {
    if (c.precision) return c.quad ? launch_form<true, true>(a, c.exact, st) : launch_form<true, false>(a, c.exact, st);
    return c.quad ? launch_form<false, true>(a, c.exact, st) : launch_form<false, false>(a, c.exact, st);
}

}  // namespace astro
