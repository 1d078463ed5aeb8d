// Headless particle splat: the scene pass of the reference's renderer
// (Astro/Spheres.metal:23-64 vertex math, Renderer.swift:780-830 draw order,
// :143-144 depth state, :276-295 pipelines) drawn into a device image.
//
// Every particle is projected as sphere_vertex / dust_point_vertex do:
//   clip = P * (V * float4(x - camera, 1))
// Stars and planets (types 0, 1) are the reference's sphere meshes (extent 1,
// scaled by the radius: world radius radius/2); here each is a disc of that
// projected radius at its centre's depth, drawn opaque. Dust (type 2) is a
// point sprite of `radius` pixels, blended with source alpha. Fragments are
// keyed (pixel, particle) in as few bits as both need, sorted with the library's radix sort, and every
// pixel folds its fragments in particle order — the reference's draw order
// (stars, planets, dust by instance) — with the depth test "less", depth
// writes on, and the colour rounded to half precision after every write (the
// rgba16Float attachment). Correctly rounded operations throughout, in the
// order of the CPU restatement (oracle/oracle_splat.cpp).
#include <algorithm>

#include <cuda_fp16.h>

#include "build_kernels.cuh"
#include "common.cuh"

namespace astro {

namespace {

__device__ __forceinline__ float mat_row(const float* m, int r, float x, float y, float z, float w) {
    // (m * v)[r] for a column-major 4x4 m, summed over columns 0..3 in order.
    float s = __fmul_rn(m[r], x);
    s = __fadd_rn(s, __fmul_rn(m[4 + r], y));
    s = __fadd_rn(s, __fmul_rn(m[8 + r], z));
    return __fadd_rn(s, __fmul_rn(m[12 + r], w));
}

__device__ __forceinline__ float to_half(float x) { return __half2float(__float2half_rn(x)); }

// One projected primitive: window x, y, depth, and the point size (pixels) or
// the disc radius (pixels); kind 0 = culled, 1 = disc, 2 = point.
__global__ void splat_project_kernel(SplatArgs a) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const float4 p = a.pos[i];
    const float rel_x = __fsub_rn(p.x, a.cam[0]), rel_y = __fsub_rn(p.y, a.cam[1]),
                rel_z = __fsub_rn(p.z, a.cam[2]);
    float v[4], c[4];
    for (int r = 0; r < 4; ++r) v[r] = mat_row(a.view, r, rel_x, rel_y, rel_z, 1.0f);
    for (int r = 0; r < 4; ++r) c[r] = mat_row(a.proj, r, v[0], v[1], v[2], v[3]);
    const uint32_t type = a.types[i];
    const float radius = a.vel[i].w;
    const bool point = type == 2u;
    uint32_t kind = point ? 2u : 1u;
    const float w = c[3];
    if (!(w > 0.0f) || !(c[2] >= 0.0f) || !(c[2] <= w)) kind = 0u;
    if (point && !(c[0] >= -w && c[0] <= w && c[1] >= -w && c[1] <= w)) kind = 0u;
    float4 out = make_float4(0.f, 0.f, 0.f, 0.f);
    if (kind) {
        const float nx = __fdiv_rn(c[0], w), ny = __fdiv_rn(c[1], w), nz = __fdiv_rn(c[2], w);
        out.x = __fmul_rn(__fmul_rn(__fadd_rn(nx, 1.0f), 0.5f), (float)a.width);
        out.y = __fmul_rn(__fmul_rn(__fsub_rn(1.0f, ny), 0.5f), (float)a.height);
        out.z = nz;
        if (point) {
            out.w = radius;
        } else {
            const float world_r = __fmul_rn(0.5f, radius);
            out.w = __fmul_rn(__fdiv_rn(__fmul_rn(world_r, a.proj[5]), w),
                              __fmul_rn(0.5f, (float)a.height));
        }
        if (!(out.w > 0.0f) || !isfinite(out.x) || !isfinite(out.y)) kind = 0u;
    }
    a.prim[i] = out;
    a.kind[i] = kind;
}

// Pixel range [lo, hi] whose centres can lie in [c - h, c + h], clamped.
__device__ __forceinline__ void span(float c, float h, uint32_t size, int& lo, int& hi) {
    const float a = floorf(__fsub_rn(__fsub_rn(c, h), 0.5f));
    const float b = ceilf(__fsub_rn(__fadd_rn(c, h), 0.5f));
    lo = a < 0.0f ? 0 : (a > (float)size ? (int)size : (int)a);
    hi = b < 0.0f ? -1 : (b >= (float)size ? (int)size - 1 : (int)b);
}

__device__ __forceinline__ bool covers(uint32_t kind, float4 q, int px, int py) {
    const float cx = __fadd_rn((float)px, 0.5f), cy = __fadd_rn((float)py, 0.5f);
    if (kind == 2u) {
        const float h = __fmul_rn(q.w, 0.5f);
        return cx >= __fsub_rn(q.x, h) && cx < __fadd_rn(q.x, h) && cy >= __fsub_rn(q.y, h) &&
               cy < __fadd_rn(q.y, h);
    }
    const float dx = __fsub_rn(cx, q.x), dy = __fsub_rn(cy, q.y);
    return __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)) < __fmul_rn(q.w, q.w);
}

// Fragments of 32 primitives per warp and round. A lane draws its own small
// primitive (a box of at most kLaneCells pixels: dust points) - it counts the
// pixels covered, the warp claims the slots of all its lanes with one atomic,
// and the lane writes its keys. Larger ones go to a list from both ends: those of
// up to kWarpCells pixels are drawn by a warp each afterwards, the rest in up to
// kSlices parts of at least kPartCells (splat_emit_large_kernel). Keys are pixel << id_bits | particle; writes past
// cap are counted, not stored.
// One atomic per fragment on the one cursor took 185 us for 500,205 particles
// (about two million fragments); one per 32 primitives 32 us. With the large ones
// drawn one after the other by the warp that met them, 3,000 points of 50 pixels took
// 31.2 ms a picture and 300 that fill it 604 ms (11.2 and 38.3 with a warp for every
// primitive); 1.9 and 15.1 now.
constexpr uint32_t kLaneCells = 64, kWarpCells = 4096, kSlices = 256, kPartCells = 1024;

struct Box {
    int x0, y0;
    uint32_t width, cells;  // (an image has at most 2^31 pixels)
};
__device__ __forceinline__ Box box_of(const SplatArgs& a, uint32_t kind, float4 q) {
    const float h = kind == 2u ? __fmul_rn(q.w, 0.5f) : q.w;
    int x0, x1, y0, y1;
    span(q.x, h, a.width, x0, x1);
    span(q.y, h, a.height, y0, y1);
    if (x1 < x0 || y1 < y0) return Box{0, 0, 0u, 0u};
    const uint32_t width = (uint32_t)(x1 - x0 + 1);
    return Box{x0, y0, width, width * (uint32_t)(y1 - y0 + 1)};
}

__global__ __launch_bounds__(256) void splat_emit_kernel(SplatArgs a) {
    const uint32_t lane = threadIdx.x & 31u, lt = lanemask_lt();
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t chunks = (a.n + 31u) / 32u;
    for (uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < chunks; c += warps) {
        const uint32_t i = c * 32u + lane;
        const uint32_t kind = i < a.n ? a.kind[i] : 0u;
        const float4 q = kind ? a.prim[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        const Box box = kind ? box_of(a, kind, q) : Box{0, 0, 0u, 0u};
        const bool small = box.cells <= kLaneCells;
        uint32_t count = 0;
        auto each = [&](auto&& draw) {
            uint32_t x = 0, y = 0;
            for (uint32_t k = 0; k < box.cells; ++k) {
                const int px = box.x0 + (int)x, py = box.y0 + (int)y;
                if (covers(kind, q, px, py)) draw(px, py);
                if (++x == box.width) x = 0, ++y;
            }
        };
        if (small) each([&](int, int) { ++count; });
        uint32_t incl = count;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        const uint32_t total = __shfl_sync(kFullMask, incl, 31);
        if (total > 0u) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(a.cursor, total);
            uint32_t slot = __shfl_sync(kFullMask, base, 0) + incl - count;
            if (count)
                each([&](int px, int py) {
                    if (slot < a.cap)
                        a.keys[slot] = ((uint64_t)((uint32_t)py * a.width + (uint32_t)px) << a.id_bits) | i;
                    ++slot;
                });
        }
        const bool huge = box.cells > kWarpCells;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const bool mine = !small && huge == (e == 1);
            const uint32_t m = __ballot_sync(kFullMask, mine);
            if (m == 0u) continue;
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(a.cursor + 1 + e, (uint32_t)__popc(m));
            const uint32_t at = __shfl_sync(kFullMask, base, 0) + __popc(m & lt);
            if (mine) a.large[e == 0 ? at : a.n - 1u - at] = i;
        }
    }
}

// The listed primitives: a warp draws one, or one part of it, 128 pixels for an
// atomic.
__global__ __launch_bounds__(256) void splat_emit_large_kernel(SplatArgs a) {
    const uint32_t lane = threadIdx.x & 31u, lt = lanemask_lt();
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t single = a.cursor[1];
    const uint64_t items = single + (uint64_t)a.cursor[2] * kSlices;
    for (uint64_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < items; t += warps) {
        const bool whole = t < single;
        const uint32_t i = a.large[whole ? (uint32_t)t : a.n - 1u - (uint32_t)((t - single) / kSlices)];
        const uint32_t kind = a.kind[i];
        const float4 q = a.prim[i];
        const Box box = box_of(a, kind, q);
        const uint32_t part = whole ? box.cells : max(kPartCells, (box.cells + kSlices - 1u) / kSlices);
        const uint32_t begin = whole ? 0u : (uint32_t)min((t - single) % kSlices * part, (uint64_t)box.cells);
        const uint32_t end = begin + min(part, box.cells - begin);
        for (uint32_t k0 = begin; k0 < end; k0 += 128u) {
            uint32_t m[4], cell[4], total = 0;
#pragma unroll
            for (uint32_t u = 0; u < 4u; ++u) {
                const uint32_t k = k0 + 32u * u + lane;
                const uint32_t y = k / box.width, x = k - y * box.width;
                const int px = box.x0 + (int)x, py = box.y0 + (int)y;
                m[u] = __ballot_sync(kFullMask, k < end && covers(kind, q, px, py));
                cell[u] = (uint32_t)py * a.width + (uint32_t)px;
                total += __popc(m[u]);
            }
            if (total == 0u) continue;
            uint32_t slot = 0;
            if (lane == 0) slot = atomicAdd(a.cursor, total);
            slot = __shfl_sync(kFullMask, slot, 0);
#pragma unroll
            for (uint32_t u = 0; u < 4u; ++u) {
                const uint32_t at = slot + __popc(m[u] & lt);
                if ((m[u] >> lane & 1u) && at < a.cap) a.keys[at] = ((uint64_t)cell[u] << a.id_bits) | i;
                slot += __popc(m[u]);
            }
        }
    }
}

__global__ void splat_clear_kernel(SplatArgs a) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.width * a.height) return;
    a.image[p] = make_float4(to_half(a.clear[0]), to_half(a.clear[1]), to_half(a.clear[2]),
                             to_half(a.clear[3]));
    a.depth[p] = a.clear_depth;
}

// One thread per pixel run of the sorted keys: depth test and blend in
// particle order.
__global__ void splat_fold_kernel(SplatArgs a, const uint64_t* __restrict__ keys, uint32_t count) {
    const uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= count) return;
    const uint32_t pix = (uint32_t)(keys[f] >> a.id_bits);
    if (f > 0 && (uint32_t)(keys[f - 1] >> a.id_bits) == pix) return;
    const uint64_t id_mask = (1ull << a.id_bits) - 1ull;
    float4 dst = a.image[pix];
    float z = a.depth[pix];
    for (uint32_t g = f; g < count && (uint32_t)(keys[g] >> a.id_bits) == pix; ++g) {
        const uint32_t i = (uint32_t)(keys[g] & id_mask);
        const float zf = a.prim[i].z;
        if (!(zf < z)) continue;
        const float4 src = a.colors[i];
        if (a.kind[i] == 2u) {
            const float inv = __fsub_rn(1.0f, src.w);
            dst.x = to_half(__fadd_rn(__fmul_rn(src.x, src.w), __fmul_rn(dst.x, inv)));
            dst.y = to_half(__fadd_rn(__fmul_rn(src.y, src.w), __fmul_rn(dst.y, inv)));
            dst.z = to_half(__fadd_rn(__fmul_rn(src.z, src.w), __fmul_rn(dst.z, inv)));
            dst.w = to_half(__fadd_rn(__fmul_rn(src.w, src.w), __fmul_rn(dst.w, inv)));
        } else {
            dst = make_float4(to_half(src.x), to_half(src.y), to_half(src.z), to_half(src.w));
        }
        z = zf;
    }
    a.image[pix] = dst;
    a.depth[pix] = z;
}

}  // namespace

cudaError_t launch_splat_project(const SplatArgs& a, cudaStream_t st) {
    if (a.n == 0) return cudaSuccess;
    splat_project_kernel<<<(a.n + 255) / 256, 256, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_splat_emit(const SplatArgs& a, cudaStream_t st) {
    if (a.n == 0) return cudaSuccess;
    const uint32_t blocks = (uint32_t)std::min<uint64_t>(((uint64_t)a.n + 255) / 256, 152u * 64u);
    splat_emit_kernel<<<blocks, 256, 0, st>>>(a);
    splat_emit_large_kernel<<<152u * 8u, 256, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_splat_clear(const SplatArgs& a, cudaStream_t st) {
    const uint32_t pixels = a.width * a.height;
    splat_clear_kernel<<<(pixels + 255) / 256, 256, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_splat_fold(const SplatArgs& a, const uint64_t* keys, uint32_t count,
                              cudaStream_t st) {
    if (count == 0) return cudaSuccess;
    splat_fold_kernel<<<(count + 255) / 256, 256, 0, st>>>(a, keys, count);
    return cudaGetLastError();
}

}  // namespace astro
