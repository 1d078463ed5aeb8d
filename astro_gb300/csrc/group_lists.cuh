// What the group walk, the far-node sums and the evaluation share: the
// order groups are taken from a queue and the reading of list chains.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "build_kernels.cuh"

namespace astro {

// Queue ticket -> group index. For a batch the groups are visited in whole
// chunks of consecutive groups in a scrambled chunk order (a bijection:
// 1000003 is prime and larger than the chunk count); the last partial chunk
// keeps its place.
__device__ __forceinline__ uint32_t group_of_ticket(uint32_t gi, uint32_t ngroups, uint32_t chunk) {
    if (chunk > 0) {
        const uint32_t nfull = ngroups / chunk;
        if (gi < nfull * chunk)
            gi = (uint32_t)(((uint64_t)(gi / chunk) * 1000003ull) % nfull) * chunk + gi % chunk;
    }
    return gi;
}

// Reads a list chain block by block.
struct ChainCursor {
    uint32_t blk;
    __device__ __forceinline__ const uint32_t* words(const TraverseArgs& a) const {
        return a.lists + (size_t)blk * kListBlockWords;
    }
    __device__ __forceinline__ void advance(const TraverseArgs& a) { blk = __ldg(&a.list_next[blk]); }
};

// The lists and the box centre of a walk's record (its first 48 bytes).
__device__ __forceinline__ GroupDesc load_desc(const GroupDesc* dp) {
    const uint4* w = reinterpret_cast<const uint4*>(dp);
    const uint4 w0 = __ldg(w), w1 = __ldg(w + 1), w2 = __ldg(w + 2);
    GroupDesc d;
    d.leaf_first = w0.x, d.n_leaf = w0.y, d.cell_first = w0.z, d.n_cell = w0.w;
    d.far_first = w1.x, d.n_far = w1.y, d.gcx = __uint_as_float(w1.z);
    d.gcy = __uint_as_float(w1.w), d.gcz = __uint_as_float(w2.x);
    return d;
}

// The group evaluation (group_eval.cu), after the walk and the far-node sums.
cudaError_t launch_group_eval(const TraverseArgs& a, const TraverseConfig& c, cudaStream_t st);

}  // namespace astro
