// Onesweep LSD radix sort of (uint64 key, uint32 value) pairs for sm_103a.
//
// Replaces MetalKernelsRadixSort.sort (Astro/RadixSort.swift:98-185), whose
// 64 one-bit split passes (split_prep / prefixSum / prefixFixup /
// split_scatter, Astro/RadixSort.metal:30-131) each move the whole key and
// index arrays. Here the key is consumed 8 bits per pass:
//   1. one histogram kernel reads the keys once and counts every digit of
//      every pass (warp-ballot peer groups, shared-memory histograms); its
//      last block turns the counts into exclusive digit offsets;
//   2. one kernel per pass: each block takes the next tile (atomic ticket),
//      ranks its keys stably with warp-ballot peer masks and per-warp digit
//      counters in shared memory, publishes its digit counts, stages the
//      tile in sorted order in shared memory, obtains the counts of all
//      earlier tiles by decoupled look-back (bounded waits), and writes each
//      digit's run of the tile with contiguous stores.
// Digits that all keys share are skipped, and where the top digits alone nearly
// tell the keys apart only those are sorted, and the few keys that share them are
// ordered in place of the remaining passes (see SortSchedule).
// Few pairs are sorted in one launch instead (sort_small.cu).
// A stable LSD sort yields the one stable permutation, so the result equals
// the reference's bit by bit, including the order of equal keys.
#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "internal.h"

namespace astro {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kRadix = 256;
constexpr int kMaxPasses = 8;
constexpr int kHistBlocksPerSm = 4, kHistCopies = 4;

// Words of the scratch's counter block: [8] histogram blocks done, [9] error
// word, from kScheduleWord on the schedule, from kTicketWord on one ticket
// counter a launch. All zero when a sort starts.
constexpr uint32_t kDoneWord = 8, kScheduleWord = 10, kTicketWord = 16;
// The schedule is worked out on the device by the last histogram block, which
// knows the digit counts: word 0 holds the number m of digits that not all keys
// share (at least 1) and in bits 8-15 the number of top digits to sort by (0: all
// m, from the lowest up); word 1 the m digits, lowest first, four bits each;
// word 4 kLongRuns and kStartOver as met on the way; word 5 the long runs listed.
//
// Top digits: stable passes over the top kTopDigits digits, then ordering by
// reading: a key finds its place among the others that share them, about
// kNeighbours at most on average (fixup_kernel). A run of more than kFixHalo of them
// is sorted by a block of its own (runs_kernel); should one be longer than kRunMax,
// all m digits are sorted from the input after all.
//
// 63-bit keys without / with it: uniform ones, 2,097,152 226 / 167 us, 16,777,216
// 1005 / 526. Keys of clustered particles do not qualify and pay for the question
// and its idle launches: 48 bits, 5,000,000 298 / 310, 1,400,000 140 / 161 (146
// before the resident passes), so not below kTopMin: uniform ones of 63 bits lose by
// that, 1,400,000 181 / 148, but no keys are slower than they were. Uniform keys of
// 48 bits but for one place that holds 500 or 5,000 of them, 2,000,000: 265 and 278
// us when every long run had all digits sorted, 161 and 191 with blocks for them (155
// without the place). (Four or five top digits let clustered 63-bit keys qualify,
// 5,000,000 399 -> 370 us, but with longer runs.)
constexpr uint32_t kTopDigits = 3, kSavedPasses = 3;  // of at least 6 digits
constexpr uint32_t kTopMin = 3u << 19;
constexpr float kNeighbours = 4.f;
constexpr uint32_t kSamples = 4096, kSampleSlots = 2 * kSamples;
constexpr uint32_t kFixTile = 2048, kFixHalo = 128;
constexpr uint32_t kRunThreads = 1024, kRunMax = 32u * kRunThreads;
constexpr uint32_t kLongRuns = 1u, kStartOver = 2u;

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// The digit of a pass. Passes start at multiples of 8 bits, so a digit lies in
// one word of the key.
__device__ __forceinline__ uint32_t digit_of(uint64_t key, uint32_t shift, uint32_t dmask) {
    const uint32_t w = (shift & 32u) ? (uint32_t)(key >> 32) : (uint32_t)key;
    return (w >> (shift & 31u)) & dmask;
}

// Lanes of the warp whose digit equals this lane's digit, among `valid`. All
// eight bits are compared, also where the last digit has fewer: the loop has to
// be unrolled (over the run-time width, with the checks that whole tiles
// do not need it cost a pass 187 instructions for 32 keys, and 16.7 M pairs 156
// us a pass against 135).
__device__ __forceinline__ uint32_t peer_mask(uint32_t digit, uint32_t valid) {
    uint32_t peers = valid;
#pragma unroll
    for (uint32_t b = 0; b < 8; ++b) {
        const bool bit = (digit & (1u << b)) != 0u;
        const uint32_t ballot = __ballot_sync(kFullMask, bit);
        peers &= bit ? ballot : ~ballot;
    }
    return peers;
}

// Stable rank of this lane's key among the keys of its digit that the warp has
// ranked so far; counts the warp's keys in `hist`.
__device__ __forceinline__ uint32_t warp_rank(uint32_t* hist, uint32_t digit, bool valid, uint32_t valid_mask,
                                              uint32_t lane, uint32_t lt) {
    const uint32_t peers = peer_mask(digit, valid_mask);
    uint32_t rank = __popc(peers & lt);
    if (valid) rank += hist[digit];
    __syncwarp();
    // The last lane of the digit has the highest rank.
    if (valid && (peers & ~lt) == (1u << lane)) hist[digit] = rank + 1u;
    __syncwarp();
    return rank;
}

// Place of sample k: spread over the input regardless of its order.
__device__ __forceinline__ uint32_t sample_place(uint32_t k, uint32_t n) {
    uint32_t h = (k + 1u) * 0x9E3779B1u;
    h = (h ^ (h >> 15)) * 0x85EBCA77u;
    h ^= h >> 13;
    return __umulhi(h, n);
}

// The bits of a key that take part.
__device__ __forceinline__ uint64_t key_mask(uint32_t key_bits) {
    return key_bits >= 64u ? ~0ull : (1ull << key_bits) - 1ull;
}

// Whether the digits from `shift` up (of the bits that take part) leave a key
// about kNeighbours others with the same ones: of S keys at random places, S^2 / 2
// times the chance that two keys agree do.
__device__ __forceinline__ bool top_suffices(const uint64_t* samples, uint32_t n, uint32_t shift, uint64_t mask) {
    extern __shared__ uint32_t slots[];  // hashes of prefixes; all ones: empty
    __shared__ uint32_t s_equal;
    const uint32_t tid = threadIdx.x;
    __syncthreads();
    if (tid == 0) s_equal = 0;
#pragma unroll 1
    for (uint32_t i = tid; i < kSampleSlots; i += kThreads) slots[i] = ~0u;
    __syncthreads();
    uint32_t equal = 0;
    // (Not unrolled: one block runs this, and fetching 16 copies of the code took
    // 45 us.)
#pragma unroll 1
    for (uint32_t k = tid; k < kSamples; k += kThreads) {
        const uint64_t prefix = (__ldcg(samples + k) & mask) >> shift;
        const uint32_t id = min((uint32_t)((prefix * 0x9E3779B97F4A7C15ull) >> 32), ~1u);
        uint32_t at = id & (kSampleSlots - 1u);
        while (true) {  // half of the slots stay empty
            const uint32_t was = atomicCAS(&slots[at], ~0u, id);
            equal += was == id ? 1u : 0u;
            if (was == ~0u || was == id) break;
            at = (at + 1u) & (kSampleSlots - 1u);
        }
    }
    equal = __reduce_add_sync(kFullMask, equal);
    if ((tid & 31) == 0) atomicAdd(&s_equal, equal);
    __syncthreads();
    return (float)s_equal <= 0.5f * (float)kSamples * (float)kSamples * kNeighbours / (float)n + 4.f;
}

// All digit histograms in one read of the keys. Two warps share a copy of the
// counters in shared memory, which they count into with atomics (16.7 M keys, 8
// digits: 87 us against 97 with a copy for each, which left 24 warps an SM); a warp whose 32 keys share a digit (the
// usual case for the high digits of Morton keys of a Morton-ordered state)
// adds 32 with a single atomic.
// The last block then schedules the passes.
__global__ __launch_bounds__(kThreads, kHistBlocksPerSm) void sort_histogram_kernel(
    const uint64_t* __restrict__ keys, const uint32_t* __restrict__ d_count, uint32_t n_est,
    uint32_t key_bits, uint32_t passes, uint32_t* __restrict__ hist, uint32_t* __restrict__ excl,
    uint32_t* __restrict__ counters, bool skip_shared, bool try_top, uint64_t* __restrict__ samples) {
    extern __shared__ uint32_t s_hist[];  // [kHistCopies][passes][kRadix]
    __shared__ bool s_last;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t n = d_count ? min(*d_count, n_est) : n_est;
    const uint32_t per_copy = passes * kRadix;
    for (uint32_t i = tid; i < kHistCopies * per_copy; i += kThreads) s_hist[i] = 0;
    __syncthreads();
    // The first blocks fetch the samples, whose scattered reads would take the
    // last block about 40 us (`samples`: the temporaries, unused until then).
    if (try_top && n != 0u && blockIdx.x < kSamples / kThreads)
        samples[blockIdx.x * kThreads + tid] = keys[sample_place(blockIdx.x * kThreads + tid, n)];
    uint32_t* my_hist = s_hist + (warp % kHistCopies) * per_copy;
    const uint32_t last_mask = key_bits == 0 ? 0u : (1u << (key_bits - 8u * (passes - 1u))) - 1u;
    // Each thread takes kHistKeys keys per round (independent loads in flight).
    constexpr int kHistKeys = 4;
    const uint64_t stride = (uint64_t)gridDim.x * kThreads * kHistKeys;
    for (uint64_t base = (uint64_t)blockIdx.x * kThreads * kHistKeys; base < n; base += stride) {
        uint64_t key[kHistKeys];
        bool valid[kHistKeys];
#pragma unroll
        for (int k = 0; k < kHistKeys; ++k) {
            const uint64_t i = base + (uint64_t)k * kThreads + tid;
            valid[k] = i < n;
            key[k] = valid[k] ? __ldcs(keys + i) : 0ull;
        }
#pragma unroll
        for (int k = 0; k < kHistKeys; ++k) {
            // Bits in which the warp's keys differ.
            const uint64_t x = key[k] ^ __shfl_sync(kFullMask, key[k], 0);
            const bool full = __all_sync(kFullMask, valid[k]);
            const uint32_t dlo = __reduce_or_sync(kFullMask, full ? (uint32_t)x : ~0u);
            const uint32_t dhi = __reduce_or_sync(kFullMask, full ? (uint32_t)(x >> 32) : ~0u);
#pragma unroll
            for (uint32_t p = 0; p < kMaxPasses; ++p) {
                if (p >= passes) break;
                const uint32_t dmask = p + 1 == passes ? last_mask : 0xFFu;
                const uint32_t digit = digit_of(key[k], 8u * p, dmask);
                const uint32_t diff = digit_of((uint64_t)dhi << 32 | dlo, 8u * p, dmask);
                if (diff == 0u) {
                    if (lane == 0) atomicAdd(&my_hist[p * kRadix + digit], 32u);
                } else if (valid[k]) {
                    atomicAdd(&my_hist[p * kRadix + digit], 1u);
                }
            }
        }
    }
    __syncthreads();
    for (uint32_t i = tid; i < per_copy; i += kThreads) {
        uint32_t c = 0;
        for (int w = 0; w < kHistCopies; ++w) c += s_hist[w * per_copy + i];
        if (c) atomicAdd(&hist[i], c);
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(counters + kDoneWord, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // A warp each turns a digit's counts into offsets, eight counts a lane (the block
    // for one digit after the other took 2 us more for six of them: 200,000 pairs of
    // 48 bits 80 -> 76).
    __shared__ float s_agree[kMaxPasses];   // chance that two keys have the same digit
    __shared__ bool s_shared[kMaxPasses];   // all keys have the same digit
    static_assert(kWarps == kMaxPasses && kRadix == 8 * 32, "a warp a pass");
    if (warp < passes) {
        const uint4* from = reinterpret_cast<const uint4*>(hist + warp * kRadix) + 2u * lane;
        uint4* to = reinterpret_cast<uint4*>(excl + warp * kRadix) + 2u * lane;
        const uint4 x = __ldcg(from), y = __ldcg(from + 1);
        const uint32_t c[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
        uint32_t o[8], run = 0;
        float agree = 0.f;
        bool all = false;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            o[k] = run;
            run += c[k];
            all |= c[k] == n;
            const float f = (float)c[k] / (float)n;
            agree += f * f;
        }
        uint32_t incl = run;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t z = __shfl_up_sync(kFullMask, incl, d);
            if (lane >= (uint32_t)d) incl += z;
        }
        const uint32_t before = incl - run;
        to[0] = make_uint4(before + o[0], before + o[1], before + o[2], before + o[3]);
        to[1] = make_uint4(before + o[4], before + o[5], before + o[6], before + o[7]);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) agree += __shfl_xor_sync(kFullMask, agree, d);
        all = __any_sync(kFullMask, all);
        if (lane == 0) s_agree[warp] = agree, s_shared[warp] = all;
    }
    __syncthreads();
    uint32_t m = 0, digits = 0;
    for (uint32_t p = 0; p < passes; ++p)
        if (!s_shared[p] || !skip_shared) digits |= p << (4u * m++);
    if (m == 0) m = 1;  // equal keys: one pass copies them
    uint32_t top = 0;
    if (try_top && n >= kTopMin && m >= kTopDigits + kSavedPasses) {
        const uint32_t lowest = (digits >> (4u * (m - kTopDigits))) & 15u;
        float others = (float)n;  // if the digits were independent
        for (uint32_t k = m - kTopDigits; k < m; ++k) others *= s_agree[(digits >> (4u * k)) & 15u];
        // Keys of clustered particles share their digits far more often.
        if (others <= 16.f * kNeighbours && top_suffices(samples, n, 8u * lowest, key_mask(key_bits))) top = kTopDigits;
    }
    if (tid == 0) {
        counters[kScheduleWord] = m | (top << 8);
        counters[kScheduleWord + 1] = digits;
    }
}

// What the launches of a sort share.
struct SortArgs {
    const uint64_t* keys_in;
    const uint32_t* vals_in;  // null: the places 0, 1, ...
    uint64_t *keys_tmp, *keys_out;
    uint32_t *vals_tmp, *vals_out;
    const uint32_t* d_count;
    uint32_t n_est, key_bits;
    const uint32_t* excl;
    uint32_t* lookback;
    size_t lookback_stride;  // words of one pass
    uint32_t* counters;
    uint32_t early;  // launches before the fix-up (0: no fix-up)
    uint32_t* runs;  // beginnings of the long runs
    uint32_t* err;
    uint32_t spin_limit;
};
// One pass: where from, where to, which digit.
struct Pass {
    const uint64_t* keys_in;
    const uint32_t* vals_in;
    uint64_t* keys_out;
    uint32_t* vals_out;
    const uint32_t* excl;
    uint32_t* lookback;
    uint32_t shift, digit_bits;
};
// The pass that launch `launch` has to run under the schedule; false: none. The
// passes alternate between the temporaries and the output so that the last one
// (or the fix-up) ends in the output.
__device__ __forceinline__ bool pick_pass(const SortArgs& a, uint32_t launch, Pass& p) {
    const uint32_t w = a.counters[kScheduleWord], digits = a.counters[kScheduleWord + 1];
    const uint32_t m = w & 255u, top = w >> 8;
    uint32_t i = launch, at = i, count = m, stages = m;
    if (top != 0u && launch < a.early) {
        count = top;
        at = m - top + i;
        stages = top + 1u;
    } else if (top != 0u) {
        if ((a.counters[kScheduleWord + 4] & kStartOver) == 0u) return false;
        at = i -= a.early;
    }
    if (i >= count) return false;
    const uint32_t digit = (digits >> (4u * at)) & 15u;
    const bool to_out = ((stages - 1u - i) & 1u) == 0u;
    p.keys_in = i == 0u ? a.keys_in : (to_out ? a.keys_tmp : a.keys_out);
    p.vals_in = i == 0u ? a.vals_in : (to_out ? a.vals_tmp : a.vals_out);
    p.keys_out = to_out ? a.keys_out : a.keys_tmp;
    p.vals_out = to_out ? a.vals_out : a.vals_tmp;
    p.excl = a.excl + digit * kRadix;
    p.lookback = a.lookback + i * a.lookback_stride;
    p.shift = 8u * digit;
    p.digit_bits = min(8u, a.key_bits - min(a.key_bits, p.shift));
    return true;
}

template <int kBlock, int kItems>
struct PassSmem {
    static constexpr int kTile = kBlock * kItems;
    uint64_t keys[kTile];  // the tile in sorted order
    uint32_t vals[kTile];
    uint32_t warp_hist[kBlock / 32][kRadix];  // per-warp digit counts, then the next slot of each
    uint32_t out_base[kRadix];  // first output slot of each digit less its first slot in the tile
    uint32_t warp_sum[kWarps];
    uint32_t next_tile;
};

// One onesweep pass. kItems pairs per thread, ranked with per-bit ballots and
// per-warp counters.
//
// A pass is a chain of latencies, not of bytes (384 MB at 16.7 M pairs are 59
// us): the ticket, the loads, the ranking, the wait for the earlier tiles'
// counts, the scatter. So the blocks stay (grid: what fits on the chip), and
//  - the next tile's ticket is taken before the look-back and its keys are
//    asked for before the scatter, so both arrive behind other work;
//  - the digits are counted (one shared atomic a key) and published before the
//    ranking, so that no look-back waits for another tile's ranking;
//  - the ranking then yields final slots of the sorted tile, and the values are
//    asked for behind it, to arrive during the look-back.
// Tickets are taken in order and each block works on its lowest first: a
// look-back only waits for tiles that running blocks hold and reach.
// 16.7 M pairs of 63-bit keys: 156 us a pass -> 124 (20 keys a thread); 524,288:
// 12.0 -> 10.2. What is left is spread over the phases: a warp's 32 keys cost an
// SM about 26 cycles of ranking (the ballots' logic runs at half rate), 22 of
// scattering and 8 of counting and staging, and the look-back 5,000 cycles a
// tile. Tried: wider windows and a look-back inside the ranking (the words to
// add up are the same, it only moves), blocks of 384 to 1,024 threads with
// larger tiles (their warps rank at once and scatter at once: 130-150 us).
template <int kBlock, int kItems, int kMinBlocks>
__global__ __launch_bounds__(kBlock, kMinBlocks) void sort_pass_kernel(SortArgs args, uint32_t launch) {
    using Smem = PassSmem<kBlock, kItems>;
    constexpr int kBlockWarps = kBlock / 32;
    constexpr int kTile = Smem::kTile;
    static_assert(kTile <= 65536, "tile-local indices fit 16 bits");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t* tile_counter = args.counters + kTicketWord + launch;
    if (tid == 0) sm.next_tile = atomicAdd(tile_counter, 1u);
    Pass pass_args;
    if (!pick_pass(args, launch, pass_args)) return;
    const uint64_t* __restrict__ keys_in = pass_args.keys_in;
    const uint32_t* __restrict__ vals_in = pass_args.vals_in;
    uint64_t* __restrict__ keys_out = pass_args.keys_out;
    uint32_t* __restrict__ vals_out = pass_args.vals_out;
    const uint32_t* excl = pass_args.excl;
    uint32_t* lookback = pass_args.lookback;
    const uint32_t shift = pass_args.shift, digit_bits = pass_args.digit_bits;
    uint32_t* err = args.err;
    const uint32_t spin_limit = args.spin_limit;
    const uint32_t n = args.d_count ? min(*args.d_count, args.n_est) : args.n_est;
    const uint32_t ntiles = n / kTile + (n % kTile != 0 ? 1u : 0u);
    const uint32_t dmask = (1u << digit_bits) - 1u;
    const uint32_t lt = lanemask_lt();
    // Warp-striped: warp w owns a contiguous 32*kItems slice of a tile, item k of
    // lane j sits at slice + 32k + j, so processing k in order keeps the ranking
    // stable.
    const uint32_t first = warp * 32u * kItems + lane;
    uint32_t* my_hist = sm.warp_hist[warp];

    uint64_t key[kItems];
    auto tile_len = [&](uint32_t t) { return min((uint32_t)kTile, n - t * (uint32_t)kTile); };
    auto load_keys = [&](uint32_t t) {
        const uint64_t* src = keys_in + (size_t)t * kTile;
        const uint32_t len = tile_len(t);
        if (len == (uint32_t)kTile) {
#pragma unroll
            for (int k = 0; k < kItems; ++k) key[k] = __ldcs(src + first + 32 * k);
        } else {
#pragma unroll
            for (int k = 0; k < kItems; ++k) key[k] = first + 32u * k < len ? __ldcs(src + first + 32 * k) : ~0ull;
        }
    };
    // Whole tiles (all but the last) take a copy of the code without checks.
    auto pass = [&](uint32_t tile, auto whole) {
        constexpr bool kWhole = decltype(whole)::value;
        const uint32_t tile_n = tile_len(tile), tile_base = tile * (uint32_t)kTile;
        const uint32_t* tile_vals = vals_in ? vals_in + tile_base : nullptr;
#pragma unroll
        for (int k = 0; k < kItems; ++k)
            if (kWhole || first + 32u * k < tile_n) atomicAdd(&my_hist[digit_of(key[k], shift, dmask)], 1u);
        __syncthreads();

        // Thread d < 256 owns digit d: the tile's count, then the first slot of
        // each warp's keys of the digit inside the sorted tile.
        uint32_t* my_word = lookback + (size_t)tile * kRadix + tid;
        uint32_t tile_cnt = 0, tile_start = 0;
        if (tid < kRadix) {
#pragma unroll
            for (int w = 0; w < kBlockWarps; ++w) tile_cnt += sm.warp_hist[w][tid];
            st_relaxed_u32(my_word, (tile == 0 ? kLbInclusive : kLbAggregate) | tile_cnt);
            tile_start = tile_cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFullMask, tile_start, o);
                if (lane >= (uint32_t)o) tile_start += y;
            }
            if (lane == 31) sm.warp_sum[warp] = tile_start;
            tile_start -= tile_cnt;
        }
        __syncthreads();
        if (tid < kRadix) {
#pragma unroll
            for (int w = 0; w < kWarps; ++w) tile_start += w < (int)warp ? sm.warp_sum[w] : 0u;
            uint32_t run = tile_start;
#pragma unroll
            for (int w = 0; w < kBlockWarps; ++w) {
                const uint32_t c = sm.warp_hist[w][tid];
                sm.warp_hist[w][tid] = run;
                run += c;
            }
        }
        __syncthreads();

        uint32_t val[kItems], pos[kItems];
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            const bool valid = kWhole || first + 32u * k < tile_n;
            const uint32_t vmask = kWhole ? kFullMask : __ballot_sync(kFullMask, valid);
            pos[k] = warp_rank(my_hist, digit_of(key[k], shift, dmask), valid, vmask, lane, lt);
        }
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            const uint32_t i = first + 32u * k;
            val[k] = (kWhole || i < tile_n) ? (tile_vals ? __ldcs(tile_vals + i) : tile_base + i) : 0u;
        }
        if (tid < kRadix) {
            uint32_t prefix = 0;
            if (tile > 0) {
                prefix = lookback_window(lookback, tile, tid, err, kRadix, spin_limit);
                st_relaxed_u32(my_word, kLbInclusive | (prefix + tile_cnt));
            }
            // Slot i of the tile goes to out_base[its digit] + i (modulo 2^32).
            sm.out_base[tid] = excl[tid] + prefix - tile_start;
        }
        if (tid == 0) sm.next_tile = atomicAdd(tile_counter, 1u);
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            if (kWhole || first + 32u * k < tile_n) {
                sm.keys[pos[k]] = key[k];
                sm.vals[pos[k]] = val[k];
            }
        }
        __syncthreads();
        const uint32_t next = sm.next_tile;
        if (next < ntiles) load_keys(next);
#pragma unroll(kWhole ? kItems : 1)
        for (int k = 0; k < kItems; ++k) {
            const uint32_t i = tid + (uint32_t)k * kBlock;
            if (kWhole || i < tile_n) {
                const uint64_t key_i = sm.keys[i];
                const uint32_t o = sm.out_base[digit_of(key_i, shift, dmask)] + i;
                keys_out[o] = key_i;
                vals_out[o] = sm.vals[i];
            }
        }
        return next;
    };

    __syncthreads();
    uint32_t tile = sm.next_tile;
    if (tile >= ntiles) return;
    load_keys(tile);
    while (true) {
#pragma unroll
        for (int w = 0; w < 8; ++w) my_hist[32 * w + lane] = 0;
        __syncthreads();  // the stage and the counters are free
        tile = tile_len(tile) == (uint32_t)kTile ? pass(tile, std::true_type{}) : pass(tile, std::false_type{});
        if (tile >= ntiles) return;
    }
}

// ------------------------------------------------------------- fix-up ----
// Orders keys that are sorted, stably, by their top digits. Where a key's run (the
// neighbours that share these digits) begins and ends is read off a bit mask of
// the runs' heads; its place is the run's beginning plus the keys of the run that
// come before it. Like the passes, all of this looks at the low key_bits bits only:
// a caller may keep anything above them (kMasked: key_bits < 64; the masks in the
// inner loop cost 11 us at 16.7 M pairs). A key sees kFixHalo keys on each side of
// its tile, so all keys of a run agree whether it has more than kFixHalo of them; the
// first one then lists it for runs_kernel.
// 16.7 M pairs, two others a run on average: 109 us, bound by its instructions
// (384 MB are 59 us); scanning left and right from each key 119 us.
template <bool kMasked>
__global__ __launch_bounds__(kThreads) void fixup_kernel(SortArgs a) {
    constexpr uint32_t kKeys = kFixTile + 2 * kFixHalo;
    __shared__ uint64_t s_key[kKeys];
    __shared__ uint32_t s_head[kKeys / 32];
    static_assert(kKeys % kThreads == 0, "whole warps look for heads");
    const uint32_t w = a.counters[kScheduleWord], digits = a.counters[kScheduleWord + 1];
    const uint32_t m = w & 255u, top = w >> 8, tid = threadIdx.x;
    if (top == 0u) return;
    const uint32_t n = a.d_count ? min(*a.d_count, a.n_est) : a.n_est;
    const uint32_t begin = blockIdx.x * kFixTile;
    if (begin >= n) return;
    const uint32_t shift = 8u * ((digits >> (4u * (m - top))) & 15u);
    const uint64_t mask = kMasked ? key_mask(a.key_bits) : ~0ull;
    const uint32_t tile = min(kFixTile, n - begin);
    const uint32_t lead = min(begin, kFixHalo), count = lead + tile + min(n - begin - tile, kFixHalo);
    const uint64_t* src = a.keys_tmp + (begin - lead);
#pragma unroll
    for (uint32_t i = tid; i < kKeys; i += kThreads)
        if (i < count) s_key[i] = __ldcs(src + i);
    __syncthreads();
#pragma unroll
    for (uint32_t i = tid; i < kKeys; i += kThreads) {
        const bool head = i >= count || i == 0u || (((s_key[i] ^ s_key[i - 1]) & mask) >> shift) != 0ull;
        const uint32_t heads = __ballot_sync(kFullMask, head);
        if ((tid & 31u) == 0u) s_head[i / 32u] = heads;
    }
    __syncthreads();
    for (uint32_t i = lead + tid; i < lead + tile; i += kThreads) {
        const uint64_t key = s_key[i], low = key & mask;
        const uint32_t val = __ldcs(a.vals_tmp + (begin - lead) + i);
        uint32_t word = i / 32u;
        uint32_t bits = s_head[word] & (0xFFFFFFFFu >> (31u - (i & 31u)));
        while (bits == 0u) bits = s_head[--word];  // entry 0 is a head
        const uint32_t from = 32u * word + 31u - __clz(bits);
        word = i / 32u;
        bits = s_head[word] & ((0xFFFFFFFEu << (i & 31u)));
        while (bits == 0u && ++word < kKeys / 32u) bits = s_head[word];
        const uint32_t to = bits == 0u ? count : min(count, 32u * word + (uint32_t)__ffs(bits) - 1u);
        if (to - from > kFixHalo) {  // of those in sight
            if (from == i) {
                const uint32_t first = begin - lead + i, past = min(n, first + kRunMax);
                const bool too_long = past < n && (((src[i + kRunMax] ^ key) & mask) >> shift) == 0ull;
                atomicOr(a.counters + kScheduleWord + 4, too_long ? kStartOver : kLongRuns);
                if (!too_long) a.runs[atomicAdd(a.counters + kScheduleWord + 5, 1u)] = first;
            }
            continue;
        }
        // Keys of a run differ by less than 2^56: the sign of a difference
        // orders them. Equal keys before i count, those behind it do not.
        uint32_t place = from;
        for (uint32_t j = from; j < to; ++j)
            place += (uint32_t)(((s_key[j] & mask) - low - (j < i ? 1ull : 0ull)) >> 63);
        a.keys_out[begin - lead + place] = key;
        a.vals_out[begin - lead + place] = val;
    }
}

// The long runs, a block each: stable passes over the digits below the top ones,
// between the temporaries and the output, where a warp ranks a contiguous part of
// the run 32 keys at a time. The keys stay in L2 and the chain of loads bounds it:
// 7 us for a run of 500 keys, 36 for one of 5,000, three digits.
// Where all digits have to be sorted after all it empties the look-back words (the
// early passes', and the list, which stands where the fourth pass has its words).
__global__ __launch_bounds__(kRunThreads) void runs_kernel(SortArgs a, size_t words) {
    const uint32_t flags = a.counters[kScheduleWord + 4];
    if (flags == 0u) return;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    if (flags & kStartOver) {
        for (size_t i = (size_t)blockIdx.x * kRunThreads + tid; i < words; i += (size_t)gridDim.x * kRunThreads)
            a.lookback[i] = 0u;
        return;
    }
    constexpr uint32_t kRunWarps = kRunThreads / 32;
    __shared__ uint32_t s_hist[kRunWarps][kRadix];
    __shared__ uint32_t s_sum[kWarps];
    const uint32_t w = a.counters[kScheduleWord], digits = a.counters[kScheduleWord + 1];
    const uint32_t m = w & 255u, low = m - (w >> 8), listed = a.counters[kScheduleWord + 5];
    const uint32_t n = a.d_count ? min(*a.d_count, a.n_est) : a.n_est;
    const uint32_t top_shift = 8u * ((digits >> (4u * low)) & 15u);
    const uint64_t mask = key_mask(a.key_bits);
    const uint32_t lt = lanemask_lt();
    uint32_t* const my_hist = s_hist[warp];
    for (uint32_t r = blockIdx.x; r < listed; r += gridDim.x) {
        // Where the run ends: its keys are a prefix of what follows, so 1,024
        // places 32 apart and then 32 places tell. (What others do to their runs
        // leaves the top digits as they are.)
        const uint32_t first = a.runs[r];
        const uint64_t head = __ldcg(a.keys_tmp + first) & mask;
        const auto belongs = [&](uint32_t i) {
            return first + i < n && (((__ldcg(a.keys_tmp + first + i) & mask) ^ head) >> top_shift) == 0ull;
        };
        const uint32_t base = 32u * ((uint32_t)__syncthreads_count(belongs(32u * tid)) - 1u);
        const uint32_t len = base + __popc(__ballot_sync(kFullMask, belongs(base + lane)));
        const uint32_t part = (len + kRunThreads - 1u) / kRunThreads * 32u;  // a warp's share
        const uint32_t begin = min(len, warp * part), end = min(len, begin + part);
        __syncthreads();  // all have read before any key moves
        uint64_t *src = a.keys_tmp + first, *dst = a.keys_out + first;
        uint32_t *src_val = a.vals_tmp + first, *dst_val = a.vals_out + first;
        for (uint32_t d = 0; d < low; ++d) {
            const uint32_t shift = 8u * ((digits >> (4u * d)) & 15u);
#pragma unroll
            for (uint32_t k = 0; k < kRadix / 32u; ++k) my_hist[32u * k + lane] = 0u;
            __syncwarp();
            for (uint32_t i = begin + lane; i < end; i += 32u)
                atomicAdd(&my_hist[digit_of(__ldcg(src + i), shift, 0xFFu)], 1u);
            __syncthreads();
            uint32_t count = 0, incl = 0;
            if (tid < kRadix) {
                for (uint32_t k = 0; k < kRunWarps; ++k) count += s_hist[k][tid];
                incl = count;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
                    if (lane >= (uint32_t)o) incl += y;
                }
                if (lane == 31u) s_sum[warp] = incl;
            }
            __syncthreads();
            if (tid < kRadix) {
                uint32_t run = incl - count;
                for (uint32_t k = 0; k < warp; ++k) run += s_sum[k];
                for (uint32_t k = 0; k < kRunWarps; ++k) {
                    const uint32_t c = s_hist[k][tid];
                    s_hist[k][tid] = run;
                    run += c;
                }
            }
            __syncthreads();
            for (uint32_t i0 = begin; i0 < end; i0 += 32u) {
                const uint32_t i = i0 + lane;
                const bool valid = i < end;
                const uint64_t key = valid ? __ldcg(src + i) : 0ull;
                const uint32_t val = valid ? __ldcg(src_val + i) : 0u;
                const uint32_t at = warp_rank(my_hist, digit_of(key, shift, 0xFFu), valid,
                                              __ballot_sync(kFullMask, valid), lane, lt);
                if (valid) {
                    dst[at] = key;
                    dst_val[at] = val;
                }
            }
            __syncthreads();
            uint64_t* const k = src;
            src = dst, dst = k;
            uint32_t* const v = src_val;
            src_val = dst_val, dst_val = v;
        }
        if (src != a.keys_out + first)
            for (uint32_t i = tid; i < len; i += kRunThreads) {
                dst[i] = __ldcg(src + i);
                dst_val[i] = __ldcg(src_val + i);
            }
        __syncthreads();
    }
}

// Pass-kernel variants (threads, items per thread, blocks per SM). The numbers
// are settings that callers keep, so the last five, which once had kernels of
// their own, stand for the shapes that took their place.
struct PassVariant {
    int threads, items;
    void (*kernel)(SortArgs, uint32_t);
    size_t smem;
};
template <int kBlock, int kItems, int kMinBlocks>
constexpr PassVariant pass_variant() {
    return {kBlock, kItems, sort_pass_kernel<kBlock, kItems, kMinBlocks>, sizeof(PassSmem<kBlock, kItems>)};
}
const PassVariant kVariants[] = {
    pass_variant<256, 16, 2>(), pass_variant<384, 12, 2>(), pass_variant<512, 12, 1>(), pass_variant<256, 8, 4>(),
    pass_variant<256, 20, 2>(), pass_variant<256, 12, 3>(), pass_variant<256, 8, 3>(),  pass_variant<256, 12, 3>(),
    pass_variant<256, 8, 4>(),  pass_variant<256, 12, 3>(), pass_variant<256, 16, 2>(), pass_variant<256, 20, 2>(),
};
constexpr int kNumVariants = sizeof(kVariants) / sizeof(kVariants[0]);
constexpr int kMinItems = 8;  // sizes the look-back words for every variant
static_assert(kThreads * kMinItems == (int)kSortPlanTile, "look-back sizing");
int g_variant = -1;  // the variant that serves where the caller names none; negative: by the number of pairs
// Small tiles while they all run at once (with room for their registers: at four
// blocks an SM a tile takes longer), then fewer and larger ones, which have fewer
// earlier tiles to look back on. 63-bit keys, 8 a thread at three / four blocks, 16,
// us: 150,000 pairs 80 / 92 / 96; 350,000 98 / 107 / 98 (110 before the resident
// passes, which at four blocks were slower than those from 400,000 to 524,287);
// 524,288 106 / 119 / 102. 16 / 20 a thread: 2,097,152 236 / 253; 16,777,216 1128 / 1091.
int variant_for(uint32_t n) { return n < (1u << 19) ? 6 : (n < (1u << 23) ? 0 : 4); }

// Per-device set-up state: the pass kernels' shared-memory attribute is set
// once on each device that sorts, and the SM count is cached per device.
constexpr int kMaxDevices = 64;
bool g_init_done[kMaxDevices] = {};
int g_num_sms[kMaxDevices] = {};
int g_resident[kMaxDevices][kNumVariants] = {};  // blocks of each pass kernel the device holds
std::mutex g_init_mutex;

int current_device() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
    return dev;
}

int num_sms() {
    const int dev = current_device();
    std::lock_guard<std::mutex> lock(g_init_mutex);
    if (g_num_sms[dev] == 0) {
        int n = 0;
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        g_num_sms[dev] = n > 0 ? n : 1;
    }
    return g_num_sms[dev];
}

// Position of the error word inside the scratch (the counters come first,
// so the word sits at the same offset for every length and key width).
constexpr size_t kErrWord = 9;

}  // namespace

// Kernel attributes (the pass kernels' shared memory exceeds the 48 KB
// default), set once per device. Safe to call repeatedly and from several
// threads; called before any stream capture.
cudaError_t sort_init() {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_init_mutex);
    if (g_init_done[dev]) return cudaSuccess;
    for (int v = 0; v < kNumVariants; ++v) {
        e = cudaFuncSetAttribute(kVariants[v].kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kVariants[v].smem);
        if (e != cudaSuccess) return e;
        int per_sm = 0, sms = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kVariants[v].kernel, kVariants[v].threads,
                                                          kVariants[v].smem);
        if (e != cudaSuccess) return e;
        if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
        g_resident[dev][v] = std::max(1, per_sm * sms);
    }
    // Tuning knob for benchmarks: ASTRO_SORT_VARIANT selects a pass variant.
    if (const char* env = getenv("ASTRO_SORT_VARIANT")) {
        const int v = atoi(env);
        if (v >= 0 && v < kNumVariants) g_variant = v;
    }
    e = cudaFuncSetAttribute(sort_histogram_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(kHistCopies * kMaxPasses * kRadix * sizeof(uint32_t)));
    if (e == cudaSuccess) e = sort_small_init(dev);
    if (e == cudaSuccess) g_init_done[dev] = true;
    return e;
}

uint32_t sort_variant_count() { return (uint32_t)kNumVariants; }
uint32_t sort_shape_count() { return 7u; }

SortPlan sort_plan(uint32_t max_len, uint32_t key_bits) {
    SortPlan p{};
    p.passes = key_bits == 0 ? 1u : (key_bits + 7u) / 8u;
    p.tile = kSortPlanTile;
    p.ntiles = (uint32_t)(((uint64_t)max_len + p.tile - 1) / p.tile);
    size_t off = 0;
    // Zeroed at the start of every sort: counters (a block of 64 words),
    // histograms and look-back words.
    p.zero_begin = off;
    p.counters = off;
    off = align_up(off + 4ull * 64, 256);
    p.hist = off;
    off = align_up(off + 4ull * kMaxPasses * kRadix, 256);
    p.lookback = off;
    off = align_up(off + 4ull * p.passes * (size_t)std::max(p.ntiles, 1u) * kRadix, 256);
    p.zero_end = off;
    p.excl = off;
    off = align_up(off + 4ull * kMaxPasses * kRadix, 256);
    p.keys_tmp = off;
    off = align_up(off + 8ull * max_len, 256);
    p.vals_tmp = off;
    off = align_up(off + 4ull * max_len, 256);
    p.total = off;
    return p;
}

namespace {

bool overlaps(const void* a, size_t na, const void* b, size_t nb) {
    const uintptr_t x = (uintptr_t)a, y = (uintptr_t)b;
    return x < y + nb && y < x + na;
}

// The sort's kernels on the scratch `temp` (laid out by sort_plan). With
// `stall_first_tile` (test hook, one pass only) the first pass hands out
// tickets from 1, so tile 0 is never processed and every later tile's
// look-back waits on a word that nobody publishes until `spin_limit` polls.
cudaError_t sort_launch(const uint64_t* keys_in, const uint32_t* vals_in, uint64_t* keys_out,
                        uint32_t* vals_out, uint32_t n_est, const uint32_t* d_count,
                        uint32_t key_bits, void* temp, size_t temp_bytes, cudaStream_t st,
                        uint32_t* err, uint32_t variant, uint32_t spin_limit,
                        bool stall_first_tile) {
    if (n_est == 0) return cudaSuccess;
    const SortPlan plan = sort_plan(n_est, key_bits);
    if (temp_bytes < plan.total || key_bits > 64 || variant > (uint32_t)kNumVariants)
        return cudaErrorInvalidValue;
    if (stall_first_tile && plan.passes != 1) return cudaErrorInvalidValue;
    cudaError_t e0 = sort_init();
    if (e0 != cudaSuccess) return e0;
    if (!stall_first_tile && n_est <= sort_small_max(current_device())) {
        char* t = static_cast<char*>(temp);
        uint32_t* own = err ? nullptr : reinterpret_cast<uint32_t*>(t + plan.counters) + kErrWord;
        return sort_small(keys_in, vals_in, keys_out, vals_out, reinterpret_cast<uint64_t*>(t + plan.keys_tmp),
                          reinterpret_cast<uint32_t*>(t + plan.vals_tmp), n_est, d_count, key_bits,
                          current_device(), st, own);
    }
    const int vi = variant != 0 ? (int)variant - 1 : (g_variant >= 0 ? g_variant : variant_for(n_est));
    const PassVariant& pv = kVariants[vi];
    const uint32_t tile = (uint32_t)(pv.threads * pv.items);
    const uint32_t ntiles = (uint32_t)(((uint64_t)n_est + tile - 1) / tile);
    const uint32_t grid = std::min(ntiles, (uint32_t)g_resident[current_device()][vi]);
    char* base = static_cast<char*>(temp);
    uint64_t* keys_tmp = reinterpret_cast<uint64_t*>(base + plan.keys_tmp);
    uint32_t* vals_tmp = reinterpret_cast<uint32_t*>(base + plan.vals_tmp);
    uint32_t* excl = reinterpret_cast<uint32_t*>(base + plan.excl);
    uint32_t* hist = reinterpret_cast<uint32_t*>(base + plan.hist);
    uint32_t* counters = reinterpret_cast<uint32_t*>(base + plan.counters);
    uint32_t* lookback = reinterpret_cast<uint32_t*>(base + plan.lookback);
    if (!err) err = counters + kErrWord;
    cudaError_t e = cudaMemsetAsync(base + plan.zero_begin, 0, plan.zero_end - plan.zero_begin, st);
    if (e != cudaSuccess) return e;
    if (stall_first_tile) {
        // The ticket counter starts at 1 (its low byte set to 1).
        e = cudaMemsetAsync(counters + kTicketWord, 1, 1, st);
        if (e != cudaSuccess) return e;
    }
    const uint32_t hist_blocks = (uint32_t)std::min<uint64_t>(
        ((uint64_t)n_est + 4 * kThreads - 1) / (4 * kThreads), (uint64_t)num_sms() * kHistBlocksPerSm);
    // The passes may be reordered or left out only if no pass overwrites the
    // input (a caller may sort in place with an even number of passes).
    const bool apart = !overlaps(keys_in, 8ull * n_est, keys_out, 8ull * n_est) &&
                       !(vals_in && overlaps(vals_in, 4ull * n_est, vals_out, 4ull * n_est)) && !stall_first_tile;
    const bool try_top = apart && n_est >= kTopMin && plan.passes >= kTopDigits + kSavedPasses;
    const uint32_t early = try_top ? kTopDigits : 0u;
    const size_t hist_smem = std::max((size_t)kHistCopies * plan.passes * kRadix * sizeof(uint32_t),
                                      try_top ? (size_t)kSampleSlots * sizeof(uint32_t) : (size_t)0);
    sort_histogram_kernel<<<hist_blocks, kThreads, hist_smem, st>>>(keys_in, d_count, n_est, key_bits, plan.passes,
                                                                    hist, excl, counters, apart, try_top, keys_tmp);
    const size_t stride = (size_t)plan.ntiles * kRadix;
    const SortArgs args{keys_in,  vals_in, keys_tmp, keys_out, vals_tmp, vals_out, d_count, n_est,
                        key_bits, excl,    lookback, stride,   counters, early,    lookback + (size_t)kTopDigits * stride,
                        err,      spin_limit};
    // Where the top digits may suffice: as many passes, the fix-up, and launches
    // for all passes, which a schedule without top digits goes on with and a run that
    // is too long starts over with. A launch with nothing to do takes about 2 us.
    for (uint32_t l = 0; l < plan.passes + early; ++l) {
        if (try_top && l == early) {
            const uint32_t tiles = (n_est - 1u) / kFixTile + 1u;
            if (key_bits < 64u) fixup_kernel<true><<<tiles, kThreads, 0, st>>>(args);
            else fixup_kernel<false><<<tiles, kThreads, 0, st>>>(args);
            runs_kernel<<<2 * num_sms(), kRunThreads, 0, st>>>(args, plan.passes * stride);
        }
        pv.kernel<<<grid, pv.threads, pv.smem, st>>>(args, l);
    }
    return cudaGetLastError();
}

}  // namespace

cudaError_t sort_pairs(const uint64_t* keys_in, const uint32_t* vals_in, uint64_t* keys_out,
                       uint32_t* vals_out, uint32_t n_est, const uint32_t* d_count,
                       uint32_t key_bits, void* temp, size_t temp_bytes, cudaStream_t st,
                       uint32_t* err, uint32_t variant) {
    return sort_launch(keys_in, vals_in, keys_out, vals_out, n_est, d_count, key_bits, temp,
                       temp_bytes, st, err, variant, kSpinLimit, false);
}

cudaError_t sort_pairs_stalled(const uint64_t* keys_in, uint64_t* keys_out, uint32_t* vals_out,
                               uint32_t n, uint32_t key_bits, void* temp, size_t temp_bytes,
                               uint32_t spin_limit, cudaStream_t st) {
    return sort_launch(keys_in, nullptr, keys_out, vals_out, n, nullptr, key_bits, temp, temp_bytes,
                       st, nullptr, 0, spin_limit, true);
}

int sort_status(const void* temp, cudaStream_t st) {
    if (!temp) return ASTRO_ERR_INVALID_ARGUMENT;
    if (cudaStreamSynchronize(st) != cudaSuccess) {
        (void)cudaGetLastError();
        return ASTRO_ERR_CUDA;
    }
    uint32_t* word = reinterpret_cast<uint32_t*>(static_cast<char*>(const_cast<void*>(temp)) +
                                                 sort_plan(0, 8).counters) + kErrWord;
    uint32_t v = 0;
    if (cudaMemcpy(&v, word, sizeof(v), cudaMemcpyDeviceToHost) != cudaSuccess) {
        (void)cudaGetLastError();
        return ASTRO_ERR_CUDA;
    }
    if (v == 0) return ASTRO_OK;
    if (cudaMemset(word, 0, sizeof(uint32_t)) != cudaSuccess) {
        (void)cudaGetLastError();
        return ASTRO_ERR_CUDA;
    }
    return (v & kErrLookbackTimeout) ? ASTRO_ERR_DEVICE_TIMEOUT : ASTRO_ERR_DEVICE_OVERFLOW;
}

}  // namespace astro

extern "C" int astro_radix_sort_temp_bytes(uint32_t max_length, uint32_t key_bits, size_t* bytes) {
    if (!bytes || key_bits > 64) return ASTRO_ERR_INVALID_ARGUMENT;
    *bytes = astro::sort_plan(max_length, key_bits).total;
    return ASTRO_OK;
}

// MetalKernelsRadixSort.sort (Astro/RadixSort.swift:98-105): input/inputIndices
// are read, output/outputIndices receive the sorted pairs, estimatedLength
// sizes the launch and actualCountBuffer (d_actual_count) holds the count.
// On the NULL stream the call waits for the sort and returns its device
// status; on any other stream astro_radix_sort_status reads it later.
extern "C" int astro_radix_sort(const uint64_t* d_input, const uint32_t* d_input_indices,
                                uint64_t* d_output, uint32_t* d_output_indices,
                                uint32_t estimated_length, const uint32_t* d_actual_count,
                                uint32_t key_bits, void* d_temp, size_t temp_bytes, void* stream) {
    if (estimated_length == 0) return ASTRO_OK;  // RadixSort.swift:106
    if (!d_input || !d_output || !d_output_indices || !d_temp || key_bits > 64)
        return ASTRO_ERR_INVALID_ARGUMENT;
    if ((const void*)d_input == (const void*)d_output ||
        (const void*)d_input_indices == (const void*)d_output_indices)
        return ASTRO_ERR_INVALID_ARGUMENT;
    if (temp_bytes < astro::sort_plan(estimated_length, key_bits).total) return ASTRO_ERR_CAPACITY;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e = astro::sort_pairs(d_input, d_input_indices, d_output, d_output_indices,
                                      estimated_length, d_actual_count, key_bits, d_temp,
                                      temp_bytes, st, nullptr);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return ASTRO_ERR_CUDA;
    }
    return st == nullptr ? astro::sort_status(d_temp, st) : ASTRO_OK;
}

extern "C" int astro_radix_sort_status(const void* d_temp, void* stream) {
    return astro::sort_status(d_temp, static_cast<cudaStream_t>(stream));
}

extern "C" int astro_test_sort_lookback_timeout(const uint64_t* d_input, uint64_t* d_output,
                                                uint32_t* d_output_indices, uint32_t n,
                                                uint32_t key_bits, uint32_t spin_limit,
                                                void* d_temp, size_t temp_bytes, void* stream) {
    if (!d_input || !d_output || !d_output_indices || n == 0 || key_bits == 0 || key_bits > 8 ||
        spin_limit == 0 || spin_limit > astro::kSpinLimit)
        return ASTRO_ERR_INVALID_ARGUMENT;
    if ((const void*)d_input == (const void*)d_output) return ASTRO_ERR_INVALID_ARGUMENT;
    if (!d_temp && astro::noalloc_scratch(&d_temp, &temp_bytes) != cudaSuccess) {
        (void)cudaGetLastError();
        return ASTRO_ERR_CUDA;
    }
    if (temp_bytes < astro::sort_plan(n, key_bits).total) return ASTRO_ERR_CAPACITY;
    cudaError_t e = astro::sort_pairs_stalled(d_input, d_output, d_output_indices, n, key_bits, d_temp,
                                              temp_bytes, spin_limit, static_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return ASTRO_ERR_CUDA;
    }
    return ASTRO_OK;
}
