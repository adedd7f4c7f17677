// hr_block.cuh -- CTA-wide scan helpers shared by the build and sort kernels.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace hr {

constexpr unsigned kFullMask = 0xffffffffu;

__device__ __forceinline__ uint2 operator+(uint2 a, uint2 b) { return make_uint2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ uint2 operator-(uint2 a, uint2 b) { return make_uint2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ uint32_t shfl_up(uint32_t x, int o) { return __shfl_up_sync(kFullMask, x, o); }
__device__ __forceinline__ uint2 shfl_up(uint2 x, int o) {
    return make_uint2(__shfl_up_sync(kFullMask, x.x, o), __shfl_up_sync(kFullMask, x.y, o));
}
template <class T> __device__ __forceinline__ T zero();
template <> __device__ __forceinline__ uint32_t zero<uint32_t>() { return 0u; }
template <> __device__ __forceinline__ uint2 zero<uint2>() { return make_uint2(0u, 0u); }

// Exclusive scan of one value per thread across a CTA of NT threads; returns the
// exclusive prefix and writes the CTA total to *total.
template <class T, int NT>
__device__ __forceinline__ T block_excl_scan(T x, T* total) {
    __shared__ T s_w[NT / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T inc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T y = shfl_up(inc, o);
        if (lane >= o) inc = inc + y;
    }
    if (lane == 31) s_w[w] = inc;
    __syncthreads();
    if (w == 0) {
        T v = lane < NT / 32 ? s_w[lane] : zero<T>();
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            T y = shfl_up(v, o);
            if (lane >= o) v = v + y;
        }
        if (lane < NT / 32) s_w[lane] = v;
    }
    __syncthreads();
    T before = w > 0 ? s_w[w - 1] : zero<T>();
    *total = s_w[NT / 32 - 1];
    __syncthreads();
    return before + (inc - x);
}

// Largest k in [0, NT) with off[k] <= j, for a non-decreasing off[] (off[0] = 0 <= j): the
// item whose output run [off[k], off[k + 1]) holds output j of a block.
template <int NT>
__device__ __forceinline__ int block_owner(const uint32_t* off, uint32_t j) {
    int k = 0;
#pragma unroll
    for (int step = NT / 2; step > 0; step >>= 1)
        if (off[k + step] <= j) k += step;
    return k;
}

// One item's run of (cell key, value) pairs: the cells of an ex x ey x ez box, x fastest,
// then y, then z, keyed key0 + dx + dy * sx + dz * sxy, all with value val.
struct PairRun { uint32_t key0, ex, ey, sx, sxy, val; };

// Adds every key of a warp's lanes to counts[key * CS], neighbouring lanes with the same key
// together: a mesh's pairs come with equal keys side by side, and a crowded cell then costs
// few atomics.  A warp of many runs whose keys also come back 12 lanes on (triangles of a few
// crowded cells in turn) adds each key once, by match: two-level builds of 100k triangles that
// alternate between two cells 129 us by runs alone, 103 so, 116 by match in every warp.  Without
// the look 12 lanes on, the match would also meet the ground plane's long runs of different
// keys (2M triangles 303 -> 312 us).  Lanes without a key pass valid = false; called by all
// lanes.
template <int CS>
__device__ __forceinline__ void count_keys(uint32_t key, bool valid, uint32_t* __restrict__ counts) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t prev = __shfl_up_sync(kFullMask, key, 1);
    const uint32_t pv = __shfl_up_sync(kFullMask, valid ? 1u : 0u, 1);
    const bool head = lane == 0u || prev != key || (pv != 0u) != valid;
    const uint32_t heads = __ballot_sync(kFullMask, head);
    if (__popc(heads) > 16 &&
        __popc(__ballot_sync(kFullMask, __shfl_up_sync(kFullMask, key, 12) == key && lane >= 12u)) >= 5) {
        const uint32_t peers = __match_any_sync(kFullMask, key);
        if (valid && lane == (uint32_t)__ffs(peers) - 1u) atomicAdd(counts + (size_t)key * CS, (uint32_t)__popc(peers));
        return;
    }
    const uint32_t after = heads & (0xfffffffeu << lane);
    const uint32_t end = after ? (uint32_t)__ffs(after) - 1u : 32u;
    if (valid && head) atomicAdd(counts + (size_t)key * CS, end - lane);
}

// Writes a block's pairs with all its threads: the runs follow one another in thread order
// from out0, and pair j of the block is stored by thread j mod NT, so consecutive threads
// store consecutive slots.  Blocks of short runs (at most kShortRun cells each, STAGE pairs
// together) put them together in shared memory, every thread its own run in turn; in the
// others, whose runs may be thousands of cells long, each thread finds the run of every pair
// it stores by binary search and two divisions.  (2M-triangle key-frame rebuild 0.368 -> 0.353
// ms with the staged blocks, the counts per run of equal keys instead of by match, and the
// staged vertex records of k_count_pairs.)  n is this thread's run length, run is read
// when n > 0.  Every thread of the block calls it.
// With `counts`, also adds every written key to counts[key * CS] (a histogram of the keys).
constexpr uint32_t kShortRun = 32u;
template <int NT, int CS = 1, uint32_t STAGE = 2048u>
__device__ __forceinline__ void block_write_runs(uint32_t n, const PairRun& run, uint32_t out0,
                                                 uint32_t* __restrict__ keys, uint32_t* __restrict__ vals,
                                                 uint32_t* __restrict__ counts = nullptr) {
    __shared__ union {
        struct { uint32_t off[NT]; PairRun run[NT]; } r;
        uint2 pair[STAGE];
    } sh;
    uint32_t tot;
    const uint32_t off = block_excl_scan<uint32_t, NT>(n, &tot);
    const uint32_t lane = threadIdx.x & 31u;
    if (__syncthreads_or(n > kShortRun) == 0 && tot <= STAGE) {
        if (n) {
            uint32_t key = run.key0, x = 0, y = 0;
            uint32_t row = run.key0, plane = run.key0;
            for (uint32_t l = 0; l < n; ++l) {
                sh.pair[off + l] = make_uint2(key, run.val);
                ++key;
                if (++x == run.ex) {
                    x = 0;
                    row += run.sx;
                    if (++y == run.ey) {
                        y = 0;
                        plane += run.sxy;
                        row = plane;
                    }
                    key = row;
                }
            }
        }
        __syncthreads();
        for (uint32_t j0 = threadIdx.x - lane; j0 < tot; j0 += NT) {   // warp-uniform trip count
            const uint32_t j = j0 + lane;
            const uint2 q = j < tot ? sh.pair[j] : make_uint2(0xffffffffu, 0u);
            if (j < tot) {
                keys[out0 + j] = q.x;
                vals[out0 + j] = q.y;
            }
            if (counts) count_keys<CS>(q.x, j < tot, counts);
        }
        return;
    }
    sh.r.off[threadIdx.x] = off;
    if (n) sh.r.run[threadIdx.x] = run;
    __syncthreads();
    for (uint32_t j0 = threadIdx.x - lane; j0 < tot; j0 += NT) {
        const uint32_t j = j0 + lane;
        const bool valid = j < tot;
        uint32_t key = 0xffffffffu;
        if (valid) {
            const int k = block_owner<NT>(sh.r.off, j);
            const PairRun q = sh.r.run[k];
            const uint32_t l = j - sh.r.off[k];
            key = q.key0;
            if (l) {
                const uint32_t a = l / q.ex, z = a / q.ey;
                key += (l - a * q.ex) + (a - z * q.ey) * q.sx + z * q.sxy;
            }
            keys[out0 + j] = key;
            vals[out0 + j] = q.val;
        }
        if (counts) count_keys<CS>(key, valid, counts);
    }
}


}  // namespace hr

namespace hr {
// largest s in [0, n) with off[s] <= x, for ascending off with off[0] = 0
__device__ __forceinline__ uint32_t find_segment(const uint32_t* __restrict__ off, uint32_t n, uint32_t x) {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1u) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(off + mid) <= x) lo = mid;
        else hi = mid;
    }
    return lo;
}
}  // namespace hr
