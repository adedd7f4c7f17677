// sort.cu -- device-wide exclusive scans and the stable LSD radix sort of (key, value)
// pairs used by the grid builders.
//
// Replaces the reference's CUB wrappers: ExclusiveScan (Scan.cu:39-58) and RadixSort
// (Sort.cu:31-53, cub::DeviceRadixSort::SortPairs over uint32 keys/values).
//
// Design: reduce-then-scan in every pass (tile digit counts, their scan over the tiles,
// rank and scatter), so no kernel waits on another CTA and nothing spins.  All element counts are read from device memory, so
// the whole pipeline is enqueued without a host round trip; grids are sized from the
// host-side capacity and surplus CTAs exit at once.
#include "hr_internal.h"
#include "hr_block.cuh"
#include "radix_tile.cuh"

namespace hr {

namespace {

// ----------------------------------------------------------------------------------
// generic exclusive scan: reduce -> scan partials -> apply

template <class T>
__global__ __launch_bounds__(kThreads) void k_scan_reduce(const T* __restrict__ data, const uint32_t* d_count,
                                                          T* partials) {
    const uint32_t n = *d_count;
    const size_t base = (size_t)blockIdx.x * kTile;
    T s = zero<T>();
    if (base < n) {
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            size_t i = base + threadIdx.x + (size_t)k * kThreads;
            if (i < n) s = s + data[i];
        }
    }
    T total;
    block_excl_scan<T, kThreads>(s, &total);
    if (threadIdx.x == 0) partials[blockIdx.x] = total;
}

// One CTA scans `n` partials (exclusive, in place); the grand total goes to d_total_*.
// If cap > 0 and the total exceeds it, `ovf_bit` is or-ed into *ovf.
template <class T>
__global__ __launch_bounds__(1024) void k_scan_partials(T* partials, uint32_t n, uint32_t* d_total_x,
                                                        uint32_t* d_total_y, uint32_t* ovf,
                                                        uint32_t cap_x, uint32_t ovf_bit_x,
                                                        uint32_t cap_y, uint32_t ovf_bit_y);

template <>
__global__ __launch_bounds__(1024) void k_scan_partials<uint32_t>(uint32_t* partials, uint32_t n,
                                                                  uint32_t* d_total_x, uint32_t*,
                                                                  uint32_t* ovf, uint32_t cap_x,
                                                                  uint32_t ovf_bit_x, uint32_t, uint32_t) {
    uint32_t carry = 0;
    for (uint32_t b = 0; b < n; b += 1024) {
        uint32_t i = b + threadIdx.x;
        uint32_t x = i < n ? partials[i] : 0u;
        uint32_t tot;
        uint32_t ex = block_excl_scan<uint32_t, 1024>(x, &tot);
        if (i < n) partials[i] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) {
        if (d_total_x) *d_total_x = carry;
        if (ovf && cap_x && carry > cap_x) atomicOr(ovf, ovf_bit_x);
    }
}

template <>
__global__ __launch_bounds__(1024) void k_scan_partials<uint2>(uint2* partials, uint32_t n, uint32_t* d_total_x,
                                                               uint32_t* d_total_y, uint32_t* ovf,
                                                               uint32_t cap_x, uint32_t ovf_bit_x,
                                                               uint32_t cap_y, uint32_t ovf_bit_y) {
    uint2 carry = make_uint2(0u, 0u);
    for (uint32_t b = 0; b < n; b += 1024) {
        uint32_t i = b + threadIdx.x;
        uint2 x = i < n ? partials[i] : make_uint2(0u, 0u);
        uint2 tot;
        uint2 ex = block_excl_scan<uint2, 1024>(x, &tot);
        if (i < n) partials[i] = carry + ex;
        carry = carry + tot;
    }
    if (threadIdx.x == 0) {
        if (d_total_x) *d_total_x = carry.x;
        if (d_total_y) *d_total_y = carry.y;
        if (ovf && cap_x && carry.x > cap_x) atomicOr(ovf, ovf_bit_x);
        if (ovf && cap_y && carry.y > cap_y) atomicOr(ovf, ovf_bit_y);
    }
}

template <class T>
__global__ __launch_bounds__(kThreads) void k_scan_apply(T* data, const uint32_t* d_count, const T* partials) {
    const uint32_t n = *d_count;
    const size_t base = (size_t)blockIdx.x * kTile;
    if (base >= n) return;
    // blocked arrangement: thread j owns items base + j*kItems .. +kItems
    T v[kItems];
    T s = zero<T>();
    const size_t b0 = base + (size_t)threadIdx.x * kItems;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        v[k] = (b0 + k < n) ? data[b0 + k] : zero<T>();
        s = s + v[k];
    }
    T total;
    T run = block_excl_scan<T, kThreads>(s, &total) + partials[blockIdx.x];
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        if (b0 + k < n) data[b0 + k] = run;
        run = run + v[k];
    }
}

// ----------------------------------------------------------------------------------
// radix sort kernels: tiles of 256 x ITEMS keys, digits of up to BITS bits.  Tile counts are
// stored tile by tile (nd = 2^digit bits words each), so that a tile writes and reads its
// counts in one run.  (The single-launch build keeps the steps of radix_tile.cuh, whose
// tiles of 2048 keys suit its few pairs.)

// The run of equal digits among neighbouring lanes that this lane begins, as a lane mask; 0
// when the lane before it holds the same digit.  A mesh's pairs come with many equal
// digits side by side, and a run then costs one shared-memory atomic.
__device__ __forceinline__ uint32_t digit_run(uint32_t dig) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t prev = __shfl_up_sync(kFullMask, dig, 1);
    const bool head = lane == 0u || prev != dig;
    const uint32_t after = __ballot_sync(kFullMask, head) & (0xfffffffeu << lane);
    return head ? ((after & (0u - after)) - 1u) & (0xffffffffu << lane) : 0u;
}

// tile digit counts, an add per run of equal digits
template <int BITS, int ITEMS>
__global__ __launch_bounds__(kThreads) void k_radix_count(const uint32_t* __restrict__ keys, const uint32_t* d_count,
                                                          int shift, uint32_t mask, uint32_t* __restrict__ tile_hist) {
    __shared__ uint32_t h[1 << BITS];
    const uint32_t n = *d_count;
    const size_t base = (size_t)blockIdx.x * (kThreads * ITEMS);
    if (base >= n) return;
    for (uint32_t d = threadIdx.x; d <= mask; d += kThreads) h[d] = 0u;
    uint32_t key[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const size_t i = base + threadIdx.x + (size_t)k * kThreads;
        key[k] = i < n ? __ldg(keys + i) : 0u;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const bool valid = base + threadIdx.x + (size_t)k * kThreads < n;
        const uint32_t dig = valid ? (key[k] >> shift) & mask : 0xffffffffu, run = digit_run(dig);
        if (valid && run) atomicAdd(&h[dig], (uint32_t)__popc(run));
    }
    __syncthreads();
    uint32_t* out = tile_hist + (size_t)blockIdx.x * (mask + 1u);
    for (uint32_t d = threadIdx.x; d <= mask; d += kThreads) out[d] = h[d];
}

// exclusive scan of the tile counts of each digit over the tiles, in place, and the digit
// totals.  Latency bounds it: a block takes 8 digits (one sector of each tile's counts, so
// that 256 digits reach 32 SMs), cuts the tiles into 128 runs and keeps the first 12 counts
// of a run, all there are up to 1536 tiles, in registers between the sum and the store.
// (32 digits a block, 32 runs and two reads of each count: kernels of a 2M-triangle rebuild
// 0.353 ms, now 0.339; 1M 0.208 and 0.195; 300k uniform 0.105 and 0.094.)
constexpr uint32_t kScanDigits = 8;
template <int ITEMS>
__global__ __launch_bounds__(1024) void k_radix_scan(uint32_t* __restrict__ tile_hist, const uint32_t* d_count, uint32_t nd,
                                                     uint32_t* __restrict__ row_total) {
    __shared__ uint32_t s[32][kScanDigits + 1];
    constexpr uint32_t kRuns = 1024u / kScanDigits, kRows = 12;   // loads in flight per thread
    const uint32_t ntiles = (uint32_t)(((size_t)*d_count + kThreads * ITEMS - 1) / (kThreads * ITEMS));
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5, dl = lane % kScanDigits;
    const uint32_t d = blockIdx.x * kScanDigits + dl, g = threadIdx.x / kScanDigits;
    const uint32_t chunk = (ntiles + kRuns - 1u) / kRuns, t0 = min(g * chunk, ntiles);
    const uint32_t t1 = d < nd ? min(t0 + chunk, ntiles) : t0;
    uint32_t* col = tile_hist + d;
    auto load = [&](uint32_t (&x)[kRows], uint32_t t) {
#pragma unroll
        for (uint32_t k = 0; k < kRows; ++k) x[k] = t + k < t1 ? __ldcg(col + (size_t)(t + k) * nd) : 0u;
    };
    uint32_t x0[kRows], x[kRows], sum = 0;
    load(x0, t0);
#pragma unroll
    for (uint32_t k = 0; k < kRows; ++k) sum += x0[k];
    for (uint32_t t = t0 + kRows; t < t1; t += kRows) {
        load(x, t);
#pragma unroll
        for (uint32_t k = 0; k < kRows; ++k) sum += x[k];
    }
    // the runs of a digit before this one: those of this warp, then the warps before it
    uint32_t inc = sum;
#pragma unroll
    for (uint32_t o = kScanDigits; o < 32u; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFullMask, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane >= 32u - kScanDigits) s[w][dl] = inc;
    __syncthreads();
    if (w < kScanDigits) {   // a warp scans a digit's 32 warp totals
        const uint32_t v = s[lane][w];
        uint32_t y, z = v;
#pragma unroll
        for (uint32_t o = 1; o < 32u; o <<= 1) {
            y = __shfl_up_sync(kFullMask, z, o);
            if (lane >= o) z += y;
        }
        s[lane][w] = z - v;
        if (lane == 31u && blockIdx.x * kScanDigits + w < nd) row_total[blockIdx.x * kScanDigits + w] = z;
    }
    __syncthreads();
    uint32_t run = s[w][dl] + (inc - sum);
    auto store = [&](const uint32_t (&x)[kRows], uint32_t t) {
#pragma unroll
        for (uint32_t k = 0; k < kRows; ++k) {
            if (t + k < t1) col[(size_t)(t + k) * nd] = run;
            run += x[k];
        }
    };
    store(x0, t0);
    for (uint32_t t = t0 + kRows; t < t1; t += kRows) {
        load(x, t);
        store(x, t);
    }
}

// stable rank and scatter of a tile: a key goes to its digit's start (the totals scanned
// here) plus the tile's scanned count plus its rank among the tile's keys of the digit.
//
// Ranks within a warp's row of 32 keys come alternately from two pipes, because each alone
// bounds the kernel: a match of the digits holds its pipe for 32 cycles a warp, and the
// other way, each run of equal digits oring its lanes into the digit's word (whose set bits
// below a lane are its rank), costs about 15 shared-memory cycles.  All three passes over
// 4.87M leaf pairs of a 2M-triangle mesh / 4.8M random keys of 23 bits: every row by match
// 203 / 258 us, by oring 219 / 218, in turn 205 / 222 (tiles of 2048 keys 209 / 239; the kernel
// before, by match over 512 counters, 209 / 337).  511k pairs: tiles of 2048 keys 92 us, 4096
// 103; 158k 52 and 62; 2.1M 134 and 130, so the line lies where both sizes fill the GPU.
template <int BITS, int ITEMS>
__global__ __launch_bounds__(kThreads, 4) void k_radix_scatter(
    const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in, uint32_t* __restrict__ keys_out,
    uint32_t* __restrict__ vals_out, const uint32_t* d_count, int shift, uint32_t mask,
    const uint32_t* __restrict__ tile_hist, const uint32_t* __restrict__ row_total) {
    constexpr int ND = 1 << BITS, TILE = kThreads * ITEMS, DPT = ND / kThreads > 0 ? ND / kThreads : 1;
    extern __shared__ __align__(16) unsigned char s_raw[];   // ranks, then the sorted tile
    uint2(*s_rank)[ND] = reinterpret_cast<uint2(*)[ND]>(s_raw);
    uint2* s_kv = reinterpret_cast<uint2*>(s_raw);
    __shared__ uint32_t s_goff[ND];   // digit's place in the output, minus its place in the tile

    const uint32_t n = *d_count;
    const size_t base = (size_t)blockIdx.x * TILE;
    if (base >= n) return;
    const uint32_t nvalid = (uint32_t)min((size_t)TILE, n - base);
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5, lt = (1u << lane) - 1u;
    uint32_t key[ITEMS];
    const uint32_t li0 = w * 32u * ITEMS + lane;
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const uint32_t li = li0 + (uint32_t)r * 32u;
        key[r] = li < nvalid ? __ldg(keys_in + base + li) : 0u;
    }
    for (uint32_t i = threadIdx.x; i < (uint32_t)(kWarps * ND); i += kThreads) (&s_rank[0][0])[i] = make_uint2(0u, 0u);
    // digit starts: exclusive scan of the totals (DPT consecutive digits per thread)
    {
        uint32_t t[DPT], sum = 0, all;
#pragma unroll
        for (int j = 0; j < DPT; ++j) {
            const uint32_t d = threadIdx.x * DPT + j;
            t[j] = d <= mask ? __ldg(row_total + d) : 0u;
            sum += t[j];
        }
        uint32_t ex = block_excl_scan<uint32_t, kThreads>(sum, &all);
        const uint32_t* col = tile_hist + (size_t)blockIdx.x * (mask + 1u);
#pragma unroll
        for (int j = 0; j < DPT; ++j) {
            const uint32_t d = threadIdx.x * DPT + j;
            if (d <= mask) s_goff[d] = ex + __ldg(col + d);
            ex += t[j];
        }
    }
    __syncthreads();
    uint32_t rank[ITEMS];
    uint2* const mine = s_rank[w];
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const bool valid = li0 + (uint32_t)r * 32u < nvalid;
        const uint32_t dig = (key[r] >> shift) & mask;
        if (r & 1) {
            const uint32_t run = digit_run(valid ? dig : 0xffffffffu);
            if (valid && run) atomicOr(&mine[dig].x, run);
            __syncwarp();
            uint2 q = make_uint2(0u, 0u);
            if (valid) q = mine[dig];
            rank[r] = q.y + __popc(q.x & lt);
            __syncwarp();
            if (valid && (q.x & lt) == 0u) mine[dig] = make_uint2(0u, q.y + __popc(q.x));   // the digit's first lane
            __syncwarp();
        } else {
            const uint32_t peers = __match_any_sync(kFullMask, valid ? dig : 0xffffffffu);
            uint32_t b = 0;
            if (valid) b = mine[dig].y;
            rank[r] = b + __popc(peers & lt);
            __syncwarp();
            if (valid && (peers & lt) == 0u) mine[dig].y = b + __popc(peers);
            __syncwarp();
        }
    }
    __syncthreads();
    // per digit: the tile-local start plus the prefix over the warps, where its keys rank
    // from; and what leads from there to its place in the output
    {
        uint32_t c[DPT][kWarps], sum = 0, all;
#pragma unroll
        for (int j = 0; j < DPT; ++j) {
            const uint32_t d = threadIdx.x * DPT + j;
#pragma unroll
            for (int ww = 0; ww < kWarps; ++ww) {
                c[j][ww] = d <= mask ? s_rank[ww][d].y : 0u;
                sum += c[j][ww];
            }
        }
        uint32_t ex = block_excl_scan<uint32_t, kThreads>(sum, &all);
#pragma unroll
        for (int j = 0; j < DPT; ++j) {
            const uint32_t d = threadIdx.x * DPT + j;
            if (d <= mask) {
                s_goff[d] -= ex;
#pragma unroll
                for (int ww = 0; ww < kWarps; ++ww) {
                    s_rank[ww][d].y = ex;
                    ex += c[j][ww];
                }
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; ++r)
        if (li0 + (uint32_t)r * 32u < nvalid) rank[r] += mine[(key[r] >> shift) & mask].y;
    __syncthreads();   // the ranks are read: the buffer takes the sorted tile
#pragma unroll
    for (int r = 0; r < ITEMS; ++r)
        if (li0 + (uint32_t)r * 32u < nvalid)
            s_kv[rank[r]] = make_uint2(key[r], __ldg(vals_in + base + li0 + (uint32_t)r * 32u));
    __syncthreads();
#pragma unroll 4
    for (uint32_t j = threadIdx.x; j < nvalid; j += kThreads) {
        const uint2 q = s_kv[j];
        const uint32_t at = s_goff[(q.x >> shift) & mask] + j;
        keys_out[at] = q.x;
        vals_out[at] = q.y;
    }
}

}  // namespace

// ----------------------------------------------------------------------------------
// host launchers

size_t scan_partials_words(size_t cap_count) { return (cap_count + kTile - 1) / kTile + 1; }

int exclusive_scan_u32(hr_ctx* c, uint32_t* data, const uint32_t* d_count, size_t cap_count,
                       uint32_t* d_total, uint32_t* partials, cudaStream_t s) {
    const uint32_t nb = (uint32_t)((cap_count + kTile - 1) / kTile);
    if (nb == 0) return 0;
    c->launches += 3;
    k_scan_reduce<uint32_t><<<nb, kThreads, 0, s>>>(data, d_count, partials);
    k_scan_partials<uint32_t><<<1, 1024, 0, s>>>(partials, nb, d_total, nullptr, nullptr, 0, 0, 0, 0);
    k_scan_apply<uint32_t><<<nb, kThreads, 0, s>>>(data, d_count, partials);
    return cuda_check(c, cudaGetLastError(), "exclusive_scan_u32");
}

int exclusive_scan_u32x2(hr_ctx* c, uint2* data, const uint32_t* d_count, size_t cap_count,
                         uint32_t* d_total_x, uint32_t* d_total_y, uint2* partials, cudaStream_t s) {
    const uint32_t nb = (uint32_t)((cap_count + kTile - 1) / kTile);
    if (nb == 0) return 0;
    c->launches += 3;
    k_scan_reduce<uint2><<<nb, kThreads, 0, s>>>(data, d_count, partials);
    k_scan_partials<uint2><<<1, 1024, 0, s>>>(partials, nb, d_total_x, d_total_y, nullptr, 0, 0, 0, 0);
    k_scan_apply<uint2><<<nb, kThreads, 0, s>>>(data, d_count, partials);
    return cuda_check(c, cudaGetLastError(), "exclusive_scan_u32x2");
}

// scan of per-block pair counts written by the count kernels (in place, exclusive).
// A total above `cap` sets `ovf_bit`, stores the total in *d_req and publishes a zero
// count, so every later stage of the build sees no work.
__global__ __launch_bounds__(1024) void k_scan_block_sums(uint32_t* sums, uint32_t n, uint32_t* d_total,
                                                          uint32_t* ovf, uint32_t cap, uint32_t ovf_bit,
                                                          uint32_t* d_req) {
    // 8 consecutive counts per thread, 8192 per round
    constexpr uint32_t kIpt = 8, kChunk = 1024 * kIpt;
    uint64_t carry = 0;
    for (uint32_t b = 0; b < n; b += kChunk) {
        const uint32_t i0 = b + threadIdx.x * kIpt;
        uint32_t x[kIpt], s = 0;
#pragma unroll
        for (uint32_t k = 0; k < kIpt; ++k) {
            x[k] = i0 + k < n ? sums[i0 + k] : 0u;
            s += x[k];
        }
        uint32_t tot;
        uint32_t run = (uint32_t)carry + block_excl_scan<uint32_t, 1024>(s, &tot);
#pragma unroll
        for (uint32_t k = 0; k < kIpt; ++k) {
            if (i0 + k < n) sums[i0 + k] = run;
            run += x[k];
        }
        carry += tot;
    }
    if (threadIdx.x == 0) {
        if (carry > cap) {
            atomicOr(ovf, ovf_bit);
            *d_req = carry > 0xffffffffull ? 0xffffffffu : (uint32_t)carry;
            *d_total = 0u;
        } else {
            *d_total = (uint32_t)carry;
        }
    }
}

int scan_block_sums(hr_ctx* c, uint32_t* sums, uint32_t n, uint32_t* d_total, uint32_t* ovf,
                    uint32_t cap, uint32_t ovf_bit, uint32_t* d_req, cudaStream_t s) {
    k_scan_block_sums<<<1, 1024, 0, s>>>(sums, n, d_total, ovf, cap, ovf_bit, d_req);
    return cuda_check(c, cudaGetLastError(), "scan_block_sums");
}

// fewest passes of at most max_db-bit digits, the bits spread evenly over them (the
// context path takes 9-bit digits: 17-18-bit cell keys sort in two passes, not three)
static void radix_plan(int key_bits, int max_db, int* passes, int* db) {
    if (key_bits < 1) key_bits = 1;
    if (key_bits > 32) key_bits = 32;
    *passes = (key_bits + max_db - 1) / max_db;
    *db = (key_bits + *passes - 1) / *passes;
}

constexpr int kMaxDigitBits = 9;   // context sorts; the allocation-free sort keeps 8 (its static scratch)

int radix_sort_passes(int key_bits) {
    int passes, db;
    radix_plan(key_bits, kMaxDigitBits, &passes, &db);
    return passes;
}

// tiles of 4096 keys halve the counts and the per-tile work, but need more keys to fill the GPU:
// four tiles of 2048 per SM (see k_radix_scatter)
int radix_items(const hr_ctx* c, size_t n, int last) {
    const size_t line = (size_t)c->num_sms * 4u * kTile;
    return n >= (last == 16 ? line - line / 8u : line) ? 16 : 8;
}

size_t radix_tile_hist_words(size_t cap_count, int key_bits) {
    int passes, db;
    radix_plan(key_bits, kMaxDigitBits, &passes, &db);
    size_t ntiles = (cap_count + kTile - 1) / kTile;   // the smaller tiles
    if (ntiles == 0) ntiles = 1;
    return ntiles * ((size_t)1 << db);
}

// one pass: counts, scan, scatter
template <int BITS, int ITEMS>
static cudaError_t radix_pass(const uint32_t* sk, const uint32_t* sv, uint32_t* dk, uint32_t* dv, const uint32_t* d_count,
                              size_t cap_count, int shift, uint32_t mask, uint32_t* tile_hist, uint32_t* row_total,
                              cudaStream_t s) {
    constexpr size_t rank = sizeof(uint2) * kWarps * (1 << BITS), sort = sizeof(uint32_t) * 2 * kThreads * ITEMS;
    constexpr size_t smem = rank > sort ? rank : sort;
    const uint32_t ntiles = (uint32_t)((cap_count + kThreads * ITEMS - 1) / (kThreads * ITEMS));
    k_radix_count<BITS, ITEMS><<<ntiles, kThreads, 0, s>>>(sk, d_count, shift, mask, tile_hist);
    k_radix_scan<ITEMS><<<(mask + kScanDigits) / kScanDigits, 1024, 0, s>>>(tile_hist, d_count, mask + 1u, row_total);
    k_radix_scatter<BITS, ITEMS><<<ntiles, kThreads, smem, s>>>(sk, sv, dk, dv, d_count, shift, mask, tile_hist, row_total);
    return cudaGetLastError();
}

// all passes of a plan with digits of at most max_db bits
static cudaError_t radix_passes(const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_tmp, uint32_t* vals_tmp,
                                uint32_t* keys_out, uint32_t* vals_out, const uint32_t* d_count, size_t cap_count,
                                int key_bits, int max_db, int items, uint32_t* tile_hist, uint32_t* row_total, cudaStream_t s,
                                uint64_t* launches) {
    int passes, db;
    radix_plan(key_bits, max_db, &passes, &db);
    const uint32_t mask = (1u << db) - 1u;
    if (cap_count == 0) return cudaSuccess;
    const uint32_t* sk = keys_in;
    const uint32_t* sv = vals_in;
    for (int p = 0; p < passes; ++p) {
        const bool last = p == passes - 1;
        uint32_t* dk = last ? keys_out : ((p % 2 == 0) ? keys_tmp : const_cast<uint32_t*>(keys_in));
        uint32_t* dv = last ? vals_out : ((p % 2 == 0) ? vals_tmp : const_cast<uint32_t*>(vals_in));
        auto pass = db <= 8 ? (items == 16 ? radix_pass<8, 16> : radix_pass<8, 8>)
                            : (items == 16 ? radix_pass<9, 16> : radix_pass<9, 8>);
        const cudaError_t e = pass(sk, sv, dk, dv, d_count, cap_count, p * db, mask, tile_hist, row_total, s);
        if (e != cudaSuccess) return e;
        if (launches) *launches += 3;
        sk = dk;
        sv = dv;
    }
    return cudaSuccess;
}

int radix_sort_pairs(hr_ctx* c, const uint32_t* keys_in, const uint32_t* vals_in,
                     uint32_t* keys_tmp, uint32_t* vals_tmp, uint32_t* keys_out, uint32_t* vals_out,
                     const uint32_t* d_count, size_t cap_count, int key_bits,
                     uint32_t* tile_hist, size_t tile_hist_bytes, uint32_t* row_total, cudaStream_t s, int items) {
    // the histogram holds 2^digit words per tile: fewer key bits can need more of them
    if (radix_tile_hist_words(cap_count, key_bits) * sizeof(uint32_t) > tile_hist_bytes)
        return set_error(c, 4, "radix sort: histogram of %zu bytes is too small for %zu keys of %d bits",
                         tile_hist_bytes, cap_count, key_bits);
    return cuda_check(c, radix_passes(keys_in, vals_in, keys_tmp, vals_tmp, keys_out, vals_out, d_count, cap_count, key_bits,
                                      kMaxDigitBits, items ? items : radix_items(c, cap_count), tile_hist, row_total, s,
                                      &c->launches), "radix_sort_pairs");
}

// Same pass sequence as radix_sort_pairs, without a context (no status text, no launch
// count); used by the allocation-free entry point, whose 2^20 pairs at most take the smaller tiles.
cudaError_t radix_sort_pairs_raw(const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_tmp,
                                 uint32_t* vals_tmp, uint32_t* keys_out, uint32_t* vals_out,
                                 const uint32_t* d_count, size_t cap_count, int key_bits, uint32_t* tile_hist,
                                 uint32_t* row_total, cudaStream_t s) {
    return radix_passes(keys_in, vals_in, keys_tmp, vals_tmp, keys_out, vals_out, d_count, cap_count, key_bits, 8, 8,
                        tile_hist, row_total, s, nullptr);
}

}  // namespace hr
