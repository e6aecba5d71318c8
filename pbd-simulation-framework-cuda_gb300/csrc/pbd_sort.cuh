// pbd_sort.cuh -- stable LSD radix sort of (Morton key, particle index) pairs.
//
// Replaces cub::DeviceRadixSort::SortPairs (kernel/SortReorder.h:39-47, temp storage
// :221-238).  CUB's sort is a stable LSD radix sort; this one is too, so the permutation is
// the one any stable sort by the uint32 key gives (checked bit for bit against the oracle).
//
// Design (one kernel per 8-bit digit, "onesweep" style):
//  - The digit histograms of every pass are counted once, fused into the predict kernel
//    (shared-memory histograms flushed with one global atomic per non-empty bin).
//  - Each pass kernel takes a tile of keys (sort_plan).  Tiles are numbered by an atomic
//    counter in launch order, so a tile only ever waits on tiles that are already running.
//  - Inside a tile every warp ranks its items (stable: item order is warp, then register slot,
//    then lane) from one ballot per digit bit; warp counts are scanned per digit in shared memory.
//  - Tile digit counts are chained across tiles with decoupled look-back (status word =
//    2 flag bits + 30 count bits), kLookBack words in flight at a time.  Every wait is bounded:
//    after SortScratch::spin_limit polls without progress (kSpinLimit by default, a few seconds)
//    the tile records PBD device error bit kErrSortTimeout and carries on, so a lost predecessor
//    can never hang the GPU.  For tests of that path, SortScratch::hold makes the first tile of
//    every pass withhold its status (a predecessor that never publishes): every wait on it runs out.
//  - Keys are scattered to shared memory in tile order first, then written out so that
//    each digit's run lands on consecutive global addresses.
//
// What bounds it: the serial chain inside a tile (load, rank item after item through the warp's
// counts, scan, look back, scatter, write), not DRAM (16 B per key and pass).  So a tile has 512
// threads with few items each and the ranks come from ballots (__match_any_sync cost ~200 cycles an
// item).  Three passes, back to back, GB300: 1,000,000 keys 64 -> 46 us, 600,001 keys 47 -> 35,
// 262,144 keys 42 -> 29, 33,000 keys 35 -> 21, 4,275 keys 31 -> 19 (256 threads x 16 items with
// __match_any_sync and one status word per look-back step, against the present passes).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace pbd {

constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;
constexpr int kMaxPasses = 4;
constexpr int kSortThreads = 512;          // threads 0..255 own a digit each
constexpr int kLookBack = 8;               // status words a look-back step reads (16 and 4: the same time)
// Keys per tile: the smallest of 1,024 / 2,048 / 4,096 that needs at most one tile per SM (152), as
// a tile's time grows with its items per thread (262,144 keys, three passes: 4 items 28 us, 8 items
// 33, 2 items and two tiles per SM 33); beyond that 6,656 keys, the most that fit in static shared
// memory with 16 warps (1,000,000 keys: 151 tiles, 46 us against 52 with 245 tiles of
// 4,096; 4,000,000 keys: 121 us against 126).
constexpr uint32_t kSortSpread = 152;
constexpr int kSortItemsMax = 13;
struct SortPlan {
    int items;        // keys per thread
    uint32_t ntiles;
};
inline SortPlan sort_plan(uint32_t n) {
    for (int items : {2, 4, 8})
        if (n <= kSortSpread * (uint32_t)(kSortThreads * items))
            return SortPlan{items, (n + kSortThreads * items - 1) / (uint32_t)(kSortThreads * items)};
    return SortPlan{kSortItemsMax, (n + kSortThreads * kSortItemsMax - 1) / (uint32_t)(kSortThreads * kSortItemsMax)};
}
// Status rows that sort_plan needs at most for up to `capacity` keys.
inline uint32_t sort_max_tiles(uint32_t capacity) {
    const uint32_t t = sort_plan(capacity).ntiles;
    return t > kSortSpread ? t : kSortSpread;
}
constexpr uint32_t kFlagAggregate = 1u << 30;
constexpr uint32_t kFlagPrefix = 2u << 30;
constexpr uint32_t kValueMask = (1u << 30) - 1u;
constexpr uint32_t kSpinLimit = 1u << 22;

// device error word bits
constexpr uint32_t kErrSortTimeout = 1u << 0;
constexpr uint32_t kErrKeyBits = 1u << 1;

struct SortScratch {
    uint32_t* hist;          // [kMaxPasses][kRadix] digit counts of the whole array
    uint32_t* status;        // [kMaxPasses][max_tiles][kRadix] look-back words
    uint32_t* tile_counter;  // [kMaxPasses]
    uint32_t* err;           // device error word
    uint32_t max_tiles;
    uint32_t spin_limit = kSpinLimit;   // polls of one look-back wait before it gives up
    uint32_t hold = 0;                  // 1: the first tile of each pass never publishes (tests)
    uint32_t key_bits = 32;             // only bits [0, key_bits) order the keys
};

// The digit of `key` in pass `pass`, counting only the bits below key_bits.
__device__ __forceinline__ uint32_t sort_digit(uint32_t key, int pass, uint32_t key_bits) {
    const uint32_t shift = (uint32_t)pass * kRadixBits;
    const uint32_t bits = key_bits - shift;          // >= 1 for every pass the sort runs
    const uint32_t mask = bits >= (uint32_t)kRadixBits ? (uint32_t)(kRadix - 1) : ((1u << bits) - 1u);
    return (key >> shift) & mask;
}

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Count a key's digits into the block's histograms sh[pass][digit].  All lanes of a warp call it; `valid`
// lanes count.  kCoherent: neighbouring keys mostly share their upper digits (Morton keys of particles
// in last frame's order), where 32 lanes adding to one word took 32 turns: the lanes that hold the first
// lane's digit are counted with one add.
template <bool kCoherent>
__device__ __forceinline__ void count_digits(uint32_t* sh, uint32_t key, bool valid, int npasses, uint32_t key_bits) {
    const uint32_t any = __ballot_sync(0xffffffffu, valid);
    if (any == 0u) return;
    const uint32_t lane = threadIdx.x & 31u, lead = (uint32_t)__ffs(any) - 1u;
    for (int ps = 0; ps < npasses; ++ps) {
        const uint32_t d = sort_digit(key, ps, key_bits);
        if (kCoherent && ps > 0) {
            const uint32_t d0 = __shfl_sync(0xffffffffu, d, lead);
            const uint32_t same = __ballot_sync(0xffffffffu, valid && d == d0);
            if (lane == lead) atomicAdd(&sh[ps * kRadix + d0], (uint32_t)__popc(same));
            else if (valid && d != d0) atomicAdd(&sh[ps * kRadix + d], 1u);
        } else if (valid) {
            atomicAdd(&sh[ps * kRadix + d], 1u);
        }
    }
}

// One LSD pass over digit `pass` (bits 8*pass .. 8*pass+7).  kFirst: values are the
// identity (initializeParticleIds, SortReorder.h:199-210) and are generated, not loaded.
template <bool kFirst, int kItems>
__global__ void __launch_bounds__(kSortThreads)
onesweep_pass(const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin,
              uint32_t* __restrict__ kout, uint32_t* __restrict__ vout, uint32_t n, int pass,
              SortScratch S) {
    constexpr int kThreads = kSortThreads, kWarps = kThreads / 32;
    constexpr int kTile = kThreads * kItems;
    static_assert(kThreads >= kRadix && kTile <= 65535, "thread d < 256 owns digit d; tile counts are 16-bit");
    __shared__ uint16_t s_whist[kWarps][kRadix];
    __shared__ uint32_t s_keys[kTile];
    __shared__ uint32_t s_vals[kTile];
    __shared__ uint32_t s_goff[kRadix];
    __shared__ uint32_t s_start[kRadix];
    __shared__ uint32_t s_wtot[2][kRadix / 32];
    __shared__ uint32_t s_tile;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_tile = atomicAdd(&S.tile_counter[pass], 1u);
    for (int k = tid; k < kWarps * kRadix / 2; k += kThreads) reinterpret_cast<uint32_t*>(&s_whist[0][0])[k] = 0u;
    const uint32_t hist = tid < kRadix ? S.hist[pass * kRadix + tid] : 0u;
    __syncthreads();
    const uint32_t tile = s_tile;
    // The previous pass has finished (stream order): clear its look-back row for this tile.
    if (pass > 0 && tid < kRadix) S.status[((size_t)(pass - 1) * S.max_tiles + tile) * kRadix + tid] = 0u;

    const uint32_t base = tile * (uint32_t)kTile;
    uint32_t key[kItems], val[kItems], rank[kItems];
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const uint32_t idx = base + warp * (32 * kItems) + k * 32 + lane;
        const bool valid = idx < n;
        key[k] = valid ? kin[idx] : 0xFFFFFFFFu;
        val[k] = kFirst ? idx : (valid ? vin[idx] : 0u);
    }
    // ---- warp-level stable ranking: the lanes holding the same digit from one ballot per bit
    uint16_t* wh = s_whist[warp];
    const uint32_t lt = lanemask_lt();
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const uint32_t idx = base + warp * (32 * kItems) + k * 32 + lane;
        const bool valid = idx < n;
        const uint32_t digit = sort_digit(key[k], pass, S.key_bits);
        uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
        for (int b = 0; b < kRadixBits; ++b) {
            const uint32_t ones = __ballot_sync(0xffffffffu, (digit >> b) & 1u);
            peers &= ((digit >> b) & 1u) ? ones : ~ones;
        }
        const uint32_t before = valid ? wh[digit] : 0u;
        __syncwarp();
        if (valid && (peers & lt) == 0u) wh[digit] = (uint16_t)(before + __popc(peers));
        __syncwarp();
        rank[k] = before + __popc(peers & lt);
    }
    __syncthreads();
    // ---- per digit (thread d): warp offsets and the tile's count, published for the tiles after
    // this one; then one scan over the digits of both the tile's counts and the whole array's
    uint32_t* st = S.status + (size_t)pass * S.max_tiles * kRadix;
    const uint32_t d = tid;
    uint32_t run = 0, rx = 0, hx = 0;
    if (tid < kRadix) {
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const uint32_t c = s_whist[w][d];
            s_whist[w][d] = (uint16_t)run;
            run += c;
        }
        if (!(tile == 0 && S.hold)) st_relaxed(&st[(size_t)tile * kRadix + d], (tile == 0 ? kFlagPrefix : kFlagAggregate) | run);
        rx = run;
        hx = hist;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t a = __shfl_up_sync(0xffffffffu, rx, o), b = __shfl_up_sync(0xffffffffu, hx, o);
            if (lane >= o) { rx += a; hx += b; }
        }
        if (lane == 31) { s_wtot[0][warp] = rx; s_wtot[1][warp] = hx; }
        rx -= run;
        hx -= hist;
    }
    __syncthreads();
    if (tid < kRadix) {
#pragma unroll
        for (int w = 0; w < kRadix / 32 - 1; ++w)
            if (w < warp) { rx += s_wtot[0][w]; hx += s_wtot[1][w]; }
        // ---- look back over the tiles before this one, kLookBack status words in flight at a time
        uint32_t excl = 0, spins = 0;
        int t = (int)tile - 1;
        while (t >= 0) {
            uint32_t w[kLookBack];
#pragma unroll
            for (int k = 0; k < kLookBack; ++k) w[k] = t >= k ? ld_relaxed(&st[(size_t)(t - k) * kRadix + d]) : 0u;
            int taken = 0;
            bool done = false, open = true;
#pragma unroll
            for (int k = 0; k < kLookBack; ++k) {
                open = open && !done && (w[k] >> 30) != 0u;
                if (open) {
                    excl += w[k] & kValueMask;
                    ++taken;
                    done = (w[k] >> 30) == 2u;
                }
            }
            if (done) break;
            t -= taken;
            if (taken != 0) { spins = 0; continue; }
            if (++spins > S.spin_limit) {
                atomicOr(S.err, kErrSortTimeout);
                break;
            }
            __nanosleep(32);
        }
        if (tile != 0) st_relaxed(&st[(size_t)tile * kRadix + d], kFlagPrefix | ((excl + run) & kValueMask));
        s_goff[d] = hx + excl - rx;
        s_start[d] = rx;
    }
    __syncthreads();
    // ---- scatter to shared memory in tile order
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const uint32_t idx = base + warp * (32 * kItems) + k * 32 + lane;
        if (idx < n) {
            const uint32_t digit = sort_digit(key[k], pass, S.key_bits);
            const uint32_t pos = s_start[digit] + s_whist[warp][digit] + rank[k];
            s_keys[pos] = key[k];
            s_vals[pos] = val[k];
        }
    }
    __syncthreads();
    const uint32_t tile_n = (n - base) < (uint32_t)kTile ? (n - base) : (uint32_t)kTile;
    for (uint32_t i = tid; i < tile_n; i += kThreads) {
        const uint32_t kk = s_keys[i];
        const uint32_t o = s_goff[sort_digit(kk, pass, S.key_bits)] + i;
        if (o < n) {            // always true unless a look-back wait gave up (error word set)
            kout[o] = kk;
            vout[o] = s_vals[i];
        }
    }
}

template <int kItems>
inline void launch_sort_pass(cudaStream_t st, uint32_t ntiles, bool first, const uint32_t* kin, const uint32_t* vin,
                             uint32_t* kout, uint32_t* vout, uint32_t n, int pass, const SortScratch& S) {
    if (first) onesweep_pass<true, kItems><<<ntiles, kSortThreads, 0, st>>>(kin, vin, kout, vout, n, pass, S);
    else onesweep_pass<false, kItems><<<ntiles, kSortThreads, 0, st>>>(kin, vin, kout, vout, n, pass, S);
}
// Queue pass `pass` of a sort of n keys (the values of the first pass are the identity).
inline void sort_pass(cudaStream_t st, const SortPlan& plan, const uint32_t* kin, const uint32_t* vin, uint32_t* kout,
                      uint32_t* vout, uint32_t n, int pass, const SortScratch& S) {
    const auto launch = plan.items == 2 ? launch_sort_pass<2> : plan.items == 4 ? launch_sort_pass<4>
                        : plan.items == 8 ? launch_sort_pass<8> : launch_sort_pass<kSortItemsMax>;
    launch(st, plan.ntiles, pass == 0, kin, vin, kout, vout, n, pass, S);
}


// All passes of a sort of few keys by one block: the keys stay in registers and shared memory, ranked as
// in onesweep_pass, and no pass waits for a launch, a histogram or another tile.  kin may be kout; *err,
// when given, is cleared.  Bound by its serial steps, ~2 us a pass with 1,024 keys, ~4 with 4,096.
constexpr int kSmallThreads = 1024;
template <int kItems>
constexpr uint32_t sort_small_smem() { return (uint32_t)kSmallThreads * kItems * 6u + 32u * kRadix * 2u; }
template <int kItems>
__global__ void __launch_bounds__(kSmallThreads)
sort_small_kernel(const uint32_t* kin, uint32_t* kout, uint32_t* vout, uint32_t n, int npasses, uint32_t key_bits,
                  uint32_t* err) {
    constexpr int kTile = kSmallThreads * kItems, kWarps = kSmallThreads / 32;
    static_assert(kTile <= 65536, "values and counts are 16-bit");
    extern __shared__ uint32_t s_keys[];
    uint16_t* s_vals = reinterpret_cast<uint16_t*>(s_keys + kTile);
    uint16_t (*s_whist)[kRadix] = reinterpret_cast<uint16_t (*)[kRadix]>(s_vals + kTile);
    __shared__ uint32_t s_start[kRadix], s_wtot[kRadix / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t first = warp * (32 * kItems) + lane, lt = lanemask_lt();
    if (err && tid == 0) *err = 0u;
    uint32_t key[kItems], val[kItems];
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const uint32_t idx = first + k * 32;
        key[k] = idx < n ? kin[idx] : 0xFFFFFFFFu;
        val[k] = idx;
    }
    uint16_t* wh = s_whist[warp];
    for (int pass = 0; pass < npasses; ++pass) {
        uint32_t rank[kItems];
#pragma unroll
        for (int b = 0; b < kRadix / 64; ++b) reinterpret_cast<uint32_t*>(wh)[b * 32 + lane] = 0u;
        __syncwarp();
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            const bool valid = first + k * 32 < n;
            const uint32_t digit = sort_digit(key[k], pass, key_bits);
            uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
            for (int b = 0; b < kRadixBits; ++b) {
                const uint32_t ones = __ballot_sync(0xffffffffu, (digit >> b) & 1u);
                peers &= ((digit >> b) & 1u) ? ones : ~ones;
            }
            const uint32_t before = valid ? wh[digit] : 0u;
            __syncwarp();
            if (valid && (peers & lt) == 0u) wh[digit] = (uint16_t)(before + __popc(peers));
            __syncwarp();
            rank[k] = before + __popc(peers & lt);
        }
        __syncthreads();
        uint32_t run = 0, rx = 0;
        if (tid < kRadix) {   // thread d: the warps' offsets of digit d and its count
            uint32_t c[kWarps];
#pragma unroll
            for (int w = 0; w < kWarps; ++w) c[w] = s_whist[w][tid];
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
                s_whist[w][tid] = (uint16_t)run;
                run += c[w];
            }
            rx = run;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t a = __shfl_up_sync(0xffffffffu, rx, o);
                if (lane >= o) rx += a;
            }
            if (lane == 31) s_wtot[warp] = rx;
        }
        __syncthreads();
        if (tid < kRadix) {
            rx -= run;
#pragma unroll
            for (int w = 0; w < kRadix / 32 - 1; ++w)
                if (w < warp) rx += s_wtot[w];
            s_start[tid] = rx;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kItems; ++k)
            if (first + k * 32 < n) {
                const uint32_t digit = sort_digit(key[k], pass, key_bits);
                const uint32_t pos = s_start[digit] + s_whist[warp][digit] + rank[k];
                s_keys[pos] = key[k];
                s_vals[pos] = (uint16_t)val[k];
            }
        __syncthreads();
        if (pass + 1 == npasses) break;
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            const uint32_t idx = first + k * 32;
            key[k] = idx < n ? s_keys[idx] : 0xFFFFFFFFu;
            val[k] = idx < n ? s_vals[idx] : 0u;
        }
    }
    for (uint32_t i = tid; i < n; i += kSmallThreads) {
        kout[i] = s_keys[i];
        vout[i] = s_vals[i];
    }
}
// Most keys of one block's sort.  A sort by itself (three passes, 21 bits), the tiles' passes against one
// block: 1,000 keys 17.4 / 7.1 us, 4,097 23.6 / (4,096) 14.3, 8,192 23.6 / 22.5 with eight keys per thread, 12,000
// 23.6 / 39 with sixteen.  Inside a frame, where the passes overlap their launches and the histogram comes
// with the keys: 1,000 particles 47.0 -> 43.6 us per frame, 2,016 48.1 -> 45.4, but 4,096 68.7 against 70.5.
constexpr uint32_t kSortSmall = 4096;
constexpr uint32_t kSortSmallFrame = 2048;
template <int kItems>
inline void launch_sort_small(cudaStream_t st, const uint32_t* kin, uint32_t* kout, uint32_t* vout, uint32_t n, int npasses,
                              uint32_t key_bits, uint32_t* err) {
    static_assert(sort_small_smem<kItems>() <= 46u * 1024u, "with the static part below the 48 KB every kernel may take");
    sort_small_kernel<kItems><<<1, kSmallThreads, sort_small_smem<kItems>(), st>>>(kin, kout, vout, n, npasses, key_bits, err);
}
// Queue a whole sort of n <= kSortSmall keys.
inline void sort_small(cudaStream_t st, const uint32_t* kin, uint32_t* kout, uint32_t* vout, uint32_t n, int npasses, uint32_t key_bits,
                       uint32_t* err) {
    const auto launch = n <= 1024u ? launch_sort_small<1> : n <= 2048u ? launch_sort_small<2> : launch_sort_small<4>;
    launch(st, kin, kout, vout, n, npasses, key_bits, err);
}

}  // namespace pbd
