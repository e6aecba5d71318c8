// pbd_passes.cuh -- the neighbour passes of a frame.
//
// The reference builds an explicit N x M list once per frame (findContacts +
// findNeighbours, kernel/Collision.h:11-160) and every density/vorticity/viscosity kernel
// loops over it (kernel/Density.h).  Here the frame's first lambda pass walks the cells in
// exactly the order the list would hold them (27 cells with the x offset outer and z inner,
// then the shells of findNeighbours), skipping self and stopping at the cap M, and stores the
// result (the full list); later passes read the stored lists, so sums run in the list's order.
//
// Each pass is split into a per-candidate contribution (`contrib`) and an in-order
// accumulation (`add`); a visitor may also name per-neighbour data (`Extra`, loaded by
// `fetch(j)`) that the walkers load together with the neighbour's position.  These walkers
// drive them:
//  - walk_seq: one thread per particle over the cells;
//  - walk_coop: one warp per particle.  Lanes evaluate 32 candidates at once and the
//    contributions are added in list order through shuffles, so the result is bit-identical
//    to walk_seq.  It takes the particles whose walk meets a cell range longer than
//    kLongRange -- in practice the range that SortReorder.h:183-184 extends to N (up to M
//    entries) -- which would otherwise serialise a whole warp behind one thread;
//  - walk_full, walk_near: one thread per particle over a stored list;
//  - walk_list_warp: one warp per particle over a stored list (the long lists, LongLists);
//  - walk_group_sums: G lanes per particle over a stored list (small simulations).
#pragma once
#include <type_traits>
#include "pbd_device.cuh"
#include "../../include/pbd.h"

namespace pbd {

// Per-neighbour data a visitor loads with the neighbour's position: V::Extra and V::fetch(j)
// when the visitor declares them, nothing otherwise.
struct NoExtra {};
template <class V, class = void> struct ExtraOf { using type = NoExtra; static constexpr bool has = false; };
template <class V> struct ExtraOf<V, std::void_t<typename V::Extra>> {
    using type = typename V::Extra;
    static constexpr bool has = true;
};
template <class V>
__device__ __forceinline__ typename ExtraOf<V>::type fetch_extra(const V& vis, uint32_t j) {
    if constexpr (ExtraOf<V>::has) return vis.fetch(j);
    else return NoExtra{};
}
template <class V>
__device__ __forceinline__ typename V::Contrib contrib_of(V& vis, uint32_t j, const float4& pj,
                                                          const typename ExtraOf<V>::type& ex, bool contact) {
    if constexpr (ExtraOf<V>::has) return vis.contrib(j, pj, ex, contact);
    else return vis.contrib(j, pj, contact);
}

// Two float4 side by side (32-byte aligned), in one load.
struct alignas(32) Pair4 { float4 a, b; };
__device__ __forceinline__ Pair4 load_pair(const Pair4* p) {
    Pair4 r;
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(r.a.x), "=f"(r.a.y), "=f"(r.a.z), "=f"(r.a.w), "=f"(r.b.x), "=f"(r.b.y), "=f"(r.b.z), "=f"(r.b.w) : "l"(p));
    return r;
}

constexpr uint32_t kLongRange = 32;
constexpr uint32_t kFullMask = 0xffffffffu;

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }
__device__ __forceinline__ float shfl_f(float v, int k) { return __shfl_sync(kFullMask, v, k); }
__device__ __forceinline__ uint32_t shfl_u(uint32_t v, int k) { return __shfl_sync(kFullMask, v, k); }
__device__ __forceinline__ uint32_t lanemask_lt_u() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Particles whose walk is handed to the warp-cooperative kernel.
struct DeferList {
    uint32_t* items;
    uint32_t* count;
    uint32_t* done;
    uint32_t cap;
};

// Stored lists, both in the reference's list order.
//  - The full list: the frame's first lambda pass walks the cells once (the cells come from the
//    frame's anchors, so the list is fixed for the frame) and stores every entry, up to the cap
//    M; the later lambda passes, omega and vorticity read it instead of the cell tables.
//  - The near list: a lambda or omega pass keeps the entries within the cut (r^2 < cut2 at the
//    positions it read); the pass right after it reads the same positions (delta after lambda,
//    viscosity after omega), so every entry left out adds an exact zero there and the short
//    list gives the full walk's sums bit for bit.
// A particle whose list does not fit (or whose walk met a long cell range) has its list stored by
// a warp (LongLists), or walks the cells when those are full.
constexpr uint32_t kListOff = 0x80000000u;   // meta: no list here (a full list's meta: | kListWalked | its set slot)
constexpr uint32_t kListWalked = 0x40000000u;   // with kListOff: the first lambda pass walked this particle itself
// The full list holds four entries side by side (entry k of particle i at full_at): a pass that
// reads every entry takes four indices per load and steps one address per four entries, a third
// fewer instructions outside the arithmetic than one load per entry.  The near list is slot-major
// (slot k of particle i at k * stride + i): its readers stop after ~6 entries, its writers run side
// by side in the slot.
struct NbList {
    uint32_t* list;      // near list: kmax x stride; full list: full_slots(kmax) x stride
    uint32_t* meta;      // per particle: count | contacts << 8, or kListOff
    uint32_t stride;
    uint32_t kmax;       // <= 255
};
__host__ __device__ __forceinline__ uint32_t full_slots(uint32_t kmax) { return (kmax + 3u) & ~3u; }
__device__ __forceinline__ uint32_t* full_at(const NbList& F, uint32_t i, uint32_t k) {
    return F.list + ((size_t)(k >> 2) * F.stride + i) * 4u + (k & 3u);
}
// The lists of the particles without a full list (the set DF, slot q of the set at row q): stored
// once per frame by the warp that finishes their first lambda pass, read by a warp in every pass
// after it.  Walking the cells again in each pass cost two dependent table loads and a position
// load per cell, one cell after the other (125 cells with two shells): on a 152k-particle dense
// frame the 125 particles around the cell-end range held up every pass by 100 us and more.
constexpr uint32_t kLongSlots = 8192;   // rows (16 MB); particles beyond them walk the cells
constexpr uint32_t kLongMax = 512;      // entries of a row: config.txt's list cap
struct LongLists {
    uint32_t* list;      // slots x kLongMax
    uint32_t* meta;      // per row: count | contacts << 16, or kListOff (longer than kLongMax)
    uint32_t slots;
};

// Enumerate the non-empty cell ranges [s, e) of particle i's list in the reference's
// order.  f(s, e, contact) returns true to stop; end_contacts(n) marks the end of the
// 27-cell part (Collision.h:38-39).  `pi` is the particle's anchor: its predicted position
// right after the frame's re-order, from which the reference builds the list once per frame
// (findContacts/findNeighbours run before the solver loop, Fluid.cu:41-47); passes later in
// the frame use the moved positions for the physics but the anchor's cells.
template <class F, class G>
__device__ __forceinline__ void for_each_range(const DevParams& P, const SceneCtx& S, float4 pi, const uint32_t* __restrict__ cs,
                                               const uint32_t* __restrict__ ce, F& f, G& end_contacts) {
    const uint32_t N = P.N;     // table starts >= N mark empty cells
    const bool quirk = (P.flags & PBD_FLAG_CELL_END_QUIRK) && S.n >= 2;
    if (P.active & PBD_ACTIVE_FIND_CONTACTS) {
        uint32_t mz[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) mz[c] = morton_axis(__fmaf_rn((float)(c - 1), P.d, pi.z));
#pragma unroll 1
        for (int a = -1; a <= 1; ++a) {
            const uint32_t hx = morton_axis(__fmaf_rn((float)a, P.d, pi.x)) << 2;
#pragma unroll 1
            for (int b = -1; b <= 1; ++b) {
                const uint32_t hxy = hx + (morton_axis(__fmaf_rn((float)b, P.d, pi.y)) << 1);
                // the column's three cells: all six table loads in flight before the walk
                uint32_t h[3], cs3[3], ce3[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    h[c] = hxy + mz[c];
                    cs3[c] = h[c] < S.cells ? __ldg(cs + S.base + h[c]) : kEmptyCell;
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) ce3[c] = h[c] < S.cells ? __ldg(ce + S.base + h[c]) : 0u;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    if (cs3[c] >= N) continue;
                    const uint32_t e = ((quirk && h[c] == S.n - 1) || ce3[c] > S.end) ? S.end : ce3[c];
                    if (f(cs3[c], e, true)) return;
                }
            }
        }
    }
    if (end_contacts()) return;
    if (P.active & PBD_ACTIVE_FIND_NEIGHBOURS) {
        const int K = (int)P.K;
#pragma unroll 1
        for (int sh = 2; sh <= K; ++sh) {
#pragma unroll 1
            for (int a = -sh; a <= sh; ++a) {
                const uint32_t hx = morton_axis(__fmaf_rn((float)a, P.d, pi.x)) << 2;
#pragma unroll 1
                for (int b = -sh; b <= sh; ++b) {
                    const uint32_t hy = morton_axis(__fmaf_rn((float)b, P.d, pi.y)) << 1;
                    const bool edge_ab = (a == sh || a == -sh || b == sh || b == -sh);
                    const int cstep = edge_ab ? 1 : 2 * sh;   // interior columns: only c = +-sh
#pragma unroll 1
                    for (int c = -sh; c <= sh; c += cstep) {
                        const uint32_t h = hx + hy + morton_axis(__fmaf_rn((float)c, P.d, pi.z));
                        if (h >= S.cells) continue;
                        const uint32_t s = __ldg(cs + S.base + h);
                        uint32_t e = __ldg(ce + S.base + h);
                        if (s >= N) continue;
                        if ((quirk && h == S.n - 1) || e > S.end) e = S.end;   // entries >= N are skipped (Collision.h:142)
                        if (f(s, e, false)) return;
                    }
                }
            }
        }
    }
}

// One thread per particle.  Returns the list length; sets *deferred (and stops) when a
// range longer than kLongRange is met and `defer` is set.  `anchor` selects the cells, `p`
// holds the current positions.
template <class V>
__device__ __forceinline__ uint32_t walk_seq(const DevParams& P, const SceneCtx& S, uint32_t i, float4 anchor,
                                             const float4* __restrict__ p, const uint32_t* __restrict__ cs,
                                             const uint32_t* __restrict__ ce, V& vis, bool defer, bool* deferred) {
    const uint32_t M = P.M;
    uint32_t cnt = 0;
    if (M == 0) return 0;
    auto range = [&](uint32_t s, uint32_t e, bool contact) -> bool {
        if (defer && e - s > kLongRange) { *deferred = true; return true; }
        for (uint32_t j = s; j < e; ++j) {
            if (j == i) continue;
            vis.add(contrib_of(vis, j, __ldg(p + j), fetch_extra(vis, j), contact), contact);
            if (++cnt == M) return true;
        }
        return false;
    };
    auto endc = [&]() -> bool { vis.end_contacts(cnt); return false; };
    for_each_range(P, S, anchor, cs, ce, range, endc);
    return cnt;
}

// One warp per particle (all 32 lanes call it with the same i).  Same list, same order.
template <class V>
__device__ __forceinline__ uint32_t walk_coop(const DevParams& P, const SceneCtx& S, uint32_t i, float4 anchor,
                                              const float4* __restrict__ p, const uint32_t* __restrict__ cs,
                                              const uint32_t* __restrict__ ce, V& vis) {
    const uint32_t M = P.M;
    const uint32_t lane = lane_id(), lt = lanemask_lt_u();
    uint32_t cnt = 0;
    if (M == 0) return 0;
    auto range = [&](uint32_t s, uint32_t e, bool contact) -> bool {
        for (uint32_t c0 = s; c0 < e; c0 += 32u) {
            const uint32_t j = c0 + lane;
            bool valid = j < e && j != i;
            const uint32_t b = __ballot_sync(kFullMask, valid);
            valid = valid && __popc(b & lt) < M - cnt;
            typename V::Contrib c = valid ? contrib_of(vis, j, __ldg(p + j), fetch_extra(vis, j), contact) : V::zero();
            const uint32_t n = __popc(__ballot_sync(kFullMask, valid));
            // only entries whose contribution changes a sum are added (in order); the others
            // are exact no-ops of add() and still count toward the cap
            uint32_t take = __ballot_sync(kFullMask, valid && V::effective(c));
            while (take) {
                const int k = __ffs(take) - 1;
                take &= take - 1u;
                vis.add(V::shfl(c, k), contact);
            }
            cnt += n;
            if (cnt == M) return true;
        }
        return false;
    };
    auto endc = [&]() -> bool { vis.end_contacts(cnt); return false; };
    for_each_range(P, S, anchor, cs, ce, range, endc);
    return cnt;
}

// Cell t of findNeighbours' shell sh, in list order (Collision.h:127-134: edge columns hold every
// c, interior columns only c = -sh and c = +sh).  The shell has side^3 - (side - 2)^3 cells.
__device__ __forceinline__ void shell_cell(int sh, int t, int& a, int& b, int& c) {
    const int side = 2 * sh + 1, slab = side * side, ring = 4 * side - 4;
    const bool last = t >= slab + (side - 2) * ring;
    if (t < slab || last) {
        if (last) t -= slab + (side - 2) * ring;
        a = last ? sh : -sh;
        b = t / side - sh;
        c = t % side - sh;
        return;
    }
    t -= slab;
    a = t / ring - sh + 1;
    t %= ring;
    if (t < side) { b = -sh; c = t - sh; return; }
    t -= side;
    if (t < 2 * (side - 2)) { b = t / 2 - sh + 1; c = (t & 1) ? sh : -sh; return; }
    b = sh;
    c = t - 2 * (side - 2) - sh;
}

// G lanes enumerate particle i's list (the entries and order of for_each_range, without i, up to
// `cap`, the list cap M or one past the room of whatever takes the entries): a lane per cell for
// the table loads, then a lane per entry, which finds its cell by a search over the group's
// offsets.  emit(k, j) gets every entry once.  long_stop: a cell range longer than kLongRange ends the
// walk (walk_seq's hand-over).  Every lane of the warp calls it; groups with on = false only take
// part in the shuffles.
struct GroupList {
    uint32_t n, nc;      // entries, contact entries
    bool handed_over;
};
template <int G, class Emit>
__device__ __forceinline__ GroupList enumerate_group(const DevParams& P, const SceneCtx& S, uint32_t i, float4 anchor, bool on,
                                                     const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce,
                                                     uint32_t cap, bool long_stop, Emit&& emit) {
    const uint32_t lane = lane_id(), t = lane & (uint32_t)(G - 1);
    const uint32_t shift = lane & ~(uint32_t)(G - 1), gmask = G == 32 ? kFullMask : (1u << G) - 1u;
    const bool quirk = (P.flags & PBD_FLAG_CELL_END_QUIRK) && S.n >= 2;
    GroupList R{0u, 0u, false};
    bool done = !on || cap == 0u;
    auto cells = [&](bool in, int a, int b, int c) {
        uint32_t s = 0, len = 0, own = 0;
        bool is_long = false;
        if (in && !done) {
            const uint32_t h = (morton_axis(__fmaf_rn((float)a, P.d, anchor.x)) << 2) +
                               (morton_axis(__fmaf_rn((float)b, P.d, anchor.y)) << 1) +
                               morton_axis(__fmaf_rn((float)c, P.d, anchor.z));
            if (h < S.cells) {
                s = __ldg(cs + S.base + h);
                uint32_t e = __ldg(ce + S.base + h);
                if (s < P.N) {
                    if ((quirk && h == S.n - 1) || e > S.end) e = S.end;
                    if (e > s) {
                        is_long = e - s > kLongRange;
                        own = (s <= i && i < e) ? 1u : 0u;
                        len = min(e - s - own, cap);
                    }
                }
            }
        }
        uint32_t off = len;
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
            const uint32_t v = __shfl_up_sync(kFullMask, off, o, G);
            if (t >= (uint32_t)o) off += v;
        }
        const uint32_t total = __shfl_sync(kFullMask, off, G - 1, G);
        off -= len;
        if (long_stop) {
            const uint32_t bad = __ballot_sync(kFullMask, is_long && R.n + off < cap);
            if ((bad >> shift) & gmask) { R.handed_over = true; done = true; }
        }
        const uint32_t mine = done ? 0u : total;
        for (uint32_t o0 = 0; __any_sync(kFullMask, o0 < mine && R.n + o0 < cap); o0 += (uint32_t)G) {
            const uint32_t o = o0 + t;
            uint32_t q = 0;   // the last lane whose offset is not beyond o
#pragma unroll
            for (uint32_t step = G / 2; step > 0; step >>= 1) {
                const uint32_t v = __shfl_sync(kFullMask, off, q + step, G);
                if (v <= o) q += step;
            }
            const uint32_t qs = __shfl_sync(kFullMask, s, q, G), qo = __shfl_sync(kFullMask, off, q, G);
            const uint32_t qi = __shfl_sync(kFullMask, own, q, G);
            uint32_t j = qs + (o - qo);
            if (qi && j >= i) ++j;
            if (o < mine && R.n + o < cap) emit(R.n + o, j);
        }
        R.n = min(R.n + mine, cap);
        done = done || R.n == cap;
    };
    if (P.active & PBD_ACTIVE_FIND_CONTACTS) {
#pragma unroll 1
        for (int t0 = 0; t0 < 27; t0 += G) {
            const int k = t0 + (int)t;
            cells(k < 27, k / 9 - 1, (k / 3) % 3 - 1, k % 3 - 1);
        }
        R.nc = R.n;
    }
    if (P.active & PBD_ACTIVE_FIND_NEIGHBOURS)
        for (int sh = 2; sh <= (int)P.K; ++sh) {
            const int side = 2 * sh + 1, count = side * side * side - (side - 2) * (side - 2) * (side - 2);
            for (int t0 = 0; t0 < count && !__all_sync(kFullMask, done); t0 += G) {
                const int k = t0 + (int)t;
                int a = 0, b = 0, c = 0;
                if (k < count) shell_cell(sh, k, a, b, c);
                cells(k < count, a, b, c);
            }
        }
    return R;
}

// One warp stores particle i's list into `row` (kLongMax entries at most).  Returns the row's meta.
__device__ __forceinline__ uint32_t store_row(const DevParams& P, const SceneCtx& S, uint32_t i, float4 anchor,
                                              const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce,
                                              uint32_t* row) {
    const GroupList R = enumerate_group<32>(P, S, i, anchor, true, cs, ce, min(P.M, kLongMax + 1u), false,
                                            [&](uint32_t k, uint32_t j) { if (k < kLongMax) row[k] = j; });
    return R.n > kLongMax ? kListOff : (R.n | (R.nc << 16));
}

// One warp per particle over a stored list (entry k at entry(k); n and nc the same in all lanes): each
// lane evaluates every 32nd entry, two position loads in flight and the next indices loaded
// meanwhile, and the contributions that change a sum are added in list order through shuffles, as
// in walk_coop, so every lane ends with the sums.
template <class E, class V>
__device__ __forceinline__ void walk_list_warp(E&& entry, uint32_t n, uint32_t nc, uint32_t i, const float4* __restrict__ p,
                                           V& vis) {
    const uint32_t t = lane_id();
    uint32_t jn[2];
#pragma unroll
    for (uint32_t b = 0; b < 2u; ++b) jn[b] = b * 32u + t < n ? *entry(b * 32u + t) : i;
    for (uint32_t kb = 0; kb < n; kb += 64u) {
        uint32_t j[2];
        float4 pj[2];
        typename ExtraOf<V>::type ex[2];
#pragma unroll
        for (uint32_t b = 0; b < 2u; ++b) {
            j[b] = jn[b];
            pj[b] = __ldg(p + j[b]);
            ex[b] = fetch_extra(vis, j[b]);
        }
#pragma unroll
        for (uint32_t b = 0; b < 2u; ++b) {
            const uint32_t k = kb + (2u + b) * 32u + t;
            jn[b] = k < n ? *entry(k) : i;
        }
#pragma unroll
        for (uint32_t b = 0; b < 2u; ++b) {
            const uint32_t k = kb + b * 32u + t;
            const typename V::Contrib c = k < n ? contrib_of(vis, j[b], pj[b], ex[b], k < nc) : V::zero();
            uint32_t take = __ballot_sync(kFullMask, k < n && V::effective(c));
            while (take) {
                const int q = __ffs(take) - 1;
                take &= take - 1u;
                vis.add(V::shfl(c, q), true);
            }
        }
    }
    vis.end_contacts(nc);
}

// A stored list with G lanes per particle and the sums split over the lanes (every lane of the warp calls
// it; a group with n = 0 only takes part in the shuffles).  Every sum
// of a visitor is a chain acc = fma(mul, val, acc) over the entries (mul = 1 where a contribution is
// added as it is: the same rounding as an addition).  Each lane puts its entry's numbers (V::rows,
// zeros where the entry has no effect, which leave a chain alone) into shared memory, a row per
// number, and lane t of the group runs the chain of sum t (t + G, ...) over them: two loads and four
// fused multiply-adds for four entries, where handing a contribution to every lane took seven
// shuffles and seven adds per entry.
constexpr uint32_t kSumStride = 68;   // two entries per lane, rows four banks apart
template <int G, class E, class V>
__device__ __forceinline__ void walk_group_sums(E&& entry, uint32_t n, uint32_t nc, uint32_t i, const float4* __restrict__ p,
                                                V& vis) {
    constexpr int kRows = V::kRows, kSums = V::kSums, kPer = (kSums + G - 1) / G;
    __shared__ float4 rows4[8][(kRows + 1) * kSumStride / 4];   // blocks of up to 256 threads
    float* rows = reinterpret_cast<float*>(rows4[threadIdx.x >> 5]);
    const uint32_t lane = lane_id(), t = lane & (uint32_t)(G - 1);
    rows[kRows * kSumStride + lane] = 1.0f;
    rows[kRows * kSumStride + 32u + lane] = 1.0f;
    float acc[kPer];
    const float4 *mul[kPer], *val[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        int m = kRows, v = kRows;
        acc[u] = 0.0f;
#pragma unroll
        for (int s = u * G; s < kSums && s < (u + 1) * G; ++s)
            if ((int)t == s - u * G) { acc[u] = vis.sum(s); m = V::mul_row(s); v = V::val_row(s); }
        mul[u] = reinterpret_cast<const float4*>(rows + m * kSumStride + (lane - t));
        val[u] = reinterpret_cast<const float4*>(rows + v * kSumStride + (lane - t));
    }
    uint32_t jn[2];
#pragma unroll
    for (uint32_t b = 0; b < 2u; ++b) jn[b] = b * G + t < n ? *entry(b * G + t) : i;
    for (uint32_t kb = 0; __any_sync(kFullMask, kb < n); kb += 2u * G) {
        uint32_t j[2];
        float4 pj[2];
        typename ExtraOf<V>::type ex[2];
#pragma unroll
        for (uint32_t b = 0; b < 2u; ++b) {
            j[b] = jn[b];
            pj[b] = __ldg(p + j[b]);
            ex[b] = fetch_extra(vis, j[b]);
        }
#pragma unroll
        for (uint32_t b = 0; b < 2u; ++b) {
            const uint32_t k = kb + (2u + b) * G + t;
            jn[b] = k < n ? *entry(k) : i;
        }
        __syncwarp();   // the last step's rows have been read
#pragma unroll
        for (uint32_t b = 0; b < 2u; ++b) {
            const uint32_t k = kb + b * G + t;
            float r[kRows];
            V::rows(contrib_of(vis, j[b], pj[b], ex[b], k < nc), k < n, r);
#pragma unroll
            for (int q = 0; q < kRows; ++q) rows[q * kSumStride + b * 32u + lane] = r[q];
        }
        __syncwarp();
#pragma unroll
        for (uint32_t b = 0; b < 2u; ++b)
#pragma unroll
            for (int q = 0; q < G / 4; ++q)
#pragma unroll
                for (int u = 0; u < kPer; ++u) {
                    const float4 m = mul[u][b * 8u + q], v = val[u][b * 8u + q];
                    acc[u] = __fmaf_rn(m.x, v.x, acc[u]);
                    acc[u] = __fmaf_rn(m.y, v.y, acc[u]);
                    acc[u] = __fmaf_rn(m.z, v.z, acc[u]);
                    acc[u] = __fmaf_rn(m.w, v.w, acc[u]);
                }
    }
#pragma unroll
    for (int s = 0; s < kSums; ++s) vis.sum(s) = __shfl_sync(kFullMask, acc[s / G], s % G, G);
}

// filter_list with G lanes per particle (entry k at entry(k), n entries, nc of them contacts; 0 for a
// group that only takes part): each lane tests every G-th entry, its slot among the group's lanes
// from a ballot.  kWalk: an entry whose distance is not a number counts as near, as a walk of the cells
// counts it.
template <int G, bool kWalk = false, class E>
__device__ __forceinline__ uint32_t filter_group(E&& entry, uint32_t n, uint32_t nc, const NbList& L, uint32_t i,
                                                 const float4& pi, float cut2, const float4* __restrict__ p) {
    const uint32_t lane = lane_id(), t = lane & (uint32_t)(G - 1);
    const uint32_t shift = lane & ~(uint32_t)(G - 1), gmask = G == 32 ? kFullMask : (1u << G) - 1u;
    uint32_t m = 0, mc = 0;
    for (uint32_t kb = 0; __any_sync(kFullMask, kb < n); kb += 4u * G) {
        uint32_t j[4];
        float4 pj[4];
#pragma unroll
        for (uint32_t b = 0; b < 4u; ++b) j[b] = kb + b * G + t < n ? *entry(kb + b * G + t) : i;
#pragma unroll
        for (uint32_t b = 0; b < 4u; ++b) pj[b] = __ldg(p + j[b]);
#pragma unroll
        for (uint32_t b = 0; b < 4u; ++b) {
            const uint32_t k = kb + b * G + t;
            const float rx = pi.x - pj[b].x, ry = pi.y - pj[b].y, rz = pi.z - pj[b].z;
            const float r2 = dist2(rx, ry, rz);
            const bool near = k < n && (kWalk ? !(r2 >= cut2) : r2 < cut2);
            const uint32_t all = (__ballot_sync(kFullMask, near) >> shift) & gmask;
            const uint32_t con = (__ballot_sync(kFullMask, near && k < nc) >> shift) & gmask;
            const uint32_t at = m + __popc(all & ((1u << t) - 1u));
            if (near && at < L.kmax) L.list[(size_t)at * L.stride + i] = j[b];
            m += __popc(all);
            mc += __popc(con);
        }
    }
    __syncwarp();
    return m > L.kmax ? kListOff : (m | (mc << 8));
}

// One thread per particle over a stored list (meta not kListOff).
// Every visitor adds its contributions with explicitly rounded operations (__fadd_rn, or
// __fmaf_rn where a product goes into the sum), which the compiler never contracts, so the sums
// get the same bits whichever walker (cells, stored list, cooperative warp) and whichever loop
// shape the compiler sees.
//
// kOwn: the list was written by this thread in this kernel, so it is read with ordinary
// (coherent) loads rather than through the read-only path.  Otherwise the list entries are
// read with the streaming hint (ld.global.cs: evict first): each is read once per pass, and
// the cache lines they would take are worth more to the neighbour positions gathered next
// (3% off the frame on fluid_1m).

// A visitor with add_if (its contributions have no side effects) is evaluated for every slot of a
// group and added under a predicate, so the group's arithmetic runs without branches; the others are
// visited entry by entry.
template <class V, class = void> struct AddIf : std::false_type {};
template <class V> struct AddIf<V, std::void_t<decltype(&V::add_if)>> : std::true_type {};
// A visitor with kAddTwo adds two entries, one after the other, by one call: the arithmetic of both in
// two-float instructions, each kernel's range tested only where its term is added.  Over full lists the
// passes are bound by instruction issue and the gathers together: 54 -> 43 instructions per entry for
// delta and 43 -> 31 for lambda made them 211 -> 185 and 169 -> 147 us (1M particles, ~124 entries;
// positions loaded a group ahead instead: 210 and 180, the registers cost warps).  i itself as an entry
// must add nothing to its sums; where it might (self_adds), the list is summed once more, entry by entry (after
// the loop, where it costs nothing: as a second loop for the last group lambda took 154 us, as a test of
// every entry 165).
template <class V, class = void> struct AddTwo : std::false_type {};
template <class V> struct AddTwo<V, std::void_t<decltype(V::kAddTwo)>> : std::bool_constant<V::kAddTwo> {};
template <class V, class = void> struct SelfAdds : std::false_type {};
template <class V> struct SelfAdds<V, std::void_t<decltype(&V::self_adds)>> : std::true_type {};
// A visitor with load(j, pj, ex) takes an entry's position and extra data from an array of its own.
template <class V, class = void> struct OwnLoad : std::false_type {};
template <class V> struct OwnLoad<V, std::void_t<decltype(&V::load)>> : std::true_type {};
template <class V, class = void> struct TestsContacts : std::false_type {};
template <class V> struct TestsContacts<V, std::void_t<decltype(V::kTestsContacts)>> : std::true_type {};

// The full list, a group of four entries at a time: the group's position (and extra) loads are all
// in flight before the first contribution, and the next group's indices are loaded meanwhile.
// Slots past the end hold anything: they are replaced by i itself and not added.
template <bool kOwn = false, class V>
__device__ __forceinline__ void walk_full(const NbList& F, uint32_t i, uint32_t meta, const float4* __restrict__ p, V& vis) {
    const uint32_t n = meta & 0xFFu, nc = (meta >> 8) & 0xFFu;
    const uint4* e = reinterpret_cast<const uint4*>(F.list) + i;
    uint4 q = make_uint4(i, i, i, i);
    if (n) q = kOwn ? *e : __ldcs(e);
    uint32_t kb = 0;
    auto group = [&](auto contacts) {
        const uint32_t j[4] = {q.x, kb + 1u < n ? q.y : i, kb + 2u < n ? q.z : i, kb + 3u < n ? q.w : i};
        float4 pj[4];
        typename ExtraOf<V>::type ex[4];
#pragma unroll
        for (uint32_t b = 0; b < 4u; ++b) {
            if constexpr (OwnLoad<V>::value) {
                vis.load(j[b], pj[b], ex[b]);
            } else {
                pj[b] = __ldg(p + j[b]);
                ex[b] = fetch_extra(vis, j[b]);
            }
        }
        e += F.stride;
        if (kb + 4u < n) q = kOwn ? *e : __ldcs(e);
        if constexpr (AddTwo<V>::value) {
            constexpr bool kC = decltype(contacts)::value;
            vis.template add_two<kC>(j[0], pj[0], kb < nc, j[1], pj[1], kb + 1u < nc);
            vis.template add_two<kC>(j[2], pj[2], kb + 2u < nc, j[3], pj[3], kb + 3u < nc);
        } else {
#pragma unroll
            for (uint32_t b = 0; b < 4u; ++b) {
                const bool contact = decltype(contacts)::value && kb + b < nc;
                if constexpr (AddIf<V>::value) vis.add_if(kb + b, n, contrib_of(vis, j[b], pj[b], ex[b], contact));
                else if (kb + b < n) vis.add(contrib_of(vis, j[b], pj[b], ex[b], contact), contact);
            }
        }
        kb += 4u;
    };
    // a visitor that tests contacts (kTestsContacts): first the groups that hold contact entries, then
    // the others without the test (with two shells 26 of ~125 entries are contacts: 322 -> 275 us)
    if constexpr (TestsContacts<V>::value) {
#pragma unroll 1
        while (kb < nc) group(std::true_type{});
#pragma unroll 1
        while (kb < n) group(std::false_type{});
    } else {
#pragma unroll 1
        while (kb < n) group(std::true_type{});
        if constexpr (SelfAdds<V>::value) {
            if (vis.self_adds()) {
                vis.reset();
#pragma unroll 1
                for (uint32_t k = 0; k < n; ++k) {
                    const uint32_t j = *full_at(F, i, k);
                    vis.add(contrib_of(vis, j, __ldg(p + j), fetch_extra(vis, j), k < nc), k < nc);
                }
            }
        }
    }
    vis.end_contacts(nc);
}

// A near list (~6 entries), B entries at a time (on fluid_1m 1; 2, 3 and 8 slower), the next
// entries' indices in flight.
template <bool kOwn = false, uint32_t B = 1, class V>
__device__ __forceinline__ void walk_near(const NbList& L, uint32_t i, uint32_t meta, const float4* __restrict__ p, V& vis) {
    const uint32_t n = meta & 0xFFu, nc = (meta >> 8) & 0xFFu;
    const size_t st = L.stride;
    const uint32_t* e = L.list + i;
    uint32_t jn[B];
#pragma unroll
    for (uint32_t b = 0; b < B; ++b) jn[b] = b < n ? (kOwn ? e[b * st] : __ldcs(e + b * st)) : i;
#pragma unroll 1
    for (uint32_t kb = 0; kb < n; kb += B) {
        uint32_t j[B];
        float4 pj[B];
        typename ExtraOf<V>::type ex[B];
#pragma unroll
        for (uint32_t b = 0; b < B; ++b) {
            j[b] = jn[b];
            pj[b] = __ldg(p + j[b]);
            ex[b] = fetch_extra(vis, j[b]);
        }
        e += B * st;
#pragma unroll
        for (uint32_t b = 0; b < B; ++b) jn[b] = kb + B + b < n ? (kOwn ? e[b * st] : __ldcs(e + b * st)) : i;
#pragma unroll
        for (uint32_t b = 0; b < B; ++b) {
            const bool contact = kb + b < nc;
            if constexpr (AddIf<V>::value) vis.add_if(kb + b, n, contrib_of(vis, j[b], pj[b], ex[b], contact));
            else if (kb + b < n) vis.add(contrib_of(vis, j[b], pj[b], ex[b], contact), contact);
        }
    }
    vis.end_contacts(nc);
}

// Particle i's near list from its full list (meta fm): the entries with r^2 < cut2 at p, in
// list order, the boundary of the contact entries kept.  No sums: a pass then walks the near
// list alone (every entry left out adds an exact zero to every sum of a lambda, omega or delta
// pass), so the warp runs the kernel arithmetic for ~6 entries per particle instead of ~32.
// Returns the near list's meta (kListOff when it does not fit).
// kCoarse: by the coarse positions, which let in at most the entries within 0.006 cells of the cut
// besides (they add the same exact zeros).  The filter is bound by the L1, which takes a turn for every
// line a gather touches: 8-byte positions touch half as many as 16-byte ones.  A position of i that is
// not finite has no near entry, as its r^2 is not below the cut.
template <bool kOwn, bool kCoarse>
__device__ __forceinline__ uint32_t filter_list(const DevParams& P, const NbList& F, uint32_t fm, const NbList& L, uint32_t i,
                                                const float4& pi, const float4* __restrict__ p) {
    using Pos = typename std::conditional<kCoarse, uint2, float4>::type;
    const uint32_t n = fm & 0xFFu, nc = (fm >> 8) & 0xFFu;
    const uint4* e = reinterpret_cast<const uint4*>(F.list) + i;
    const Pos* __restrict__ pos;
    Pos own;
    float cut2 = 0.0f;
    uint32_t limit = 0u;
    if constexpr (kCoarse) {
        pos = P.coarse;
        own = coarse_pos(pi);
        limit = (fabsf(pi.x) + fabsf(pi.y) + fabsf(pi.z) < __int_as_float(0x7f800000)) ? P.near_coarse : 0u;
    } else {
        pos = p;
        own = pi;
        cut2 = P.cut2;
    }
    uint32_t* o = L.list + i;
    const size_t ost = L.stride;
    uint32_t m = 0, mc = 0;
    uint4 q = make_uint4(i, i, i, i);
    if (n) q = kOwn ? *e : __ldcs(e);
#pragma unroll 1
    for (uint32_t kb = 0; kb < n; kb += 4u) {
        const uint32_t j[4] = {q.x, kb + 1u < n ? q.y : i, kb + 2u < n ? q.z : i, kb + 3u < n ? q.w : i};
        Pos pj[4];
#pragma unroll
        for (uint32_t b = 0; b < 4u; ++b) pj[b] = __ldg(pos + j[b]);
        e += F.stride;
        if (kb + 4u < n) q = kOwn ? *e : __ldcs(e);
#pragma unroll
        for (uint32_t b = 0; b < 4u; ++b) {
            if (kb + b == nc) mc = m;
            bool near;
            if constexpr (kCoarse) near = coarse_near(own, pj[b], limit);
            else near = dist2(own.x - pj[b].x, own.y - pj[b].y, own.z - pj[b].z) < cut2;
            if (kb + b < n && near) {
                if (m < L.kmax) {
                    *o = j[b];
                    o += ost;
                }
                ++m;
            }
        }
    }
    if (nc >= n) mc = m;
    return m > L.kmax ? kListOff : (m | (mc << 8));
}

// Wraps the visitor of a walking pass and keeps particle i's near list as the walk goes.  Holds
// everything by value so the visitor stays in registers.
template <class V>
struct Recorder {
    using Contrib = typename V::Contrib;
    using Extra = typename ExtraOf<V>::type;
    V inner;
    uint32_t* list;
    uint32_t stride, kmax, i;
    float4 pi;
    float cut2;
    uint32_t n = 0, nc = 0xFFFFFFFFu;
    __device__ Recorder(const V& v, const NbList& L, uint32_t i_, float4 p_i, float c2)
        : inner(v), list(L.list), stride(L.stride), kmax(L.kmax), i(i_), pi(p_i), cut2(c2) {}
    __device__ static Contrib zero() { return V::zero(); }
    __device__ __forceinline__ void end_contacts(uint32_t c) { nc = n; inner.end_contacts(c); }
    __device__ __forceinline__ Extra fetch(uint32_t j) const { return fetch_extra(inner, j); }
    __device__ __forceinline__ Contrib contrib(uint32_t j, const float4& pj, const Extra& ex, bool contact) {
        const float rx = pi.x - pj.x, ry = pi.y - pj.y, rz = pi.z - pj.z;
        if (dist2(rx, ry, rz) < cut2) {
            if (n < kmax) list[(size_t)n * stride + i] = j;
            ++n;
        }
        return contrib_of(inner, j, pj, ex, contact);
    }
    __device__ __forceinline__ void add(const Contrib& c, bool contact) { inner.add(c, contact); }
    __device__ __forceinline__ uint32_t meta() const {
        const uint32_t c = nc == 0xFFFFFFFFu ? n : nc;
        return n > kmax ? kListOff : (n | (c << 8));
    }
};

// A walk that only stores particle i's full list: indices, no positions (the walk's position
// loads are dead and vanish), the boundary of the contact entries kept.
struct ListRecorder {
    struct Contrib {};
    const NbList& F;
    uint32_t i;
    uint32_t n = 0, nc = 0xFFFFFFFFu;
    __device__ ListRecorder(const NbList& F_, uint32_t i_) : F(F_), i(i_) {}
    __device__ static Contrib zero() { return Contrib{}; }
    __device__ static bool effective(const Contrib&) { return false; }
    __device__ static Contrib shfl(const Contrib& c, int) { return c; }
    __device__ __forceinline__ void end_contacts(uint32_t) { nc = n; }
    __device__ __forceinline__ Contrib contrib(uint32_t j, const float4&, bool) {
        if (n < F.kmax) *full_at(F, i, n) = j;
        ++n;
        return Contrib{};
    }
    __device__ __forceinline__ void add(const Contrib&, bool) {}
    __device__ __forceinline__ uint32_t meta() const {
        const uint32_t c = nc == 0xFFFFFFFFu ? n : nc;
        return n > F.kmax ? kListOff : (n | (c << 8));
    }
};

// Appends entries to particle i's full list: four collect in registers and go out as one store.
struct FullWriter {
    uint4 q = make_uint4(0u, 0u, 0u, 0u);   // the last four entries, the newest in w
    uint4* o;
    size_t st;
    uint32_t n = 0;                          // entries appended
    __device__ FullWriter(const NbList& F, uint32_t i) : o(reinterpret_cast<uint4*>(F.list) + i), st(F.stride) {}
    __device__ __forceinline__ void push(uint32_t j) {
        q.x = q.y; q.y = q.z; q.z = q.w; q.w = j;
        if ((++n & 3u) == 0u) {
            *o = q;
            o += st;
        }
    }
    __device__ __forceinline__ void flush() {   // the last 1 to 3 entries
        const uint32_t r = n & 3u;
        if (r == 1u) *o = make_uint4(q.w, 0u, 0u, 0u);
        if (r == 2u) *o = make_uint4(q.z, q.w, 0u, 0u);
        if (r == 3u) *o = make_uint4(q.y, q.z, q.w, 0u);
    }
};

// The cells of one group of particle i's list (store_column's), cell by cell: the entries in list
// order, skipping self, with the cap M, the list's room and the long-range hand-over of walk_seq.  Returns true when the walk ends here
// (cap reached or handed over).
template <int kMax>
__device__ __forceinline__ bool store_cells(const DevParams& P, const SceneCtx& S, uint32_t i, const uint32_t* h,
                                            const uint32_t* s, const uint32_t* e, const NbList& F, bool quirk,
                                            FullWriter& out, uint32_t& n, bool* deferred) {
    const uint32_t N = P.N, M = P.M;
    uint32_t len[kMax];
    uint32_t reach = n;   // entries stored before the cell: the walk reaches it while below the cap
#pragma unroll
    for (int c = 0; c < kMax; ++c) {
        const bool valid = s[c] < N;
        const uint32_t ec = ((quirk && h[c] == S.n - 1) || e[c] > S.end) ? S.end : e[c];
        len[c] = valid ? ec - s[c] : 0u;
        if (valid && reach < M && len[c] > kLongRange) { *deferred = true; return true; }
        reach += len[c] - ((valid && s[c] <= i && i < ec) ? 1u : 0u);
    }
#pragma unroll
    for (int c = 0; c < kMax; ++c)
#pragma unroll 1
        for (uint32_t t = 0; t < len[c]; ++t) {
            const uint32_t j = s[c] + t;
            if (j == i) continue;
            if (n < F.kmax) out.push(j);
            if (++n == M) return true;
        }
    return false;
}

// Append the entries of kRuns runs of particles without i, by one loop without a check per entry, where
// no run is longer than kLongRange and the cap and the list's room are out of reach; false otherwise.
template <int kRuns>
__device__ __forceinline__ bool push_runs(const DevParams& P, uint32_t i, const uint32_t* rs, const uint32_t* len, const NbList& F,
                                          FullWriter& out, uint32_t& n) {
    uint32_t end[kRuns], off[kRuns];   // run r: entries [end[r - 1], end[r]) of the column; entry t is particle off[r] + t
    uint32_t T = 0, longest = 0;
#pragma unroll
    for (int r = 0; r < kRuns; ++r) {
        longest = max(longest, len[r]);
        off[r] = rs[r] - T;
        T += len[r];
        end[r] = T;
    }
    if (!(longest <= kLongRange && n + T < P.M && n + T <= F.kmax)) return false;
#pragma unroll 1
    for (uint32_t t = 0; t < T; ++t) {
        uint32_t o = off[kRuns - 1];
#pragma unroll
        for (int r = kRuns - 2; r >= 0; --r) o = t < end[r] ? off[r] : o;
        const uint32_t j = o + t;
        if (j != i) out.push(j);
    }
    n = out.n;
    return true;
}

// One column of particle i's list: the 3 cells of a findContacts column or the cells of a
// findNeighbours column (2 sh + 1 on an edge column, 2 otherwise), keys h in list order; the table
// loads are all in flight first.  Cells z, z + 1 with z even have consecutive Morton keys, so their
// particles lie side by side: where the cells' z follow each other (`consecutive`; rounding or a diameter
// other than 1 can break it) each such pair is one run and the column has 2 to 4, else a run per cell.
// A column with a range longer than kLongRange, the cell-end range, or near the cap or the list's room
// goes cell by cell.  (One loop per cell, each with its checks, was 604 us for 1M dense particles, this
// 451; for 27 cells 154 -> 143.  With the sums' two-float arithmetic the pass takes 409 and 138.)  Returns true when the walk ends here (cap reached or handed over).
template <int kCells>
__device__ __forceinline__ bool store_column(const DevParams& P, const SceneCtx& S, uint32_t i, const uint32_t* h,
                                             bool odd, bool consecutive, const uint32_t* __restrict__ cs,
                                             const uint32_t* __restrict__ ce, const NbList& F, bool quirk,
                                             FullWriter& out, uint32_t& n, bool* deferred) {
    constexpr int kRuns = kCells == 2 ? 2 : (kCells + 1) / 2;
    uint32_t s[kCells], e[kCells];
#pragma unroll
    for (int c = 0; c < kCells; ++c) s[c] = h[c] < S.cells ? __ldg(cs + S.base + h[c]) : kEmptyCell;
#pragma unroll
    for (int c = 0; c < kCells; ++c) e[c] = h[c] < S.cells ? __ldg(ce + S.base + h[c]) : 0u;
    bool cell_end = false;
    if (quirk) {
#pragma unroll
        for (int c = 0; c < kCells; ++c) cell_end = cell_end || h[c] == S.n - 1u;
    }
    if (!cell_end) {
        if (kCells == 2 || !consecutive) {
            uint32_t len[kCells];
#pragma unroll
            for (int c = 0; c < kCells; ++c) len[c] = s[c] < P.N ? e[c] - s[c] : 0u;
            if (push_runs<kCells>(P, i, s, len, F, out, n)) return false;
        } else {
            const bool even_first = odd == (((kCells - 1) / 2) & 1);   // the column's first cell has an even z
            uint32_t rs[kRuns], len[kRuns];
#pragma unroll
            for (int r = 0; r < kRuns; ++r) {   // cells (2 r, 2 r + 1) or (2 r - 1, 2 r), those that exist
                const uint32_t s0 = r > 0 ? s[2 * r - 1] : kEmptyCell, e0 = r > 0 ? e[2 * r - 1] : 0u;
                const uint32_t s2 = 2 * r + 1 < kCells ? s[2 * r + 1] : kEmptyCell, e2 = 2 * r + 1 < kCells ? e[2 * r + 1] : 0u;
                const uint32_t slo = even_first ? s[2 * r] : s0, elo = even_first ? e[2 * r] : e0;
                const uint32_t shi = even_first ? s2 : s[2 * r], ehi = even_first ? e2 : e[2 * r];
                const bool lo = slo < P.N, hi = shi < P.N;
                rs[r] = lo ? slo : shi;
                len[r] = (lo || hi) ? (hi ? ehi : elo) - rs[r] : 0u;
            }
            if (push_runs<kRuns>(P, i, rs, len, F, out, n)) return false;
        }
    }
    return store_cells<kCells>(P, S, i, h, s, e, F, quirk, out, n, deferred);
}

// The frame's full list of particle i, indices only (findContacts on; kShells: with findNeighbours'
// shells, kernelWidthNeighbours 2 or 3): the entries, order, cap M, self-skip and long-range hand-over
// of walk_seq over for_each_range, column by column.  Returns the list's meta (kListOff when it does not
// fit or the particle is handed over; *deferred tells which).
template <bool kShells>
__device__ __forceinline__ uint32_t store_full_list(const DevParams& P, const SceneCtx& S, uint32_t i, float4 pa,
                                                    const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce,
                                                    const NbList& F, bool* deferred) {
    if (P.M == 0) return 0u;
    constexpr int R = kShells ? 3 : 1;
    const bool quirk = (P.flags & PBD_FLAG_CELL_END_QUIRK) && S.n >= 2;
    const int K = kShells ? (int)P.K : 1;
    uint32_t mz[2 * R + 1];
    int zc = 0;
    bool consecutive = true;
#pragma unroll
    for (int c = -R; c <= R; ++c) {
        const float z = fminf(fmaxf(__fmaf_rn((float)c, P.d, pa.z), 0.0f), 1023.0f);   // morton_axis
        const int cell = (int)(uint32_t)z;
        mz[c + R] = expand_bits((uint32_t)cell);
        if (c > -R && c > -K && c <= K) consecutive = consecutive && cell == zc + 1;
        zc = cell;
    }
    const bool odd = (mz[R] & 1u) != 0u;
    uint32_t n = 0, nc = 0xFFFFFFFFu;
    FullWriter out(F, i);
    auto meta = [&]() -> uint32_t {
        const uint32_t c = nc == 0xFFFFFFFFu ? n : nc;
        out.flush();
        return n > F.kmax ? kListOff : (n | (c << 8));
    };
    uint32_t h[7];
#pragma unroll 1
    for (int a = -1; a <= 1; ++a) {
        const uint32_t hx = morton_axis(__fmaf_rn((float)a, P.d, pa.x)) << 2;
#pragma unroll 1
        for (int b = -1; b <= 1; ++b) {
            const uint32_t hxy = hx + (morton_axis(__fmaf_rn((float)b, P.d, pa.y)) << 1);
#pragma unroll
            for (int c = 0; c < 3; ++c) h[c] = hxy + mz[R - 1 + c];
            if (store_column<3>(P, S, i, h, odd, consecutive, cs, ce, F, quirk, out, n, deferred)) return *deferred ? kListOff : meta();
        }
    }
    if constexpr (kShells) {
        nc = n;
#pragma unroll 1
        for (int sh = 2; sh <= K; ++sh)
#pragma unroll 1
            for (int a = -sh; a <= sh; ++a) {
                const uint32_t hx = morton_axis(__fmaf_rn((float)a, P.d, pa.x)) << 2;
#pragma unroll 1
                for (int b = -sh; b <= sh; ++b) {
                    const uint32_t hxy = hx + (morton_axis(__fmaf_rn((float)b, P.d, pa.y)) << 1);
                    const bool edge = a == sh || a == -sh || b == sh || b == -sh;
                    bool ends;
                    if (!edge) {   // interior columns: only c = -sh and c = +sh
                        h[0] = hxy + (sh == 2 ? mz[1] : mz[0]);
                        h[1] = hxy + (sh == 2 ? mz[5] : mz[6]);
                        ends = store_column<2>(P, S, i, h, odd, consecutive, cs, ce, F, quirk, out, n, deferred);
                    } else if (sh == 2) {
#pragma unroll
                        for (int c = 0; c < 5; ++c) h[c] = hxy + mz[1 + c];
                        ends = store_column<5>(P, S, i, h, odd, consecutive, cs, ce, F, quirk, out, n, deferred);
                    } else {
#pragma unroll
                        for (int c = 0; c < 7; ++c) h[c] = hxy + mz[c];
                        ends = store_column<7>(P, S, i, h, odd, consecutive, cs, ce, F, quirk, out, n, deferred);
                    }
                    if (ends) return *deferred ? kListOff : meta();
                }
            }
    }
    return meta();
}

// A visitor that sums nothing: a walk with Recorder<NullVisit> only stores the near list.
struct NullVisit {
    struct Contrib {};
    __device__ static Contrib zero() { return Contrib{}; }
    __device__ static bool effective(const Contrib&) { return false; }
    __device__ static Contrib shfl(const Contrib& c, int) { return c; }
    __device__ __forceinline__ void end_contacts(uint32_t) {}
    __device__ __forceinline__ Contrib contrib(uint32_t, const float4&, bool) const { return Contrib{}; }
    __device__ __forceinline__ void add(const Contrib&, bool) {}
};


// Hand particle i to the cooperative kernel; if the list is full, walk it here.
__device__ __forceinline__ bool defer_particle(const DeferList& D, uint32_t i) {
    const uint32_t k = atomicAdd(D.count, 1u);
    if (k < D.cap) { D.items[k] = i; return true; }
    return false;
}

// Grid-stride loop of the cooperative kernels over the deferred particles, then the last
// block to finish empties the list for the next pass.
template <class F>
__device__ __forceinline__ void for_each_deferred(const DeferList& D, F&& f) {
    const uint32_t n = min(*((volatile uint32_t*)D.count), D.cap);
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < n; w += warps) f(D.items[w]);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(D.done, 1u) == gridDim.x - 1) {
            *D.count = 0u;
            *D.done = 0u;
            __threadfence();
        }
    }
}

// The leading `blocks` blocks of a list kernel walk a set of particles over the cells (one warp
// per particle, walk_coop) while the other blocks walk the stored lists.  The particles without
// a list are known before such a kernel starts (the frame's first lambda pass, or the pass
// that recorded the near lists), so their long walks run beside the list walks instead of in a
// kernel after them.  With `reset`, the last of these blocks empties the set for its producer.
struct CoopSet {
    const uint32_t* items;
    uint32_t* count;
    uint32_t* done;
    uint32_t cap;
    uint32_t blocks;
    uint32_t reset;
};
template <class F>
__device__ __forceinline__ void run_coop_set(const CoopSet& C, F&& f) {
    const uint32_t n = min(*((volatile uint32_t*)C.count), C.cap);
    const uint32_t wpb = blockDim.x >> 5;
    const uint32_t warps = C.blocks * wpb;
    for (uint32_t w = blockIdx.x * wpb + (threadIdx.x >> 5); w < n; w += warps) f(C.items[w]);
    if (C.reset) {
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            if (atomicAdd(C.done, 1u) == C.blocks - 1) {
                *C.count = 0u;
                *C.done = 0u;
                __threadfence();
            }
        }
    }
}
// Append i to a set when the set is given (items non-null); returns its slot there.  The sets hold
// every particle of the simulation, so there is always room.
__device__ __forceinline__ uint32_t note_particle(const DeferList& D, uint32_t i) {
    if (!D.items) return 0u;
    const uint32_t k = atomicAdd(D.count, 1u);
    if (k < D.cap) D.items[k] = i;
    return k;
}

// Particle i's stored list as a warp reads it: its full list, else its long row; none: walk the cells.
struct WarpList {
    const uint32_t* row;   // null: no list
    bool grouped;          // a full list (groups of four), else a row
    uint32_t n, nc;
};
__device__ __forceinline__ WarpList warp_list(const LongLists& LL, const NbList& F, uint32_t i) {
    const uint32_t fm = F.list ? F.meta[i] : kListOff;
    if (!(fm & kListOff)) return WarpList{F.list, true, fm & 0xFFu, (fm >> 8) & 0xFFu};
    const uint32_t q = fm & ~(kListOff | kListWalked);
    const uint32_t m = (F.list && q < LL.slots) ? LL.meta[q] : kListOff;
    if (m == kListOff) return WarpList{nullptr, false, 0u, 0u};
    return WarpList{LL.list + (size_t)q * kLongMax, false, m & 0xFFFFu, m >> 16};
}
// One warp runs particle i's walk in a pass after the frame's first lambda pass.
template <class V>
__device__ __forceinline__ void walk_warp(const DevParams& P, const SceneCtx& S, uint32_t i, float4 anchor,
                                          const float4* __restrict__ p, const uint32_t* __restrict__ cs,
                                          const uint32_t* __restrict__ ce, const LongLists& LL, const NbList& F, V& vis) {
    const WarpList W = warp_list(LL, F, i);
    if (W.row) walk_list_warp([&](uint32_t k) { return W.grouped ? full_at(F, i, k) : W.row + k; }, W.n, W.nc, i, p, vis);
    else walk_coop(P, S, i, anchor, p, cs, ce, vis);
}

// ======================================================================================
// computeLambda (Density.h:48-93)
// ======================================================================================
// kUnitW: every p.w is 1 (DevParams::unit_w), so the entries' w difference is 0: it adds nothing to |r|_4
// and nothing to the gradient sum's w, and is left out.
template <bool kUnitW>
struct LambdaVisitT {
    // a = W, b = |grad|^2 = s^2 |r|^2; the gradient sum takes s * r by explicit FMAs, so every
    // walker rounds it the same way
    struct Contrib { float a, b, s, rx, ry, rz, rw, r2; bool near; };
    const DevParams& P;
    float4 pi;
    float A = 0.f, B = 0.f, Cx = 0.f, Cy = 0.f, Cz = 0.f, Cw = 0.f;
    __device__ LambdaVisitT(const DevParams& P_, float4 pi_) : P(P_), pi(pi_) {}
    __device__ void reset() { A = B = Cx = Cy = Cz = Cw = 0.f; }
    __device__ static Contrib zero() { return Contrib{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, false}; }
    __device__ static bool effective(const Contrib& c) { return c.near; }
    __device__ static Contrib shfl(const Contrib& c, int k) {
        return Contrib{shfl_f(c.a, k), shfl_f(c.b, k), shfl_f(c.s, k), shfl_f(c.rx, k), shfl_f(c.ry, k),
                       shfl_f(c.rz, k), shfl_f(c.rw, k), 0.f, shfl_u(c.near, k) != 0u};
    }
    __device__ __forceinline__ void end_contacts(uint32_t) {}
    __device__ __forceinline__ Contrib contrib(uint32_t, const float4& pj, bool) const {
        const float rx = pi.x - pj.x, ry = pi.y - pj.y, rz = pi.z - pj.z, rw = kUnitW ? 0.0f : pi.w - pj.w;
        const float r2 = dist2(rx, ry, rz);
        const float dist = sqrt_fast(r2);
        const float r2w = kUnitW ? r2 : __fmaf_rn(rw, rw, r2);
        const float s = spiky_scale(P, dist, r2w);
        // beyond the cut every kernel is exactly 0: add() leaves the sums alone
        return Contrib{poly6(P, dist), __fmul_rn(__fmul_rn(s, s), r2w), s, rx, ry, rz, rw, r2, !(r2 >= P.cut2)};
    }
    __device__ __forceinline__ void add(const Contrib& c, bool) {
        if (!c.near) return;
        A = __fadd_rn(A, c.a); B = __fadd_rn(B, c.b);
        Cx = __fmaf_rn(c.s, c.rx, Cx); Cy = __fmaf_rn(c.s, c.ry, Cy);
        Cz = __fmaf_rn(c.s, c.rz, Cz);
        if constexpr (!kUnitW) Cw = __fmaf_rn(c.s, c.rw, Cw);
    }
    // add() of entry k when k < n, as predicated instructions: as a branch the compiler moves the
    // contribution's arithmetic into it, and the entries of a group run one after the other. The tests
    // belong to the same block of instructions: as a flag handed to it they cost a select and a compare
    // per entry more (1M particles, full lists: delta 244 -> 211 us, lambda 173 -> 169).  Near lists only: an
    // entry whose distance is not a number is left out, as the test of exact positions leaves it out.
    __device__ __forceinline__ void add_if(uint32_t k, uint32_t n, const Contrib& c) {
        asm("{ .reg .pred q; setp.lt.u32 q, %5, %6; setp.lt.and.f32 q, %7, %8, q;"
            " @q add.rn.f32 %0, %0, %9; @q add.rn.f32 %1, %1, %10; @q fma.rn.f32 %2, %11, %12, %2;"
            " @q fma.rn.f32 %3, %11, %13, %3; @q fma.rn.f32 %4, %11, %14, %4; }"
            : "+f"(A), "+f"(B), "+f"(Cx), "+f"(Cy), "+f"(Cz)
            : "r"(k), "r"(n), "f"(c.r2), "f"(P.cut2), "f"(c.a), "f"(c.b), "f"(c.s), "f"(c.rx), "f"(c.ry), "f"(c.rz));
        if constexpr (!kUnitW)
            asm("{ .reg .pred q; setp.lt.u32 q, %1, %2; setp.lt.and.f32 q, %3, %4, q; @q fma.rn.f32 %0, %5, %6, %0; }"
                : "+f"(Cw) : "r"(k), "r"(n), "f"(c.r2), "f"(P.cut2), "f"(c.s), "f"(c.rw));
    }
    // The kernels are tested where they are added: within spiky's range (or NaN, which add() passes on)
    // r^2 < cut2 holds, and i itself (r = 0) is in neither range unless its position is infinite (r NaN).
    static constexpr bool kAddTwo = true;
    __device__ __forceinline__ bool self_adds() const {
        return !(fabsf(pi.x) + fabsf(pi.y) + fabsf(pi.z) < __int_as_float(0x7f800000));
    }
    template <bool>
    __device__ __forceinline__ void add_two(uint32_t, const float4& p0, bool, uint32_t, const float4& p1, bool) {
        float x[2], y[2], z[2], w[2], d[2], a[2], W[2], s[2], B2[2];
        f2_split(sub2(f2(pi.x, pi.y), f2(p0.x, p0.y)), x[0], y[0]);
        f2_split(sub2(f2(pi.x, pi.y), f2(p1.x, p1.y)), x[1], y[1]);
        z[0] = pi.z - p0.z; z[1] = pi.z - p1.z;
        const float r0 = dist2(x[0], y[0], z[0]), r1 = dist2(x[1], y[1], z[1]);
        float q0 = r0, q1 = r1;
        if constexpr (!kUnitW) {
            w[0] = pi.w - p0.w; w[1] = pi.w - p1.w;
            q0 = __fmaf_rn(w[0], w[0], r0); q1 = __fmaf_rn(w[1], w[1], r1);
        }
        d[0] = sqrt_fast(r0); d[1] = sqrt_fast(r1);
        const F2 dd = f2(d[0], d[1]), aa = sub2(f2(P.hs, P.hs), dd);
        f2_split(poly6_open(P, dd), W[0], W[1]);
        const F2 ss = spiky_open(P, aa, f2(rsqrt_fast(q0), rsqrt_fast(q1)));
        f2_split(mul2(mul2(ss, ss), f2(q0, q1)), B2[0], B2[1]);
        f2_split(aa, a[0], a[1]);
        f2_split(ss, s[0], s[1]);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            asm("{ .reg .pred q; setp.gt.f32 q, %1, %2; setp.lt.and.f32 q, %1, %3, q; @q add.rn.f32 %0, %0, %4; }"
                : "+f"(A) : "f"(d[b]), "f"(0.001f), "f"(P.hp_lim), "f"(W[b]));
            if constexpr (kUnitW)
                asm("{ .reg .pred q; setp.gtu.f32 q, %4, %6; setp.gtu.and.f32 q, %5, %6, q; @q add.rn.f32 %0, %0, %7;"
                    " @q fma.rn.f32 %1, %8, %9, %1; @q fma.rn.f32 %2, %8, %10, %2; @q fma.rn.f32 %3, %8, %11, %3; }"
                    : "+f"(B), "+f"(Cx), "+f"(Cy), "+f"(Cz)
                    : "f"(d[b]), "f"(a[b]), "f"(0.0001f), "f"(B2[b]), "f"(s[b]), "f"(x[b]), "f"(y[b]), "f"(z[b]));
            else
                asm("{ .reg .pred q; setp.gtu.f32 q, %5, %7; setp.gtu.and.f32 q, %6, %7, q; @q add.rn.f32 %0, %0, %8;"
                    " @q fma.rn.f32 %1, %9, %10, %1; @q fma.rn.f32 %2, %9, %11, %2; @q fma.rn.f32 %3, %9, %12, %3;"
                    " @q fma.rn.f32 %4, %9, %13, %4; }"
                    : "+f"(B), "+f"(Cx), "+f"(Cy), "+f"(Cz), "+f"(Cw)
                    : "f"(d[b]), "f"(a[b]), "f"(0.0001f), "f"(B2[b]), "f"(s[b]), "f"(x[b]), "f"(y[b]), "f"(z[b]), "f"(w[b]));
        }
    }
    // walk_group_sums: A, B, C from the rows a, b, s, r
    static constexpr int kRows = 7, kSums = 6;
    __device__ static constexpr int mul_row(int s) { return s < 2 ? kRows : 2; }
    __device__ static constexpr int val_row(int s) { return s < 2 ? s : s + 1; }
    __device__ __forceinline__ float& sum(int s) {
        return s == 0 ? A : (s == 1 ? B : (s == 2 ? Cx : (s == 3 ? Cy : (s == 4 ? Cz : Cw))));
    }
    __device__ __forceinline__ static void rows(const Contrib& c, bool live, float* r) {
        const bool on = live && c.near;
        r[0] = on ? c.a : 0.f; r[1] = on ? c.b : 0.f; r[2] = on ? c.s : 0.f;
        r[3] = on ? c.rx : 0.f; r[4] = on ? c.ry : 0.f; r[5] = on ? c.rz : 0.f; r[6] = on ? c.rw : 0.f;
    }
    // the sums the reverse pass needs: aux[i] = (rho, B, S.x, S.y), aux[N + i] = (S.z, S.w, 0, 0)
    __device__ __forceinline__ void store_aux(float4* __restrict__ aux, uint32_t N, uint32_t i) const {
        aux[i] = make_float4(A, B, Cx, Cy);
        aux[N + i] = make_float4(Cz, Cw, 0.f, 0.f);
    }
    __device__ __forceinline__ float finish(float rho0) const {
        // correctly rounded: every kernel that finishes a lambda gets the same bits
        const float a = __fsub_rn(__fdiv_rn(A, rho0), 1.0f);
        const float b = __fdiv_rn(B, rho0);
        const float s2 = __fadd_rn(__fadd_rn(__fmul_rn(Cx, Cx), __fmul_rn(Cy, Cy)), __fadd_rn(__fmul_rn(Cz, Cz), __fmul_rn(Cw, Cw)));
        const float c = __fdiv_rn(s2, rho0);
        return __fdiv_rn(-a, __fadd_rn(__fadd_rn(b, c), P.lambda_eps));
    }
};
using LambdaVisit = LambdaVisitT<false>;

template <bool kUnitW>
__global__ void __launch_bounds__(256, 4)   // 5 (48 registers) spills: 4% slower on 1M dense particles
lambda_kernel(DevParams P, const float4* __restrict__ p, const float4* __restrict__ pa, const uint32_t* __restrict__ cs,
              const uint32_t* __restrict__ ce, float* __restrict__ lambda, DeferList D, float4* __restrict__ aux,
              NbList L, NbList F, DeferList DF, DeferList DN, uint32_t long_slots, float4* __restrict__ pl) {
    // walks the cells; L.list: record the near lists for the delta pass that follows (the
    // particles left without one noted in DN); pl: also leave (p, lambda) there; F.list: store the full lists (the frame's first
    // lambda pass; the particles left without one noted in DF and finished by lambda_long_kernel,
    // which stores the lists of the first long_slots of them)
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    const SceneCtx S = scene_ctx(P, i);
    const float4 pi = p[i];
    LambdaVisitT<kUnitW> vis(P, pi);
    bool deferred = false;
    if (F.list) {
        // the walk stores the full list (indices only), the filter the near list; the sums then
        // run over the shortest list that fits
        uint32_t fm;
        const bool shells = (P.active & PBD_ACTIVE_FIND_NEIGHBOURS) && P.K >= 2;
        if (!shells && (P.active & PBD_ACTIVE_FIND_CONTACTS)) {
            fm = store_full_list<false>(P, S, i, pa[i], cs, ce, F, &deferred);
        } else if (shells && P.K <= 3 && (P.active & PBD_ACTIVE_FIND_CONTACTS)) {
            fm = store_full_list<true>(P, S, i, pa[i], cs, ce, F, &deferred);
        } else {
            ListRecorder rec(F, i);
            walk_seq(P, S, i, pa[i], p, cs, ce, rec, true, &deferred);
            fm = deferred ? kListOff : rec.meta();
        }
        uint32_t q = 0;
        if (fm == kListOff) {
            q = note_particle(DF, i);
            fm |= q | ((!deferred && q >= long_slots) ? kListWalked : 0u);
        }
        F.meta[i] = fm;
        const bool listed = !(fm & kListOff);
        if (!listed && !(fm & kListWalked)) return;
        const uint32_t lm = (L.list && listed) ? filter_list<true, kUnitW>(P, F, fm, L, i, pi, p) : kListOff;
        if (L.list) {
            L.meta[i] = lm;
            if (lm == kListOff) note_particle(DN, i);
        }
        if (lm != kListOff) walk_near<true>(L, i, lm, p, vis);
        else if (listed) walk_full<true>(F, i, fm, p, vis);
        else walk_seq(P, S, i, pa[i], p, cs, ce, vis, false, &deferred);
        const float li = vis.finish(S.rho0);
        lambda[i] = li;
        if (pl) pl[i] = make_float4(pi.x, pi.y, pi.z, li);
        if (aux) vis.store_aux(aux, P.N, i);
        return;
    } else if (L.list) {
        // the walk stores the near list; the sums then run over it when it fits
        Recorder<NullVisit> rec(NullVisit{}, L, i, pi, P.cut2);
        walk_seq(P, S, i, pa[i], p, cs, ce, rec, true, &deferred);
        const uint32_t lm = deferred ? kListOff : rec.meta();
        L.meta[i] = lm;
        if (lm == kListOff) note_particle(DN, i);
        if (!deferred) {
            if (lm != kListOff) walk_near<true>(L, i, lm, p, vis);
            else walk_seq(P, S, i, pa[i], p, cs, ce, vis, false, &deferred);
            const float li = vis.finish(S.rho0);
            lambda[i] = li;
            if (pl) pl[i] = make_float4(pi.x, pi.y, pi.z, li);
            if (aux) vis.store_aux(aux, P.N, i);
            return;
        }
    } else {
        walk_seq(P, S, i, pa[i], p, cs, ce, vis, true, &deferred);
    }
    if (deferred) {
        if (defer_particle(D, i)) return;
        vis.reset();
        walk_seq(P, S, i, pa[i], p, cs, ce, vis, false, &deferred);
    }
    const float li = vis.finish(S.rho0);
    lambda[i] = li;
    if (pl) pl[i] = make_float4(pi.x, pi.y, pi.z, li);
    if (aux) vis.store_aux(aux, P.N, i);
}

// One warp computes lambda_i.  With L, it also leaves the particle's near list for the delta pass (and
// sums over that), or notes the particle in DN: the cell-end range's 512 entries hold ~6 near ones, and
// walked again in the delta pass they held it up (21 us against 13 for lambda_list with 33k particles).  Which
// particles have a row is a matter of which came first: the sums are those of the walk, also of positions that
// are not numbers.
__device__ __noinline__ void coop_lambda(const DevParams& P, const float4* __restrict__ p, const float4* __restrict__ pa,
                                            const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce,
                                            float* __restrict__ lambda, float4* __restrict__ aux, uint32_t i,
                                            const LongLists& LL, const NbList& F, const NbList& L, const DeferList& DN,
                                            float4* __restrict__ pl) {
    const SceneCtx S = scene_ctx(P, i);
    const float4 pi = p[i];
    LambdaVisit vis(P, pi);
    uint32_t lm = kListOff;
    if (L.list) {
        const WarpList W = warp_list(LL, F, i);
        if (W.row) lm = filter_group<32, true>([&](uint32_t k) { return W.grouped ? full_at(F, i, k) : W.row + k; }, W.n, W.nc, L, i, pi, P.cut2, p);
        if (lane_id() == 0) {
            L.meta[i] = lm;
            if (lm == kListOff) note_particle(DN, i);
        }
    }
    if (lm != kListOff) walk_list_warp([&](uint32_t k) { return L.list + (size_t)k * L.stride + i; }, lm & 0xFFu, lm >> 8, i, p, vis);
    else walk_warp(P, S, i, pa[i], p, cs, ce, LL, F, vis);
    if (lane_id() == 0) {
        const float li = vis.finish(S.rho0);
        lambda[i] = li;
        if (pl) pl[i] = make_float4(pi.x, pi.y, pi.z, li);
        if (aux) vis.store_aux(aux, P.N, i);
    }
}

__global__ void __launch_bounds__(128)
lambda_coop_kernel(const __grid_constant__ DevParams P, const float4* __restrict__ p, const float4* __restrict__ pa, const uint32_t* __restrict__ cs,
                   const uint32_t* __restrict__ ce, float* __restrict__ lambda, DeferList D, float4* __restrict__ aux) {
    for_each_deferred(D, [&](uint32_t i) { coop_lambda(P, p, pa, cs, ce, lambda, aux, i, LongLists{}, NbList{}, NbList{}, DeferList{}, nullptr); });
}

// After lambda_kernel stored the full lists: the particles left without one (the set DF), a warp
// each.  Stores their long rows, computes their lambda and leaves their near lists.
__global__ void __launch_bounds__(128)
lambda_long_kernel(const __grid_constant__ DevParams P, const float4* __restrict__ p, const float4* __restrict__ pa, const uint32_t* __restrict__ cs,
                   const uint32_t* __restrict__ ce, float* __restrict__ lambda, DeferList DF, float4* __restrict__ aux,
                   const __grid_constant__ LongLists LL, const __grid_constant__ NbList F, const __grid_constant__ NbList L,
                   const __grid_constant__ DeferList DN, float4* __restrict__ pl) {
    const uint32_t n = min(*DF.count, DF.cap);
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t q = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); q < n; q += warps) {
        const uint32_t i = DF.items[q];
        if (F.meta[i] & kListWalked) continue;
        if (q < LL.slots) {
            const uint32_t m = store_row(P, scene_ctx(P, i), i, pa[i], cs, ce, LL.list + (size_t)q * kLongMax);
            if (lane_id() == 0) LL.meta[q] = m;
            __syncwarp();
        }
        coop_lambda(P, p, pa, cs, ce, lambda, aux, i, LL, F, L, DN, pl);
    }
}

// The frame's later lambda passes: read the full list (no cell tables), record the near list.
// The particles without a full list (the set C) are walked by the leading blocks; the ones left
// without a near list are noted in DN for the delta pass.  Kept apart from lambda_kernel so that
// its register budget is the list walk's alone.
// kNear: with near lists (L).  Blocks of 256 per SM: 6 with them (62 us with 1M particles; 5 66, 4 74), 5
// over full lists (147 us with 1M dense particles; 4 155, 6 167).
template <bool kUnitW, bool kNear>
__global__ void __launch_bounds__(256, kNear ? 6 : 5)
lambda_list_kernel(const __grid_constant__ DevParams P, const float4* __restrict__ p, const float4* __restrict__ pa,
                   const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce, float* __restrict__ lambda,
                   CoopSet C, const __grid_constant__ DeferList DN, float4* __restrict__ aux, const __grid_constant__ NbList L, const __grid_constant__ NbList F, const __grid_constant__ LongLists LL,
                   float4* __restrict__ pl) {
    if (blockIdx.x < C.blocks) {
        run_coop_set(C, [&](uint32_t i) { coop_lambda(P, p, pa, cs, ce, lambda, aux, i, LL, F, L, DN, pl); });
        return;
    }
    const uint32_t i = (blockIdx.x - C.blocks) * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    const uint32_t fm = F.meta[i];
    if (fm & kListOff) return;   // in the set C
    const SceneCtx S = scene_ctx(P, i);
    const float4 pi = p[i];
    LambdaVisitT<kUnitW> vis(P, pi);
    uint32_t lm = kListOff;
    if constexpr (kNear) {
        lm = filter_list<false, kUnitW>(P, F, fm, L, i, pi, p);
        L.meta[i] = lm;
        if (lm == kListOff) note_particle(DN, i);
        if (lm != kListOff) walk_near<true>(L, i, lm, p, vis);
    }
    if (lm == kListOff) walk_full(F, i, fm, p, vis);
    const float li = vis.finish(S.rho0);
    lambda[i] = li;
    if (pl) pl[i] = make_float4(pi.x, pi.y, pi.z, li);
    if (aux) vis.store_aux(aux, P.N, i);
}

// The passes of a small simulation: G lanes per particle.  With a thread per particle a 4,275-particle
// pass is 34 blocks on 152 SMs, each thread a serial chain of list loads, position loads and adds; a
// group takes the loads of G entries at a time.  The sums are added in list order all the same.
//
// The frame's first lambda pass (lambda_kernel with full lists): the list enumerated, stored and
// filtered by the group.  Particles without a full list go to lambda_long_kernel.
template <int G>
__global__ void __launch_bounds__(256)
lambda_group_kernel(const __grid_constant__ DevParams P, const float4* __restrict__ p, const float4* __restrict__ pa,
                    const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce, float* __restrict__ lambda,
                    float4* __restrict__ aux, const __grid_constant__ NbList L, const __grid_constant__ NbList F,
                    DeferList DF, DeferList DN) {
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    const bool on = tid / G < P.N, first = on && tid % G == 0u;
    const uint32_t i = on ? tid / G : P.N - 1u;
    const SceneCtx S = scene_ctx(P, i);
    const float4 pi = p[i];
    const GroupList R = enumerate_group<G>(P, S, i, pa[i], on, cs, ce, min(P.M, F.kmax + 1u), true,
                                           [&](uint32_t k, uint32_t j) { if (k < F.kmax) *full_at(F, i, k) = j; });
    __syncwarp();
    const bool listed = on && !R.handed_over && R.n <= F.kmax;
    if (first) F.meta[i] = listed ? (R.n | (R.nc << 8)) : (kListOff | note_particle(DF, i));
    uint32_t lm = kListOff;
    if (L.list) {
        lm = filter_group<G>([&](uint32_t k) { return full_at(F, i, k); }, listed ? R.n : 0u, R.nc, L, i, pi, P.cut2, p);
        if (!listed) lm = kListOff;
        if (first && listed) {
            L.meta[i] = lm;
            if (lm == kListOff) note_particle(DN, i);
        }
    }
    LambdaVisit vis(P, pi);
    const bool near = lm != kListOff;
    walk_group_sums<G>([&](uint32_t k) { return near ? L.list + (size_t)k * L.stride + i : full_at(F, i, k); },
                  !listed ? 0u : (near ? lm & 0xFFu : R.n), 0u, i, p, vis);
    if (first && listed) {
        lambda[i] = vis.finish(S.rho0);
        if (aux) vis.store_aux(aux, P.N, i);
    }
}

// lambda_list_kernel with G lanes per particle.
template <int G>
__global__ void __launch_bounds__(256)
lambda_list_group_kernel(const __grid_constant__ DevParams P, const float4* __restrict__ p, const float4* __restrict__ pa,
                         const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce, float* __restrict__ lambda,
                         CoopSet C, const __grid_constant__ DeferList DN, float4* __restrict__ aux, const __grid_constant__ NbList L,
                         const __grid_constant__ NbList F, const __grid_constant__ LongLists LL) {
    if (blockIdx.x < C.blocks) {
        run_coop_set(C, [&](uint32_t i) { coop_lambda(P, p, pa, cs, ce, lambda, aux, i, LL, F, L, DN, nullptr); });
        return;
    }
    const uint32_t tid = (blockIdx.x - C.blocks) * blockDim.x + threadIdx.x;
    const bool on = tid / G < P.N, first = on && tid % G == 0u;
    const uint32_t i = on ? tid / G : P.N - 1u;
    const uint32_t fm = F.meta[i];
    const bool listed = on && !(fm & kListOff);
    const float4 pi = p[i];
    uint32_t lm = kListOff;
    if (L.list) {
        lm = filter_group<G>([&](uint32_t k) { return full_at(F, i, k); }, listed ? fm & 0xFFu : 0u, (fm >> 8) & 0xFFu, L, i, pi, P.cut2, p);
        if (!listed) lm = kListOff;
        if (first && listed) {
            L.meta[i] = lm;
            if (lm == kListOff) note_particle(DN, i);
        }
    }
    LambdaVisit vis(P, pi);
    const bool near = lm != kListOff;
    walk_group_sums<G>([&](uint32_t k) { return near ? L.list + (size_t)k * L.stride + i : full_at(F, i, k); },
                  !listed ? 0u : (near ? lm & 0xFFu : fm & 0xFFu), 0u, i, p, vis);
    if (first && listed) {
        lambda[i] = vis.finish(scene_ctx(P, i).rho0);
        if (aux) vis.store_aux(aux, P.N, i);
    }
}

// ======================================================================================
// computeDeltaPositions (Density.h:104-145) + solveCollisions type 0 (Collision.h:171-242,
// Jacobi: contacts read the frame's snapshot, the adds of particle i apply in list order)
// + applyDeltaPositions (Density.h:156-168) + updatePositions (Update.h:11-32).
// ======================================================================================
enum DeltaMode : uint32_t {
    kDoDelta = 1u << 0,      // compute delta p from lambda
    kDoCollide = 1u << 1,    // one solveCollisions pass over the contacts
    kDoApply = 1u << 2,      // p -= delta
    kLoadDelta = 1u << 3,    // delta from the buffer (not computed in this pass)
    kStoreDelta = 1u << 4,   // keep delta in the buffer
    kDoUpdate = 1u << 5,     // v = (p - x)/dt; x = p
};

// What a delta visitor knows at compile time: kDeltaAny nothing (the mode, the inverse masses, the
// exponent and far_pairs_zero are looked at for every entry); kDeltaPlain a pass with the density
// part, the contacts, config.txt's nSCorr = 4, far pairs exactly zero, every p.w 1 (LambdaVisitT's
// kUnitW) and no inverse masses; kDeltaMass the same with inverse masses.  These two take a neighbour's
// lambda from the w of its position (the lambda pass's pl), one gather per entry instead of two.  The
// arithmetic is the same.
enum DeltaKnown : uint32_t { kDeltaAny = 0, kDeltaPlain = 1, kDeltaMass = 2 };

template <uint32_t kKnown>
struct DeltaVisitT {
    // coef * r is the density part, t * (-r) the contact part; add() applies both with explicit
    // FMAs, so every walker (cells, lists, cooperative warp) rounds them the same way
    struct Contrib { float coef, rx, ry, rz, rw, t, r2, s; bool d, c; };   // d: the density part adds, c: the contact part
    static constexpr bool kKnow = kKnown != kDeltaAny;
    static constexpr bool kTestsContacts = true;
    const DevParams& P;
    const float* __restrict__ lambda;
    const float* __restrict__ w;       // inverse masses, or null (all 1, the reference)
    float4 pi;
    float li, wi;
    bool do_delta, do_collide, all_pairs;
    float ax = 0.f, ay = 0.f, az = 0.f, aw = 0.f;   // sum of (li + lj + sCorr) * grad
    float4 pacc, xacc;                               // positions with the contact corrections added in order
    float4 xi;
    __device__ DeltaVisitT(const DevParams& P_, const float* lam, const float* w_, float4 pi_, float li_, float wi_,
                           bool dd, bool dc, float4 xi_)
        : P(P_), lambda(lam), w(w_), pi(pi_), li(li_), wi(wi_), do_delta(kKnow || dd), do_collide(kKnow || dc),
          all_pairs(!kKnow && P_.far_pairs_zero == 0u), pacc(pi_), xacc(xi_), xi(xi_) {}
    __device__ void reset() { ax = ay = az = aw = 0.f; pacc = pi; xacc = xi; }
    __device__ static Contrib zero() { return Contrib{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, false, false}; }
    __device__ static bool effective(const Contrib& c) { return c.d || c.c; }
    __device__ static Contrib shfl(const Contrib& c, int k) {
        const uint32_t f = shfl_u((c.d ? 1u : 0u) | (c.c ? 2u : 0u), k);
        return Contrib{shfl_f(c.coef, k), shfl_f(c.rx, k), shfl_f(c.ry, k), shfl_f(c.rz, k), shfl_f(c.rw, k),
                       shfl_f(c.t, k), 0.f, 0.f, (f & 1u) != 0u, (f & 2u) != 0u};
    }
    __device__ __forceinline__ void end_contacts(uint32_t) {}
    using Extra = float;   // lambda_j
    __device__ __forceinline__ float fetch(uint32_t j) const { return (!kKnow && do_delta) ? __ldg(lambda + j) : 0.f; }
    __device__ __forceinline__ bool masses() const { return kKnown == kDeltaPlain ? false : (kKnown == kDeltaMass ? true : w != nullptr); }
    // the contact part's t of an entry at distance dist; false when they do not touch
    __device__ __forceinline__ bool contact_t(uint32_t j, float dist, float& t) const {
        const float overlap = P.d - dist;
        if (!(overlap > 0.0f && dist > 0.00001f)) return false;
        // share of the overlap this particle takes: inverseMass1 / (inverseMass1 + inverseMass2)
        // (Collision.h:223-225, where both are forced to 1); solids have inverse mass 0
        float share = 0.5f;
        if (masses()) {
            const float wj = __ldg(w + j);
            share = (wi + wj) > 0.0f ? wi / (wi + wj) : 0.0f;
        }
        // -share * overlap * (1 - stiffness) along -r / |r|
        t = __fmul_rn(__fmul_rn(-share * overlap, rcp_fast(dist)), P.one_minus_stiffness);
        return share != 0.0f;
    }
    __device__ __forceinline__ void add_contact(float rx, float ry, float rz, float t) {
        pacc.x = __fmaf_rn(-rx, t, pacc.x); xacc.x = __fmaf_rn(-rx, t, xacc.x);
        pacc.y = __fmaf_rn(-ry, t, pacc.y); xacc.y = __fmaf_rn(-ry, t, xacc.y);
        pacc.z = __fmaf_rn(-rz, t, pacc.z); xacc.z = __fmaf_rn(-rz, t, xacc.z);
    }
    __device__ __forceinline__ Contrib contrib(uint32_t j, const float4& pj, float lj_, bool contact) const {
        const float rx = pi.x - pj.x, ry = pi.y - pj.y, rz = pi.z - pj.z, rw = kKnow ? 0.0f : pi.w - pj.w;
        const float lj = kKnow ? pj.w : lj_;
        const float r2 = dist2(rx, ry, rz);
        const float dist = sqrt_fast(r2);
        const bool near = all_pairs || !(r2 >= P.cut2);
        Contrib c{0.f, rx, ry, rz, rw, 0.f, r2, 0.f, false, false};
        if (do_delta) {
            const float s = spiky_scale(P, dist, kKnow ? r2 : __fmaf_rn(rw, rw, r2));
            const float q = __fmul_rn(poly6(P, dist), P.inv_wq);
            const float sc = __fmul_rn(-P.k_scorr, kKnow ? ((q * q) * q) * q : powi(q, P.n_scorr));
            c.coef = __fmul_rn(__fadd_rn(__fadd_rn(li, lj), sc), s);
            c.s = s;
            c.d = near && (s != 0.0f || all_pairs);
        }
        if (contact && do_collide && near) c.c = contact_t(j, dist, c.t);
        return c;
    }
    __device__ __forceinline__ void add(const Contrib& c, bool) {
        if (c.d) {
            ax = __fmaf_rn(c.coef, c.rx, ax); ay = __fmaf_rn(c.coef, c.ry, ay);
            az = __fmaf_rn(c.coef, c.rz, az);
            if constexpr (!kKnow) aw = __fmaf_rn(c.coef, c.rw, aw);
        }
        if (c.c) add_contact(c.rx, c.ry, c.rz, c.t);
    }
    // the density part predicated (LambdaVisitT::add_if); contacts are rare enough for a branch
    __device__ __forceinline__ void add_if(uint32_t k, uint32_t n, const Contrib& c) {
        if constexpr (kKnow) {
            asm("{ .reg .pred q; setp.lt.u32 q, %3, %4; setp.ltu.and.f32 q, %5, %6, q; setp.neu.and.f32 q, %7, 0f00000000, q;"
                " @q fma.rn.f32 %0, %8, %9, %0; @q fma.rn.f32 %1, %8, %10, %1; @q fma.rn.f32 %2, %8, %11, %2; }"
                : "+f"(ax), "+f"(ay), "+f"(az)
                : "r"(k), "r"(n), "f"(c.r2), "f"(P.cut2), "f"(c.s), "f"(c.coef), "f"(c.rx), "f"(c.ry), "f"(c.rz));
        } else {
            asm("{ .reg .pred q; setp.ne.u32 q, %4, 0; @q fma.rn.f32 %0, %5, %6, %0; @q fma.rn.f32 %1, %5, %7, %1;"
                " @q fma.rn.f32 %2, %5, %8, %2; @q fma.rn.f32 %3, %5, %9, %3; }"
                : "+f"(ax), "+f"(ay), "+f"(az), "+f"(aw)
                : "r"((k < n && c.d) ? 1u : 0u), "f"(c.coef), "f"(c.rx), "f"(c.ry), "f"(c.rz), "f"(c.rw));
        }
        if (c.c && k < n) add_contact(c.rx, c.ry, c.rz, c.t);
    }
    // LambdaVisitT::add_two (a NaN adds nothing here, so i itself never does); a pass of unknown kind
    // (kDeltaAny) adds every entry by itself
    static constexpr bool kAddTwo = kKnow;
    template <bool kContacts>   // some entry of the group is a contact (k0, k1: this one)
    __device__ __forceinline__ void add_two(uint32_t j0, const float4& p0, bool k0, uint32_t j1, const float4& p1, bool k1) {
        float x[2], y[2], z[2], d[2], a[2], c[2], s[2], l[2];
        f2_split(sub2(f2(pi.x, pi.y), f2(p0.x, p0.y)), x[0], y[0]);
        f2_split(sub2(f2(pi.x, pi.y), f2(p1.x, p1.y)), x[1], y[1]);
        z[0] = pi.z - p0.z; z[1] = pi.z - p1.z;
        const float r0 = dist2(x[0], y[0], z[0]), r1 = dist2(x[1], y[1], z[1]);
        d[0] = sqrt_fast(r0); d[1] = sqrt_fast(r1);
        const F2 dd = f2(d[0], d[1]), aa = sub2(f2(P.hs, P.hs), dd);
        const F2 ss = spiky_open(P, aa, f2(rsqrt_fast(r0), rsqrt_fast(r1)));
        const F2 q = mul2(poly6_open(P, dd), f2(P.inv_wq, P.inv_wq));
        f2_split(mul2(f2(-P.k_scorr, -P.k_scorr), mul2(mul2(mul2(q, q), q), q)), c[0], c[1]);
        f2_split(aa, a[0], a[1]);
        l[0] = __fadd_rn(li, p0.w); l[1] = __fadd_rn(li, p1.w);   // w: the entry's lambda
#pragma unroll
        for (int b = 0; b < 2; ++b)
            asm("{ .reg .pred q; setp.gt.f32 q, %1, %2; setp.lt.and.f32 q, %1, %3, q; @q add.rn.f32 %0, %0, %4; }"
                : "+f"(l[b]) : "f"(d[b]), "f"(0.001f), "f"(P.hp_lim), "f"(c[b]));
        f2_split(mul2(f2(l[0], l[1]), ss), c[0], c[1]);
        f2_split(ss, s[0], s[1]);
#pragma unroll
        for (int b = 0; b < 2; ++b)
            asm("{ .reg .pred q; setp.gt.f32 q, %3, %5; setp.gt.and.f32 q, %4, %5, q; setp.neu.and.f32 q, %6, 0f00000000, q;"
                " @q fma.rn.f32 %0, %7, %8, %0; @q fma.rn.f32 %1, %7, %9, %1; @q fma.rn.f32 %2, %7, %10, %2; }"
                : "+f"(ax), "+f"(ay), "+f"(az)
                : "f"(d[b]), "f"(a[b]), "f"(0.0001f), "f"(s[b]), "f"(c[b]), "f"(x[b]), "f"(y[b]), "f"(z[b]));
        if constexpr (kContacts) {
            float t;
            if (k0 && contact_t(j0, d[0], t)) add_contact(x[0], y[0], z[0], t);
            if (k1 && contact_t(j1, d[1], t)) add_contact(x[1], y[1], z[1], t);
        }
    }
    // walk_group_sums: the density part's sums, then the contacts' on p* and x, from coef, -t and r.  The parts
    // share r, times 0 in the sums that an entry is not part of: only for passes whose far pairs are exactly
    // zero, where an entry of either part is in reach and its r finite (else a NaN position, which every pair
    // beyond the kernels has a part in, would reach the contacts' sums, and x).
    static constexpr int kRows = 6, kSums = 10;
    __device__ static constexpr int mul_row(int s) { return s < 4 ? 0 : 1; }
    __device__ static constexpr int val_row(int s) { return s < 4 ? 2 + s : (s < 7 ? s - 2 : s - 5); }
    __device__ __forceinline__ float& sum(int s) {
        return s == 0 ? ax : (s == 1 ? ay : (s == 2 ? az : (s == 3 ? aw : (s == 4 ? pacc.x : (s == 5 ? pacc.y : (s == 6 ? pacc.z
               : (s == 7 ? xacc.x : (s == 8 ? xacc.y : xacc.z))))))));
    }
    __device__ __forceinline__ static void rows(const Contrib& c, bool live, float* r) {
        const bool f = live && (c.d || c.c);
        r[0] = (live && c.d) ? c.coef : 0.f;
        r[1] = (live && c.c) ? -c.t : 0.f;
        r[2] = f ? c.rx : 0.f; r[3] = f ? c.ry : 0.f; r[4] = f ? c.rz : 0.f;
        r[5] = (live && c.d) ? c.rw : 0.f;
    }
};
using DeltaVisit = DeltaVisitT<kDeltaAny>;

template <class V>
__device__ __forceinline__ void delta_finish(const DevParams& P, float rho0, uint32_t mode, uint32_t i, const V& vis,
                                             float4* __restrict__ pout, float4* __restrict__ x, float4* __restrict__ v,
                                             float4* __restrict__ delta) {
    // a solid (inverse mass 0) takes no density correction
    float4 pn = vis.pacc, xn = vis.xacc;
    float4 dp = make_float4(0.f, 0.f, 0.f, 0.f);
    if (mode & kDoDelta)   // correctly rounded: the list and the walking kernels store the same bits
        dp = make_float4(__fdiv_rn(vis.ax, rho0), __fdiv_rn(vis.ay, rho0), __fdiv_rn(vis.az, rho0), __fdiv_rn(vis.aw, rho0));
    else if (mode & kLoadDelta) dp = delta[i];
    if (mode & kStoreDelta) delta[i] = dp;
    if (mode & kDoApply) {
        if (vis.masses()) { dp.x *= vis.wi; dp.y *= vis.wi; dp.z *= vis.wi; dp.w *= vis.wi; }
        pn.x -= dp.x; pn.y -= dp.y; pn.z -= dp.z; pn.w -= dp.w;
    }
    if (mode & kDoUpdate) {
        const float r = P.inv_dt;
        v[i] = make_float4((pn.x - xn.x) * r, (pn.y - xn.y) * r, (pn.z - xn.z) * r, (pn.w - xn.w) * r);
        xn = pn;
    }
    pout[i] = pn;
    if (P.coarse) P.coarse[i] = coarse_pos(pn);
    if (mode & (kDoCollide | kDoUpdate)) x[i] = xn;
}

__global__ void __launch_bounds__(256, 2)
delta_kernel(DevParams P, uint32_t mode, const float4* __restrict__ pin, const float4* __restrict__ pa, float4* __restrict__ pout,
             float4* __restrict__ x, float4* __restrict__ v, const float* __restrict__ lambda, const float* __restrict__ w,
             float4* __restrict__ delta, const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce,
             DeferList D) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    const float4 pi = pin[i];
    const bool need_x = (mode & (kDoCollide | kDoUpdate)) != 0;
    const float4 xi = need_x ? x[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float li = (mode & kDoDelta) ? lambda[i] : 0.f;
    const SceneCtx S = scene_ctx(P, i);
    DeltaVisit vis(P, lambda, w, pi, li, w ? w[i] : 1.0f, (mode & kDoDelta) != 0, (mode & kDoCollide) != 0, xi);
    if (mode & (kDoDelta | kDoCollide)) {
        bool deferred = false;
        walk_seq(P, S, i, pa[i], pin, cs, ce, vis, true, &deferred);
        if (deferred) {
            if (defer_particle(D, i)) return;
            vis.reset();
            walk_seq(P, S, i, pa[i], pin, cs, ce, vis, false, &deferred);
        }
    }
    delta_finish(P, S.rho0, mode, i, vis, pout, x, v, delta);
}

// One warp runs the delta pass for particle i.
__device__ __noinline__ void coop_delta(const DevParams& P, uint32_t mode, const float4* __restrict__ pin,
                                           const float4* __restrict__ pa, float4* __restrict__ pout, float4* __restrict__ x,
                                           float4* __restrict__ v, const float* __restrict__ lambda, const float* __restrict__ w,
                                           float4* __restrict__ delta, const uint32_t* __restrict__ cs,
                                           const uint32_t* __restrict__ ce, uint32_t i, const LongLists& LL,
                                           const NbList& F) {
    const float4 pi = pin[i];
    const bool need_x = (mode & (kDoCollide | kDoUpdate)) != 0;
    const float4 xi = need_x ? x[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float li = (mode & kDoDelta) ? lambda[i] : 0.f;
    const SceneCtx S = scene_ctx(P, i);
    DeltaVisit vis(P, lambda, w, pi, li, w ? w[i] : 1.0f, (mode & kDoDelta) != 0, (mode & kDoCollide) != 0, xi);
    walk_warp(P, S, i, pa[i], pin, cs, ce, LL, F, vis);
    if (lane_id() == 0) delta_finish(P, S.rho0, mode, i, vis, pout, x, v, delta);
}

// delta pass 0 of an iteration over the near lists its lambda pass recorded (kFull = false), or
// any delta pass over the frame's full list when there are no near lists (kFull = true); the
// particles without one (the set C) walk the cells.  kMode != 0: the pass
// mode fixed at compile time (the two passes of a fluid frame), kMode = 0: `mode` at run time; kKnown:
// what else is fixed (DeltaKnown).
// Blocks of 256 per SM by the list it walks (1M particles, GB300): 6 over the near lists (31.3 us;
// 5 33.2), 4 over the full lists, whose groups of four entries take 64 registers (185 us; 5 210 with
// spills, 3 186).
template <uint32_t kMode, bool kFull, uint32_t kKnown>
__global__ void __launch_bounds__(256, kFull ? 4 : 6)
delta_list_kernel(const __grid_constant__ DevParams P, uint32_t mode_rt, const float4* __restrict__ pin, const float4* __restrict__ pa,
                  float4* __restrict__ pout, float4* __restrict__ x, float4* __restrict__ v,
                  const float* __restrict__ lambda, const float* __restrict__ w, float4* __restrict__ delta,
                  const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce, CoopSet C, const __grid_constant__ NbList L, const __grid_constant__ NbList F,
                  const __grid_constant__ LongLists LL, const float4* __restrict__ pl) {
    const uint32_t mode = kMode ? kMode : mode_rt;
    if (blockIdx.x < C.blocks) {
        run_coop_set(C, [&](uint32_t i) { coop_delta(P, mode, pin, pa, pout, x, v, lambda, w, delta, cs, ce, i, LL, F); });
        return;
    }
    const uint32_t i = (blockIdx.x - C.blocks) * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    const uint32_t meta = L.meta[i];
    if (meta & kListOff) return;
    float4 pi;
    float li;
    if constexpr (kKnown != kDeltaAny) {   // p.w is 1
        pi = pl[i];
        li = pi.w;
        pi.w = 1.0f;
    } else {
        pi = pin[i];
        li = (mode & kDoDelta) ? lambda[i] : 0.f;
    }
    const bool need_x = (mode & (kDoCollide | kDoUpdate)) != 0;
    const float4 xi = need_x ? x[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const SceneCtx S = scene_ctx(P, i);
    DeltaVisitT<kKnown> vis(P, lambda, w, pi, li, w ? w[i] : 1.0f, (mode & kDoDelta) != 0, (mode & kDoCollide) != 0, xi);
    const float4* pj = kKnown != kDeltaAny ? pl : pin;
    if constexpr (kFull) walk_full(L, i, meta, pj, vis);
    else walk_near(L, i, meta, pj, vis);
    // the w of the sums: 0 times each coefficient, which is 0 until a coefficient is not finite
    if constexpr (kKnown != kDeltaAny) vis.aw = 0.0f * vis.ax + 0.0f * vis.ay + 0.0f * vis.az;
    delta_finish(P, S.rho0, mode, i, vis, pout, x, v, delta);
}

// delta_list_kernel with G lanes per particle (small simulations, see lambda_group_kernel).
template <bool kFull, int G>
__global__ void __launch_bounds__(256)
delta_list_group_kernel(const __grid_constant__ DevParams P, uint32_t mode, const float4* __restrict__ pin,
                        const float4* __restrict__ pa, float4* __restrict__ pout, float4* __restrict__ x,
                        float4* __restrict__ v, const float* __restrict__ lambda, const float* __restrict__ w,
                        float4* __restrict__ delta, const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce,
                        CoopSet C, const __grid_constant__ NbList L, const __grid_constant__ NbList F,
                        const __grid_constant__ LongLists LL) {
    if (blockIdx.x < C.blocks) {
        run_coop_set(C, [&](uint32_t i) { coop_delta(P, mode, pin, pa, pout, x, v, lambda, w, delta, cs, ce, i, LL, F); });
        return;
    }
    const uint32_t tid = (blockIdx.x - C.blocks) * blockDim.x + threadIdx.x;
    const bool on = tid / G < P.N;
    const uint32_t i = on ? tid / G : P.N - 1u;
    const uint32_t meta = L.meta[i];
    const bool listed = on && !(meta & kListOff);
    const float4 pi = pin[i];
    const bool need_x = (mode & (kDoCollide | kDoUpdate)) != 0;
    const float4 xi = need_x ? x[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float li = (mode & kDoDelta) ? lambda[i] : 0.f;
    DeltaVisit vis(P, lambda, w, pi, li, w ? w[i] : 1.0f, (mode & kDoDelta) != 0, (mode & kDoCollide) != 0, xi);
    walk_group_sums<G>([&](uint32_t k) { return kFull ? full_at(L, i, k) : L.list + (size_t)k * L.stride + i; },
                  listed ? meta & 0xFFu : 0u, (meta >> 8) & 0xFFu, i, pin, vis);
    if (listed && tid % G == 0u) delta_finish(P, scene_ctx(P, i).rho0, mode, i, vis, pout, x, v, delta);
}

__global__ void __launch_bounds__(128)
delta_coop_kernel(const __grid_constant__ DevParams P, uint32_t mode, const float4* __restrict__ pin, const float4* __restrict__ pa, float4* __restrict__ pout,
                  float4* __restrict__ x, float4* __restrict__ v, const float* __restrict__ lambda, const float* __restrict__ w,
                  float4* __restrict__ delta, const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce,
                  DeferList D) {
    for_each_deferred(D, [&](uint32_t i) {
        coop_delta(P, mode, pin, pa, pout, x, v, lambda, w, delta, cs, ce, i, LongLists{}, NbList{});
    });
}

// updatePositions on its own (Update.h:11-32), when no delta pass can carry it.
__global__ void __launch_bounds__(256)
update_kernel(DevParams P, const float4* __restrict__ p, float4* __restrict__ x, float4* __restrict__ v) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    const float4 pp = p[i], xx = x[i];
    const float r = P.inv_dt;
    v[i] = make_float4((pp.x - xx.x) * r, (pp.y - xx.y) * r, (pp.z - xx.z) * r, (pp.w - xx.w) * r);
    x[i] = pp;
}

// ======================================================================================
// computeOmega (Density.h:232-269): omega_i = sum_j (v_j - v_i) x spiky(p_i, p_j)
// ======================================================================================
template <bool kUnitW>   // LambdaVisitT
struct OmegaVisitT {
    struct Contrib { float ox, oy, oz, r2, s; bool near; };
    const DevParams& P;
    const float4* __restrict__ v;
    float4 pi, vi;
    float ox = 0.f, oy = 0.f, oz = 0.f;
    __device__ OmegaVisitT(const DevParams& P_, const float4* v_, float4 pi_, float4 vi_) : P(P_), v(v_), pi(pi_), vi(vi_) {}
    __device__ void reset() { ox = oy = oz = 0.f; }
    __device__ static Contrib zero() { return Contrib{0.f, 0.f, 0.f, 0.f, 0.f, false}; }
    __device__ static bool effective(const Contrib& c) { return c.near; }
    __device__ static Contrib shfl(const Contrib& c, int k) {
        return Contrib{shfl_f(c.ox, k), shfl_f(c.oy, k), shfl_f(c.oz, k), 0.f, 0.f, shfl_u(c.near, k) != 0u};
    }
    __device__ __forceinline__ void end_contacts(uint32_t) {}
    using Extra = float4;   // v_j
    __device__ __forceinline__ float4 fetch(uint32_t j) const { return __ldg(v + j); }
    __device__ __forceinline__ Contrib contrib(uint32_t, const float4& pj, const float4& vj, bool) const {
        const float rx = pi.x - pj.x, ry = pi.y - pj.y, rz = pi.z - pj.z, rw = kUnitW ? 0.0f : pi.w - pj.w;
        const float r2 = dist2(rx, ry, rz);
        const float s = spiky_scale(P, sqrt_fast(r2), kUnitW ? r2 : __fmaf_rn(rw, rw, r2));
        const float wx = vj.x - vi.x, wy = vj.y - vi.y, wz = vj.z - vi.z;
        const float gx = s * rx, gy = s * ry, gz = s * rz;
        return Contrib{__fsub_rn(__fmul_rn(wy, gz), __fmul_rn(wz, gy)), __fsub_rn(__fmul_rn(wz, gx), __fmul_rn(wx, gz)),
                       __fsub_rn(__fmul_rn(wx, gy), __fmul_rn(wy, gx)), r2, s, !(r2 >= P.cut2 || s == 0.0f)};
    }
    __device__ __forceinline__ void add(const Contrib& c, bool) {
        if (!c.near) return;
        ox = __fadd_rn(ox, c.ox); oy = __fadd_rn(oy, c.oy); oz = __fadd_rn(oz, c.oz);
    }
    __device__ __forceinline__ void add_if(uint32_t k, uint32_t n, const Contrib& c) {   // LambdaVisitT::add_if
        asm("{ .reg .pred q; setp.lt.u32 q, %3, %4; setp.ltu.and.f32 q, %5, %6, q; setp.neu.and.f32 q, %7, 0f00000000, q;"
            " @q add.rn.f32 %0, %0, %8; @q add.rn.f32 %1, %1, %9; @q add.rn.f32 %2, %2, %10; }"
            : "+f"(ox), "+f"(oy), "+f"(oz)
            : "r"(k), "r"(n), "f"(c.r2), "f"(P.cut2), "f"(c.s), "f"(c.ox), "f"(c.oy), "f"(c.oz));
    }
    static constexpr int kRows = 3, kSums = 3;   // walk_group_sums
    __device__ static constexpr int mul_row(int) { return kRows; }
    __device__ static constexpr int val_row(int s) { return s; }
    __device__ __forceinline__ float& sum(int s) { return s == 0 ? ox : (s == 1 ? oy : oz); }
    __device__ __forceinline__ static void rows(const Contrib& c, bool live, float* r) {
        const bool on = live && c.near;
        r[0] = on ? c.ox : 0.f; r[1] = on ? c.oy : 0.f; r[2] = on ? c.oz : 0.f;
    }
};
using OmegaVisit = OmegaVisitT<false>;

__global__ void __launch_bounds__(256)
omega_kernel(DevParams P, const float4* __restrict__ p, const float4* __restrict__ pa, const float4* __restrict__ v,
             const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce, float4* __restrict__ omega, DeferList D,
             NbList L, DeferList DN) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    const SceneCtx S = scene_ctx(P, i);
    // walks the cells; L.list: record the near lists for a viscosity pass without vorticity (the
    // particles left without one noted in DN when DN is given)
    const float4 pi = p[i];
    OmegaVisit vis(P, v, pi, v[i]);
    bool deferred = false;
    if (L.list) {
        Recorder<OmegaVisit> rec(vis, L, i, pi, P.cut2);
        walk_seq(P, S, i, pa[i], p, cs, ce, rec, true, &deferred);
        L.meta[i] = deferred ? kListOff : rec.meta();
        if (L.meta[i] == kListOff) note_particle(DN, i);
        if (!deferred) {
            omega[i] = make_float4(rec.inner.ox, rec.inner.oy, rec.inner.oz, 0.f);
            return;
        }
    } else {
        walk_seq(P, S, i, pa[i], p, cs, ce, vis, true, &deferred);
    }
    if (deferred) {
        if (defer_particle(D, i)) return;
        vis.reset();
        walk_seq(P, S, i, pa[i], p, cs, ce, vis, false, &deferred);
    }
    omega[i] = make_float4(vis.ox, vis.oy, vis.oz, 0.f);
}

// One warp computes omega_i.
__device__ __noinline__ void coop_omega(const DevParams& P, const float4* __restrict__ p, const float4* __restrict__ pa,
                                           const float4* __restrict__ v, const uint32_t* __restrict__ cs,
                                           const uint32_t* __restrict__ ce, float4* __restrict__ omega, uint32_t i,
                                           const LongLists& LL, const NbList& F, Pair4* __restrict__ pairs) {
    const SceneCtx S = scene_ctx(P, i);
    const float4 pi = p[i];
    OmegaVisit vis(P, v, pi, v[i]);
    walk_warp(P, S, i, pa[i], p, cs, ce, LL, F, vis);
    if (lane_id() == 0) {
        const float4 o = make_float4(vis.ox, vis.oy, vis.oz, 0.f);
        omega[i] = o;
        if (pairs) pairs[i] = Pair4{pi, o};
    }
}

// omega over the full list (recording the near list when L.list, and noting the particles left
// without one in DN when DN is given); the particles without a full list (the set C) are walked
// by the leading blocks.
// kNear: the pass filters the full list into omega's near list (5 blocks of 256 per SM: 69 us with 1M
// particles; 4 76, 6 71); else it walks the full list (4: 205 us; 3 and 5 4 to 9% slower).
template <bool kNear, bool kUnitW>
__global__ void __launch_bounds__(256, kNear ? 5 : 4)
omega_list_kernel(const __grid_constant__ DevParams P, const float4* __restrict__ p, const float4* __restrict__ pa, const float4* __restrict__ v,
                  const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce, float4* __restrict__ omega,
                  CoopSet C, DeferList DN, const __grid_constant__ NbList L, const __grid_constant__ NbList F, const __grid_constant__ LongLists LL,
                  Pair4* __restrict__ pairs) {
    if (blockIdx.x < C.blocks) {
        run_coop_set(C, [&](uint32_t i) { coop_omega(P, p, pa, v, cs, ce, omega, i, LL, F, pairs); });
        return;
    }
    const uint32_t i = (blockIdx.x - C.blocks) * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    const uint32_t fm = F.meta[i];
    if (fm & kListOff) {
        if (L.list) {
            L.meta[i] = kListOff;
            note_particle(DN, i);
        }
        return;
    }
    const float4 pi = p[i];
    OmegaVisitT<kUnitW> vis(P, v, pi, v[i]);
    const uint32_t lm = L.list ? filter_list<false, kUnitW>(P, F, fm, L, i, pi, p) : kListOff;
    if (L.list) {
        L.meta[i] = lm;
        if (lm == kListOff) note_particle(DN, i);
    }
    if (lm != kListOff) walk_near<true>(L, i, lm, p, vis);
    else walk_full(F, i, fm, p, vis);
    const float4 o = make_float4(vis.ox, vis.oy, vis.oz, 0.f);
    omega[i] = o;
    if (pairs) pairs[i] = Pair4{pi, o};
}

// omega_list_kernel with G lanes per particle (small simulations, see lambda_group_kernel).
template <int G>
__global__ void __launch_bounds__(256)
omega_list_group_kernel(const __grid_constant__ DevParams P, const float4* __restrict__ p, const float4* __restrict__ pa,
                        const float4* __restrict__ v, const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce,
                        float4* __restrict__ omega, CoopSet C, DeferList DN, const __grid_constant__ NbList L,
                        const __grid_constant__ NbList F, const __grid_constant__ LongLists LL) {
    if (blockIdx.x < C.blocks) {
        run_coop_set(C, [&](uint32_t i) { coop_omega(P, p, pa, v, cs, ce, omega, i, LL, F, nullptr); });
        return;
    }
    const uint32_t tid = (blockIdx.x - C.blocks) * blockDim.x + threadIdx.x;
    const bool on = tid / G < P.N, first = on && tid % G == 0u;
    const uint32_t i = on ? tid / G : P.N - 1u;
    const uint32_t fm = F.meta[i];
    const bool listed = on && !(fm & kListOff);
    const float4 pi = p[i];
    uint32_t lm = kListOff;
    if (L.list) {
        lm = filter_group<G>([&](uint32_t k) { return full_at(F, i, k); }, listed ? fm & 0xFFu : 0u, (fm >> 8) & 0xFFu, L, i, pi, P.cut2, p);
        if (!listed) lm = kListOff;
        if (first) {
            L.meta[i] = lm;
            if (lm == kListOff) note_particle(DN, i);
        }
    }
    OmegaVisit vis(P, v, pi, v[i]);
    const bool near = lm != kListOff;
    walk_group_sums<G>([&](uint32_t k) { return near ? L.list + (size_t)k * L.stride + i : full_at(F, i, k); },
                  !listed ? 0u : (near ? lm & 0xFFu : fm & 0xFFu), 0u, i, p, vis);
    if (first && listed) omega[i] = make_float4(vis.ox, vis.oy, vis.oz, 0.f);
}

__global__ void __launch_bounds__(128)
omega_coop_kernel(const __grid_constant__ DevParams P, const float4* __restrict__ p, const float4* __restrict__ pa, const float4* __restrict__ v,
                  const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce, float4* __restrict__ omega,
                  DeferList D) {
    for_each_deferred(D, [&](uint32_t i) { coop_omega(P, p, pa, v, cs, ce, omega, i, LongLists{}, NbList{}, nullptr); });
}

// ======================================================================================
// computeVorticity (Density.h:179-221) + computeViscosity (Density.h:280-310, Jacobi).
// Vorticity sums |omega_j - omega_i| / (p_j - p_i + 1e-8) componentwise over EVERY list
// entry (no kernel weight), so with vorticity on no pair may be skipped.
// ======================================================================================
// kTerms: the terms this visitor may run (1 vorticity, 2 viscosity, 3 either, as the run-time
// flags say); a visitor for one term loads one neighbour vector per entry.
template <uint32_t T> struct VortViscExtra { float4 oj, vj; };
template <> struct VortViscExtra<1u> { float4 oj; };
template <> struct VortViscExtra<2u> { float4 vj; };
template <uint32_t kTerms = 3u>
struct VortViscVisitT {
    struct Contrib { float gx, gy, gz, sx, sy, sz, sw, r2, w; bool vo, vs; };   // which terms add
    const DevParams& P;
    const float4* __restrict__ v;
    const float4* __restrict__ omega;
    float4 pi, vi, oi;
    bool vort, visc;
    float gx = 0.f, gy = 0.f, gz = 0.f;
    float sx = 0.f, sy = 0.f, sz = 0.f, sw = 0.f;
    __device__ VortViscVisitT(const DevParams& P_, const float4* v_, const float4* om, float4 pi_, float4 vi_, float4 oi_,
                              bool vo, bool vs)
        : P(P_), v(v_), omega(om), pi(pi_), vi(vi_), oi(oi_), vort(vo && (kTerms & 1u)), visc(vs && (kTerms & 2u)) {}
    __device__ void reset() { gx = gy = gz = sx = sy = sz = sw = 0.f; }
    __device__ static Contrib zero() { return Contrib{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, false, false}; }
    __device__ static bool effective(const Contrib& c) { return c.vo || c.vs; }
    __device__ static Contrib shfl(const Contrib& c, int k) {
        const uint32_t f = shfl_u((c.vo ? 1u : 0u) | (c.vs ? 2u : 0u), k);
        return Contrib{shfl_f(c.gx, k), shfl_f(c.gy, k), shfl_f(c.gz, k), shfl_f(c.sx, k),
                       shfl_f(c.sy, k), shfl_f(c.sz, k), shfl_f(c.sw, k), 0.f, 0.f, (f & 1u) != 0u, (f & 2u) != 0u};
    }
    __device__ __forceinline__ void end_contacts(uint32_t) {}
    using Extra = VortViscExtra<kTerms>;
    __device__ __forceinline__ Extra fetch(uint32_t j) const {
        Extra e;
        if constexpr ((kTerms & 1u) != 0u) e.oj = vort ? __ldg(omega + j) : make_float4(0.f, 0.f, 0.f, 0.f);
        if constexpr ((kTerms & 2u) != 0u) e.vj = visc ? __ldg(v + j) : make_float4(0.f, 0.f, 0.f, 0.f);
        return e;
    }
    __device__ __forceinline__ Contrib contrib(uint32_t, const float4& pj, const Extra& ex, bool) const {
        Contrib c = zero();
        if constexpr ((kTerms & 1u) != 0u) if (vort) {
            const float4 oj = ex.oj;
            const float dx = oj.x - oi.x, dy = oj.y - oi.y, dz = oj.z - oi.z;
            const float ol = sqrtf(dist2(dx, dy, dz));   // not sqrt_fast: omegas may differ by less than 1e-19
            // the fast division: the divisors (position differences + 1e-8) stay far below 2^126
            c.gx = __fdividef(ol, (pj.x - pi.x) + 0.00000001f);
            c.gy = __fdividef(ol, (pj.y - pi.y) + 0.00000001f);
            c.gz = __fdividef(ol, (pj.z - pi.z) + 0.00000001f);
            c.vo = true;
        }
        if constexpr ((kTerms & 2u) != 0u) if (visc) {
            const float rx = pi.x - pj.x, ry = pi.y - pj.y, rz = pi.z - pj.z;
            const float r2 = dist2(rx, ry, rz);
            const float W = poly6(P, sqrt_fast(r2));
            const float4 vj = ex.vj;
            c.sx = (vj.x - vi.x) * W; c.sy = (vj.y - vi.y) * W;
            c.sz = (vj.z - vi.z) * W; c.sw = (vj.w - vi.w) * W;
            c.r2 = r2;
            c.w = W;
            c.vs = !(r2 >= P.hp2) && W != 0.0f;
        }
        return c;
    }
    __device__ __forceinline__ void add(const Contrib& c, bool) {
        if (c.vo) { gx = __fadd_rn(gx, c.gx); gy = __fadd_rn(gy, c.gy); gz = __fadd_rn(gz, c.gz); }
        if (c.vs) { sx = __fadd_rn(sx, c.sx); sy = __fadd_rn(sy, c.sy); sz = __fadd_rn(sz, c.sz); sw = __fadd_rn(sw, c.sw); }
    }
    __device__ __forceinline__ void add_if(uint32_t k, uint32_t n, const Contrib& c) {   // LambdaVisitT::add_if
        if constexpr ((kTerms & 1u) != 0u) if (vort)
            asm("{ .reg .pred q; setp.lt.u32 q, %3, %4; @q add.rn.f32 %0, %0, %5; @q add.rn.f32 %1, %1, %6; @q add.rn.f32 %2, %2, %7; }"
                : "+f"(gx), "+f"(gy), "+f"(gz) : "r"(k), "r"(n), "f"(c.gx), "f"(c.gy), "f"(c.gz));
        if constexpr ((kTerms & 2u) != 0u) if (visc)
            asm("{ .reg .pred q; setp.lt.u32 q, %4, %5; setp.ltu.and.f32 q, %6, %7, q; setp.neu.and.f32 q, %8, 0f00000000, q;"
                " @q add.rn.f32 %0, %0, %9; @q add.rn.f32 %1, %1, %10; @q add.rn.f32 %2, %2, %11; @q add.rn.f32 %3, %3, %12; }"
                : "+f"(sx), "+f"(sy), "+f"(sz), "+f"(sw)
                : "r"(k), "r"(n), "f"(c.r2), "f"(P.hp2), "f"(c.w), "f"(c.sx), "f"(c.sy), "f"(c.sz), "f"(c.sw));
    }
    static constexpr int kRows = 7, kSums = 7;   // walk_group_sums
    __device__ static constexpr int mul_row(int) { return kRows; }
    __device__ static constexpr int val_row(int s) { return s; }
    __device__ __forceinline__ float& sum(int s) {
        return s == 0 ? gx : (s == 1 ? gy : (s == 2 ? gz : (s == 3 ? sx : (s == 4 ? sy : (s == 5 ? sz : sw)))));
    }
    __device__ __forceinline__ static void rows(const Contrib& c, bool live, float* r) {
        const bool vo = live && c.vo, vs = live && c.vs;
        r[0] = vo ? c.gx : 0.f; r[1] = vo ? c.gy : 0.f; r[2] = vo ? c.gz : 0.f;
        r[3] = vs ? c.sx : 0.f; r[4] = vs ? c.sy : 0.f; r[5] = vs ? c.sz : 0.f; r[6] = vs ? c.sw : 0.f;
    }
};

using VortViscVisit = VortViscVisitT<3u>;

// The same with an entry's position and omega from the omega pass's pairs: one 32-byte gather instead
// of two of 16 (vorticity on).
template <uint32_t kTerms>
struct VortPairVisitT : VortViscVisitT<kTerms> {
    using Base = VortViscVisitT<kTerms>;
    using Extra = typename Base::Extra;
    const Pair4* __restrict__ pairs;
    __device__ VortPairVisitT(const Base& b, const Pair4* q) : Base(b), pairs(q) {}
    __device__ __forceinline__ void load(uint32_t j, float4& pj, Extra& ex) const {
        const Pair4 q = load_pair(pairs + j);
        pj = q.a;
        ex.oj = q.b;
        if constexpr ((kTerms & 2u) != 0u) ex.vj = this->visc ? __ldg(this->v + j) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
};

// The vorticity force from the vorticity sums of `vo` and the viscosity update from the sums of
// `vs` (the same visitor when one walk summed both terms).  Explicitly rounded, so every kernel
// that finishes a particle stores the same bits.  `vhost` (mapped pinned host memory, or null)
// also receives the new velocity: a frame that reads its state back gets v without a copy after
// the pass.
template <class VO, class VS>
__device__ __forceinline__ void vort_visc_finish(const DevParams& P, uint32_t i, const VO& vo, const VS& vs,
                                                 float4* __restrict__ vout, float4* __restrict__ fext,
                                                 const float* __restrict__ w, float4* __restrict__ vhost = nullptr) {
    if (vo.vort) {
        if (P.eta_tape) P.eta_tape[i] = make_float4(vo.gx, vo.gy, vo.gz, 0.f);
        const float EPS = 0.00000001f;
        const float gl = sqrtf(__fmaf_rn(vo.gz, vo.gz, __fmaf_rn(vo.gy, vo.gy, __fmul_rn(vo.gx, vo.gx))));
        const float inv = 1.0f / __fadd_rn(gl, EPS);
        const float nx = __fmul_rn(inv, __fadd_rn(vo.gx, EPS)), ny = __fmul_rn(inv, __fadd_rn(vo.gy, EPS)),
                    nz = __fmul_rn(inv, __fadd_rn(vo.gz, EPS));
        const float e = P.e_vort;
        const float4 oi = vo.oi;
        fext[i] = make_float4(__fmul_rn(e, __fmaf_rn(ny, oi.z, -__fmul_rn(nz, oi.y))),
                              __fmul_rn(e, __fmaf_rn(nz, oi.x, -__fmul_rn(nx, oi.z))),
                              __fmul_rn(e, __fmaf_rn(nx, oi.y, -__fmul_rn(ny, oi.x))), 0.f);
    }
    if (vs.visc) {
        const float c = w ? __fmul_rn(w[i], P.c_visc) : P.c_visc;   // a solid keeps its velocity
        const float4 vi = vs.vi;
        const float4 vn = make_float4(__fmaf_rn(c, vs.sx, vi.x), __fmaf_rn(c, vs.sy, vi.y), __fmaf_rn(c, vs.sz, vi.z),
                                      __fmaf_rn(c, vs.sw, vi.w));
        vout[i] = vn;
        if (vhost) vhost[i] = vn;
    }
}

__global__ void __launch_bounds__(256, 2)
vort_visc_kernel(DevParams P, const float4* __restrict__ p, const float4* __restrict__ pa, const float4* __restrict__ vin,
                 float4* __restrict__ vout, const float4* __restrict__ omega, float4* __restrict__ fext,
                 const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce, int do_vort, int do_visc,
                 const float* __restrict__ w, DeferList D) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    const float4 oi = do_vort ? omega[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const SceneCtx S = scene_ctx(P, i);
    VortViscVisit vis(P, vin, omega, p[i], vin[i], oi, do_vort != 0, do_visc != 0);
    bool deferred = false;
    walk_seq(P, S, i, pa[i], p, cs, ce, vis, true, &deferred);
    if (deferred) {
        if (defer_particle(D, i)) return;
        vis.reset();
        walk_seq(P, S, i, pa[i], p, cs, ce, vis, false, &deferred);
    }
    vort_visc_finish(P, i, vis, vis, vout, fext, w);
}

// One warp runs vorticity + viscosity for particle i.
__device__ __noinline__ void coop_vort_visc(const DevParams& P, const float4* __restrict__ p, const float4* __restrict__ pa,
                                               const float4* __restrict__ vin, float4* __restrict__ vout,
                                               const float4* __restrict__ omega, float4* __restrict__ fext,
                                               const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce,
                                               int do_vort, int do_visc, const float* __restrict__ w, uint32_t i,
                                               float4* __restrict__ vhost, const LongLists& LL, const NbList& F) {
    const float4 oi = do_vort ? omega[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const SceneCtx S = scene_ctx(P, i);
    VortViscVisit vis(P, vin, omega, p[i], vin[i], oi, do_vort != 0, do_visc != 0);
    walk_warp(P, S, i, pa[i], p, cs, ce, LL, F, vis);
    if (lane_id() == 0) vort_visc_finish(P, i, vis, vis, vout, fext, w, vhost);
}

// vorticity + viscosity over a stored list (the full list with vorticity, else the omega pass's
// near list); the particles without one (the set C) are walked by the leading blocks.  With both
// terms and the omega pass's near list Ln at hand, vorticity runs over the full list and
// viscosity over the near list (its entries beyond the cut add exact zeros): the two sums keep
// their own order.
// Blocks of 256 per SM: with viscosity over omega's near list 4 (113 us with 1M particles; 3 119, 5 141);
// both terms over the full list's groups 3 (80 registers: 340 us; 2 9% slower, 4 46% with spills).
enum VortViscLists : uint32_t { kVortViscFull, kVortVisc, kViscNear };   // Lv, Ln: full, none; full, near; near, none
template <uint32_t kLists>
__global__ void __launch_bounds__(256, kLists == kVortViscFull ? 3 : 4)
vort_visc_list_kernel(const __grid_constant__ DevParams P, const float4* __restrict__ p, const float4* __restrict__ pa,
                      const float4* __restrict__ vin, float4* __restrict__ vout, const float4* __restrict__ omega,
                      float4* __restrict__ fext, const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce,
                      int do_vort, int do_visc, const float* __restrict__ w, CoopSet C, const __grid_constant__ NbList Lv, const __grid_constant__ NbList Ln,
                      float4* __restrict__ vhost, const __grid_constant__ NbList F, const __grid_constant__ LongLists LL,
                      const Pair4* __restrict__ pairs) {
    if (blockIdx.x < C.blocks) {
        run_coop_set(C, [&](uint32_t i) {
            coop_vort_visc(P, p, pa, vin, vout, omega, fext, cs, ce, do_vort, do_visc, w, i, vhost, LL, F);
        });
        return;
    }
    const uint32_t i = (blockIdx.x - C.blocks) * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    const uint32_t meta = Lv.meta[i];
    if (meta & kListOff) return;
    const float4 oi = do_vort ? omega[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const uint32_t nm = (do_vort && do_visc && Ln.list) ? Ln.meta[i] : kListOff;
    if (nm != kListOff) {
        VortViscVisitT<1u> vo(P, vin, omega, p[i], vin[i], oi, true, false);
        walk_full(Lv, i, meta, p, vo);
        VortViscVisitT<2u> vs(P, vin, omega, p[i], vin[i], oi, false, true);
        walk_near(Ln, i, nm, p, vs);
        vort_visc_finish(P, i, vo, vs, vout, fext, w, vhost);
        return;
    }
    VortViscVisit vis(P, vin, omega, p[i], vin[i], oi, do_vort != 0, do_visc != 0);
    if constexpr (kLists == kVortViscFull) {
        if (pairs) {
            VortPairVisitT<3u> vp(vis, pairs);
            walk_full(Lv, i, meta, p, vp);
            vort_visc_finish(P, i, vp, vp, vout, fext, w, vhost);
            return;
        }
    }
    if constexpr (kLists == kViscNear) walk_near<false, 2>(Lv, i, meta, p, vis);
    else walk_full(Lv, i, meta, p, vis);
    vort_visc_finish(P, i, vis, vis, vout, fext, w, vhost);
}

// vort_visc_list_kernel with G lanes per particle (small simulations, see lambda_group_kernel); both
// terms in one walk of Lv, the full list (kFull) or omega's near list.
template <bool kFull, int G>
__global__ void __launch_bounds__(256)
vort_visc_list_group_kernel(const __grid_constant__ DevParams P, const float4* __restrict__ p, const float4* __restrict__ pa,
                            const float4* __restrict__ vin, float4* __restrict__ vout, const float4* __restrict__ omega,
                            float4* __restrict__ fext, const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce,
                            int do_vort, int do_visc, const float* __restrict__ w, CoopSet C,
                            const __grid_constant__ NbList Lv, float4* __restrict__ vhost,
                            const __grid_constant__ NbList F, const __grid_constant__ LongLists LL) {
    if (blockIdx.x < C.blocks) {
        run_coop_set(C, [&](uint32_t i) {
            coop_vort_visc(P, p, pa, vin, vout, omega, fext, cs, ce, do_vort, do_visc, w, i, vhost, LL, F);
        });
        return;
    }
    const uint32_t tid = (blockIdx.x - C.blocks) * blockDim.x + threadIdx.x;
    const bool on = tid / G < P.N;
    const uint32_t i = on ? tid / G : P.N - 1u;
    const uint32_t meta = Lv.meta[i];
    const bool listed = on && !(meta & kListOff);
    const float4 oi = do_vort ? omega[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    VortViscVisit vis(P, vin, omega, p[i], vin[i], oi, do_vort != 0, do_visc != 0);
    walk_group_sums<G>([&](uint32_t k) { return kFull ? full_at(Lv, i, k) : Lv.list + (size_t)k * Lv.stride + i; },
                  listed ? meta & 0xFFu : 0u, (meta >> 8) & 0xFFu, i, p, vis);
    if (listed && tid % G == 0u) vort_visc_finish(P, i, vis, vis, vout, fext, w, vhost);
}

__global__ void __launch_bounds__(128)
vort_visc_coop_kernel(const __grid_constant__ DevParams P, const float4* __restrict__ p, const float4* __restrict__ pa, const float4* __restrict__ vin,
                      float4* __restrict__ vout, const float4* __restrict__ omega, float4* __restrict__ fext,
                      const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce, int do_vort, int do_visc,
                      const float* __restrict__ w, DeferList D) {
    for_each_deferred(D, [&](uint32_t i) {
        coop_vort_visc(P, p, pa, vin, vout, omega, fext, cs, ce, do_vort, do_visc, w, i, nullptr, LongLists{}, NbList{});
    });
}

// ======================================================================================
// Density constraint after a frame: C_i = rho_i / rho0 - 1 with rho_i the poly6 sum over the
// frame's list (no self term, Density.h:67-84) at the current positions.
// ======================================================================================
struct DensityVisit {
    struct Contrib { float a; uint32_t near; };
    const DevParams& P;
    float4 pi;
    float A = 0.f;
    __device__ DensityVisit(const DevParams& P_, float4 pi_) : P(P_), pi(pi_) {}
    __device__ static Contrib zero() { return Contrib{0.f, 0u}; }
    __device__ static bool effective(const Contrib& c) { return c.near != 0u; }
    __device__ static Contrib shfl(const Contrib& c, int k) { return Contrib{shfl_f(c.a, k), shfl_u(c.near, k)}; }
    __device__ __forceinline__ void end_contacts(uint32_t) {}
    __device__ __forceinline__ Contrib contrib(uint32_t, const float4& pj, bool) const {
        const float rx = pi.x - pj.x, ry = pi.y - pj.y, rz = pi.z - pj.z;
        const float r2 = dist2(rx, ry, rz);
        if (r2 >= P.cut2) return zero();
        return Contrib{poly6(P, sqrt_fast(r2)), 1u};
    }
    __device__ __forceinline__ void add(const Contrib& c, bool) { if (c.near) A = __fadd_rn(A, c.a); }
};

// err[i] = C_i; acc[0] += |C_i| (double), acc[1] = max |C_i| (double bits, non-negative); over the
// interior particles (list length >= min_nb and position at least `margin` inside the enclosure on
// every axis: their kernel support lies in the fluid) acc[2] += |C_i|, acc[3] = max |C_i|,
// acc[4] += 1.
__global__ void __launch_bounds__(128)
density_error_kernel(DevParams P, const float4* __restrict__ p, const float4* __restrict__ pa,
                     const uint32_t* __restrict__ cs, const uint32_t* __restrict__ ce, float* __restrict__ err,
                     double* acc, uint32_t min_nb, float margin) {
    __shared__ double sred[5][4];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    double a = 0.0, ai = 0.0, ni = 0.0;
    if (i < P.N) {
        const SceneCtx S = scene_ctx(P, i);
        const float4 pi = p[i];
        DensityVisit vis(P, pi);
        bool deferred = false;
        const uint32_t n = walk_seq(P, S, i, pa[i], p, cs, ce, vis, false, &deferred);
        const float c = vis.A / S.rho0 - 1.0f;
        err[i] = c;
        a = fabs((double)c);
        const float* bmn = P.batched ? P.scenes[P.scene_of[i]].bmin : P.bmin;
        const float* bmx = P.batched ? P.scenes[P.scene_of[i]].bmax : P.bmax;
        const bool inside = pi.x > bmn[0] + margin && pi.x < bmx[0] - margin && pi.y > bmn[1] + margin &&
                            pi.y < bmx[1] - margin && pi.z > bmn[2] + margin && pi.z < bmx[2] - margin;
        if (inside && n >= min_nb) { ai = a; ni = 1.0; }
    }
    double sm = a, mx = a, smi = ai, mxi = ai, cnt = ni;
    for (int o = 16; o > 0; o >>= 1) {
        sm += __shfl_down_sync(0xffffffffu, sm, o);
        mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, o));
        smi += __shfl_down_sync(0xffffffffu, smi, o);
        mxi = fmax(mxi, __shfl_down_sync(0xffffffffu, mxi, o));
        cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    }
    if ((threadIdx.x & 31u) == 0u) {
        const int w = threadIdx.x >> 5;
        sred[0][w] = sm; sred[1][w] = mx; sred[2][w] = smi; sred[3][w] = mxi; sred[4][w] = cnt;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0, m = 0.0, ti = 0.0, mi = 0.0, c = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            t += sred[0][w]; m = fmax(m, sred[1][w]); ti += sred[2][w]; mi = fmax(mi, sred[3][w]); c += sred[4][w];
        }
        atomicAdd(acc, t);
        atomicMax(reinterpret_cast<unsigned long long*>(acc + 1), (unsigned long long)__double_as_longlong(m));
        atomicAdd(acc + 2, ti);
        atomicMax(reinterpret_cast<unsigned long long*>(acc + 3), (unsigned long long)__double_as_longlong(mi));
        atomicAdd(acc + 4, c);
    }
}

// ======================================================================================
// Debug: materialise the neighbour list (findContacts + findNeighbours, Collision.h:11-160)
// ======================================================================================
struct ListVisit {
    struct Contrib { uint32_t j; };
    uint32_t* out;
    uint32_t cap, n = 0, contacts = 0xFFFFFFFFu;
    __device__ ListVisit(uint32_t* o, uint32_t c) : out(o), cap(c) {}
    __device__ static Contrib zero() { return Contrib{0u}; }
    __device__ static bool effective(const Contrib&) { return true; }
    __device__ static Contrib shfl(const Contrib& c, int k) { return Contrib{shfl_u(c.j, k)}; }
    __device__ __forceinline__ void end_contacts(uint32_t c) { contacts = c; }
    __device__ __forceinline__ Contrib contrib(uint32_t j, const float4&, bool) const { return Contrib{j}; }
    __device__ __forceinline__ void add(const Contrib& c, bool) {
        if (n < cap) out[n] = c.j;
        ++n;
    }
};

__global__ void list_kernel(DevParams P, const float4* __restrict__ p, const uint32_t* __restrict__ cs,
                            const uint32_t* __restrict__ ce, uint32_t cap, uint32_t* list,
                            uint32_t* count, uint32_t* contacts, float4* col, int coop) {
    // coop = 0: one thread per particle; coop = 1: one warp per particle (checks walk_coop)
    const uint32_t i = coop ? (blockIdx.x * blockDim.x + threadIdx.x) >> 5 : blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    ListVisit vis(list + (size_t)i * cap, cap);
    uint32_t n;
    if (coop) {
        ListVisit lv(lane_id() == 0 ? list + (size_t)i * cap : nullptr, lane_id() == 0 ? cap : 0u);
        n = walk_coop(P, scene_ctx(P, i), i, p[i], p, cs, ce, lv);
        vis.contacts = lv.contacts;
        if (lane_id() != 0) return;
    } else {
        bool deferred = false;
        n = walk_seq(P, scene_ctx(P, i), i, p[i], p, cs, ce, vis, false, &deferred);
    }
    if (vis.contacts == 0xFFFFFFFFu) vis.contacts = n;   // cap reached inside the 27 cells
    count[i] = n;
    contacts[i] = vis.contacts;
    if (col) {
        const float f = (float)n / (float)P.M;
        col[i] = make_float4(f, f, f, 1.0f);
    }
}

}  // namespace pbd
