// pbd_contacts.cuh -- collisionType 1: contact constraints solved in batches of disjoint pairs
// (kernel/Collision.h:288-436, Fluid.cu:37-38,65-72).
//
// The reference claims contacts with a __syncthreads inside divergent code and lets blocks race
// on the claims, so its batches are undefined across blocks.  Here the batches are defined as
// locally dominant matching:
//  - the constraints are the frame's list entries c = i * M + k (partner = entry k of particle
//    i's list; the reference fills the same array, findContacts + findNeighbours);
//  - in each batch, a constraint not yet solved in this stabilization pass competes when its
//    particles overlap at the batch's start (diameter - |p_j - p_i| > 0, |p_j - p_i| > 1e-5, a
//    movable particle); its key is lowbias32(c + 1) (C. Wellons' published 32-bit integer mix)
//    above c; every particle takes its highest competing key (atomicMax over both ends) and a
//    constraint both of whose particles took it is solved -- a batch is a matching, so its
//    projections touch disjoint particles and run in parallel (Gauss-Seidel across batches);
//  - solving follows setupCollisionConstraintBatchesCheck (Collision.h:389-436): d = p2 - p1
//    (w = 0), half = (diameter - |d|) / 2, p1 and x1 move by -n half (1 - stiffness), p2 and x2 by
//    +n half (1 - stiffness), and both p* are written back with w = 0.  With unified solids the
//    overlap is split by inverse mass (1/2 each for unit masses, the same bits as half).
// The oracle (solve_collisions_batched) restates the same definition.
#pragma once
#include "pbd_passes.cuh"

namespace pbd {

struct ContactStore {
    uint32_t* list;      // partner indices, four entries side by side as in a full list (full_at)
    uint32_t* count;     // entries per particle
    uint32_t* solved;    // ceil(M / 32) x stride words: bit k of particle i = constraint (i, k) solved
    unsigned long long* best;   // each particle's chosen constraint key in this batch (0: none)
    unsigned long long* best_next;   // the next batch's keys: cleared by this batch's solve pass
    uint32_t* long_items;   // particles with more than kClaimLong entries (any order)
    uint32_t* long_count;   // zeroed before the frame's contact_list_kernel
    uint32_t stride;
    uint32_t M;
};

// Lists longer than kClaimLong (up to M = 512 entries where the cell-end quirk stretches a cell's
// range, against ~26 on average) go to a whole warp in the claim pass's leading blocks, so they do not
// hold up the pass.
constexpr uint32_t kClaimLong = 64;
constexpr uint32_t kClaimCoopBlocks = 4;

__device__ __forceinline__ uint32_t lowbias32(uint32_t x) {
    x ^= x >> 16;
    x *= 0x7feb352du;
    x ^= x >> 15;
    x *= 0x846ca68bu;
    x ^= x >> 16;
    return x;
}

// |p_j - p_i| of a contact pair, with explicit FMAs: the claim and the solve pass round it the
// same way, so they agree on which contacts act.
__device__ __forceinline__ float contact_len(float dx, float dy, float dz) {
    return sqrtf(__fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx))));
}
// Whether the contact of i and j at distance len acts: an overlap, not coincident, and not two
// immovable particles.
__device__ __forceinline__ bool contact_acts(const DevParams& P, const float* __restrict__ w, uint32_t i, uint32_t j,
                                             float len) {
    if (w && !(w[i] + w[j] > 0.f)) return false;
    const float overlap = P.d - len;
    return (overlap * 0.5f > 0.f) && len > 0.00001f;
}

// The contact between particles i and j at the current positions: false when it does not act.
__device__ __forceinline__ bool contact_geometry(const DevParams& P, const float4* __restrict__ p,
                                                 const float* __restrict__ w, uint32_t i, uint32_t j,
                                                 float4& n, float& h1, float& h2) {
    const float4 p1 = p[i], p2 = p[j];
    const float dx = p2.x - p1.x, dy = p2.y - p1.y, dz = p2.z - p1.z;
    const float len = contact_len(dx, dy, dz);
    if (!contact_acts(P, w, i, j, len)) return false;
    float s1 = 0.5f, s2 = 0.5f;
    if (w) {
        const float w1 = w[i], w2 = w[j];
        s1 = w1 / (w1 + w2);
        s2 = w2 / (w1 + w2);
    }
    const float overlap = P.d - len;
    n = make_float4(dx / len, dy / len, dz / len, 0.f);
    h1 = overlap * s1;
    h2 = overlap * s2;
    return true;
}

__device__ __forceinline__ NbList contact_entries(const ContactStore& C) { return NbList{C.list, nullptr, C.stride, C.M}; }

// Every entry of particle i's list, in list order, up to the cap M.
struct ContactListVisit {
    struct Contrib { uint32_t j; };
    NbList L;
    uint32_t i, n = 0;
    __device__ ContactListVisit(const ContactStore& C, uint32_t i_) : L(contact_entries(C)), i(i_) {}
    __device__ static Contrib zero() { return Contrib{0u}; }
    __device__ static bool effective(const Contrib&) { return true; }
    __device__ static Contrib shfl(const Contrib& c, int k) { return Contrib{shfl_u(c.j, k)}; }
    __device__ __forceinline__ void end_contacts(uint32_t) {}
    __device__ __forceinline__ Contrib contrib(uint32_t j, const float4&, bool) const { return Contrib{j}; }
    __device__ __forceinline__ void add(const Contrib& c, bool) { *full_at(L, i, n) = c.j; ++n; }
};

// The same by one thread, four entries a store.
struct ContactWriteVisit {
    struct Contrib { uint32_t j; };
    FullWriter out;
    __device__ ContactWriteVisit(const ContactStore& C, uint32_t i) : out(contact_entries(C), i) {}
    __device__ static Contrib zero() { return Contrib{0u}; }
    __device__ static bool effective(const Contrib&) { return true; }
    __device__ __forceinline__ void end_contacts(uint32_t) {}
    __device__ __forceinline__ Contrib contrib(uint32_t j, const float4&, bool) const { return Contrib{j}; }
    __device__ __forceinline__ void add(const Contrib& c, bool) { out.push(c.j); }
};

__device__ __forceinline__ void contact_list_done(const ContactStore& C, uint32_t i, uint32_t n) {
    C.count[i] = n;
    if (n > kClaimLong) C.long_items[atomicAdd(C.long_count, 1u)] = i;
}

// After the re-order: each particle's constraint list (the walk stops at the cap M itself).  A
// particle whose walk meets a cell range longer than one thread's walk takes is listed again by
// a warp of its block (walk_coop: the same entries in the same order) once the block's threads
// are done.  Blocks of 256 threads.
__global__ void __launch_bounds__(256)
contact_list_kernel(DevParams P, const float4* __restrict__ pa, const uint32_t* __restrict__ cs,
                    const uint32_t* __restrict__ ce, ContactStore C) {
    __shared__ uint32_t left[256];
    __shared__ uint32_t nleft;
    if (threadIdx.x == 0) nleft = 0u;
    __syncthreads();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < P.N) {
        ContactWriteVisit vis(C, i);
        bool deferred = false;
        walk_seq(P, scene_ctx(P, i), i, pa[i], pa, cs, ce, vis, true, &deferred);
        if (deferred) left[atomicAdd(&nleft, 1u)] = i;
        else {
            vis.out.flush();
            contact_list_done(C, i, vis.out.n);
        }
    }
    __syncthreads();
    const uint32_t nl = nleft;
    for (uint32_t k = threadIdx.x >> 5; k < nl; k += blockDim.x >> 5) {
        const uint32_t q = left[k];
        ContactListVisit vis(C, q);
        walk_coop(P, scene_ctx(P, q), q, pa[q], pa, cs, ce, vis);
        if (lane_id() == 0) contact_list_done(C, q, vis.n);
    }
}

// Offer constraint (i, k)'s key to its partner j and to `own`, i's own best, when the contact acts.
__device__ __forceinline__ void offer(const DevParams& P, const ContactStore& C, const float* __restrict__ w, uint32_t i,
                                      uint32_t k, uint32_t j, const float4& pi, const float4& pj, unsigned long long& own) {
    if (!contact_acts(P, w, i, j, contact_len(pj.x - pi.x, pj.y - pi.y, pj.z - pi.z))) return;
    const uint32_t c = i * C.M + k;
    const unsigned long long key = ((unsigned long long)lowbias32(c + 1u) << 32) | c;
    own = key > own ? key : own;          // i's own offers: one atomic per particle
    atomicMax(C.best + j, key);           // the partner's (no read first: fire and forget)
}

// One thread offers the keys of particle i's pending overlapping constraints (n of them at most) and
// returns the highest.  32 entries at a time: first only the squared distances (a superset of the
// overlap test, |r| < diameter), four entries per index load, into a mask without the solved ones;
// then the exact test, key and atomic for the entries in the mask.  About 12% of the entries compete:
// with the test of every entry followed by its offer, some lane of a warp took almost every offer
// (2,400 warp instructions per 32 particles against 1,150).
__device__ __forceinline__ unsigned long long claim_entries(const DevParams& P, const ContactStore& C,
                                                            const float4* __restrict__ p, const float* __restrict__ w,
                                                            uint32_t i, uint32_t n) {
    const NbList L = contact_entries(C);
    const float4 pi = p[i];
    const float reach2 = P.d * P.d * 1.0001f;
    unsigned long long own = 0ull;
    for (uint32_t k0 = 0; k0 < n; k0 += 32u) {
        const uint32_t solved = C.solved[(size_t)(k0 >> 5) * C.stride + i];
        const uint32_t m = min(n - k0, 32u);
        const uint4* e = reinterpret_cast<const uint4*>(L.list) + (size_t)(k0 >> 2) * L.stride + i;
        uint4 q = __ldg(e);
        uint32_t mask = 0;
#pragma unroll 1
        for (uint32_t kb = 0; kb < m; kb += 4u) {
            const uint32_t j[4] = {q.x, kb + 1u < m ? q.y : i, kb + 2u < m ? q.z : i, kb + 3u < m ? q.w : i};
            float4 pj[4];
#pragma unroll
            for (uint32_t b = 0; b < 4u; ++b) pj[b] = __ldg(p + j[b]);
            e += L.stride;
            if (kb + 4u < m) q = __ldg(e);
            uint32_t four = 0;
#pragma unroll
            for (uint32_t b = 0; b < 4u; ++b) {
                const float dx = pj[b].x - pi.x, dy = pj[b].y - pi.y, dz = pj[b].z - pi.z;
                if (kb + b < m && dist2(dx, dy, dz) < reach2) four |= 1u << b;
            }
            mask |= four << kb;
        }
        mask &= ~solved;
        uint32_t k = k0 + (uint32_t)__ffs(mask) - 1u;
        uint32_t j = mask ? __ldg(full_at(L, i, k)) : i;
        while (mask) {   // the next entry's index in flight
            mask &= mask - 1u;
            const uint32_t kn = k0 + (uint32_t)__ffs(mask) - 1u;
            const float4 pj = __ldg(p + j);
            const uint32_t jn = mask ? __ldg(full_at(L, i, kn)) : i;
            offer(P, C, w, i, k, j, pi, pj, own);
            k = kn;
            j = jn;
        }
    }
    return own;
}

// The same for a long list by the 32 lanes of a warp (lane t takes entries t, t + 32, ...): a lane's
// highest own offer.
__device__ __forceinline__ unsigned long long claim_entries_warp(const DevParams& P, const ContactStore& C,
                                                                 const float4* __restrict__ p, const float* __restrict__ w,
                                                                 uint32_t i, uint32_t t, uint32_t n) {
    const NbList L = contact_entries(C);
    const float4 pi = p[i];
    const float reach2 = P.d * P.d * 1.0001f;
    unsigned long long own = 0ull;
    for (uint32_t k0 = 0; k0 < n; k0 += 64u) {
        uint32_t j[2], solved[2];
        float4 pj[2];
#pragma unroll
        for (uint32_t b = 0; b < 2u; ++b) {
            const uint32_t k = k0 + b * 32u + t;
            j[b] = k < n ? __ldg(full_at(L, i, k)) : i;
            solved[b] = k < n ? C.solved[(size_t)(k >> 5) * C.stride + i] : kFullMask;
        }
#pragma unroll
        for (uint32_t b = 0; b < 2u; ++b) pj[b] = __ldg(p + j[b]);
#pragma unroll
        for (uint32_t b = 0; b < 2u; ++b) {
            const uint32_t k = k0 + b * 32u + t;
            if ((solved[b] >> t) & 1u) continue;
            if (dist2(pj[b].x - pi.x, pj[b].y - pi.y, pj[b].z - pi.z) < reach2) offer(P, C, w, i, k, j[b], pi, pj[b], own);
        }
    }
    return own;
}

// Each pending overlapping constraint offers its key to both of its particles.  The first
// kClaimCoopBlocks blocks take the long lists, a warp each; the others take every other particle, a
// thread each.  kPerSm blocks of 256 per SM (claim_blocks_per_sm).
template <int kPerSm>
__global__ void __launch_bounds__(256, kPerSm)
contact_claim_kernel(DevParams P, ContactStore C, const float4* __restrict__ p, const float* __restrict__ w) {
    if (blockIdx.x < kClaimCoopBlocks) {
        const uint32_t nl = *C.long_count;
        const uint32_t wpb = blockDim.x >> 5, lane = threadIdx.x & 31u;
        for (uint32_t q = blockIdx.x * wpb + (threadIdx.x >> 5); q < nl; q += kClaimCoopBlocks * wpb) {
            const uint32_t i = C.long_items[q];
            unsigned long long own = claim_entries_warp(P, C, p, w, i, lane, C.count[i]);
#pragma unroll
            for (uint32_t s = 1; s < 32u; s <<= 1) {
                const unsigned long long o = __shfl_xor_sync(kFullMask, own, s);
                own = o > own ? o : own;
            }
            if (lane == 0 && own) atomicMax(C.best + i, own);
        }
        return;
    }
    const uint32_t i = (blockIdx.x - kClaimCoopBlocks) * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    const uint32_t n = C.count[i];
    if (n > kClaimLong) return;                  // a long list: a leading block's warp takes it
    const unsigned long long own = claim_entries(P, C, p, w, i, n);
    if (own) atomicMax(C.best + i, own);
}

// Four blocks per SM have the L1 to themselves, whose hits the pass lives on; six run it in fewer waves and
// hide the L2's and memory's latency.  So four where they need at most two waves, and no more than six
// would.  Ten frames of 16 batches, ms per frame, four / six: 130,000 particles (1 wave each) 1.28 / 1.31,
// 175,616 (2, 1) 1.94 / 1.64, 262,144 (2, 2) 2.17 / 2.37, 323,680 (3, 2) 2.69 / 2.63, 512,000 (4, 3)
// 4.22 / 3.98, 1,000,000 (7, 5) 7.63 / 6.94.
inline int claim_blocks_per_sm(uint32_t blocks, uint32_t sms) {
    const uint32_t w4 = (blocks + 4u * sms - 1u) / (4u * sms), w6 = (blocks + 6u * sms - 1u) / (6u * sms);
    return (w4 <= 2u && w4 <= w6) ? 4 : 6;
}

// A constraint both of whose particles took it is solved by its partner's thread: the key holds
// the constraint c = a * M + k, so the partner finds the owner a without reading the list.  Each
// thread also clears its particle's key for the next batch (that buffer was the previous batch's
// and is read by no one here).
__global__ void __launch_bounds__(256)
contact_solve_kernel(DevParams P, ContactStore C, float4* __restrict__ p, float4* __restrict__ x,
                     const float* __restrict__ w) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    C.best_next[i] = 0ull;
    const unsigned long long key = C.best[i];
    if (key == 0ull) return;
    const uint32_t c = (uint32_t)key;
    const uint32_t a = c / C.M;                  // the owner; i is its partner unless a == i
    if (a == i || C.best[a] != key) return;
    const uint32_t k = c - a * C.M;
    C.solved[(size_t)(k >> 5) * C.stride + a] |= 1u << (k & 31u);   // a is in one solved constraint
    float4 n;
    float h1, h2;
    if (!contact_geometry(P, p, w, a, i, n, h1, h2)) return;
    const float om = P.one_minus_stiffness;
    const float4 a1 = make_float4(-n.x * h1 * om, -n.y * h1 * om, -n.z * h1 * om, -n.w * h1 * om);
    const float4 a2 = make_float4(n.x * h2 * om, n.y * h2 * om, n.z * h2 * om, n.w * h2 * om);
    const float4 p1 = p[a], p2 = p[i];
    p[a] = make_float4(p1.x + a1.x, p1.y + a1.y, p1.z + a1.z, 0.f + a1.w);
    p[i] = make_float4(p2.x + a2.x, p2.y + a2.y, p2.z + a2.z, 0.f + a2.w);
    const float4 x1 = x[a], x2 = x[i];
    x[a] = make_float4(x1.x + a1.x, x1.y + a1.y, x1.z + a1.z, x1.w + a1.w);
    x[i] = make_float4(x2.x + a2.x, x2.y + a2.y, x2.z + a2.z, x2.w + a2.w);
}

}  // namespace pbd
