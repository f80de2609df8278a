// PBF step kernels.  This file is compiled twice:
//   pbf_exact.cu: PBF_FAST=0, built with -fmad=false and IEEE div/sqrt, so
//                 every expression below rounds exactly like the reference's
//                 float code (pbf_solver.cpp, sph_kernel.h) term by term;
//   pbf_fast.cu:  PBF_FAST=1, built with FMA contraction, approximate
//                 division and square root, and rsqrt in the spiky gradient.
// Summation order is the reference's in both builds: for particle i the
// candidates are visited bucket by bucket over the 27 neighbour cells in
// (dz, dy, dx) order and, inside a bucket, by ascending particle index
// (neighbor_search.cpp:14-22, :36-48).
#pragma once

#include <cstdint>
#include <type_traits>

#include <cuda_fp16.h>

#include "exact_pair.cuh"
#include "exact_repeat.h"
#include "pbf_types.cuh"
#include "radix_sort.cuh"

#ifndef PBF_FAST
#error "define PBF_FAST before including pbf_kernels.cuh"
#endif
#ifndef PBF_NS
#error "define PBF_NS before including pbf_kernels.cuh"
#endif

namespace pbf {
namespace PBF_NS {

constexpr int kBlock = 128;
// Single scenes of at least this many particles look for runs of identical
// particles (k_segments).
constexpr int kBigScene = 1 << 17;
// The fewest candidates a row or bucket must hold before a walk looks for
// runs of identical candidates in it (rows of ordinary fluid hold a few
// hundred).
constexpr uint32_t kRunRow = 1024;
constexpr uint32_t kNoBucket = 0xffffffffu;
// Flags in a particle's owner word (StepBuffers::sown) for runs of identical
// particles (k_segments): the particle only copies the results of its run's
// first particle (kCopyBit), or it is a run's first particle (kLeadBit).  The
// owner row itself takes the low 30 bits.
constexpr uint32_t kCopyBit = 0x40000000u;
constexpr uint32_t kLeadBit = 0x80000000u;
constexpr uint32_t kOwnerMask = 0x3fffffffu;
// Bits of a slot's alias byte (StepBuffers::slot_alias): the slot holds a
// particle from outside the grid box; a run's first particle; particles whose
// reference bucket holds more than their run of cells.
constexpr unsigned char kAliasSlot = 1;
constexpr unsigned char kRunSlot = 2;
constexpr unsigned char kMergedSlot = 4;

// ---------------------------------------------------------------------------
// SPH kernels (include/novaphy/fluid/sph_kernel.h:24-46)

// e0 + (e1 + e2): the 3-term reduction order of Vector3f::squaredNorm.
__device__ __forceinline__ float sqn(float x, float y, float z) { return x * x + (y * y + z * z); }

// r = x_i - x_j of a candidate and sqn(r), with (r.x, r.y) as one paired
// operation: fma(x_j, -1, x_i) rounds once, exactly as x_i - x_j, so the
// result is the reference's subtraction bit for bit.  The exact build also
// squares (r.x, r.y) as a pair; the _rn forms are never contracted, so the
// sum keeps sqn's separately rounded terms.  With with_w, rw = x_i.w + x_j.w
// (the lambda sum) comes from the same paired operation as r.z.
template <bool with_w = false>
__device__ __forceinline__ float rel_sq(const float4& xi, const float4& xj, float& rx, float& ry,
                                        float& rz, float* rw = nullptr) {
    const float2 dxy = __ffma2_rn(make_float2(xj.x, xj.y), make_float2(-1.0f, -1.0f),
                                  make_float2(xi.x, xi.y));
    rx = dxy.x;
    ry = dxy.y;
    if constexpr (with_w) {
        const float2 dzw = __ffma2_rn(make_float2(xj.z, xj.w), make_float2(-1.0f, 1.0f),
                                      make_float2(xi.z, xi.w));
        rz = dzw.x;
        *rw = dzw.y;
    } else {
        rz = xi.z - xj.z;
    }
#if PBF_FAST
    return sqn(rx, ry, rz);
#else
    const float2 sq = __fmul2_rn(dxy, dxy);
    return sq.x + (sq.y + rz * rz);
#endif
}

__device__ __forceinline__ float poly6(float r_sq, const StepConsts& C) {
    if (r_sq >= C.h2) return 0.0f;
    const float diff = C.h2 - r_sq;
    return C.k_poly * diff * diff * diff;
}

// Spiky gradient of r (= x_i - x_j) given r_sq = sqn(r); returns the scalar
// coefficient c so that grad = c * r (0 outside 1e-7 < |r| < h).
__device__ __forceinline__ float spiky_coeff(float r_sq, const StepConsts& C) {
#if PBF_FAST
    if (r_sq >= C.h2 || r_sq <= 1e-14f) return 0.0f;
    const float ir = rsqrtf(r_sq);
    const float diff = C.h - r_sq * ir;
    return C.k_spiky * diff * diff * ir;
#else
    const float r_len = sqrtf(r_sq);
    if (r_len <= 1e-7f || r_len >= C.h) return 0.0f;
    const float diff = C.h - r_len;
    return C.k_spiky * diff * diff / r_len;
#endif
}

// Adding a term to a running sum m times in a row (a run of identical
// candidates): the float that m single additions of t leave, bit for bit.  A
// call for long runs: inlined, its loop cost the neighbour passes' hot loops
// registers.
constexpr uint32_t kAddSingly = 12;
__device__ __noinline__ float rep_add_call(float s, float t, uint32_t m) { return rep_add(s, t, m); }
template <int K>
__device__ __forceinline__ void add_times(float (&s)[K], const float (&t)[K], uint32_t m) {
    if (m > kAddSingly) {
#pragma unroll
        for (int k = 0; k < K; ++k) s[k] = rep_add_call(s[k], t[k], m);
        return;
    }
#pragma unroll 1
    for (; m; --m) {
#pragma unroll
        for (int k = 0; k < K; ++k) s[k] = s[k] + t[k];
    }
}

// ---------------------------------------------------------------------------
// Grid helpers

__device__ __forceinline__ int wrap(int c, int o, int g) {
    int t = (c - o) % g;
    return t < 0 ? t + g : t;
}

// Global slot of a cell: the grid's base plus its wrapped local index.
__device__ __forceinline__ uint32_t slot_of(int cx, int cy, int cz, const GridDesc& G) {
    return G.base + (uint32_t)wrap(cx, G.ox, G.gx) +
           (uint32_t)G.gx * ((uint32_t)wrap(cy, G.oy, G.gy) + (uint32_t)G.gy * (uint32_t)wrap(cz, G.oz, G.gz));
}

__device__ __forceinline__ bool in_grid(int cx, int cy, int cz, const GridDesc& G) {
    return (unsigned)(cx - G.ox) < (unsigned)G.gx && (unsigned)(cy - G.oy) < (unsigned)G.gy &&
           (unsigned)(cz - G.oz) < (unsigned)G.gz;
}

__device__ __forceinline__ void cell_of(float x, float y, float z, float inv, int& cx, int& cy,
                                        int& cz) {
    cx = (int)floorf(x * inv);
    cy = (int)floorf(y * inv);
    cz = (int)floorf(z * inv);
}

// Reference cell hash (neighbor_search.cpp:89-97).
__device__ __forceinline__ unsigned long long ref_hash(int cx, int cy, int cz) {
    return ((unsigned long long)(long long)cx * 73856093ULL) ^
           ((unsigned long long)(long long)cy * 19349663ULL) ^
           ((unsigned long long)(long long)cz * 83492791ULL);
}

// An index of cell-sorted points that walks visit: cell-order offsets of the
// slots, and the reference buckets (see BucketTable) of the dirty cells' rows.
struct WalkIndex {
    uint32_t n;
    const uint32_t* __restrict__ off;
    const uint32_t* __restrict__ merged;
    const uint32_t* __restrict__ end;
    const uint32_t* __restrict__ btab;
    // The cell-order position of bucket position q.
    __device__ __forceinline__ uint32_t at(uint32_t q) const {
        return q < n ? q : __ldg(merged + (q - n));
    }
};

// Visits the candidate sorted positions q of a particle whose step-start cell
// is `cell`, in the reference's order.  The particle itself is among them:
// the reference skips j == i in every pass but the density, and the kernels
// rely on its terms being exact zeros instead (spiky_grad(0) = 0 and the
// velocity / |omega| differences vanish), which leaves every sum unchanged.
//
// cell.w == 0 (clean): every neighbour bucket holds exactly the particles of
// that cell, so each (dz, dy) row of three cells is one contiguous range of
// the cell-sorted order.  cell.w == o + 1 (dirty: a neighbour key is shared
// with another occupied cell, or a slot holds wrapped aliases): the 27 bucket
// starts are row o of `btab`.
template <class F>
__device__ __forceinline__ void for_each_candidate(const int4 cell, const WalkIndex& I,
                                                   const StepConsts& C, F&& f) {
    const GridDesc& G = C.grid;
    if (cell.w == 0) {
        for (int dz = -1; dz <= 1; ++dz) {
            const uint32_t wz = (uint32_t)wrap(cell.z + dz, G.oz, G.gz);
            for (int dy = -1; dy <= 1; ++dy) {
                const uint32_t wy = (uint32_t)wrap(cell.y + dy, G.oy, G.gy);
                const uint32_t row = G.base + (uint32_t)G.gx * (wy + (uint32_t)G.gy * wz);
                const int wx = wrap(cell.x - 1, G.ox, G.gx);
                if (wx + 2 < G.gx) {
                    const uint32_t q1 = __ldg(I.off + row + wx + 3);
#pragma unroll 4
                    for (uint32_t q = __ldg(I.off + row + wx); q < q1; ++q) f(q);
                } else {
                    for (int d = 0; d < 3; ++d) {
                        const uint32_t s = row + (uint32_t)wrap(cell.x - 1 + d, G.ox, G.gx);
                        const uint32_t q1 = __ldg(I.off + s + 1);
                        for (uint32_t q = __ldg(I.off + s); q < q1; ++q) f(q);
                    }
                }
            }
        }
    } else {
        const uint32_t* row = I.btab + (size_t)(uint32_t)(cell.w - 1) * 27u;
        for (int k = 0; k < 27; ++k) {
            const uint32_t b0 = __ldg(row + k);
            if (b0 == kNoBucket) continue;
            const uint32_t b1 = __ldg(I.end + b0);
            for (uint32_t q = b0; q < b1; ++q) f(I.at(q));
        }
    }
}

// ---------------------------------------------------------------------------
// Where a kernel finds its step constants and particle state.  One scene: the
// constants and the state arrays travel by value in the kernel parameters.
// A batch of scenes: tables with one entry per scene, indexed by the scene of
// the particle (sid, in the order the kernel walks); batch particle i of a
// scene whose particles start at `first` is the scene's particle i - first.

struct OneScene {
    StepConsts C;
    StateRef S;
    __device__ __forceinline__ const StepConsts& at(const uint32_t*, uint32_t) const { return C; }
    __device__ __forceinline__ const StateRef& state(const uint32_t*, uint32_t) const { return S; }
};

struct SceneTable {
    const StepConsts* __restrict__ tab;
    const StateRef* __restrict__ refs;
    __device__ __forceinline__ StepConsts at(const uint32_t* __restrict__ sid, uint32_t i) const {
        return tab[__ldg(sid + i)];
    }
    __device__ __forceinline__ StateRef state(const uint32_t* __restrict__ sid, uint32_t i) const {
        return refs[__ldg(sid + i)];
    }
};

// Scene ids of a step: per particle in particle order (pid) and in the
// cell-sorted order (spid); null for a single scene.
struct SceneIds {
    const uint32_t* __restrict__ pid;
    uint32_t* __restrict__ spid;
};

// ---------------------------------------------------------------------------
// Grid construction kernels

// v' = v + g dt;  x* = x + v' dt  (pbf_solver.cpp:31-32), rounded product
// then sum in both builds so that cell assignment is bit-exact.
__device__ __forceinline__ void predict(const float4 xi, const float4 vi, const StepConsts& C,
                                        float& px, float& py, float& pz) {
    const float vx = __fadd_rn(vi.x, __fmul_rn(C.g[0], C.dt));
    const float vy = __fadd_rn(vi.y, __fmul_rn(C.g[1], C.dt));
    const float vz = __fadd_rn(vi.z, __fmul_rn(C.g[2], C.dt));
    px = __fadd_rn(xi.x, __fmul_rn(vx, C.dt));
    py = __fadd_rn(xi.y, __fmul_rn(vy, C.dt));
    pz = __fadd_rn(xi.z, __fmul_rn(vz, C.dt));
}

// Predict + cell slot per particle (particle order), with the digits of the
// slots counted for the sort.  Also turns this step's density-pass counts of
// the last step (dhist, where there are any) into the previous step's, and
// begins the step's record of missing lists (ListRecord).
template <class P>
__global__ void __launch_bounds__(kCountThreads)
k_predict_key(uint32_t* __restrict__ keys, uint32_t* __restrict__ dhist, ListRecord* __restrict__ missing,
              int n, const SortCounts counts, const SceneIds S, const P prm) {
    __shared__ BlockCounts B;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    static_assert(4 * kWalkHist <= kCountThreads, "one thread per count");
    if (dhist && t < 4 * kWalkHist) {
        uint32_t* const d = dhist + (t / (2 * kWalkHist)) * 4 * kWalkHist + t % (2 * kWalkHist);
        d[0] = d[2 * kWalkHist];
        d[2 * kWalkHist] = 0u;
    }
    if (missing && t == 0) {
        const uint32_t off = missing->off;
        missing->off = off ? off - 1u : (2u * missing->failed > missing->tried ? kListsOff : 0u);
        missing->any = missing->tried = missing->failed = 0u;
    }
    B.begin(counts);
    for (int i = t; i < n; i += gridDim.x * blockDim.x) {
        const StepConsts& C = prm.at(S.pid, i);
        const StateRef& R = prm.state(S.pid, i);
        const uint32_t l = (uint32_t)i - R.first;
        float px, py, pz;
        predict(R.x[l], R.v[l], C, px, py, pz);
        int cx, cy, cz;
        cell_of(px, py, pz, C.inv_cell, cx, cy, cz);
        const uint32_t key = slot_of(cx, cy, cz, C.grid);
        keys[i] = key;
        B.count(counts, key);
    }
    B.end(counts);
}

// off[s] = lower_bound(skeys, s) for s in [0, nslots].
__device__ __forceinline__ void slot_offset(uint32_t s, const uint32_t* __restrict__ skeys, int n,
                                            uint32_t* __restrict__ off, uint32_t nslots) {
    if (s > nslots) return;
    int a = 0, b = n;
    while (a < b) {
        const int m = (a + b) >> 1;
        if (skeys[m] < s) a = m + 1;
        else b = m;
    }
    off[s] = (uint32_t)a;
}

// A launch of `points` blocks over the n points and more over the slots: the
// offsets' searches (a chain of log n loads each) run beside the points' work.
struct SlotOffsets {
    const uint32_t* skeys;
    uint32_t* off;
    uint32_t nslots;
    int points;
    // Whether the block is one of the slots' (and has done its work then).
    __device__ __forceinline__ bool block(int n) const {
        if ((int)blockIdx.x < points) return false;
        slot_offset((blockIdx.x - (uint32_t)points) * blockDim.x + threadIdx.x, skeys, n, off, nslots);
        return true;
    }
};

// Gather particle state into cell-sorted order; recompute x* exactly as
// predicted.  Records each particle's scene, empties the bucket chains and
// flags slots that receive a particle from outside the grid box (wrapped
// alias).
template <class P>
__global__ void __launch_bounds__(kBlock)
k_gather(const uint32_t* __restrict__ sidx, float4* __restrict__ sx, float4* __restrict__ xa,
         float* __restrict__ srho, int4* __restrict__ scell, uint32_t* __restrict__ link,
         unsigned char* __restrict__ slot_alias, uint32_t* __restrict__ err, int n,
         const SlotOffsets offsets, const SceneIds S, const P prm) {
    if (offsets.block(n)) return;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    uint32_t i = sidx[p];
    if (i >= (uint32_t)n) {  // only after a failed sort; keep every access in range
        atomicOr(err, 2u);
        i = 0;
    }
    const StepConsts& C = prm.at(S.pid, i);
    const StateRef& R = prm.state(S.pid, i);
    const uint32_t l = i - R.first;
    const float4 xi = R.x[l];
    float px, py, pz;
    predict(xi, R.v[l], C, px, py, pz);
    int cx, cy, cz;
    cell_of(px, py, pz, C.inv_cell, cx, cy, cz);
    sx[p] = make_float4(xi.x, xi.y, xi.z, __uint_as_float(i));
    xa[p] = make_float4(px, py, pz, R.lam[l]);
    srho[p] = R.rho[l];
    scell[p] = make_int4(cx, cy, cz, 0);
    link[p] = kNoBucket;
    if (S.spid) S.spid[p] = S.pid[i];
    if (!in_grid(cx, cy, cz, C.grid)) slot_alias[slot_of(cx, cy, cz, C.grid)] = kAliasSlot;
}

// Runs of particles with bit-identical step state (x, x* and lambda and rho
// as gathered) next to each other in cell order.  Everything a step computes
// for a particle follows from that state and from its candidates, which are
// those of its cell, so the particles of a run come out identical in every
// pass: only the run's first particle computes, and writes its results for
// the others too (their owner words get kCopyBit, the first one's segend the
// run's end).  Such runs form where the domain clamp piles fluid into a box
// corner, bit for bit: tens of thousands of particles, each of which would
// otherwise sum over all the others.  One warp per 32 positions; a warp with
// a run's first particle finds the run's end, 256 positions per round.
struct StepState {
    const float4* __restrict__ sx;
    const float4* __restrict__ xa;
    const float* __restrict__ srho;
    int n;
    __device__ __forceinline__ bool same(int a, int b) const {
        const float4 x0 = sx[a], x1 = sx[b], y0 = xa[a], y1 = xa[b];
        return __float_as_uint(x0.x) == __float_as_uint(x1.x) &&
               __float_as_uint(x0.y) == __float_as_uint(x1.y) &&
               __float_as_uint(x0.z) == __float_as_uint(x1.z) &&
               __float_as_uint(y0.x) == __float_as_uint(y1.x) &&
               __float_as_uint(y0.y) == __float_as_uint(y1.y) &&
               __float_as_uint(y0.z) == __float_as_uint(y1.z) &&
               __float_as_uint(y0.w) == __float_as_uint(y1.w) &&
               __float_as_uint(srho[a]) == __float_as_uint(srho[b]);
    }
};

__global__ void __launch_bounds__(256)
k_segments(const StepState S, const int4* __restrict__ scell, const GridDesc Gd,
           int* __restrict__ sown, unsigned char* __restrict__ slot_alias,
           uint32_t* __restrict__ segend) {
    const unsigned full = 0xffffffffu;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const bool in = p < S.n;
    const bool prev = in && p > 0 && S.same(p, p - 1);
    const bool next = in && p + 1 < S.n && S.same(p + 1, p);
    if (prev) sown[p] = (int)((uint32_t)sown[p] | kCopyBit);
    if (in && !prev && next) {
        sown[p] = (int)((uint32_t)sown[p] | kLeadBit);
        const int4 c = scell[p];
        unsigned char* a = slot_alias + slot_of(c.x, c.y, c.z, Gd);
        *a = (unsigned char)(*a | kRunSlot);
    }
    uint32_t end = 0u;
    uint32_t firsts = __ballot_sync(full, in && !prev && next);
    while (firsts) {
        const int l = __ffs(firsts) - 1;
        firsts &= firsts - 1u;
        // Positions from the first one's successor on, 8 per lane per round,
        // while each equals its predecessor.
        int base = (p - lane) + l + 1;
        int e = S.n;
        for (;;) {
            int fail = 8;
#pragma unroll
            for (int j = 7; j >= 0; --j) {
                const int q = base + lane * 8 + j;
                if (!(q < S.n && S.same(q, q - 1))) fail = j;
            }
            const uint32_t m = __ballot_sync(full, fail < 8);
            if (m) {
                const int fl = __ffs(m) - 1;
                e = base + fl * 8 + __shfl_sync(full, fail, fl);
                break;
            }
            base += 256;
        }
        if (lane == l) end = (uint32_t)e;
    }
    if (in) segend[p] = end;
}

// Reference buckets over cell-sorted points (see BucketTable), in three
// launches.  With scene ids (sid, in cell order) a bucket never crosses a
// scene: every scene has its own hash grid.  This took the place of a radix
// sort of the points by 64-bit reference key (eight passes) and of binary
// searches over the sorted keys: a step's neighbour structure has as many runs
// as occupied cells, a few per cent of its points, and few buckets merge.
struct CellRuns {
    const int4* __restrict__ scell;
    const uint32_t* __restrict__ sid;
    int n;
    __device__ __forceinline__ bool same(int a, int b) const {
        const int4 c = scell[a], d = scell[b];
        return c.x == d.x && c.y == d.y && c.z == d.z && (!sid || sid[a] == sid[b]);
    }
    // First position after p outside p's run, and the run's first position, in
    // a slot without aliases (where a cell has one run).  Both gallop, so a run
    // of L points costs O(log L) per thread: fluid piled into a corner by the
    // domain clamp makes runs of tens of thousands.
    __device__ __forceinline__ int end_of(int p) const {
        int lo = p, step = 1, hi = p + 1;
        while (hi < n && same(hi, p)) {
            lo = hi;
            step <<= 1;
            hi = (n - p > step) ? p + step : n;
        }
        while (hi - lo > 1) {
            const int mid = lo + ((hi - lo) >> 1);
            if (same(mid, p)) lo = mid;
            else hi = mid;
        }
        return hi;
    }
    __device__ __forceinline__ int start_of(int p) const {
        int hi = p, step = 1, lo = p - 1;
        while (lo >= 0 && same(lo, p)) {
            hi = lo;
            step <<= 1;
            lo = (p >= step) ? p - step : -1;
        }
        while (hi - lo > 1) {
            const int mid = lo + ((hi - lo) >> 1);
            if (same(mid, p)) hi = mid;
            else lo = mid;
        }
        return hi;
    }
    __device__ __forceinline__ unsigned long long key(int p) const {
        const int4 c = scell[p];
        return ref_hash(c.x, c.y, c.z);
    }
};

__device__ __forceinline__ uint32_t table_slot(unsigned long long key, uint32_t sid, uint32_t slots) {
    const unsigned long long h = (key ^ (key >> 29)) * 0x9e3779b97f4a7c15ull + (unsigned long long)sid * 0x632be59bd9b4e019ull;
    return (uint32_t)(h >> 32) & (slots - 1u);
}

// T with the slots that a build over n of its points uses.
inline BucketTable sized_for(BucketTable T, int n) {
    T.slots = bucket_slots((uint32_t)n);
    return T;
}

inline ClearRange bucket_clear(const BucketTable& T, int n) {
    return ClearRange{T.table, (size_t)bucket_slots((uint32_t)n) + 1, 0xffffffffu};
}
inline ClearRange slot_clear(const StepBuffers& B) { return ClearRange{reinterpret_cast<uint32_t*>(B.slot_alias), B.slot_bytes / 4, 0u}; }

// The first run of the bucket with this key (and scene), kNoBucket if none.
__device__ __forceinline__ uint32_t find_bucket(const BucketTable& T, const CellRuns& R,
                                                unsigned long long key, uint32_t sid) {
    uint32_t h = table_slot(key, sid, T.slots);
    for (uint32_t k = 0; k < T.slots; ++k) {
        const uint32_t e = T.table[h];
        if (e == kNoBucket) return kNoBucket;
        if (R.key((int)e) == key && (!R.sid || R.sid[e] == sid)) return e;
        h = (h + 1u) & (T.slots - 1u);
    }
    return kNoBucket;
}

// The points of a cell in a slot that holds aliases, where the cells' runs
// may alternate: positions [b0, b1) of the cell order, run start p.  Called by
// a warp together, 128 positions a round.  Returns whether p is the first of
// its cell; then the cell's other points get kMember | p, and T.end[p] is the
// end of its only run, or kListed | at where `merged` holds several (with
// their end in T.end[n + at]).  A pile of L points among aliases takes L / 128
// rounds for each cell in its slot.  One thread per run stepping through it,
// and every point of a merged bucket stepping back to its run's start and
// searching all runs of the bucket, took 17.5 ms for 60,000 points of two
// cells in turn (2.5 ms now).
__device__ __forceinline__ bool alias_cell(const BucketTable& T, const CellRuns& R, int p, int b0, int b1) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    b1 = min(b1, R.n);
    for (int b = p; b > b0; b -= 128) {
        bool found = false;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int q = b - 1 - 32 * j - lane;
            found |= q >= b0 && R.same(q, p);
        }
        if (__any_sync(full, found)) return false;
    }
    int count = 0, last = p;
    for (int b = p; b < b1; b += 128) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int q = b + 32 * j + lane;
            const bool in = q < b1 && R.same(q, p);
            if (in && q != p) T.rep[q] = kMember | (uint32_t)p;
            const uint32_t m = __ballot_sync(full, in);
            if (m) last = b + 32 * j + 31 - __clz(m);
            count += __popc(m);
        }
    }
    uint32_t at = 0u;
    const bool listed = count != last - p + 1;
    if (listed && lane == 0) at = atomicAdd(T.table + T.slots, (uint32_t)count) + 1u;
    at = __shfl_sync(full, at, 0);
    // (No room only after a failed sort; keep every access in range.)
    if (!listed || at + (uint32_t)count > 2u * (uint32_t)R.n) {
        if (lane == 0) T.end[p] = (uint32_t)(listed ? p + 1 : last + 1);
        return true;
    }
    if (lane == 0) {
        T.end[p] = kListed | at;
        T.end[(uint32_t)R.n + at] = (uint32_t)R.n + at + (uint32_t)count;
    }
    for (int b = p; b <= last; b += 128) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int q = b + 32 * j + lane;
            const bool in = q <= last && R.same(q, p);
            const uint32_t m = __ballot_sync(full, in);
            if (in) T.merged[at + (uint32_t)__popc(m & ((1u << lane) - 1u))] = (uint32_t)q;
            at += (uint32_t)__popc(m);
        }
    }
    return true;
}

// Every cell's points (T.end at the first one), and its place in the table.
template <class P>
__global__ void __launch_bounds__(256, 6)
k_cell_runs(const BucketTable T, const CellRuns R, const uint32_t* __restrict__ off,
            const unsigned char* __restrict__ slot_alias, const P prm) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    bool first = p < R.n && !(p > 0 && R.same(p, p - 1));
    int4 c = make_int4(0, 0, 0, 0);
    uint32_t slot = 0u;
    bool alias = false;
    if (first) {
        c = R.scell[p];
        const StepConsts& C = prm.at(R.sid, (uint32_t)p);
        slot = slot_of(c.x, c.y, c.z, C.grid);
        alias = (slot_alias[slot] & kAliasSlot) != 0;
        if (!alias) T.end[p] = (uint32_t)R.end_of(p);
    }
    uint32_t todo = __ballot_sync(0xffffffffu, alias);
    while (todo) {
        const int l = __ffs(todo) - 1;
        todo &= todo - 1u;
        const uint32_t s = __shfl_sync(0xffffffffu, slot, l);
        const bool leads = alias_cell(T, R, __shfl_sync(0xffffffffu, p, l), (int)off[s], (int)off[s + 1]);
        if ((int)(threadIdx.x & 31) == l) first = leads;
    }
    if (!first) return;
    const unsigned long long key = ref_hash(c.x, c.y, c.z);
    const uint32_t sid = R.sid ? R.sid[p] : 0u;
    uint32_t rep = (uint32_t)p;
    uint32_t h = table_slot(key, sid, T.slots);
    for (uint32_t k = 0; k < T.slots; ++k) {
        const uint32_t e = atomicCAS(T.table + h, kNoBucket, (uint32_t)p);
        if (e == kNoBucket) break;
        if (R.key((int)e) == key && (!R.sid || R.sid[e] == sid)) {
            rep = e;
            T.link[p] = atomicExch(T.link + e, (uint32_t)p);
            break;
        }
        h = (h + 1u) & (T.slots - 1u);
    }
    T.rep[p] = rep;
    if (rep != (uint32_t)p) return;
    uint32_t lo = (uint32_t)p, hi;
    if (alias) T.points(lo, (uint32_t)R.n, lo, hi);
    T.start[p] = lo;
}

// Room for the buckets of more than one cell.
template <class P>
__global__ void __launch_bounds__(256)
k_merge_room(const BucketTable T, const CellRuns R, unsigned char* __restrict__ slot_alias, const P prm) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= R.n || (p > 0 && R.same(p, p - 1))) return;
    if (T.rep[p] != (uint32_t)p || T.link[p] == kNoBucket) return;
    uint32_t total = 0u;
    const StepConsts& C = prm.at(R.sid, (uint32_t)p);
    for (uint32_t s = (uint32_t)p; s != kNoBucket; s = T.link[s]) {
        uint32_t lo, hi;
        T.points(s, (uint32_t)R.n, lo, hi);
        total += hi - lo;
        const int4 c = R.scell[s];
        unsigned char* const a = slot_alias + slot_of(c.x, c.y, c.z, C.grid);
        *a = (unsigned char)(*a | kMergedSlot);
    }
    const uint32_t at = (uint32_t)R.n + atomicAdd(T.table + T.slots, total) + 1u;
    T.start[p] = at;
    T.end[at] = at + total;
}

// The members of those buckets, in ascending point index: a point's place is
// the number of members before it, by a search in each of the cells.
template <class P>
__global__ void __launch_bounds__(256)
k_merge_runs(const BucketTable T, const CellRuns R, const uint32_t* __restrict__ sidx,
             const unsigned char* __restrict__ slot_alias, const P prm) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= R.n) return;
    const int4 c = R.scell[p];
    const StepConsts& C = prm.at(R.sid, (uint32_t)p);
    const unsigned char a = slot_alias[slot_of(c.x, c.y, c.z, C.grid)];
    if (!(a & kMergedSlot)) return;
    const uint32_t n = (uint32_t)R.n;
    uint32_t own = (uint32_t)p;
    if (!(a & kAliasSlot)) own = (uint32_t)R.start_of(p);
    else if (T.rep[p] & kMember) own = T.rep[p] & ~kMember;
    const uint32_t rep = T.rep[own];
    if (T.link[rep] == kNoBucket) return;
    const uint32_t i = sidx[p];
    uint32_t rank = 0u;
    for (uint32_t s = rep; s != kNoBucket; s = T.link[s]) {
        uint32_t first, lo, hi;
        T.points(s, n, first, hi);
        lo = first;
        while (lo < hi) {
            const uint32_t m = lo + ((hi - lo) >> 1);
            if (sidx[m < n ? m : T.merged[m - n]] < i) lo = m + 1u;
            else hi = m;
        }
        rank += lo - first;
    }
    const uint32_t at = T.start[rep] - n + rank;
    if (at < 2u * n) T.merged[at] = (uint32_t)p;
}

// T: sized_for n, its table cleared (bucket_clear).
template <class P>
inline cudaError_t enqueue_buckets(const BucketTable& T, const int4* scell, const uint32_t* sidx,
                                   const uint32_t* sid, const uint32_t* off, unsigned char* slot_alias, int n,
                                   const P& prm, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const CellRuns R{scell, sid, n};
    const int nb = (n + 255) / 256;
    k_cell_runs<P><<<nb, 256, 0, st>>>(T, R, off, slot_alias, prm);
    k_merge_room<P><<<nb, 256, 0, st>>>(T, R, slot_alias, prm);
    k_merge_runs<P><<<nb, 256, 0, st>>>(T, R, sidx, slot_alias, prm);
    return cudaGetLastError();
}

// Marks query points whose neighbourhood differs from the reference's
// buckets over a source point set (qown[p] = owner + 1, else 0) and stores
// their 27 bucket starts in row `owner` of btab.  Query cells are qcell[0..nq)
// (scenes qsid), the source's cells scell (scenes ssid) with buckets T and
// slot flags of the source's grid.  Within a warp, one lane per distinct cell
// (and scene) does the 27 lookups; the other lanes reuse its row.
template <class P>
__global__ void __launch_bounds__(kBlock)
k_classify(const int4* __restrict__ qcell, int nq, const int4* __restrict__ scell,
           const uint32_t* __restrict__ ssid, const BucketTable T,
           const unsigned char* __restrict__ slot_alias, uint32_t* __restrict__ btab,
           int* __restrict__ qown, const uint32_t* __restrict__ qsid, const P prm) {
    const CellRuns R{scell, ssid, 0};
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = p < (uint32_t)nq;
    const int lane = threadIdx.x & 31;
    const int4 cell = active ? qcell[p] : make_int4(0x7fffffff, 0x7fffffff, 0x7fffffff, 0);
    const uint32_t sc = (active && qsid) ? qsid[p] : 0xffffffffu;
    const unsigned long long kxy =
        ((unsigned long long)(unsigned)cell.x << 32) | (unsigned long long)(unsigned)cell.y;
    const unsigned full = 0xffffffffu;
    const uint32_t same = __match_any_sync(full, kxy) & __match_any_sync(full, (unsigned)cell.z) &
                          __match_any_sync(full, sc) & __ballot_sync(full, active);
    const int leader = same ? __ffs(same) - 1 : lane;
    // Each distinct cell of the warp in turn (its first lane is the owner of
    // its bucket row); lanes 0..26 look up one neighbour bucket each, m =
    // 9 (dz + 1) + 3 (dy + 1) + (dx + 1), so the 27 searches run side by side.
    uint32_t todo = __ballot_sync(full, active && lane == leader);
    int own = 0;
    while (todo) {
        const int L = __ffs(todo) - 1;
        todo &= todo - 1u;
        const uint32_t lp = __shfl_sync(full, p, L);
        const int cx = __shfl_sync(full, cell.x, L);
        const int cy = __shfl_sync(full, cell.y, L);
        const int cz = __shfl_sync(full, cell.z, L);
        const uint32_t grp = __shfl_sync(full, same, L);
        const uint32_t ls = __shfl_sync(full, sc, L);
        const StepConsts& C = prm.at(qsid, lp);
        int dirty = 0;
        if (C.hash_compat) {
            uint32_t t = kNoBucket;
            if (lane < 27) {
                const int nx = cx + lane % 3 - 1, ny = cy + (lane / 3) % 3 - 1, nz = cz + lane / 9 - 1;
                const uint32_t e = find_bucket(T, R, ref_hash(nx, ny, nz), ssid ? ls : 0u);
                if (e != kNoBucket) {
                    t = T.start[e];
                    const int4 c0 = scell[e];
                    if (T.link[e] != kNoBucket || c0.x != nx || c0.y != ny || c0.z != nz) dirty = 1;
                }
                if (slot_alias[slot_of(nx, ny, nz, C.grid)] & kAliasSlot) dirty = 1;
            }
            dirty = __any_sync(full, dirty);
            if (dirty && lane < 27) btab[(size_t)lp * 27u + (uint32_t)lane] = t;
        }
        if ((grp >> lane) & 1u) own = dirty ? (int)(lp + 1u) : 0;
    }
    if (active) qown[p] = own;
}

// ---------------------------------------------------------------------------
// Constraint and velocity kernels (a lane or part of a team per cell-sorted particle)

struct Grid {
    const int4* __restrict__ scell;
    const int* __restrict__ sown;
    WalkIndex ix;
    const uint32_t* __restrict__ spid;  // scene of each sorted particle (batches)
    uint32_t* moved;                     // per slot, see StepBuffers::moved
    uint32_t* lamnz;                     // per slot, see StepBuffers::lamnz
    BoundaryGrid bg;                     // two-way coupled steps only
    uint32_t* dhist;                     // see StepBuffers::dhist
    const uint32_t* segend;              // see StepBuffers::segend (large single scenes)
    const unsigned char* slot_alias;     // with kRunSlot where segend is set
    uint2* lists;                        // see StepBuffers::lists (null: none are kept)
    uint32_t* listed;
    ListRecord* missing;
};

// for_each_candidate over a single scene's step with runs of identical
// particles (k_segments): in a cell range or a one-cell bucket of at least
// kRunRow candidates, a run's first particle q calls fr(q, L) for the run's L
// particles, which come next in the candidate order (the run lies in one
// cell, in cell order), and the walk goes on after them.
template <bool kRuns, class F, class FR>
__device__ __forceinline__ void for_each_candidate_runs(const int4 cell, const Grid& G,
                                                        const StepConsts& C, F&& f, FR&& fr) {
    if constexpr (!kRuns) {
        for_each_candidate(cell, G.ix, C, f);
        return;
    }
    if (!G.segend) {
        for_each_candidate(cell, G.ix, C, f);
        return;
    }
    const GridDesc& Gd = C.grid;
    // Slots [s, s + k) of a cell range [q, q1): only ranges with a run's
    // first particle read the run flags of their candidates.
    auto range = [&](uint32_t q, uint32_t q1, uint32_t s, int k) {
        bool any = false;
        if (q1 - q >= kRunRow)
            for (int d = 0; d < k; ++d) any |= (__ldg(G.slot_alias + s + d) & kRunSlot) != 0;
        if (!any) {
#pragma unroll 4
            for (; q < q1; ++q) f(q);
            return;
        }
        while (q < q1) {
            if ((uint32_t)__ldg(G.sown + q) & kLeadBit) {
                const uint32_t e = __ldg(G.segend + q);
                fr(q, e - q);
                q = e;
            } else {
                f(q);
                ++q;
            }
        }
    };
    if (cell.w == 0) {
        for (int dz = -1; dz <= 1; ++dz) {
            const uint32_t wz = (uint32_t)wrap(cell.z + dz, Gd.oz, Gd.gz);
            for (int dy = -1; dy <= 1; ++dy) {
                const uint32_t wy = (uint32_t)wrap(cell.y + dy, Gd.oy, Gd.gy);
                const uint32_t row = Gd.base + (uint32_t)Gd.gx * (wy + (uint32_t)Gd.gy * wz);
                const int wx = wrap(cell.x - 1, Gd.ox, Gd.gx);
                if (wx + 2 < Gd.gx) {
                    range(__ldg(G.ix.off + row + wx), __ldg(G.ix.off + row + wx + 3), row + wx, 3);
                } else {
                    for (int d = 0; d < 3; ++d) {
                        const uint32_t s = row + (uint32_t)wrap(cell.x - 1 + d, Gd.ox, Gd.gx);
                        range(__ldg(G.ix.off + s), __ldg(G.ix.off + s + 1), s, 1);
                    }
                }
            }
        }
    } else {
        const uint32_t* row = G.ix.btab + (size_t)(uint32_t)(cell.w - 1) * 27u;
        for (int k = 0; k < 27; ++k) {
            const uint32_t b0 = __ldg(row + k);
            if (b0 == kNoBucket) continue;
            const uint32_t b1 = __ldg(G.ix.end + b0);
            if (b0 < G.ix.n) {
                const int4 c = G.scell[b0];
                range(b0, b1, slot_of(c.x, c.y, c.z, Gd), 1);
            } else {
                for (uint32_t q = b0; q < b1; ++q) f(G.ix.at(q));
            }
        }
    }
}

// The run flags of sorted particle p (kCopyBit, kLeadBit).
__device__ __forceinline__ uint32_t run_flags(const Grid& G, uint32_t p) {
    return (uint32_t)G.sown[p] & ~kOwnerMask;
}

// One past the last particle of the run p leads (p + 1 when it leads none).
__device__ __forceinline__ uint32_t run_end(const Grid& G, uint32_t p, uint32_t flags) {
    return (flags & kLeadBit) ? __ldg(G.segend + p) : p + 1;
}

// The cell of sorted particle p against the boundary index (two-way steps).
__device__ __forceinline__ int4 boundary_cell(const Grid& G, uint32_t p, const int4 cell) {
    const uint32_t i = __float_as_uint(__ldg(&G.bg.sx[p].w));
    return make_int4(cell.x, cell.y, cell.z, __ldg(G.bg.own + i));
}

__device__ __forceinline__ int4 cell_at(const Grid& G, uint32_t p) {
    int4 c = G.scell[p];
    c.w = (int)((uint32_t)G.sown[p] & kOwnerMask);
    return c;
}

// Load of a step array that the Jacobi loop rewrites.  Per-pass kernels read
// it through the read-only cache (nothing writes it during their launch); the
// persistent loop, whose other blocks rewrite it between its passes, uses
// plain loads, which its grid barrier orders after those writes.
template <bool kPersist, class T>
__device__ __forceinline__ T ld_step(const T* p) {
    if constexpr (kPersist) return *p;
    else return __ldg(p);
}

// ---------------------------------------------------------------------------
// The neighbour walks: a pass's sums over the candidates of each particle.
//
// Particles next to each other in cell order usually sit in one cell, or in
// a few cells next to each other along x.  Those of one (y, z) row of cells
// within three cells in x form a group: their candidate sequences are
// sub-sequences of one sequence, the 9 rows (dz, dy) of cells
// [xmin - 1, xmax + 1], each in slot order, which is the reference's order
// (cells in (dz, dy, dx) order, ascending particle index inside a cell).
// Particles of one cell whose reference buckets are merged (dirty) form a
// group too: their sequence is the cell's 27 buckets.  A walk takes its
// groups one after another, each in two phases:
//
//  1. listing: the sequence is cut into words of up to 32 candidates, each a
//     contiguous range of one row or bucket.  A warp stages four words in
//     shared memory as fp16 rows, and the tensor core computes
//     r^2 - support^2 of all pairs of the 128 candidates and the group's
//     particles (see Rows below); the signs of the accumulators are the
//     words' masks, one bit per candidate and particle.  The test is
//     conservative, so it keeps every in-support candidate; every term
//     re-tests the exact r^2 itself;
//  2. evaluation, once enough is listed or the sequence ends: each
//     particle's terms, two at a time, in list order.
//
// Every sum thus sees exactly the nonzero terms of the one-thread walk, in
// the same order, so it is bit-identical.
//
// Why: the exact terms (an IEEE square root and division each) should only
// run for candidates in support, with all lanes busy, and the distance test,
// which runs for every candidate (1,600 per particle at h = 4 r for about
// 250 terms), should cost little.  Lane by lane a test costs about seven
// instructions per candidate and particle; here 32 candidates x 32 particles
// cost two fragment loads, eight mma and 32 shifts, about one instruction
// and a quarter per candidate of a warp.
//
// Two forms:
//  * the warp walk (walk_group): a warp has 32 particles, one a lane, and a
//    lane adds its particle's terms itself.  The cheapest per particle.  Scenes
//    with kept lists (below) only list this way and sum in readers;
//  * the team walk (team_walk): four warps share TP = 8 or 16 particles.
//    The warps list different words, then 128 / TP lanes evaluate each
//    particle's terms side by side and pass them through shared memory to
//    the lanes that add them in order.  For scenes whose particles would
//    leave most of the chip idle, or its warps waiting on one chain each,
//    with one lane per particle (team_size).

// Words listed before an evaluation, in a warp walk and in a team walk.  With 16
// the lanes of a warp wait for the longest list twice as often (250,000
// particles 3,346 us a step against 2,995).
constexpr int kWalkWords = 32;
constexpr int kTeamWords = 64;
// Terms a team lists per particle before an evaluation: room for a round of
// its four warps (16 words of 32 candidates).
constexpr int kTeamTerms = 512;
constexpr int kTeamWarps = 4;
// Warps with more groups than this take the one-thread walk (sparse spray: a
// group's listing costs a warp about as much as a few dozen candidates of a
// one-thread walk).
constexpr int kMaxGroups = 6;
// Warps with more than this many have no lists (as many as 32 measured the
// same: 14,808 us against 14,790 for three steps of 394,831).
constexpr int kMaxListGroups = 16;

// A group's candidate sequence: ranges [start, start + len) in cell order (key
// order for a dirty cell), their rows' first slots, and the number of words of
// the ranges before each.
struct RangeList {
    uint32_t start[32], len[32], slot[32];
    int before[32];
};
constexpr uint32_t kRunRange = 0x80000000u;

// Kept lists.  The candidates that a listing finds for a particle, in the
// reference's order, two to a row (cell-order positions).  The delta pass reads
// the lists of the density pass, whose candidates sit where they sat; the
// vorticity pass those of the XSPH-omega pass.
//
// Warps of 32 particles list in a kernel of its own (k_list) and read in every
// pass (read_lists).  Their rows lie side by side (row r of particle p at
// (p / 32 kListRows + r) 32 + p % 32), and StepBuffers::listed holds the number
// of candidates, or kNoList where there were too many, where identical
// particles count more than once (k_segments) or where the warp had too many
// groups: those walk.  Teams list and sum in the density and XSPH-omega pass
// and read in the others; their rows lie one particle after another (p
// kListRows + r) and are counted, and an odd candidate's partner is the
// particle itself, whose terms are exact zeros in the passes that read.
//
// What it saves: listing and scanning are half of a walk's instructions
// (density of 300,000 particles: 180 of 318 million), and a warp walks its
// groups one after another with the lanes of the others idle (1.5 to 2 groups
// in moving fluid); a reader has one coalesced 8-byte load per row, all lanes
// busy, no shared memory and 64 registers, so 32 warps an SM instead of 20.
// The rows of a million particles are 1 GB written and read per iteration, a
// third of the memory bandwidth while the passes are bound by their
// instructions.  Measured (us a call; walking / lists kept by a walking
// density pass / k_list and readers): 1,000 particles 105 / 96 / -; 8,000 235 /
// 204 / -; 4 steps of 43,993 3,989 / 3,332 / -; 65,565 (fast build) 1,862 /
// 1,603 / -; 3 steps of 394,831 21,180 / 18,450 / 14,170; a million 6,263 /
// 5,528 / 3,974; 250,000 with bodies 3,642 / 3,133 / 2,857; a batch of 352,901
// 3,121 / 2,928 / 2,187.
__device__ __forceinline__ size_t list_at(uint32_t p) {
    return (size_t)(p >> 5) * (32u * kListRows) + (p & 31u);
}

// Shared memory of a warp walk.
struct WalkSmem {
    RangeList ranges;
    // One fp16 row of eight per candidate: x, y, z, |u|^2 (high, low), 1, 1, 0.
    alignas(16) uint32_t stage[128 * 4];
    uint32_t base[kWalkWords];  // first candidate (cell order, or key order in buckets)
    uint32_t info[kWalkWords];  // candidates | row << 8 | kRunWord
    uint32_t mask[kWalkWords * 32];
    // The mask of word w and particle p.  The exclusive-or spreads the four
    // words that a store instruction touches over the banks.
    static __device__ __forceinline__ int at(int w, int p) { return w * 32 + (p ^ ((w & 3) << 3)); }
    // The candidates of word w that a run's first particle counts
    // (k_segments), until its masks are there.
    __device__ __forceinline__ uint32_t& skip(int w) { return mask[at(w, 0)]; }
};

// In WalkSmem::info: a word of a range with runs, whose first particles stand
// for them; in the other ranges every candidate counts once.
constexpr uint32_t kRunWord = 1u << 16;

// Shared memory of a team walk.  During an evaluation the stage holds the
// terms on their way to the adding lanes, one row of float2 (two quantities)
// per pair of quantities and, in the fast build, their factors; rows are 66
// apart so that the lanes that add read without conflicts.
template <int TP>
struct TeamSmem {
    static constexpr int kRow = 66;
    static constexpr int kTermBytes = (PBF_FAST ? 6 : 3) * kRow * 8;
    static constexpr int kWarpBytes = kTermBytes > 2048 ? kTermBytes : 2048;
    static constexpr int kListRow = kTeamTerms + 2;
    alignas(16) unsigned char warp[kTeamWarps][(kWarpBytes + 15) / 16 * 16];
    RangeList ranges;
    uint32_t base[kTeamWords];
    uint32_t info[kTeamWords];
    uint32_t mask[kTeamWarps][4 * TP];
    uint32_t count[kTeamWarps][TP];  // a round's terms of each warp's words
    uint32_t total[TP];              // terms listed
    int flag[TP];
    alignas(4) unsigned short list[TP * kListRow];  // word << 5 | candidate
};

// Blocks per SM the neighbour-pass kernels are compiled for: 24 warps per SM
// (80 registers a thread).
template <int BS>
constexpr int kPassMinBlocks = 768 / BS;
// Threads per SM of the kernels that only list (640: 1M step 4,385 us against
// 4,230) and of those that read lists: 64 registers, or 72 with a batch's
// tables (16 scenes 2,310 us against 2,360 with 64).
constexpr int kListThreads = 768;
template <class P>
constexpr int kReadThreads = std::is_same<P, OneScene>::value ? 1024 : 896;
// The teams' kernels: of 8 particles seven blocks (72 registers), so that up to
// 8,500 particles run in one wave (8,000: 239 us a step against 258 with six).
template <int TP>
constexpr int kTeamMinBlocks = TP == 8 ? 7 : 6;

// A group: the cells [cx, cx + W - 3] of row (cy, cz), or one dirty cell
// (own: its bucket row + 1).  split: the row would wrap in x, so its cells
// are visited one by one (W = 3 then).
struct WalkGroup {
    int cx, cy, cz, W;
    uint32_t own;
    bool split;
};

__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ uint32_t pack_half2(__half a, __half b) {
    const __half2 h = __halves2half2(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// D = A B for one 16 x 8 tile, K = 8 (fp16 inputs, fp32 accumulators): lane
// (g = lane / 4, t = lane % 4) holds rows g and g + 8 of A (columns 2t,
// 2t + 1), column g of B (rows 2t, 2t + 1), and of D rows g (d0, d1) and
// g + 8 (d2, d3) in columns 2t, 2t + 1.
__device__ __forceinline__ void mma_16x8x8(float& d0, float& d1, float& d2, float& d3, uint32_t a0,
                                           uint32_t a1, uint32_t b0) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, "
        "{%7, %7, %7, %7};"
        : "=f"(d0), "=f"(d1), "=f"(d2), "=f"(d3)
        : "r"(a0), "r"(a1), "r"(b0), "f"(0.0f));
}

// Rows.  With positions u relative to the group's centre in units of h and
// rounded to fp16, r^2 - lim = |u_j|^2 - 2 u_i.u_j + (|u_i|^2 - lim) is a
// dot product of length seven: the candidate's row
//   (x, y, z, hi|u|^2, lo|u|^2, 1, 1, 0)
// times the particle's column
//   (-2x, -2y, -2z, 1, 1, hi(|u|^2 - lim), lo(|u|^2 - lim), 0),
// with each square split into two halves.  For |u| <= U per component the
// rounding of the positions moves a distance by at most
// 2 sqrt(3) U 2^-11 < 0.0018 U, and the split squares and the accumulation
// (fp32) move r^2 by less than 4e-5 U^2: lim = (1 + 0.0018 U)^2 + 4e-5 U^2 +
// 1e-5 keeps every candidate within h of a particle.  U is half the extent
// of the group's box plus one (a candidate farther out is in nobody's
// support, so its test may say anything); a group wider than kWalkReach
// lists every candidate instead.
constexpr float kWalkReach = 64.0f;
constexpr float kHalfFar = 60000.0f;  // |u|^2 of a row or column that is never in support

__device__ __forceinline__ uint4 candidate_row(float ux, float uy, float uz) {
    const __half2 xy = __floats2half2_rn(ux, uy);
    const __half z = __float2half_rn(uz);
    const float2 f = __half22float2(xy);
    const float fz = __half2float(z);
    const float n = fmaf(f.x, f.x, fmaf(f.y, f.y, fz * fz));
    const __half nh = __float2half_rn(n);
    const __half nl = __float2half_rn(n - __half2float(nh));
    return make_uint4(*reinterpret_cast<const uint32_t*>(&xy), pack_half2(z, nh),
                      pack_half2(nl, __float2half_rn(1.0f)),
                      pack_half2(__float2half_rn(1.0f), __float2half_rn(0.0f)));
}

__device__ __forceinline__ uint4 particle_column(float ux, float uy, float uz, float lim) {
    const __half2 xy = __floats2half2_rn(ux, uy);
    const __half z = __float2half_rn(uz);
    const float2 f = __half22float2(xy);
    const float fz = __half2float(z);
    const float m = fmaf(f.x, f.x, fmaf(f.y, f.y, fz * fz)) - lim;
    const __half mh = __float2half_rn(m);
    const __half ml = __float2half_rn(m - __half2float(mh));
    return make_uint4(pack_half2(-2.0f * f.x, -2.0f * f.y),
                      pack_half2(__float2half_rn(-2.0f * fz), __float2half_rn(1.0f)),
                      pack_half2(__float2half_rn(1.0f), mh), pack_half2(ml, __float2half_rn(0.0f)));
}

// Bits [lo, hi) of a word, for 0 <= lo, hi <= 32.
__device__ __forceinline__ uint32_t bit_range(uint32_t lo, uint32_t hi) {
    if (lo >= hi) return 0u;
    return (0xffffffffu >> (32u - (hi - lo))) << lo;
}

// The box of the wanting lanes' positions: its centre, the test's limit and
// whether it is too wide for the test.
struct WalkBox {
    float ox, oy, oz, lim;
    bool wide;
};

__device__ __forceinline__ WalkBox walk_box(bool want, const float4 xi, float inv_h) {
    const unsigned full = 0xffffffffu;
    const float inf = __int_as_float(0x7f800000);
    float lx = want ? xi.x : inf, ly = want ? xi.y : inf, lz = want ? xi.z : inf;
    float hx = want ? xi.x : -inf, hy = want ? xi.y : -inf, hz = want ? xi.z : -inf;
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        lx = fminf(lx, __shfl_xor_sync(full, lx, o));
        ly = fminf(ly, __shfl_xor_sync(full, ly, o));
        lz = fminf(lz, __shfl_xor_sync(full, lz, o));
        hx = fmaxf(hx, __shfl_xor_sync(full, hx, o));
        hy = fmaxf(hy, __shfl_xor_sync(full, hy, o));
        hz = fmaxf(hz, __shfl_xor_sync(full, hz, o));
    }
    WalkBox B;
    B.ox = 0.5f * (lx + hx);
    B.oy = 0.5f * (ly + hy);
    B.oz = 0.5f * (lz + hz);
    const float U = 0.5f * fmaxf(hx - lx, fmaxf(hy - ly, hz - lz)) * inv_h + 1.01f;
    B.wide = !(U <= kWalkReach);
    const float reach = 1.0f + 0.0018f * U;
    B.lim = reach * reach + 4e-5f * U * U + 1e-5f;
    return B;
}

// Finds the candidate sequence of a group, one range per lane, and writes it to
// L where `keep` is set (a team's first warp; the caller syncs).  Returns the
// number of its words, and with kRuns sets `runs` where a range holds runs (at
// least kRunRow candidates in slots with a run's first particle; kRunRange in
// its len).
template <bool kRuns>
__device__ __forceinline__ int walk_ranges(RangeList& L, const WalkGroup& Gr, const WalkIndex& I,
                                           const GridDesc& Gd, const Grid& G, bool keep, bool& runs) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    uint32_t start = 0u, len = 0u, slot = 0u;
    bool has_runs = false;
    if (Gr.own) {
        if (lane < 27) {
            const uint32_t b0 = __ldg(I.btab + (size_t)(Gr.own - 1u) * 27u + (uint32_t)lane);
            if (b0 != kNoBucket) {
                start = b0;
                len = __ldg(I.end + b0) - b0;
                if constexpr (kRuns) {
                    if (G.segend && len >= kRunRow && b0 < I.n) {
                        const int4 c = G.scell[b0];
                        has_runs = (__ldg(G.slot_alias + slot_of(c.x, c.y, c.z, Gd)) & kRunSlot) != 0;
                    }
                }
            }
        }
    } else if (Gr.split ? lane < 27 : lane < 9) {
        const int dx = Gr.split ? lane % 3 : 0;
        const int yz = Gr.split ? lane / 3 : lane;
        const int k = Gr.split ? 1 : Gr.W;
        slot = slot_of(Gr.cx - 1 + dx, Gr.cy + yz % 3 - 1, Gr.cz + yz / 3 - 1, Gd);
        start = __ldg(I.off + slot);
        len = __ldg(I.off + slot + k) - start;
        if constexpr (kRuns) {
            if (G.segend && len >= kRunRow)
                for (int d = 0; d < k; ++d) has_runs |= (__ldg(G.slot_alias + slot + d) & kRunSlot) != 0;
        }
    }
    const int words = (int)((len + 31u) >> 5);
    int sum = words;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(full, sum, o);
        if (lane >= o) sum += v;
    }
    if (keep) {
        L.start[lane] = start;
        L.len[lane] = len | (has_runs ? kRunRange : 0u);
        L.slot[lane] = slot;
        L.before[lane] = sum - words;
    }
    runs = kRuns && __any_sync(full, has_runs);
    return __shfl_sync(full, sum, 31);
}

// Lists words [done, done + room) of a sequence without runs.
__device__ __forceinline__ void list_words(const RangeList& L, int done, int room, uint32_t* base,
                                           uint32_t* info) {
    const int lane = threadIdx.x & 31;
    const uint32_t start = L.start[lane], len = L.len[lane];
    const int before = L.before[lane], words = (int)((len + 31u) >> 5);
    for (int k = max(0, done - before); k < words && before + k < done + room; ++k) {
        const int w = before + k - done;
        base[w] = start + 32u * (uint32_t)k;
        info[w] = min(32u, len - 32u * (uint32_t)k) | ((uint32_t)lane << 8);
    }
}

// Stages four words of candidates and tests them against the 8 NT particles
// whose columns the lanes hold (col): on return, half words of the masks, as
// 16 bits for particles 8 c + 2 t4 (h0[c]) and 8 c + 2 t4 + 1 (h1[c]) in lane
// (g, t4), for the candidates 16 g + [0, 16) of the 128.
template <int NT>
__device__ __forceinline__ void test_words(uint32_t* stage, const float4 (&xj)[4],
                                           const uint32_t (&sel)[4], const WalkBox& B, float inv_h,
                                           const uint32_t (&col)[NT], uint32_t (&h0)[NT],
                                           uint32_t (&h1)[NT]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const bool in = (sel[j] >> lane) & 1u;
        uint4 r = candidate_row((xj[j].x - B.ox) * inv_h, (xj[j].y - B.oy) * inv_h,
                                (xj[j].z - B.oz) * inv_h);
        if (!in)
            r = make_uint4(0u, pack_half2(0.0f, kHalfFar), pack_half2(0.0f, 1.0f), pack_half2(1.0f, 0.0f));
        // Candidate 16 gg + jj of the 128 (bit jj of group gg's half word) is
        // row 8 jj + (gg ^ (jj & 7)): stores and fragment loads both touch
        // every bank.
        const int jj = lane & 15, gg = 2 * j + (lane >> 4);
        reinterpret_cast<uint4*>(stage)[8 * jj + (gg ^ (jj & 7))] = r;
    }
    __syncwarp();
#pragma unroll
    for (int c = 0; c < NT; ++c) h0[c] = h1[c] = 0u;
#pragma unroll
    for (int k = 7; k >= 0; --k) {
        const uint32_t a0 = stage[32 * (2 * k) + (lane ^ (((2 * k) & 7) << 2))];
        const uint32_t a1 = stage[32 * (2 * k + 1) + (lane ^ (((2 * k + 1) & 7) << 2))];
#pragma unroll
        for (int c = 0; c < NT; ++c) {
            float d0, d1, d2, d3;
            mma_16x8x8(d0, d1, d2, d3, a0, a1, col[c]);
            // Sign bits in from the right: candidate 2k ends at bit 2k.
            h0[c] = __funnelshift_l(__float_as_uint(d2), h0[c], 1);
            h1[c] = __funnelshift_l(__float_as_uint(d3), h1[c], 1);
            h0[c] = __funnelshift_l(__float_as_uint(d0), h0[c], 1);
            h1[c] = __funnelshift_l(__float_as_uint(d1), h1[c], 1);
        }
    }
}

// The candidates of word w of a row of more than three cells that lie in the
// three cells around the particle's own (x coordinate ci); slot is the row's
// first slot.
__device__ __forceinline__ uint32_t own_cells(const WalkIndex& I, uint32_t slot, int dx, uint32_t bs) {
    const uint32_t a = __ldg(I.off + slot + (uint32_t)dx), e = __ldg(I.off + slot + (uint32_t)dx + 3u);
    return bit_range(a > bs ? min(a - bs, 32u) : 0u, e > bs ? min(e - bs, 32u) : 0u);
}

// The warp walk of one group (every lane of the warp calls it; at least one
// lane wants).  xi is the lane's x*, ci the x of its cell; lanes with `want`
// false list no candidates.  xin holds the candidates' positions in cell order
// and inv_h = 1 / support radius.  kLam (the delta pass): a candidate whose
// lambda sum with the lane, xi.w + xj.w, is zero adds an exact zero to the
// lane's sums (no s_corr either, which needs a negative sum) and the sums,
// started at +0, never are -0, so a lane whose lambda is zero lists
// candidates with a nonzero one only.  kRuns: in ranges that hold runs of
// identical particles (k_segments) a run is listed as its first particle,
// whose term is added as many times as the run is long (a step of the 1M dam
// break with a corner cell of 44,000 particles in 27,000 runs takes 229 ms;
// 434 when a word ended with each run, 255 in the one-thread walks before that,
// 265 with the runs' particles listed one by one, which costs later steps
// three times as much).  kList: nothing is
// summed; the lane's candidates go to the kept list of its particle p, whose
// rows so far are `kept`.
template <bool kPersist, bool kLam, bool kRuns, bool kList, class Sums>
__device__ __forceinline__ void walk_group(WalkSmem& sm, const WalkGroup& Gr, bool want, int ci,
                                           const float4 xi, const float4* xin, float inv_h,
                                           const GridDesc& Gd, const WalkIndex& I, const Grid& G,
                                           uint32_t p, uint32_t& kept, Sums& sums) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, t4 = lane & 3;
    const WalkBox B = walk_box(want, xi, inv_h);
    uint32_t col[4];
    {
        uint4 c = particle_column((xi.x - B.ox) * inv_h, (xi.y - B.oy) * inv_h, (xi.z - B.oz) * inv_h, B.lim);
        if (!want) c = make_uint4(0u, 0u, pack_half2(0.0f, kHalfFar), 0u);
        reinterpret_cast<uint4*>(sm.stage)[lane] = c;
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 4; ++j) col[j] = sm.stage[(8 * j + g) * 4 + t4];
        __syncwarp();
    }
    const bool key = Gr.own != 0u;
    const bool multi = Gr.W > 3;
    bool in_runs;
    const int total = walk_ranges<kRuns>(sm.ranges, Gr, I, Gd, G, true, in_runs);
    __syncwarp();
    if (kList && in_runs) {  // a row has no way to say how often its term counts
        if (want) kept = kNoList;
        return;
    }
    const bool runs = kRuns && !kList && in_runs;
    // Position of the listing with runs: range and candidate.
    int at_r = 0;
    uint32_t at_q = 0u;
    int done = 0;
    // Lists the next words; returns how many.
    auto fill = [&]() -> int {
        if (!runs) {
            const int nw = min(kWalkWords, total - done);
            list_words(sm.ranges, done, kWalkWords, sm.base, sm.info);
            done += nw;
            return nw;
        }
        int nw = 0;
        const int nr = key || Gr.split ? 27 : 9;
        while (nw < kWalkWords && at_r < nr) {
            const uint32_t st = sm.ranges.start[at_r], ln = sm.ranges.len[at_r];
            const uint32_t len_r = ln & ~kRunRange;
            if (at_q >= len_r) {
                ++at_r;
                at_q = 0u;
                continue;
            }
            // A word of up to 32 candidates without those to skip; the next one
            // begins at `next`.
            auto word = [&](uint32_t skip, uint32_t next) {
                if (lane == 0) {
                    sm.base[nw] = st + at_q;
                    sm.info[nw] = min(32u, len_r - at_q) | ((uint32_t)at_r << 8) | (ln & kRunRange ? kRunWord : 0u);
                    sm.skip(nw) = skip;
                }
                ++nw;
                at_q = next;
            };
            if (!(ln & kRunRange)) {
                word(0u, at_q + 32u);
                continue;
            }
            // A range with runs: a word starts past the runs of the words before
            // it.  The flags of four words at a time, so that their loads overlap.
            const uint32_t q0 = at_q;
            uint32_t end[4], copy[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t o = q0 + 32u * (uint32_t)j + (uint32_t)lane;
                end[j] = o < len_r ? __ldg(G.segend + st + o) : 0u;
                copy[j] = o < len_r ? (uint32_t)__ldg(G.sown + st + o) & kCopyBit : 0u;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (nw >= kWalkWords || at_q != q0 + 32u * (uint32_t)j || at_q >= len_r) break;
                const uint32_t far = __reduce_max_sync(full, end[j]);
                word(__ballot_sync(full, copy[j] != 0u), max(at_q + 32u, far > st ? far - st : 0u));
            }
        }
        return nw;
    };

    const bool lam_zero = kLam && xi.w == 0.0f;
    const bool all_zero = kLam && !__any_sync(full, want && xi.w != 0.0f);
    for (;;) {
        const int nw = fill();
        if (nw <= 0) break;
        __syncwarp();
        int cnt = 0;          // the lane's listed terms
        uint32_t filled = 0;  // words with any of them
        // --- phase 1, four words at a time
        for (int b = 0; b < nw; b += 4) {
            uint32_t sel[4], nz[4];  // candidates of each word, and those with a nonzero lambda
            uint32_t any_nz = 0u;
            float4 xj[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t n = b + j < nw ? sm.info[b + j] & 63u : 0u;
                sel[j] = bit_range(0u, n);
                if (kRuns && runs && b + j < nw) sel[j] &= ~sm.skip(b + j);
                xj[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if ((uint32_t)lane < n) {
                    uint32_t q = sm.base[b + j] + (uint32_t)lane;
                    if (key) q = I.at(q);
                    xj[j] = ld_step<kPersist>(xin + q);
                }
                if constexpr (kLam) {
                    nz[j] = __ballot_sync(full, xj[j].w != 0.0f);
                    any_nz |= nz[j];
                }
            }
            if (kRuns && runs) __syncwarp();  // the masks take the place of skip
            const bool test = !B.wide && (!kLam || !all_zero || any_nz != 0u);
            if (test) {
                uint32_t h0[4], h1[4];
                test_words<4>(sm.stage, xj, sel, B, inv_h, col, h0, h1);
                unsigned short* const mh = reinterpret_cast<unsigned short*>(sm.mask);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int w = b + (g >> 1), p = 8 * c + 2 * t4;
                    mh[2 * sm.at(w, p) + (g & 1)] = (unsigned short)h0[c];
                    mh[2 * sm.at(w, p + 1) + (g & 1)] = (unsigned short)h1[c];
                }
                __syncwarp();
            }
            // The bits that count: the word's candidates, for a lane whose
            // lambda is zero those with a nonzero one, and in a row of more
            // than three cells those of the lane's own three.
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int w = b + j;
                uint32_t m = B.wide ? 0xffffffffu : (test ? sm.mask[sm.at(w, lane)] : 0u);
                m &= sel[j];
                if constexpr (kLam)
                    if (lam_zero) m &= nz[j];
                if (!want) m = 0u;
                if (multi) {
                    if (m) m &= own_cells(I, sm.ranges.slot[(sm.info[w] >> 8) & 31u], ci - Gr.cx, sm.base[w]);
                }
                sm.mask[sm.at(w, lane)] = m;
                cnt += __popc(m);
                if (m) filled |= 1u << w;
            }
            __syncwarp();
        }
        // --- phase 2
        const int most = (int)__reduce_max_sync(full, (unsigned)cnt);
        uint32_t bits = 0u, bq = 0u;
        int w = 0;
        // The next listed candidate (there is one).
        auto next_q = [&]() -> uint32_t {
            if (bits == 0u) {
                w = __ffs(filled) - 1;
                filled &= filled - 1u;
                bits = sm.mask[sm.at(w, lane)];
                bq = sm.base[w];
            }
            const uint32_t k = (uint32_t)__ffs(bits) - 1u;
            bits &= bits - 1u;
            return bq + k;
        };
        if constexpr (kList) {
            auto take = [&]() {
                const uint32_t q = next_q();
                return key ? I.at(q) : q;
            };
            if (kept + (uint32_t)cnt <= 2u * kListRows) {
                uint2* to = G.lists + list_at(p) + 32u * (kept >> 1);
                int t = 0;
                if ((kept & 1u) && cnt > 0) {
                    to->y = take();
                    to += 32;
                    t = 1;
                }
                for (; t < cnt; t += 2) {
                    const uint32_t qa = take(), qb = t + 1 < cnt ? take() : p;
                    __stcs(to, make_uint2(qa, qb));
                    to += 32;
                }
                kept += (uint32_t)cnt;
            } else {
                kept = kNoList;
            }
            // A pile whose lists all overflowed is left to the walk at once.
            if (!__any_sync(full, want && kept != kNoList)) return;
        } else if (kRuns && runs) {
            float4 xa = make_float4(0.0f, 0.0f, 0.0f, 0.0f), xb = xa, ea = xa, eb = xa;
            uint32_t la = 0u, lb = 0u;  // ends of the runs they lead, 0 without one
            uint32_t qa = 0u, qb = 0u;
            auto load = [&](uint32_t& q, float4& x, float4& e, uint32_t& end) {
                q = next_q();
                end = sm.info[w] & kRunWord ? __ldg(G.segend + q) : 0u;
                if (key) q = I.at(q);
                x = ld_step<kPersist>(xin + q);
                if constexpr (Sums::kExtra) e = sums.extra(q);
            };
            if (cnt > 0) load(qa, xa, ea, la);
            if (cnt > 1) load(qb, xb, eb, lb);
            for (int t = 0; t < most; t += 2) {
                const float4 x0 = xa, x1 = xb, e0 = ea, e1 = eb;
                const uint32_t n0 = t < cnt ? (la ? la - qa : 1u) : 0u;
                const uint32_t n1 = t + 1 < cnt ? (lb ? lb - qb : 1u) : 0u;
                if (t + 2 < cnt) load(qa, xa, ea, la);
                if (t + 3 < cnt) load(qb, xb, eb, lb);
                if (__any_sync(full, n0 > 1u || n1 > 1u)) sums.add2_times(x0, x1, e0, e1, n0, n1);
                else sums.add2(x0, x1, e0, e1, n0 != 0u, n1 != 0u);
            }
        } else {
            float4 xa = make_float4(0.0f, 0.0f, 0.0f, 0.0f), xb = xa, ea = xa, eb = xa;
            auto load = [&](float4& x, float4& e) {
                uint32_t q = next_q();
                if (key) q = I.at(q);
                x = ld_step<kPersist>(xin + q);
                if constexpr (Sums::kExtra) e = sums.extra(q);
            };
            if (cnt > 0) load(xa, ea);
            if (cnt > 1) load(xb, eb);
            for (int t = 0; t < most; t += 2) {
                const float4 x0 = xa, x1 = xb, e0 = ea, e1 = eb;
                if (t + 2 < cnt) load(xa, ea);
                if (t + 3 < cnt) load(xb, eb);
                sums.add2(x0, x1, e0, e1, t < cnt, t + 1 < cnt);
            }
        }
        __syncwarp();
    }
}

// A pass's sums.  A quantity k of a particle is the sum over its candidates of
// factor x value, each product rounded before it is added (or fused, in the
// fast build, as the one-thread walk's expressions are).  The term D says:
// kQuantities; kFactors and factor_of(k), the factor of quantity k (-1: none);
// kTermFactor, whether the factors come with the term (else const_factor(k));
// kExtra and extra(q), per-candidate data besides the position; eval, the
// values and factors of one candidate and whether it is in support; and in the
// exact build products, the products of two candidates at once.
//
// Terms whose candidates may have to be evaluated wherever they are (the
// coupling's, for values that are not finite) set kSpecials and say which:
// special(x_j).
template <class D, class = void>
struct HasSpecials : std::false_type {};
template <class D>
struct HasSpecials<D, std::void_t<decltype(D::kSpecials)>> : std::integral_constant<bool, D::kSpecials> {};

// No sums (a walk that only lists).
struct NoSums {
    static constexpr bool kExtra = false;
};

// The sums of one lane (warp walk).
template <class D>
struct LaneSums {
    static constexpr int kNq = D::kQuantities;
    static constexpr bool kExtra = D::kExtra;
    float sum[kNq];
    const D d;
    __device__ __forceinline__ explicit LaneSums(const D& def) : d(def) {
#pragma unroll
        for (int k = 0; k < kNq; ++k) sum[k] = 0.0f;
    }
    // Continues from sums that are there already.
    __device__ __forceinline__ void start(const float* from) {
#pragma unroll
        for (int k = 0; k < kNq; ++k) sum[k] = from[k];
    }
    __device__ __forceinline__ float4 extra(uint32_t q) const { return d.extra(q); }
    __device__ __forceinline__ void add(const float4& xj, const float4& ej) {
        float v[kNq], f[D::kFactors];
        if (d.eval(xj, ej, v, f)) {
#pragma unroll
            for (int k = 0; k < kNq; ++k) {
                if (D::factor_of(k) < 0) sum[k] = sum[k] + v[k];
                else sum[k] = sum[k] + f[D::factor_of(k) < 0 ? 0 : D::factor_of(k)] * v[k];
            }
        }
    }
    // The term of a run of L identical candidates: added L times, exactly.
    __device__ __forceinline__ void add_run(const float4& xj, const float4& ej, uint32_t L) {
        float v[kNq], f[D::kFactors];
        if (d.eval(xj, ej, v, f)) {
#pragma unroll
            for (int k = 0; k < kNq; ++k)
                if (D::factor_of(k) >= 0) v[k] = f[D::factor_of(k) < 0 ? 0 : D::factor_of(k)] * v[k];
            add_times(sum, v, L);
        }
    }
    // The terms of two candidates, the first one na times, then the other nb
    // times.
    __device__ __forceinline__ void add2_times(const float4& xa, const float4& xb, const float4& ea,
                                               const float4& eb, uint32_t na, uint32_t nb) {
#if !PBF_FAST
        if (d.C.paired) {
            float2 v[kNq];
            bool in_a, in_b;
            d.products(xa, xb, ea, eb, v, in_a, in_b);
            float a[kNq], b[kNq];
#pragma unroll
            for (int k = 0; k < kNq; ++k) {
                a[k] = v[k].x;
                b[k] = v[k].y;
            }
            add_times(sum, a, in_a ? na : 0u);
            add_times(sum, b, in_b ? nb : 0u);
            return;
        }
#endif
        if (na) add_run(xa, ea, na);
        if (nb) add_run(xb, eb, nb);
    }
    // The terms of two candidates, the first one first, where they are there.
    __device__ __forceinline__ void add2(const float4& xa, const float4& xb, const float4& ea,
                                         const float4& eb, bool has_a, bool has_b) {
#if PBF_FAST
        if (has_a) add(xa, ea);
        if (has_b) add(xb, eb);
#else
        if (!d.C.paired) {
            if (has_a) add(xa, ea);
            if (has_b) add(xb, eb);
            return;
        }
        float2 v[kNq];
        bool in_a, in_b;
        d.products(xa, xb, ea, eb, v, in_a, in_b);
        if (has_a && in_a) {
#pragma unroll
            for (int k = 0; k < kNq; ++k) sum[k] = sum[k] + v[k].x;
        }
        if (has_b && in_b) {
#pragma unroll
            for (int k = 0; k < kNq; ++k) sum[k] = sum[k] + v[k].y;
        }
#endif
    }
    __device__ __forceinline__ float get(int k) const { return sum[k]; }
};

// The sums of a particle of a team: S lanes evaluate two candidates each, and
// lane j < kPairs of the S adds quantities 2 j and 2 j + 1 in list order.
template <class D, int S>
struct TeamSums {
    static constexpr int kNq = D::kQuantities;
    static constexpr int kPairs = (kNq + 1) / 2;
    static constexpr int kRow = 66;
    static constexpr bool kExtra = D::kExtra;
    static constexpr bool kSpecials = HasSpecials<D>::value;
    using Term = D;
    static_assert(kPairs <= S, "a lane per pair of quantities");
    float2 sum;
    const D d;
    __device__ __forceinline__ explicit TeamSums(const D& def) : sum(make_float2(0.0f, 0.0f)), d(def) {}
    __device__ __forceinline__ void start(const float* from) {
        const int s = (int)threadIdx.x & (S - 1);
#pragma unroll
        for (int k = 0; k < kNq; ++k) {
            if (s == k / 2) {
                if (k & 1) sum.y = from[k];
                else sum.x = from[k];
            }
        }
    }
    __device__ __forceinline__ float4 extra(uint32_t q) const { return d.extra(q); }
    // The lane's two terms into the rows, zeros where there are none (a sum
    // started at +0 never is -0, so adding +0 keeps its bits).
    __device__ __forceinline__ void put(float2* rows, const float4& xa, const float4& xb, const float4& ea,
                                        const float4& eb, bool has_a, bool has_b) const {
        float4* const at = reinterpret_cast<float4*>(rows + 2 * ((int)threadIdx.x & 31));
#if !PBF_FAST
        if (d.C.paired) {
            float2 v[kNq];
            bool in_a, in_b;
            d.products(xa, xb, ea, eb, v, in_a, in_b);
            in_a = in_a && has_a;
            in_b = in_b && has_b;
#pragma unroll
            for (int j = 0; j < kPairs; ++j) {
                const float2 lo = v[2 * j];
                const float2 hi = 2 * j + 1 < kNq ? v[2 * j + 1 < kNq ? 2 * j + 1 : 0] : make_float2(0.0f, 0.0f);
                at[j * (kRow / 2)] = make_float4(in_a ? lo.x : 0.0f, in_a ? hi.x : 0.0f,
                                                 in_b ? lo.y : 0.0f, in_b ? hi.y : 0.0f);
            }
            return;
        }
#endif
        float va[kNq], vb[kNq], fa[D::kFactors], fb[D::kFactors];
        const bool in_a = has_a && d.eval(xa, ea, va, fa);
        const bool in_b = has_b && d.eval(xb, eb, vb, fb);
        // Value, or its product in the exact build, of quantity k; factor in
        // the fast build, whose sums fuse the product and the addition.
        auto value = [&](bool in, const float* v, const float* f, int k) {
            if (k >= kNq || !in) return 0.0f;
            const int c = D::factor_of(k);
            return PBF_FAST || c < 0 ? v[k] : f[c < 0 ? 0 : c] * v[k];
        };
        auto factor = [&](bool in, const float* f, int k) {
            const int c = k < kNq ? D::factor_of(k) : -1;
            return c < 0 ? 1.0f : (in ? f[c < 0 ? 0 : c] : 0.0f);
        };
#pragma unroll
        for (int j = 0; j < kPairs; ++j) {
            const int k0 = 2 * j, k1 = 2 * j + 1;
            at[j * (kRow / 2)] = make_float4(value(in_a, va, fa, k0), value(in_a, va, fa, k1),
                                             value(in_b, vb, fb, k0), value(in_b, vb, fb, k1));
            if (PBF_FAST)
                at[(kPairs + j) * (kRow / 2)] =
                    make_float4(factor(in_a, fa, k0), factor(in_a, fa, k1), factor(in_b, fb, k0),
                                factor(in_b, fb, k1));
        }
    }
    __device__ __forceinline__ void fold(const float2* rows) {
        const int lane = (int)threadIdx.x & 31, s = lane & (S - 1);
        if (s < kPairs) {
            const float4* const v = reinterpret_cast<const float4*>(rows + s * kRow + 2 * (lane - s));
#if PBF_FAST
            const float4* const f =
                reinterpret_cast<const float4*>(rows + (kPairs + s) * kRow + 2 * (lane - s));
#endif
#pragma unroll
            for (int i = 0; i < S; ++i) {
                const float4 t = v[i];
#if PBF_FAST
                const float4 c = f[i];
                sum = make_float2(fmaf(c.x, t.x, sum.x), fmaf(c.y, t.y, sum.y));
                sum = make_float2(fmaf(c.z, t.z, sum.x), fmaf(c.w, t.w, sum.y));
#else
                sum = __fadd2_rn(sum, make_float2(t.x, t.y));
                sum = __fadd2_rn(sum, make_float2(t.z, t.w));
#endif
            }
        }
    }
    // Sum k, in every lane of the particle (warp-collective).
    __device__ __forceinline__ float get(int k) const {
        return __shfl_sync(0xffffffffu, k & 1 ? sum.y : sum.x, ((int)threadIdx.x & (32 - S)) + k / 2);
    }
};

// The team walk of one group (every lane of the team's four warps calls it).
// In the listing, lane l of each warp stands for the team's particle
// l / (32 / TP): xi, ci, want as in walk_group.  In the evaluation, thread t
// stands for particle t / (128 / TP) of the team, sorted position p, which is
// the one that `sums` and (with kKeep) the kept list are about.
template <int TP, bool kLam, bool kKeep, class Sums>
__device__ __forceinline__ void team_group(TeamSmem<TP>& sm, const WalkGroup& Gr, bool want, int ci,
                                           const float4 xi, const float4* __restrict__ xin, float inv_h,
                                           const GridDesc& Gd, const WalkIndex& I, const Grid& G,
                                           uint32_t p, uint32_t& kept, Sums& sums) {
    constexpr int NT = TP / 8;
    constexpr int LPP = 32 / TP;  // listing lanes per particle
    constexpr int WPL = 4 / LPP;  // words of a batch that a lane settles
    constexpr int S = 128 / TP;   // evaluating lanes per particle
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int g = lane >> 2, t4 = lane & 3;
    const int pl = lane / LPP, j0 = (lane % LPP) * WPL;
    uint32_t* const stage = reinterpret_cast<uint32_t*>(sm.warp[wid]);
    const WalkBox B = walk_box(want, xi, inv_h);
    uint32_t col[NT];
    {
        uint4 c = particle_column((xi.x - B.ox) * inv_h, (xi.y - B.oy) * inv_h, (xi.z - B.oz) * inv_h, B.lim);
        if (!want) c = make_uint4(0u, 0u, pack_half2(0.0f, kHalfFar), 0u);
        if (lane % LPP == 0) reinterpret_cast<uint4*>(stage)[pl] = c;
        __syncwarp();
#pragma unroll
        for (int j = 0; j < NT; ++j) col[j] = stage[(8 * j + g) * 4 + t4];
        __syncwarp();
    }
    const bool key = Gr.own != 0u;
    const bool multi = Gr.W > 3;
    bool runs;
    const int words = walk_ranges<false>(sm.ranges, Gr, I, Gd, G, wid == 0, runs);
    __syncwarp();
    // A particle all of whose candidates are special.
    const bool every = Sums::kSpecials && !(isfinite(xi.x) && isfinite(xi.y) && isfinite(xi.z));
    const bool lam_zero = kLam && xi.w == 0.0f && !every;
    const bool all_zero = kLam && !__any_sync(full, want && xi.w != 0.0f);
    uint32_t run = 0u;  // terms of particle pl listed so far

    // Phase 2 of everything listed; every thread of the team calls it.
    auto evaluate = [&]() {
        if (wid == 0 && lane % LPP == 0) sm.total[pl] = run;
        __syncthreads();
        const int pe = threadIdx.x / S, s = threadIdx.x & (S - 1);
        const int cnt = (int)sm.total[pe];
        const int most = (int)__reduce_max_sync(full, (unsigned)cnt);
        const unsigned short* const my = sm.list + pe * TeamSmem<TP>::kListRow;
        float2* const rows = reinterpret_cast<float2*>(sm.warp[wid]);
        float4 xa = make_float4(0.0f, 0.0f, 0.0f, 0.0f), xb = xa, ea = xa, eb = xa;
        uint2* to = nullptr;
        if constexpr (kKeep) {
            const uint32_t rows = ((uint32_t)cnt + 1u) / 2u;
            if (kept + rows <= kListRows) {
                to = G.lists + (size_t)p * kListRows + kept;
                kept += rows;
            } else {
                kept = kNoList;
            }
        }
        // Candidates t and t + 1 of the list (t < cnt).
        auto load = [&](int t) {
            const uint32_t two = *reinterpret_cast<const uint32_t*>(my + t);
            uint32_t qa = sm.base[(two >> 5) & (kTeamWords - 1)] + (two & 31u), qb = p;
            if (key) qa = I.at(qa);
            xa = __ldg(xin + qa);
            if constexpr (Sums::kExtra) ea = sums.extra(qa);
            if (t + 1 < cnt) {
                qb = sm.base[(two >> 21) & (kTeamWords - 1)] + ((two >> 16) & 31u);
                if (key) qb = I.at(qb);
                xb = __ldg(xin + qb);
                if constexpr (Sums::kExtra) eb = sums.extra(qb);
            }
            if constexpr (kKeep) {
                if (to) to[t >> 1] = make_uint2(qa, qb);
            }
        };
        if (2 * s < cnt) load(2 * s);
        for (int t0 = 0; t0 < most; t0 += 2 * S) {
            const int t = t0 + 2 * s;
            const float4 x0 = xa, x1 = xb, e0 = ea, e1 = eb;
            if (t + 2 * S < cnt) load(t + 2 * S);
            sums.put(rows, x0, x1, e0, e1, t < cnt, t + 1 < cnt);
            __syncwarp();
            sums.fold(rows);
            __syncwarp();
        }
        run = 0u;
        __syncthreads();
    };

    for (int done = 0; done < words; done += kTeamWords) {
        const int nw = min(kTeamWords, words - done);
        if (wid == 0) list_words(sm.ranges, done, kTeamWords, sm.base, sm.info);
        __syncthreads();
        for (int b0 = 0; b0 < nw; b0 += 4 * kTeamWarps) {
            // --- phase 1: this warp's four words
            const int b = b0 + 4 * wid;
            uint32_t m[WPL];
#pragma unroll
            for (int i = 0; i < WPL; ++i) m[i] = 0u;
            if (b < nw) {
                uint32_t sel[4], nz[4], sp[4];  // words, those with a nonzero w, special ones
                uint32_t any_nz = 0u;
                float4 xj[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t n = b + j < nw ? sm.info[b + j] & 63u : 0u;
                    sel[j] = bit_range(0u, n);
                    xj[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if ((uint32_t)lane < n) {
                        uint32_t q = sm.base[b + j] + (uint32_t)lane;
                        if (key) q = I.at(q);
                        xj[j] = __ldg(xin + q);
                    }
                    if constexpr (kLam) {
                        nz[j] = __ballot_sync(full, xj[j].w != 0.0f);
                        any_nz |= nz[j];
                    }
                    if constexpr (Sums::kSpecials)
                        sp[j] = __ballot_sync(full, Sums::Term::special(xj[j], sums.d.C));
                }
                const bool test = !B.wide && (!kLam || !all_zero || any_nz != 0u);
                if (test) {
                    uint32_t h0[NT], h1[NT];
                    test_words<NT>(stage, xj, sel, B, inv_h, col, h0, h1);
                    unsigned short* const mh = reinterpret_cast<unsigned short*>(sm.mask[wid]);
#pragma unroll
                    for (int c = 0; c < NT; ++c) {
                        const int at = (g >> 1) * TP + 8 * c + 2 * t4;
                        mh[2 * at + (g & 1)] = (unsigned short)h0[c];
                        mh[2 * at + 2 + (g & 1)] = (unsigned short)h1[c];
                    }
                    __syncwarp();
                }
#pragma unroll
                for (int i = 0; i < WPL; ++i) {
                    const int j = j0 + i;
                    uint32_t in = 0u, innz = 0u, insp = 0u;
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        if (c == j) in = sel[c];
                        if (kLam && c == j) innz = nz[c];
                        if (Sums::kSpecials && c == j) insp = sp[c];
                    }
                    uint32_t v = B.wide || every ? 0xffffffffu : (test ? sm.mask[wid][j * TP + pl] : 0u);
                    if (kLam && lam_zero) v &= innz;
                    v = (v | insp) & in;
                    if (!want) v = 0u;
                    if (multi) {
                        const int w = b + j;
                        if (v) v &= own_cells(I, sm.ranges.slot[(sm.info[w] >> 8) & 31u], ci - Gr.cx, sm.base[w]);
                    }
                    m[i] = v;
                }
            }
            uint32_t mine = 0u;
#pragma unroll
            for (int i = 0; i < WPL; ++i) mine += (uint32_t)__popc(m[i]);
            uint32_t upto = mine;  // this lane's and the particle's lanes before it
#pragma unroll
            for (int o = 1; o < LPP; o <<= 1) {
                const uint32_t v = __shfl_up_sync(full, upto, o);
                if (lane % LPP >= o) upto += v;
            }
            if (lane % LPP == LPP - 1) sm.count[wid][pl] = upto;
            __syncthreads();
            uint32_t before = 0u, round = 0u;
#pragma unroll
            for (int v = 0; v < kTeamWarps; ++v) {
                const uint32_t c = sm.count[v][pl];
                if (v < wid) before += c;
                round += c;
            }
            if (__syncthreads_or(run + round > (uint32_t)kTeamTerms)) evaluate();
            uint32_t at = (uint32_t)(pl * TeamSmem<TP>::kListRow) + run + before + upto - mine;
#pragma unroll
            for (int i = 0; i < WPL; ++i) {
                uint32_t v = m[i];
                while (v) {
                    sm.list[at++] = (unsigned short)(((b + j0 + i) << 5) | (__ffs(v) - 1));
                    v &= v - 1u;
                }
            }
            run += round;
        }
        evaluate();
    }
}

// Scene of sorted particle p (0 for a single scene).
__device__ __forceinline__ uint32_t scene_at(const Grid& G, uint32_t p) {
    return G.spid ? __ldg(G.spid + p) : 0u;
}

// The group of the first lane in `todo`, and whether the lane is in it
// (warp-collective).  p, cell (w = bucket row + 1, 0 when clean): the lane's
// particle and candidate cell; sid: its scene.
template <class P>
__device__ __forceinline__ WalkGroup next_group(uint32_t todo, const Grid& G, const P& prm, uint32_t p,
                                                uint32_t sid, const int4 cell, bool& mem, float& inv_h,
                                                GridDesc& Gd) {
    const unsigned full = 0xffffffffu;
    const int L = __ffs(todo) - 1;
    WalkGroup Gr;
    Gr.cx = __shfl_sync(full, cell.x, L);
    Gr.cy = __shfl_sync(full, cell.y, L);
    Gr.cz = __shfl_sync(full, cell.z, L);
    Gr.own = (uint32_t)__shfl_sync(full, cell.w, L);
    Gr.W = 3;
    Gr.split = false;
    mem = ((todo >> (threadIdx.x & 31)) & 1u) && cell.y == Gr.cy && cell.z == Gr.cz;
    uint32_t pl = 0u;
    if constexpr (!std::is_same<P, OneScene>::value) {
        pl = __shfl_sync(full, p, L);
        const uint32_t sl = __shfl_sync(full, sid, L);
        mem = mem && sid == sl;
    }
    const StepConsts& C = prm.at(G.spid, pl);
    Gd = C.grid;
    inv_h = C.inv_cell;
    if (Gr.own) {
        mem = mem && cell.w != 0 && cell.x == Gr.cx;
    } else {
        const int wx0 = wrap(Gr.cx - 1, Gd.ox, Gd.gx);
        const uint32_t d = (uint32_t)cell.x - (uint32_t)Gr.cx;
        mem = mem && cell.w == 0 && d <= 2u;
        const int far = (int)__reduce_max_sync(full, mem ? d : 0u);
        if (wx0 + far + 3 > Gd.gx || Gr.cx <= -(1 << 30) || Gr.cx >= (1 << 30)) {
            mem = mem && d == 0u;
            Gr.split = wx0 + 3 > Gd.gx;
        } else {
            Gr.W = far + 3;
        }
    }
    return Gr;
}

// The warp walk over the candidates, in index I with positions xin, of every
// lane that wants (every lane of the warp calls it): the lane's particle has
// sorted position p (any valid one where it does not want), candidate cell
// `cell` (w = its bucket row + 1, 0 when clean) and x* xi.  Returns false,
// with nothing summed, when the warp's particles sit in too many cells (the
// caller walks lane by lane then).
template <bool kPersist, bool kLam, bool kRuns, bool kList, class P, class Sums>
__device__ __forceinline__ bool warp_walk(WalkSmem& sm, const Grid& G, const WalkIndex& I, const P& prm,
                                          uint32_t p, const int4 cell, bool want, const float4 xi,
                                          const float4* xin, uint32_t& kept, Sums& sums) {
    const unsigned full = 0xffffffffu;
    uint32_t todo = __ballot_sync(full, want);
    if (!todo) return true;
    const uint32_t sid = scene_at(G, p);
    {
        const uint32_t x = cell.w ? (uint32_t)cell.x * 3u + 1u : ((uint32_t)cell.x + 0x30000000u) / 3u * 3u;
        const uint32_t k = (((uint32_t)cell.y * 73856093u) ^ ((uint32_t)cell.z * 19349663u) ^
                            (sid * 2654435761u)) + x * 83492791u;
        const uint32_t same = __match_any_sync(full, want ? k : 0u) & todo;
        const bool first = want && (int)(threadIdx.x & 31) == __ffs(same) - 1;
        if (__popc(__ballot_sync(full, first)) > (kList ? kMaxListGroups : kMaxGroups)) return false;
    }
    while (todo) {
        bool mem;
        float inv_h;
        GridDesc Gd;
        const WalkGroup Gr = next_group(todo, G, prm, p, sid, cell, mem, inv_h, Gd);
        todo &= ~__ballot_sync(full, mem);
        walk_group<kPersist, kLam, kRuns, kList>(sm, Gr, mem, cell.x, xi, xin, inv_h, Gd, I, G, p, kept,
                                                 sums);
    }
    return true;
}

// The team walk (every thread of the team calls it; p, cell, want and xi as
// in warp_walk, of the listing's particle, the same in all four warps).
// team_walk_keep keeps the lists of the evaluation's particles pe, see team_group.
template <int TP, bool kLam, bool kKeep, class P, class Sums>
__device__ __forceinline__ void team_walk_keep(TeamSmem<TP>& sm, const Grid& G, const WalkIndex& I,
                                               const P& prm, uint32_t p, const int4 cell, bool want,
                                               const float4 xi, const float4* __restrict__ xin, uint32_t pe,
                                               uint32_t& kept, Sums& sums) {
    const unsigned full = 0xffffffffu;
    uint32_t todo = __ballot_sync(full, want);
    const uint32_t sid = scene_at(G, p);
    while (todo) {
        bool mem;
        float inv_h;
        GridDesc Gd;
        const WalkGroup Gr = next_group(todo, G, prm, p, sid, cell, mem, inv_h, Gd);
        todo &= ~__ballot_sync(full, mem);
        team_group<TP, kLam, kKeep>(sm, Gr, mem, cell.x, xi, xin, inv_h, Gd, I, G, pe, kept, sums);
    }
}

template <int TP, bool kLam, class P, class Sums>
__device__ __forceinline__ void team_walk(TeamSmem<TP>& sm, const Grid& G, const WalkIndex& I, const P& prm,
                                          uint32_t p, const int4 cell, bool want, const float4 xi,
                                          const float4* __restrict__ xin, Sums& sums) {
    uint32_t kept = 0u;
    team_walk_keep<TP, kLam, false>(sm, G, I, prm, p, cell, want, xi, xin, 0u, kept, sums);
}

__device__ __forceinline__ WalkIndex fluid_index(const Grid& G) {
    return G.ix;
}

__device__ __forceinline__ WalkIndex boundary_index(const Grid& G) {
    return WalkIndex{G.bg.n, G.bg.off, G.bg.merged, G.bg.end, G.bg.btab};
}

// Whether a slot among the 27 around a clean particle's cell holds the stamp
// `it`: with the moved stamps and it, whether a candidate moved in the delta
// pass of Jacobi iteration it - 1 (when none did, the candidates all sit
// where they sat for the previous density pass, so the particle's rho and
// lambda would come out bit for bit the same); with the lambda stamps and
// it + 1, whether a candidate has a nonzero lambda in iteration it.  Only
// the z planes [c0, c1) of the three are looked at.
template <bool kPersist>
__device__ __forceinline__ bool neighbourhood_stamped(const int4 cell, const GridDesc& Gd,
                                                      const uint32_t* stamps, uint32_t it, int c0, int c1) {
    // The slots from wrapped coordinates per axis; the loads are independent,
    // so they overlap.
    uint32_t wx[3], wy[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        wx[d] = (uint32_t)wrap(cell.x + d - 1, Gd.ox, Gd.gx);
        wy[d] = (uint32_t)wrap(cell.y + d - 1, Gd.oy, Gd.gy);
    }
    bool any = false;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        if (c < c0 || c >= c1) continue;
        const uint32_t wz = (uint32_t)wrap(cell.z + c - 1, Gd.oz, Gd.gz);
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const uint32_t row = Gd.base + (uint32_t)Gd.gx * (wy[b] + (uint32_t)Gd.gy * wz);
#pragma unroll
            for (int a = 0; a < 3; ++a) any |= ld_step<kPersist>(stamps + row + wx[a]) == it;
        }
    }
    return any;
}

// The same for a team: whether each listing lane's particle (asking ones)
// has a stamped slot; three warps look at a plane each.
template <int TP>
__device__ __forceinline__ bool team_stamped(TeamSmem<TP>& sm, bool ask, const int4 cell, const GridDesc& Gd,
                                             const uint32_t* stamps, uint32_t it) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, pl = lane / (32 / TP);
    if (threadIdx.x < TP) sm.flag[threadIdx.x] = 0;
    __syncthreads();
    if (ask && wid < 3 && neighbourhood_stamped<false>(cell, Gd, stamps, it, wid, wid + 1)) sm.flag[pl] = 1;
    __syncthreads();
    return ask && sm.flag[pl] != 0;
}

#if !PBF_FAST
// r = x_i - x_j and r^2 of two candidates (xa, xb), as rel_sq's.
struct PairRel {
    float2 x, y, z, r2;
    __device__ __forceinline__ PairRel(const float4& xi, const float4& xa, const float4& xb, float one) {
        x = make_float2(xi.x - xa.x, xi.x - xb.x);
        y = make_float2(xi.y - xa.y, xi.y - xb.y);
        z = make_float2(xi.z - xa.z, xi.z - xb.z);
        r2 = pbf::add2(mul2(x, x), pbf::add2(mul2(y, y), mul2(z, z), one), one);
    }
};

__device__ __forceinline__ float2 not_below_zero(float2 a) {
    return make_float2(fmaxf(a.x, 0.0f), fmaxf(a.y, 0.0f));
}

// poly6 of two squared distances below the support's.
__device__ __forceinline__ float2 poly6_2(float2 r2, const StepConsts& C) {
    const float2 d = not_below_zero(sub2(both(C.h2), r2));
    return mul2(mul2(mul2(both(C.k_poly), d), d), d);
}

// spiky_coeff of two squared distances below C.cut (C.paired).
__device__ __forceinline__ float2 spiky_coeff_2(float2 r2, const StepConsts& C) {
    float2 len, inv;
    root_and_inverse(r2, len, inv);
    const float2 d = not_below_zero(sub2(both(C.h), len));
    const float2 c = quotient(mul2(mul2(both(C.k_spiky), d), d), len, inv);
    return make_float2(r2.x > C.r2_min ? c.x : 0.0f, r2.y > C.r2_min ? c.y : 0.0f);
}
#endif

// compute_density + compute_lambda (pbf_solver.cpp:129-179): the density, the
// gradient sum and the sum of the squared gradients in one candidate pass.
struct DensityGradTerm {
    static constexpr int kQuantities = 5, kFactors = 2;
    static constexpr bool kExtra = false;
    const StepConsts& C;
    const float4 xi;
    static __host__ __device__ constexpr int factor_of(int k) { return k == 0 ? 0 : (k < 4 ? 1 : -1); }
    __device__ __forceinline__ bool eval(const float4& xj, const float4&, float* v, float* f) const {
        float rx, ry, rz;
        const float r_sq = rel_sq(xi, xj, rx, ry, rz);
        if (!(r_sq < C.cut)) return false;
        v[0] = poly6(r_sq, C);
        const float c = spiky_coeff(r_sq, C);
        v[1] = c * rx;
        v[2] = c * ry;
        v[3] = c * rz;
        v[4] = sqn(C.mr * v[1], C.mr * v[2], C.mr * v[3]);
        f[0] = C.mass;
        f[1] = C.mr;
        return true;
    }
#if !PBF_FAST
    __device__ __forceinline__ void products(const float4& xa, const float4& xb, const float4&,
                                             const float4&, float2* v, bool& in_a, bool& in_b) const {
        const PairRel r(xi, xa, xb, C.one);
        in_a = r.r2.x < C.cut;
        in_b = r.r2.y < C.cut;
        v[0] = mul2(both(C.mass), poly6_2(r.r2, C));
        const float2 c = spiky_coeff_2(r.r2, C), mr = both(C.mr);
        v[1] = mul2(mr, mul2(c, r.x));
        v[2] = mul2(mr, mul2(c, r.y));
        v[3] = mul2(mr, mul2(c, r.z));
        v[4] = pbf::add2(mul2(v[1], v[1]), pbf::add2(mul2(v[2], v[2]), mul2(v[3], v[3]), C.one), C.one);
    }
#endif
};

// The density alone, and the gradient sums alone (density-first walks).
struct DensityTerm {
    static constexpr int kQuantities = 1, kFactors = 1;
    static constexpr bool kExtra = false;
    const StepConsts& C;
    const float4 xi;
    static __host__ __device__ constexpr int factor_of(int) { return 0; }
    __device__ __forceinline__ bool eval(const float4& xj, const float4&, float* v, float* f) const {
        float rx, ry, rz;
        const float r_sq = rel_sq(xi, xj, rx, ry, rz);
        if (!(r_sq < C.cut)) return false;
        v[0] = poly6(r_sq, C);
        f[0] = C.mass;
        return true;
    }
#if !PBF_FAST
    __device__ __forceinline__ void products(const float4& xa, const float4& xb, const float4&,
                                             const float4&, float2* v, bool& in_a, bool& in_b) const {
        const PairRel r(xi, xa, xb, C.one);
        in_a = r.r2.x < C.cut;
        in_b = r.r2.y < C.cut;
        v[0] = mul2(both(C.mass), poly6_2(r.r2, C));
    }
#endif
};

struct GradTerm {
    static constexpr int kQuantities = 4, kFactors = 1;
    static constexpr bool kExtra = false;
    const StepConsts& C;
    const float4 xi;
    static __host__ __device__ constexpr int factor_of(int k) { return k < 3 ? 0 : -1; }
    __device__ __forceinline__ bool eval(const float4& xj, const float4&, float* v, float* f) const {
        float rx, ry, rz;
        const float r_sq = rel_sq(xi, xj, rx, ry, rz);
        if (!(r_sq < C.cut)) return false;
        const float c = spiky_coeff(r_sq, C);
        v[0] = c * rx;
        v[1] = c * ry;
        v[2] = c * rz;
        v[3] = sqn(C.mr * v[0], C.mr * v[1], C.mr * v[2]);
        f[0] = C.mr;
        return true;
    }
#if !PBF_FAST
    __device__ __forceinline__ void products(const float4& xa, const float4& xb, const float4&,
                                             const float4&, float2* v, bool& in_a, bool& in_b) const {
        const PairRel r(xi, xa, xb, C.one);
        in_a = r.r2.x < C.cut;
        in_b = r.r2.y < C.cut;
        const float2 c = spiky_coeff_2(r.r2, C), mr = both(C.mr);
        v[0] = mul2(mr, mul2(c, r.x));
        v[1] = mul2(mr, mul2(c, r.y));
        v[2] = mul2(mr, mul2(c, r.z));
        v[3] = pbf::add2(mul2(v[0], v[0]), pbf::add2(mul2(v[1], v[1]), mul2(v[2], v[2]), C.one), C.one);
    }
#endif
};

// The boundary's share of the same sums (two-way coupling, no counterpart in
// the reference): rho0 psi_b W and its gradient psi_b grad W (= (rho0 psi_b /
// rho0) grad W).  The boundary does not move, so it adds nothing to the sum
// of the neighbours' squared gradients.
struct BoundaryDensityTerm {
    static constexpr int kQuantities = 4, kFactors = 2;
    static constexpr bool kExtra = false;
    const StepConsts& C;
    const float4 xi;
    static __host__ __device__ constexpr int factor_of(int k) { return k == 0 ? 0 : 1; }
    __device__ __forceinline__ bool eval(const float4& b, const float4&, float* v, float* f) const {
        const float rx = xi.x - b.x, ry = xi.y - b.y, rz = xi.z - b.z;
        const float r_sq = sqn(rx, ry, rz);
        if (!(r_sq < C.cut)) return false;
        v[0] = poly6(r_sq, C);
        const float c = spiky_coeff(r_sq, C);
        v[1] = c * rx;
        v[2] = c * ry;
        v[3] = c * rz;
        f[0] = C.rho0 * b.w;
        f[1] = b.w;
        return true;
    }
#if !PBF_FAST
    __device__ __forceinline__ void products(const float4& xa, const float4& xb, const float4&,
                                             const float4&, float2* v, bool& in_a, bool& in_b) const {
        const PairRel r(xi, xa, xb, C.one);
        in_a = r.r2.x < C.cut;
        in_b = r.r2.y < C.cut;
        const float2 psi = make_float2(xa.w, xb.w);
        v[0] = mul2(mul2(both(C.rho0), psi), poly6_2(r.r2, C));
        const float2 c = spiky_coeff_2(r.r2, C);
        v[1] = mul2(psi, mul2(c, r.x));
        v[2] = mul2(psi, mul2(c, r.y));
        v[3] = mul2(psi, mul2(c, r.z));
    }
#endif
};

// compute_delta_position (pbf_solver.cpp:181-223).  A zero lambda sum adds an
// exact zero (no s_corr either); the sum, started at +0, never becomes -0, so
// skipping it keeps every bit.
struct DeltaTerm {
    static constexpr int kQuantities = 3, kFactors = 1;
    static constexpr bool kExtra = false;
    const StepConsts& C;
    const float4 xi;
    static __host__ __device__ constexpr int factor_of(int) { return 0; }
    __device__ __forceinline__ bool eval(const float4& xj, const float4&, float* v, float* f) const {
        float rx, ry, rz, lambda_sum;
        const float r_sq = rel_sq<true>(xi, xj, rx, ry, rz, &lambda_sum);
        if (!(r_sq < C.cut && lambda_sum != 0.0f)) return false;
        float s_corr = 0.0f;
        if (lambda_sum < -1e-10f && C.scorr_on) {
            float ratio = poly6(r_sq, C) / C.w_dq;
            ratio = (1.0f < ratio) ? 1.0f : ratio;
            float rp = ratio * ratio;
            if (C.corr_n4) rp = rp * rp;
            s_corr = C.neg_corr_k * rp;
        }
        const float c = spiky_coeff(r_sq, C);
        f[0] = (lambda_sum + s_corr) * C.mass;
        v[0] = c * rx;
        v[1] = c * ry;
        v[2] = c * rz;
        return true;
    }
#if !PBF_FAST
    __device__ __forceinline__ void products(const float4& xa, const float4& xb, const float4&,
                                             const float4&, float2* v, bool& in_a, bool& in_b) const {
        const PairRel r(xi, xa, xb, C.one);
        float2 lam = make_float2(xi.w + xa.w, xi.w + xb.w);
        in_a = r.r2.x < C.cut && lam.x != 0.0f;
        in_b = r.r2.y < C.cut && lam.y != 0.0f;
        if (C.scorr_on) {
            float2 ratio = quotient(poly6_2(r.r2, C), both(C.w_dq), both(C.inv_w_dq));
            ratio.x = (1.0f < ratio.x) ? 1.0f : ratio.x;
            ratio.y = (1.0f < ratio.y) ? 1.0f : ratio.y;
            float2 rp = mul2(ratio, ratio);
            if (C.corr_n4) rp = mul2(rp, rp);
            const float2 s = mul2(both(C.neg_corr_k), rp);
            lam.x = lam.x + (lam.x < -1e-10f ? s.x : 0.0f);
            lam.y = lam.y + (lam.y < -1e-10f ? s.y : 0.0f);
        }
        const float2 a = mul2(lam, both(C.mass));
        const float2 c = spiky_coeff_2(r.r2, C);
        v[0] = mul2(a, mul2(c, r.x));
        v[1] = mul2(a, mul2(c, r.y));
        v[2] = mul2(a, mul2(c, r.z));
    }
#endif
};

// The boundary's share of the position correction (two-way coupling):
// lambda_i (rho0 psi_b) grad W.
struct BoundaryDeltaTerm {
    static constexpr int kQuantities = 3, kFactors = 1;
    static constexpr bool kExtra = false;
    const StepConsts& C;
    const float4 xi;
    static __host__ __device__ constexpr int factor_of(int) { return 0; }
    __device__ __forceinline__ bool eval(const float4& b, const float4&, float* v, float* f) const {
        const float rx = xi.x - b.x, ry = xi.y - b.y, rz = xi.z - b.z;
        const float r_sq = sqn(rx, ry, rz);
        if (!(r_sq < C.cut)) return false;
        const float c = spiky_coeff(r_sq, C);
        f[0] = xi.w * (C.rho0 * b.w);
        v[0] = c * rx;
        v[1] = c * ry;
        v[2] = c * rz;
        return true;
    }
#if !PBF_FAST
    __device__ __forceinline__ void products(const float4& xa, const float4& xb, const float4&,
                                             const float4&, float2* v, bool& in_a, bool& in_b) const {
        const PairRel r(xi, xa, xb, C.one);
        in_a = r.r2.x < C.cut;
        in_b = r.r2.y < C.cut;
        const float2 c = spiky_coeff_2(r.r2, C);
        const float2 a = mul2(both(xi.w), mul2(both(C.rho0), make_float2(xa.w, xb.w)));
        v[0] = mul2(a, mul2(c, r.x));
        v[1] = mul2(a, mul2(c, r.y));
        v[2] = mul2(a, mul2(c, r.z));
    }
#endif
};

// apply_xsph_viscosity (pbf_solver.cpp:225-250).
struct XsphTerm {
    static constexpr int kQuantities = 3, kFactors = 1;
    static constexpr bool kExtra = true;
    const StepConsts& C;
    const float4 xi, vi;
    const float4* __restrict__ sv;
    static __host__ __device__ constexpr int factor_of(int) { return 0; }
    __device__ __forceinline__ float4 extra(uint32_t q) const { return __ldg(sv + q); }
    __device__ __forceinline__ bool eval(const float4& xj, const float4& vj, float* v, float* f) const {
        float rx, ry, rz;
        const float r_sq = rel_sq(xi, xj, rx, ry, rz);
        if (!(r_sq < C.h2)) return false;
        f[0] = poly6(r_sq, C);
        v[0] = vj.w * (vj.x - vi.x);
        v[1] = vj.w * (vj.y - vi.y);
        v[2] = vj.w * (vj.z - vi.z);
        return true;
    }
#if !PBF_FAST
    __device__ __forceinline__ void products(const float4& xa, const float4& xb, const float4& va,
                                             const float4& vb, float2* v, bool& in_a, bool& in_b) const {
        const PairRel r(xi, xa, xb, C.one);
        in_a = r.r2.x < C.h2;
        in_b = r.r2.y < C.h2;
        const float2 w = poly6_2(r.r2, C), m = make_float2(va.w, vb.w);
        v[0] = mul2(mul2(m, make_float2(va.x - vi.x, vb.x - vi.x)), w);
        v[1] = mul2(mul2(m, make_float2(va.y - vi.y, vb.y - vi.y)), w);
        v[2] = mul2(mul2(m, make_float2(va.z - vi.z, vb.z - vi.z)), w);
    }
#endif
};

// XSPH and the SPH curl of the velocities in one pass (Macklin & Mueller
// 2013, section 5, with its volume factor):
//   omega_i = sum_j (m/rho_j') spiky_grad(x*_i - x*_j) x (v_j - v_i).
struct XsphOmegaTerm {
    static constexpr int kQuantities = 6, kFactors = 2;
    static constexpr bool kExtra = true;
    const StepConsts& C;
    const float4 xi, vi;
    const float4* __restrict__ sv;
    static __host__ __device__ constexpr int factor_of(int k) { return k < 3 ? 0 : 1; }
    __device__ __forceinline__ float4 extra(uint32_t q) const { return __ldg(sv + q); }
    __device__ __forceinline__ bool eval(const float4& xj, const float4& vj, float* v, float* f) const {
        float rx, ry, rz;
        const float r_sq = rel_sq(xi, xj, rx, ry, rz);
        if (!(r_sq < C.cut)) return false;
        const float ux = vj.x - vi.x;
        const float uy = vj.y - vi.y;
        const float uz = vj.z - vi.z;
        f[0] = poly6(r_sq, C);
        v[0] = vj.w * ux;
        v[1] = vj.w * uy;
        v[2] = vj.w * uz;
        const float c = spiky_coeff(r_sq, C);
        const float gx = c * rx, gy = c * ry, gz = c * rz;
        f[1] = vj.w;
        v[3] = gy * uz - gz * uy;
        v[4] = gz * ux - gx * uz;
        v[5] = gx * uy - gy * ux;
        return true;
    }
#if !PBF_FAST
    __device__ __forceinline__ void products(const float4& xa, const float4& xb, const float4& va,
                                             const float4& vb, float2* v, bool& in_a, bool& in_b) const {
        const PairRel r(xi, xa, xb, C.one);
        in_a = r.r2.x < C.cut;
        in_b = r.r2.y < C.cut;
        const float2 m = make_float2(va.w, vb.w);
        const float2 ux = make_float2(va.x - vi.x, vb.x - vi.x);
        const float2 uy = make_float2(va.y - vi.y, vb.y - vi.y);
        const float2 uz = make_float2(va.z - vi.z, vb.z - vi.z);
        const float2 w = poly6_2(r.r2, C);
        v[0] = mul2(mul2(m, ux), w);
        v[1] = mul2(mul2(m, uy), w);
        v[2] = mul2(mul2(m, uz), w);
        const float2 c = spiky_coeff_2(r.r2, C);
        const float2 gx = mul2(c, r.x), gy = mul2(c, r.y), gz = mul2(c, r.z);
        // a b - c d with both products rounded: (-c d) + a b, the negation exact.
        auto cross = [&](float2 p, float2 q, float2 s, float2 t) {
            return pbf::add2(mul2(p, q), mul2(mul2(s, both(-1.0f)), t), C.one);
        };
        v[3] = mul2(m, cross(gy, uz, gz, uy));
        v[4] = mul2(m, cross(gz, ux, gx, uz));
        v[5] = mul2(m, cross(gx, uy, gy, ux));
    }
#endif
};

// The gradient of |omega| (vorticity confinement):
//   eta_i = sum_j (m/rho_j') (|omega_j| - |omega_i|) spiky_grad(x*_i - x*_j).
// The extras are (m / rho_j', |omega_j|) of the candidate.
struct VorticityTerm {
    static constexpr int kQuantities = 3, kFactors = 1;
    static constexpr bool kExtra = true;
    const StepConsts& C;
    const float4 xi;
    const float wi;
    const float4* __restrict__ sv;
    const float4* __restrict__ som;
    static __host__ __device__ constexpr int factor_of(int) { return 0; }
    __device__ __forceinline__ float4 extra(uint32_t q) const {
        return make_float4(__ldg(&sv[q].w), __ldg(&som[q].w), 0.0f, 0.0f);
    }
    __device__ __forceinline__ bool eval(const float4& xj, const float4& e, float* v, float* f) const {
        float rx, ry, rz;
        const float r_sq = rel_sq(xi, xj, rx, ry, rz);
        if (!(r_sq < C.cut)) return false;
        const float c = spiky_coeff(r_sq, C);
        f[0] = e.x * (e.y - wi);
        v[0] = c * rx;
        v[1] = c * ry;
        v[2] = c * rz;
        return true;
    }
#if !PBF_FAST
    __device__ __forceinline__ void products(const float4& xa, const float4& xb, const float4& ea,
                                             const float4& eb, float2* v, bool& in_a, bool& in_b) const {
        const PairRel r(xi, xa, xb, C.one);
        in_a = r.r2.x < C.cut;
        in_b = r.r2.y < C.cut;
        const float2 c = spiky_coeff_2(r.r2, C);
        const float2 a = mul2(make_float2(ea.x, eb.x), make_float2(ea.y - wi, eb.y - wi));
        v[0] = mul2(a, mul2(c, r.x));
        v[1] = mul2(a, mul2(c, r.y));
        v[2] = mul2(a, mul2(c, r.z));
    }
#endif
};

// ---------------------------------------------------------------------------
// The passes.  A pass's kernel comes in two forms, over warps of 32 particles
// and over teams of TP; both find the same sums and share what follows them.

// The sums over the fluid's candidates of every lane that wants: the warp
// walk, or lane by lane where the warp's particles are scattered.
template <bool kPersist, bool kLam, class P, class Sums>
__device__ __forceinline__ void sum_candidates(WalkSmem& sm, const Grid& G, const P& prm, uint32_t p,
                                               const int4 cell, bool want, const float4 xi,
                                               const float4* xin, const StepConsts& C, Sums& sums) {
    constexpr bool kRuns = std::is_same<P, OneScene>::value;
    uint32_t kept = 0u;
    if (warp_walk<kPersist, kLam, kRuns, false>(sm, G, fluid_index(G), prm, p, cell, want, xi, xin, kept,
        sums))
        return;
    if (!want) return;
    for_each_candidate_runs<kRuns>(
        cell, G, C,
        [&](uint32_t q) {
            float4 e{};
            if constexpr (Sums::kExtra) e = sums.extra(q);
            sums.add(ld_step<kPersist>(xin + q), e);
        },
        [&](uint32_t q, uint32_t L) {
            float4 e{};
            if constexpr (Sums::kExtra) e = sums.extra(q);
            sums.add_run(ld_step<kPersist>(xin + q), e, L);
        });
}

// The same sums of a warp from the lanes' kept lists of `cnt` candidates (of
// lanes that want).  kLam: in a warp whose lambdas are all zero, pairs of candidates
// whose lambdas are zero too are passed over (see walk_group).
template <bool kLam, class Sums>
__device__ __forceinline__ void read_lists(const Grid& G, uint32_t p, bool want, uint32_t cnt,
                                           const float4 xi, const float4* __restrict__ xin, Sums& sums) {
    const unsigned full = 0xffffffffu;
    if (!want) cnt = 0u;
    const uint32_t most = __reduce_max_sync(full, cnt);
    const bool all_zero = kLam && !__any_sync(full, want && xi.w != 0.0f);
    const uint2* from = G.lists + list_at(p);
    float4 xa = xi, xb = xi, ea = make_float4(0.0f, 0.0f, 0.0f, 0.0f), eb = ea;
    uint2 q = make_uint2(p, p);
    auto load = [&]() {
        xa = __ldg(xin + q.x);
        xb = __ldg(xin + q.y);
        if constexpr (Sums::kExtra) {
            ea = sums.extra(q.x);
            eb = sums.extra(q.y);
        }
    };
    if (cnt > 0u) {
        q = __ldcs(from);
        load();
    }
    if (cnt > 2u) q = __ldcs(from + 32);
    from += 64;
    for (uint32_t t = 0; t < most; t += 2u) {
        const float4 x0 = xa, x1 = xb, e0 = ea, e1 = eb;
        if (t + 2u < cnt) load();
        if (t + 4u < cnt) q = __ldcs(from);
        // Lists come from HBM once they outgrow the L2: four rows ahead the
        // loads found them there (a density pass of 250,000 waited for them
        // nine cycles in eleven; 1M step 4,230 -> 3,974 us; 8 and 16 rows
        // ahead 3,987 and 4,013).
        if (t + 12u < cnt) asm volatile("prefetch.global.L2 [%0];" ::"l"(from + 128));
        from += 32;
        if (all_zero && !__any_sync(full, t < cnt && (x0.w != 0.0f || x1.w != 0.0f))) continue;
        sums.add2(x0, x1, e0, e1, t < cnt, t + 1u < cnt);
    }
}

// Candidates of the kept list of a particle that wants (kNoList: no list), 0
// where it does not.
__device__ __forceinline__ uint32_t list_rows(const Grid& G, uint32_t p, bool want) {
    return want ? G.listed[p] & kNoList : 0u;
}

// The same over the boundary of a two-way coupled step; `cell` is the
// particle's cell in the fluid's grid.
template <class P, class Sums>
__device__ __forceinline__ void sum_boundary(WalkSmem& sm, const Grid& G, const P& prm, uint32_t p,
                                             const int4 cell, bool want, const float4 xi,
                                             const StepConsts& C, Sums& sums) {
    const int4 bc = boundary_cell(G, p, cell);
    uint32_t kept = 0u;
    if (warp_walk<false, false, false, false>(sm, G, boundary_index(G), prm, p, bc, want, xi, G.bg.spos, kept,
                                              sums))
        return;
    if (!want) return;
    for_each_candidate(bc, boundary_index(G), C,
                       [&](uint32_t q) { sums.add(__ldg(G.bg.spos + q), float4{}); });
}

// A thread of a team: its particle in the listing (pl; the same in all four
// warps) and in the evaluation (pe), and whether it writes pe's results.
template <int TP>
struct TeamThread {
    uint32_t pl, pe;
    bool al, ae, writer;
    __device__ __forceinline__ explicit TeamThread(int n) {
        const uint32_t first = blockIdx.x * (uint32_t)TP;
        pl = first + (threadIdx.x & 31u) / (32u / TP);
        pe = first + threadIdx.x / (128u / TP);
        al = pl < (uint32_t)n;
        ae = pe < (uint32_t)n;
        writer = ae && threadIdx.x % (128u / TP) == 0u;
        if (!al) pl = 0u;
        if (!ae) pe = 0u;
    }
    // Hands a flag of the listing's particles to the evaluation's threads.
    __device__ __forceinline__ bool hand_over(TeamSmem<TP>& sm, bool v) const {
        __syncthreads();
        if (threadIdx.x < 32u && threadIdx.x % (32u / TP) == 0u) sm.flag[threadIdx.x / (32u / TP)] = v;
        __syncthreads();
        return sm.flag[threadIdx.x / (128u / TP)] != 0;
    }
};

// The team's sums, keeping the lists (where there is room for any) of the
// evaluation's particles that want (elive).
template <int TP, class P, class Sums>
__device__ __forceinline__ void team_keeping(TeamSmem<TP>& sm, const Grid& G, const P& prm,
                                             const TeamThread<TP>& T, bool want, bool ewant, const float4 xl,
                                             const float4* __restrict__ xin, Sums& sums) {
    const int4 cell = cell_at(G, T.pl);
    if (G.lists) {
        uint32_t kept = 0u;
        team_walk_keep<TP, false, true>(sm, G, fluid_index(G), prm, T.pl, cell, want, xl, xin, T.pe, kept, sums);
        if (ewant && T.writer) G.listed[T.pe] = kept;
    } else {
        team_walk<TP, false>(sm, G, fluid_index(G), prm, T.pl, cell, want, xl, xin, sums);
    }
}

// The team's sums from the kept lists, where every particle that wants has
// one; the warps then need nothing from each other.
template <int TP, bool kLam, class P, class Sums>
__device__ __forceinline__ void team_listed(TeamSmem<TP>& sm, const Grid& G, const P& prm,
                                            const TeamThread<TP>& T, bool want, bool ewant, const float4 xl,
                                            const float4* __restrict__ xin, Sums& sums) {
    constexpr int S = 128 / TP;
    const unsigned full = 0xffffffffu;
    if (G.lists) {
        const int rows = ewant ? (int)G.listed[T.pe] : 0;
        if (!__syncthreads_or(rows == (int)kNoList)) {
            const int s = threadIdx.x & (S - 1);
            const int most = (int)__reduce_max_sync(full, (unsigned)rows);
            const uint2* const from = G.lists + (size_t)T.pe * kListRows;
            float2* const buf = reinterpret_cast<float2*>(sm.warp[threadIdx.x >> 5]);
            float4 xa = make_float4(0.0f, 0.0f, 0.0f, 0.0f), xb = xa, ea = xa, eb = xa;
            uint2 q = make_uint2(0u, 0u);
            auto load = [&]() {
                xa = __ldg(xin + q.x);
                xb = __ldg(xin + q.y);
                if constexpr (Sums::kExtra) {
                    ea = sums.extra(q.x);
                    eb = sums.extra(q.y);
                }
            };
            if (s < rows) {
                q = __ldcs(from + s);
                load();
            }
            if (s + S < rows) q = __ldcs(from + s + S);
            for (int r0 = 0; r0 < most; r0 += S) {
                const int r = r0 + s;
                const float4 x0 = xa, x1 = xb, e0 = ea, e1 = eb;
                if (r + S < rows) load();
                if (r + 2 * S < rows) q = __ldcs(from + r + 2 * S);
                sums.put(buf, x0, x1, e0, e1, r < rows, r < rows);
                __syncwarp();
                sums.fold(buf);
                __syncwarp();
            }
            return;
        }
    }
    team_walk<TP, kLam>(sm, G, fluid_index(G), prm, T.pl, cell_at(G, T.pl), want, xl, xin, sums);
}

// What the density pass writes for particle p and the rest of its run.
__device__ __forceinline__ void keep_lambda(uint32_t p, uint32_t rf, const int4 cell, const float4* xin,
                                            float4* xout, int it, const Grid& G, const StepConsts& C) {
    // Nothing around moved since the last density pass: keep its rho (srho)
    // and lambda (x*.w, which the delta pass carried through).
    const float4 keep = xin[p];
    xout[p] = keep;
    for (uint32_t m = p + 1, e = run_end(G, p, rf); m < e; ++m) xout[m] = keep;
    if (G.lamnz && keep.w != 0.0f) G.lamnz[slot_of(cell.x, cell.y, cell.z, C.grid)] = (uint32_t)it + 1u;
}

__device__ __forceinline__ void store_lambda(uint32_t p, uint32_t rf, const int4 cell, const float4 xi,
                                             float density, float Ci, float gix, float giy, float giz,
                                             float sum_grad_sq, float4* xout, float* __restrict__ srho,
                                             int it, const Grid& G, const StepConsts& C) {
    sum_grad_sq += sqn(gix, giy, giz);
    const float lam = (Ci < 0.0f) ? 0.0f : -Ci / (sum_grad_sq + C.eps);
    if (G.lamnz && lam != 0.0f) G.lamnz[slot_of(cell.x, cell.y, cell.z, C.grid)] = (uint32_t)it + 1u;
    srho[p] = density;
    xout[p] = make_float4(xi.x, xi.y, xi.z, lam);
    for (uint32_t m = p + 1, e = run_end(G, p, rf); m < e; ++m) {
        srho[m] = density;
        xout[m] = make_float4(xi.x, xi.y, xi.z, lam);
    }
}

// How a pass of a warp finds its sums: by walking; from kept lists; from kept
// lists and, over a two-way coupled step's boundary, by walking.
enum PassMode { kWalk, kListed, kListedTwoWay };

// The density pass for sorted particle p.  Reads x* from xin, writes
// (x*, lambda) to xout and rho to srho.  Scenes whose `iters` are done by
// iteration `it` are left untouched.  Warp-collective: every lane of the warp
// calls it, with `active` false past the last particle.
template <bool kPersist, PassMode kMode, class P>
__device__ __forceinline__ void density_lambda_at(uint32_t p, bool active, const float4* xin,
                                                  float4* xout, float* __restrict__ srho, int it,
                                                  const Grid& G, const P& prm, WalkSmem* sm) {
    const uint32_t pa = active ? p : 0u;
    const StepConsts& C = prm.at(G.spid, pa);
    const int4 cell = cell_at(G, pa);
    const uint32_t rf = run_flags(G, pa);
    bool live = active && it < C.iters && !(rf & kCopyBit);
    uint32_t rows = 0u;
    if constexpr (kMode != kWalk) {
        // k_list has kept lambda where nothing around moved.
        const uint32_t word = live ? G.listed[pa] : 0u;
        if (word & kIdle) live = false;
        rows = live ? word : 0u;
        if (__reduce_max_sync(0xffffffffu, rows) == kNoList) return;
    } else if (live && it > 0 && G.moved && cell.w == 0 &&
               !neighbourhood_stamped<kPersist>(cell, C.grid, G.moved, (uint32_t)it, 0, 3)) {
        keep_lambda(p, rf, cell, xin, xout, it, G, C);
        live = false;
    }
    if (!__any_sync(0xffffffffu, live)) return;
    const float4 xi = xin[pa];
    auto sum = [&](bool want, auto& sums) {
        if constexpr (kMode != kWalk) read_lists<false>(G, pa, want, rows, xi, xin, sums);
        else sum_candidates<kPersist, false>(*sm, G, prm, pa, cell, want, xi, xin, C, sums);
    };
    float density, gix = 0.0f, giy = 0.0f, giz = 0.0f, sum_grad_sq = 0.0f;
    // Density first: when C_i < 0 lambda_i is 0 whatever the gradient sums,
    // so a warp can sum the densities alone (poly6 terms, no square root or
    // division), then walk again, in the same candidate order, for the
    // gradients of its lanes with C_i >= 0 only.  Each sum sees the same
    // terms in the same order as the single walk: same bits.  It pays where
    // most warps have no such lane; which way a warp goes follows the share
    // of warps that needed gradients in the same iteration of the last step.
    // Where there are lists, the warps that walk (in piles, or scattered) are
    // not like the others and follow their own share: with one share for all, a
    // corner pile of the 1M dam break walked twice (58 ms a pass instead of 25).
    constexpr bool kHist = std::is_same<P, OneScene>::value;
    uint32_t* const hist = G.dhist && kMode == kWalk && G.lists ? G.dhist + 4 * kWalkHist : G.dhist;
    bool dfirst = false;
    if constexpr (kHist) {
        if (hist && it < kWalkHist && !G.bg.spos) {
            const uint32_t need = __ldg(hist + it), ran = __ldg(hist + kWalkHist + it);
            dfirst = ran > 0 && 3u * need < ran;
        }
    }
    if (kHist && dfirst) {
        LaneSums<DensityTerm> ds(DensityTerm{C, xi});
        sum(live, ds);
        density = ds.get(0);
        const bool want = live && !(density * C.inv_rho0 - 1.0f < 0.0f);
        LaneSums<GradTerm> gs(GradTerm{C, xi});
        sum(want, gs);
        gix = gs.get(0);
        giy = gs.get(1);
        giz = gs.get(2);
        sum_grad_sq = gs.get(3);
    } else {
        LaneSums<DensityGradTerm> sums(DensityGradTerm{C, xi});
        sum(live, sums);
        density = sums.get(0);
        gix = sums.get(1);
        giy = sums.get(2);
        giz = sums.get(3);
        sum_grad_sq = sums.get(4);
    }
    if constexpr (kHist && kMode != kListed) {
        if (G.bg.spos) {
            // Two-way coupling: after the fluid terms, the boundary's in the
            // boundary index's bucket order.
            LaneSums<BoundaryDensityTerm> bsums(BoundaryDensityTerm{C, xi});
            const float from[4] = {density, gix, giy, giz};
            bsums.start(from);
            sum_boundary(*sm, G, prm, pa, cell, live, xi, C, bsums);
            density = bsums.get(0);
            gix = bsums.get(1);
            giy = bsums.get(2);
            giz = bsums.get(3);
        }
    }
    const float Ci = density * C.inv_rho0 - 1.0f;
    if constexpr (kHist) {
        if (hist && it < kWalkHist) {
            const bool need = __any_sync(0xffffffffu, live && !(Ci < 0.0f));
            if ((threadIdx.x & 31) == 0) {
                atomicAdd(hist + 3 * kWalkHist + it, 1u);
                if (need) atomicAdd(hist + 2 * kWalkHist + it, 1u);
            }
        }
    }
    if (live) store_lambda(p, rf, cell, xi, density, Ci, gix, giy, giz, sum_grad_sq, xout, srho, it, G, C);
}

// The passes' kernels for warps of 32 particles.  Each comes twice: walking,
// for scenes without kept lists and (rest) for the warps in which some particle
// has none; and _listed, for the other warps of scenes with lists.  The readers
// have neither a walk's registers nor its shared memory, so more warps are in
// flight and the whole L1 holds candidates.
// Blocks of a walking launch for the rest, whose blocks go on to the next warps:
// four waves, so that one with nothing to do costs 5 us at any size and piles
// spread over the chip (ten steps of the 1M dam break into its corners, before a
// word held runs: 4.74 M particle-steps/s, 4.21 M with one wave, which saved 25
// us of a 1M step).
constexpr int kRestBlocks = 152 * 24;

// Whether the walking launch `rest` leaves this warp out.
__device__ __forceinline__ bool leave_out(int rest, const Grid& G, uint32_t p, bool want) {
    return rest && __reduce_max_sync(0xffffffffu, list_rows(G, p, want)) != kNoList;
}

// Lists the candidates of a pass for its listed kernels.  it >= 0: of Jacobi
// iteration it's density and delta pass (particles around which nothing moved
// keep their list and lambda).  it < 0: of the velocity passes; lists of
// particles around which the last delta pass moved nothing still hold.
template <int BS, class P>
__global__ void __launch_bounds__(BS, kListThreads / BS)
k_list(const float4* __restrict__ xin, float4* __restrict__ xout, int it, int n, const Grid G, const P prm) {
    __shared__ WalkSmem sm[BS / 32];
    constexpr bool kRuns = std::is_same<P, OneScene>::value;
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = p < (uint32_t)n;
    const uint32_t pa = active ? p : 0u;
    const uint32_t off = G.missing->off;  // (waited for with the loads that follow)
    const StepConsts& C = prm.at(G.spid, pa);
    const int4 cell = cell_at(G, pa);
    const uint32_t rf = run_flags(G, pa);
    bool live = active && !(rf & kCopyBit);
    if (off) {
        if (active) G.listed[p] = kNoList;
        if (threadIdx.x == 0) G.missing->any = 1u;
        return;
    }
    if (it >= 0) {
        live = live && it < C.iters;
        if (live && it > 0 && G.moved && cell.w == 0 &&
            !neighbourhood_stamped<false>(cell, C.grid, G.moved, (uint32_t)it, 0, 3)) {
            keep_lambda(p, rf, cell, xin, xout, it, G, C);
            G.listed[p] |= kIdle;
            live = false;
        }
    } else {
        live = live && (C.vort_on || C.xsph_on);
        if (live && C.iters > 0 && G.moved && cell.w == 0 &&
            !neighbourhood_stamped<false>(cell, C.grid, G.moved, (uint32_t)C.iters, 0, 3))
            live = false;
    }
    if (!__any_sync(0xffffffffu, live)) return;
    uint32_t kept = 0u;
    NoSums none;
    if (!warp_walk<false, false, kRuns, true>(sm[threadIdx.x >> 5], G, fluid_index(G), prm, pa, cell, live,
                                              xin[pa], xin, kept, none))
        kept = kNoList;
    if (live) G.listed[p] = kept;
    if (live && kept == kNoList) G.missing->any = 1u;
}

template <int BS, class P>
__global__ void __launch_bounds__(BS, kPassMinBlocks<BS>)
k_density_lambda(const float4* __restrict__ xin, float4* __restrict__ xout, float* __restrict__ srho,
                 int it, int n, int rest, const Grid G, const P prm) {
    __shared__ WalkSmem sm[BS / 32];
    if (rest && G.missing->any == 0u) return;
    for (uint32_t b = blockIdx.x; b * BS < (uint32_t)n; b += gridDim.x) {
        const uint32_t p = b * BS + threadIdx.x;
        const uint32_t pa = p < (uint32_t)n ? p : 0u;
        const bool out = leave_out(rest, G, pa, p < (uint32_t)n && it < prm.at(G.spid, pa).iters &&
                                                    !(run_flags(G, pa) & kCopyBit) &&
                                                    !(rest && (G.listed[pa] & kIdle)));
        if (rest && (p & (32u * kListSample - 1u)) == 0u) {
            atomicAdd(&G.missing->tried, 1u);
            if (!out) atomicAdd(&G.missing->failed, 1u);
        }
        if (!out)
            density_lambda_at<false, kWalk>(p, p < (uint32_t)n, xin, xout, srho, it, G, prm,
                                            &sm[threadIdx.x >> 5]);
    }
}

template <int BS, PassMode kMode, class P>
__global__ void __launch_bounds__(BS, kReadThreads<P> / BS)
k_density_lambda_listed(const float4* __restrict__ xin, float4* __restrict__ xout, float* __restrict__ srho,
                        int it, int n, const Grid G, const P prm) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    WalkSmem* sm = nullptr;
    if constexpr (kMode == kListedTwoWay) {
        __shared__ WalkSmem walk[BS / 32];
        sm = &walk[threadIdx.x >> 5];
    }
    density_lambda_at<false, kMode>(p, p < (uint32_t)n, xin, xout, srho, it, G, prm, sm);
}

template <int TP, class P>
__global__ void __launch_bounds__(128, kTeamMinBlocks<TP>)
k_density_lambda_team(const float4* __restrict__ xin, float4* __restrict__ xout,
                      float* __restrict__ srho, int it, int n, const Grid G, const P prm) {
    __shared__ TeamSmem<TP> sm;
    const TeamThread<TP> T(n);
    const int4 cell = cell_at(G, T.pl);
    bool live;
    {
        const StepConsts& C = prm.at(G.spid, T.pl);
        live = T.al && it < C.iters;
        if (it > 0 && G.moved) {
            const bool ask = live && cell.w == 0;
            const bool near = team_stamped(sm, ask, cell, C.grid, G.moved, (uint32_t)it);
            if (ask && !near) {
                if (threadIdx.x < 32u && threadIdx.x % (32u / TP) == 0u)
                    keep_lambda(T.pl, 0u, cell, xin, xout, it, G, C);
                live = false;
            }
        }
    }
    if (!__any_sync(0xffffffffu, live)) return;
    const bool elive = T.hand_over(sm, live);
    const StepConsts& C = prm.at(G.spid, T.pe);
    const float4 xl = xin[T.pl], xi = xin[T.pe];
    TeamSums<DensityGradTerm, 128 / TP> sums(DensityGradTerm{C, xi});
    team_keeping<TP>(sm, G, prm, T, live, elive, xl, xin, sums);
    float density = sums.get(0), gix = sums.get(1), giy = sums.get(2), giz = sums.get(3);
    const float sum_grad_sq = sums.get(4);
    if constexpr (std::is_same<P, OneScene>::value) {
        if (G.bg.spos) {
            TeamSums<BoundaryDensityTerm, 128 / TP> bsums(BoundaryDensityTerm{C, xi});
            const float from[4] = {density, gix, giy, giz};
            bsums.start(from);
            team_walk<TP, false>(sm, G, boundary_index(G), prm, T.pl, boundary_cell(G, T.pl, cell), live, xl,
                                 G.bg.spos, bsums);
            density = bsums.get(0);
            gix = bsums.get(1);
            giy = bsums.get(2);
            giz = bsums.get(3);
        }
    }
    if (elive && T.writer)
        store_lambda(T.pe, 0u, cell_at(G, T.pe), xi, density, density * C.inv_rho0 - 1.0f, gix, giy, giz,
                     sum_grad_sq, xout, srho, it, G, C);
}

// Velocity update with speed clamp (pbf_solver.cpp:81-93) for sorted p; w is
// the XSPH weight m / rho' (pbf_solver.cpp:240-241).
__device__ __forceinline__ float4 update_velocity(float px, float py, float pz, const float4 x0,
                                                  float rho, const StepConsts& C) {
    float a = (px - x0.x) * C.inv_dt;
    float b = (py - x0.y) * C.inv_dt;
    float c = (pz - x0.z) * C.inv_dt;
    const float speed_sq = sqn(a, b, c);
    if (speed_sq > C.max_speed_sq) {
        const float s = C.max_speed / sqrtf(speed_sq);
        a *= s;
        b *= s;
        c *= s;
    }
    const float rho_j = (rho > 1e-6f) ? rho : C.rho0;
    return make_float4(a, b, c, C.mass / rho_j);
}

// What the delta pass writes for particle p and the rest of its run: (x* + dp,
// lambda) and, on the scene's last iteration, the updated velocity.
__device__ __forceinline__ void store_delta(uint32_t p, uint32_t rf, const int4 cell, const float4 xi, float dx,
                                            float dy, float dz, float4* xout, const float4* __restrict__ sx,
                                            const float* __restrict__ srho, float4* __restrict__ sv, int it,
                                            const Grid& G, const StepConsts& C) {
    const float px = xi.x + dx * C.inv_rho0;
    const float py = xi.y + dy * C.inv_rho0;
    const float pz = xi.z + dz * C.inv_rho0;
    xout[p] = make_float4(px, py, pz, xi.w);
    if (G.moved && (__float_as_uint(px) != __float_as_uint(xi.x) ||
                    __float_as_uint(py) != __float_as_uint(xi.y) ||
                    __float_as_uint(pz) != __float_as_uint(xi.z)))
        G.moved[slot_of(cell.x, cell.y, cell.z, C.grid)] = (uint32_t)it + 1u;
    float4 vu = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (it == C.iters - 1) sv[p] = vu = update_velocity(px, py, pz, sx[p], srho[p], C);
    for (uint32_t m = p + 1, e = run_end(G, p, rf); m < e; ++m) {
        xout[m] = make_float4(px, py, pz, xi.w);
        if (it == C.iters - 1) sv[m] = vu;
    }
}

// compute_delta_position + apply_delta (pbf_solver.cpp:181-223, :74-76) for
// sorted particle p.  Reads (x*, lambda) from xin, writes (x* + dp, lambda_i)
// to xout; on the scene's last iteration also the updated velocity into sv.
// Warp-collective like density_lambda_at.
template <bool kPersist, PassMode kMode, class P>
__device__ __forceinline__ void delta_at(uint32_t p, bool active, const float4* xin, float4* xout,
                                         const float4* __restrict__ sx,
                                         const float* __restrict__ srho, float4* __restrict__ sv,
                                         int it, const Grid& G, const P& prm, WalkSmem* sm) {
    const uint32_t pa = active ? p : 0u;
    const StepConsts& C = prm.at(G.spid, pa);
    const int4 cell = cell_at(G, pa);
    const uint32_t rf = run_flags(G, pa);
    const bool live = active && it < C.iters && !(rf & kCopyBit);
    uint32_t rows = 0u;
    if constexpr (kMode != kWalk) {
        rows = list_rows(G, pa, live);
        if (__reduce_max_sync(0xffffffffu, rows) == kNoList) return;
    }
    float4 xi = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (live) xi = xin[p];
    bool walk = live;
    // A clean particle with a zero lambda whose 27 cells hold no nonzero
    // lambda in this iteration has only zero terms: no walk.
    if (live && G.lamnz && cell.w == 0 && xi.w == 0.0f &&
        !neighbourhood_stamped<kPersist>(cell, C.grid, G.lamnz, (uint32_t)it + 1u, 0, 3))
        walk = false;
    LaneSums<DeltaTerm> sums(DeltaTerm{C, xi});
    if constexpr (kMode != kWalk) read_lists<true>(G, pa, walk, rows, xi, xin, sums);
    else sum_candidates<kPersist, true>(*sm, G, prm, pa, cell, walk, xi, xin, C, sums);
    float dx = sums.get(0), dy = sums.get(1), dz = sums.get(2);
    if constexpr (std::is_same<P, OneScene>::value && kMode != kListed) {
        if (G.bg.spos) {
            // Two-way coupling: the boundary's share after the fluid terms
            // (zero when lambda_i is).
            LaneSums<BoundaryDeltaTerm> bsums(BoundaryDeltaTerm{C, xi});
            const float from[3] = {dx, dy, dz};
            bsums.start(from);
            sum_boundary(*sm, G, prm, pa, cell, live && xi.w != 0.0f, xi, C, bsums);
            dx = bsums.get(0);
            dy = bsums.get(1);
            dz = bsums.get(2);
        }
    }
    if (live) store_delta(p, rf, cell, xi, dx, dy, dz, xout, sx, srho, sv, it, G, C);
}

template <int BS, class P>
__global__ void __launch_bounds__(BS, kPassMinBlocks<BS>)
k_delta(const float4* __restrict__ xin, float4* __restrict__ xout, const float4* __restrict__ sx,
        const float* __restrict__ srho, float4* __restrict__ sv, int it, int n, int rest, const Grid G,
        const P prm) {
    __shared__ WalkSmem sm[BS / 32];
    if (rest && G.missing->any == 0u) return;
    for (uint32_t b = blockIdx.x; b * BS < (uint32_t)n; b += gridDim.x) {
        const uint32_t p = b * BS + threadIdx.x;
        const uint32_t pa = p < (uint32_t)n ? p : 0u;
        if (!leave_out(rest, G, pa, p < (uint32_t)n && it < prm.at(G.spid, pa).iters &&
                                           !(run_flags(G, pa) & kCopyBit)))
            delta_at<false, kWalk>(p, p < (uint32_t)n, xin, xout, sx, srho, sv, it, G, prm,
                                   &sm[threadIdx.x >> 5]);
    }
}

template <int BS, PassMode kMode, class P>
__global__ void __launch_bounds__(BS, kReadThreads<P> / BS)
k_delta_listed(const float4* __restrict__ xin, float4* __restrict__ xout, const float4* __restrict__ sx,
               const float* __restrict__ srho, float4* __restrict__ sv, int it, int n, const Grid G,
               const P prm) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    WalkSmem* sm = nullptr;
    if constexpr (kMode == kListedTwoWay) {
        __shared__ WalkSmem walk[BS / 32];
        sm = &walk[threadIdx.x >> 5];
    }
    delta_at<false, kMode>(p, p < (uint32_t)n, xin, xout, sx, srho, sv, it, G, prm, sm);
}

template <int TP, class P>
__global__ void __launch_bounds__(128, kTeamMinBlocks<TP>)
k_delta_team(const float4* __restrict__ xin, float4* __restrict__ xout, const float4* __restrict__ sx,
             const float* __restrict__ srho, float4* __restrict__ sv, int it, int n, const Grid G,
             const P prm) {
    __shared__ TeamSmem<TP> sm;
    const TeamThread<TP> T(n);
    const int4 cell = cell_at(G, T.pl);
    const float4 xl = xin[T.pl], xi = xin[T.pe];
    bool live, walk, ewalk;
    {
        const StepConsts& C = prm.at(G.spid, T.pl);
        live = walk = T.al && it < C.iters;
        if (G.lamnz) {
            const bool ask = live && cell.w == 0 && xl.w == 0.0f;
            const bool near = team_stamped(sm, ask, cell, C.grid, G.lamnz, (uint32_t)it + 1u);
            if (ask && !near) walk = false;
        }
    }
    const StepConsts& C = prm.at(G.spid, T.pe);
    // The evaluation's particle: team_stamped left the answers in the flags.
    ewalk = T.ae && it < C.iters &&
            !(G.lamnz && cell_at(G, T.pe).w == 0 && xi.w == 0.0f && !sm.flag[threadIdx.x / (128u / TP)]);
    TeamSums<DeltaTerm, 128 / TP> sums(DeltaTerm{C, xi});
    __syncthreads();
    team_listed<TP, true>(sm, G, prm, T, walk, ewalk, xl, xin, sums);
    float dx = sums.get(0), dy = sums.get(1), dz = sums.get(2);
    if constexpr (std::is_same<P, OneScene>::value) {
        if (G.bg.spos) {
            TeamSums<BoundaryDeltaTerm, 128 / TP> bsums(BoundaryDeltaTerm{C, xi});
            const float from[3] = {dx, dy, dz};
            bsums.start(from);
            team_walk<TP, false>(sm, G, boundary_index(G), prm, T.pl, boundary_cell(G, T.pl, cell),
                                 live && xl.w != 0.0f, xl, G.bg.spos, bsums);
            dx = bsums.get(0);
            dy = bsums.get(1);
            dz = bsums.get(2);
        }
    }
    if (T.writer && it < C.iters)
        store_delta(T.pe, 0u, cell_at(G, T.pe), xi, dx, dy, dz, xout, sx, srho, sv, it, G, C);
}

// ---------------------------------------------------------------------------
// Persistent Jacobi loop: all iterations of a step in one cooperative launch.
// Every thread keeps the same particles (grid stride) in both passes, and the
// grid meets at a barrier after each pass.

// Grid barrier for a cooperative launch (all blocks resident).  `count` must
// be 0 when the launch starts.  Every wait is bounded: after kBarrierSpins
// polls or kBarrierNs of global time a block records bit 4 in *err and the
// loop returns, so a barrier that cannot complete ends the launch instead of
// hanging it.
struct GridSync {
    unsigned int* count;
    unsigned int* gen;
    uint32_t* err;
};

constexpr uint32_t kBarrierSpins = 1u << 24;
constexpr unsigned long long kBarrierNs = 10ull * 1000 * 1000 * 1000;

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ bool grid_sync(const GridSync& S) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = 1;
        const unsigned int g = *(volatile unsigned int*)S.gen;
        __threadfence();  // this block's writes before its arrival
        if (atomicAdd(S.count, 1u) == gridDim.x - 1u) {
            atomicExch(S.count, 0u);
            __threadfence();
            atomicAdd(S.gen, 1u);
        } else {
            const unsigned long long t0 = global_ns();
            for (uint32_t k = 0; *(volatile unsigned int*)S.gen == g; ++k) {
                if (k > kBarrierSpins || global_ns() - t0 > kBarrierNs) {
                    atomicOr(S.err, 4u);
                    ok = 0;
                    break;
                }
                __nanosleep(128);
            }
        }
        __threadfence();  // the other blocks' writes before this block's reads
    }
    __syncthreads();
    return ok != 0;
}

template <class P>
__global__ void __launch_bounds__(kBlock, kPassMinBlocks<kBlock>)
k_iterate(float4* xa, float4* xb, float* __restrict__ srho, const float4* __restrict__ sx,
          float4* __restrict__ sv, int max_iters, int n, const Grid G, const P prm,
          const GridSync S) {
    __shared__ WalkSmem sm[kBlock / 32];
    const uint32_t stride = gridDim.x * blockDim.x;
    // The warp strides as a whole, so that its lanes meet in every
    // warp-collective pass call.
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t w0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u);
    auto& my = sm[threadIdx.x >> 5];
    for (int it = 0; it < max_iters; ++it) {
        for (uint32_t pw = w0; pw < (uint32_t)n; pw += stride)
            density_lambda_at<true, kWalk>(pw + lane, pw + lane < (uint32_t)n, xa, xb, srho, it, G, prm, &my);
        if (!grid_sync(S)) return;
        for (uint32_t pw = w0; pw < (uint32_t)n; pw += stride)
            delta_at<true, kWalk>(pw + lane, pw + lane < (uint32_t)n, xb, xa, sx, srho, sv, it, G, prm, &my);
        if (it + 1 < max_iters && !grid_sync(S)) return;
    }
}

// Velocity update alone, for scenes with solver_iterations == 0.
template <int BS, class P>
__global__ void __launch_bounds__(BS)
k_velocity(const float4* __restrict__ xin, const float4* __restrict__ sx, const float* __restrict__ srho,
           float4* __restrict__ sv, int n, const Grid G, const P prm) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (uint32_t)n) return;
    const StepConsts& C = prm.at(G.spid, p);
    if (C.iters > 0) return;
    const float4 xi = xin[p];
    sv[p] = update_velocity(xi.x, xi.y, xi.z, sx[p], srho[p], C);
}

// Domain clamp + commit (pbf_solver.cpp:102-126), scattered to particle order.
__device__ __forceinline__ void commit(uint32_t p, float px, float py, float pz, float vx, float vy,
                                       float vz, float lam, const float4* __restrict__ sx,
                                       const float* __restrict__ srho, const StateRef& R, int n,
                                       const StepConsts& C) {
    if (C.clamp) {
        if (px < C.lo[0]) { px = C.lo[0]; vx = 0.0f; } else if (px > C.hi[0]) { px = C.hi[0]; vx = 0.0f; }
        if (py < C.lo[1]) { py = C.lo[1]; vy = 0.0f; } else if (py > C.hi[1]) { py = C.hi[1]; vy = 0.0f; }
        if (pz < C.lo[2]) { pz = C.lo[2]; vz = 0.0f; } else if (pz > C.hi[2]) { pz = C.hi[2]; vz = 0.0f; }
    }
    uint32_t i = __float_as_uint(sx[p].w);
    if (i >= (uint32_t)n) i = 0;
    const uint32_t l = i - R.first;
    if (R.bad && !(isfinite(px) && isfinite(py) && isfinite(pz) && isfinite(vx) && isfinite(vy) &&
                   isfinite(vz)))
        atomicOr(R.bad, 1u);
    R.x[l] = make_float4(px, py, pz, 0.0f);
    R.v[l] = make_float4(vx, vy, vz, 0.0f);
    R.rho[l] = srho[p];
    R.lam[l] = lam;
}

// Boundary friction of two-way steps (StepConsts::bfric), one thread per
// cell-sorted particle after the velocity update and before XSPH:
//   v_i += bfric * sum_b psi_b (v_b - v_i) W(x*_i - x_b),
// an XSPH term against the surface velocity v_b = v_k + w_k x (x_b - p_k) of
// boundary particle b's body k (zero for world-owned particles), over the
// boundary buckets of the particle's cell.  Each thread reads and writes only
// its own velocity.
__global__ void __launch_bounds__(kBlock)
k_boundary_friction(const float4* __restrict__ xin, float4* __restrict__ sv, int n, const Grid G,
                    const StepConsts C) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (uint32_t)n) return;
    const float4 xi = xin[p];
    const float4 vi = sv[p];
    float fx = 0.0f, fy = 0.0f, fz = 0.0f;
    for_each_candidate(boundary_cell(G, p, cell_at(G, p)), boundary_index(G), C, [&](uint32_t q) {
                              const float4 b = __ldg(G.bg.spos + q);
                              const float rx = xi.x - b.x, ry = xi.y - b.y, rz = xi.z - b.z;
                              const float r_sq = sqn(rx, ry, rz);
                              if (r_sq >= C.h2) return;
                              const int k = __ldg(G.bg.body + __ldg(G.bg.sidx + q));
                              float ux = 0.0f, uy = 0.0f, uz = 0.0f;
                              if (k >= 0 && k < G.bg.nbodies) {
                                  const float4 c = __ldg(G.bg.body_pos + k);
                                  const float4 l = __ldg(G.bg.body_lin + k);
                                  const float4 a = __ldg(G.bg.body_ang + k);
                                  const float dx = b.x - c.x, dy = b.y - c.y, dz = b.z - c.z;
                                  ux = l.x + (a.y * dz - a.z * dy);
                                  uy = l.y + (a.z * dx - a.x * dz);
                                  uz = l.z + (a.x * dy - a.y * dx);
                              }
                              const float w = b.w * poly6(r_sq, C);
                              fx += (ux - vi.x) * w;
                              fy += (uy - vi.y) * w;
                              fz += (uz - vi.z) * w;
                          });
    sv[p] = make_float4(vi.x + C.bfric * fx, vi.y + C.bfric * fy, vi.z + C.bfric * fz, vi.w);
}

// apply_xsph_viscosity (pbf_solver.cpp:225-250) + commit, no vorticity.
// With skip_vort set, scenes with vorticity are left to the vorticity pair.
template <class P>
__device__ __forceinline__ void store_xsph(uint32_t p, uint32_t rf, const float4 xi, const float4 vi, float cx,
                                           float cy, float cz, const float4* __restrict__ sx,
                                           const float* __restrict__ srho, int n, const Grid& G, const P& prm,
                                           const StepConsts& C) {
    float vx = vi.x, vy = vi.y, vz = vi.z;
    if (C.xsph_on) {
        vx = vi.x + C.xsph_c * cx;
        vy = vi.y + C.xsph_c * cy;
        vz = vi.z + C.xsph_c * cz;
    }
    for (uint32_t m = p, e = run_end(G, p, rf); m < e; ++m)
        commit(m, xi.x, xi.y, xi.z, vx, vy, vz, xi.w, sx, srho, prm.state(G.spid, m), n, C);
}

template <PassMode kMode, class P>
__device__ __forceinline__ void xsph_commit_at(uint32_t p, const float4* __restrict__ xin,
                                               const float4* __restrict__ sv, const float4* __restrict__ sx,
                                               const float* __restrict__ srho, int n, int skip_vort,
                                               const Grid& G, const P& prm, WalkSmem* sm) {
    const bool active = p < (uint32_t)n;
    const uint32_t pa = active ? p : 0u;
    const StepConsts& C = prm.at(G.spid, pa);
    const uint32_t rf = run_flags(G, pa);
    const bool live = active && !(skip_vort && C.vort_on) && !(rf & kCopyBit);
    const bool want = live && C.xsph_on;
    uint32_t rows = 0u;
    if constexpr (kMode != kWalk) {
        rows = list_rows(G, pa, want);
        if (__reduce_max_sync(0xffffffffu, rows) == kNoList) return;
    }
    const float4 xi = xin[pa];
    const float4 vi = sv[pa];
    LaneSums<XsphTerm> sums(XsphTerm{C, xi, vi, sv});
    if constexpr (kMode != kWalk) read_lists<false>(G, pa, want, rows, xi, xin, sums);
    else sum_candidates<false, false>(*sm, G, prm, pa, cell_at(G, pa), want, xi, xin, C, sums);
    if (live) store_xsph(p, rf, xi, vi, sums.get(0), sums.get(1), sums.get(2), sx, srho, n, G, prm, C);
}

template <int BS, class P>
__global__ void __launch_bounds__(BS, kPassMinBlocks<BS>)
k_xsph_commit(const float4* __restrict__ xin, const float4* __restrict__ sv, const float4* __restrict__ sx,
              const float* __restrict__ srho, int n, int skip_vort, int rest, const Grid G, const P prm) {
    __shared__ WalkSmem sm[BS / 32];
    if (rest && G.missing->any == 0u) return;
    for (uint32_t b = blockIdx.x; b * BS < (uint32_t)n; b += gridDim.x) {
        const uint32_t p = b * BS + threadIdx.x;
        const uint32_t pa = p < (uint32_t)n ? p : 0u;
        const StepConsts& C = prm.at(G.spid, pa);
        const bool live = p < (uint32_t)n && !(skip_vort && C.vort_on) && !(run_flags(G, pa) & kCopyBit);
        if (!leave_out(rest, G, pa, live && C.xsph_on)) xsph_commit_at<kWalk>(p, xin, sv, sx, srho, n,
            skip_vort, G, prm, &sm[threadIdx.x >> 5]);
    }
}

template <int BS, class P>
__global__ void __launch_bounds__(BS, kReadThreads<P> / BS)
k_xsph_commit_listed(const float4* __restrict__ xin, const float4* __restrict__ sv,
                     const float4* __restrict__ sx, const float* __restrict__ srho, int n, int skip_vort,
                     const Grid G, const P prm) {
    xsph_commit_at<kListed>(blockIdx.x * blockDim.x + threadIdx.x, xin, sv, sx, srho, n, skip_vort, G, prm,
                            nullptr);
}

template <int TP, class P>
__global__ void __launch_bounds__(128, kTeamMinBlocks<TP>)
k_xsph_commit_team(const float4* __restrict__ xin, const float4* __restrict__ sv,
                   const float4* __restrict__ sx, const float* __restrict__ srho, int n, int skip_vort,
                   const Grid G, const P prm) {
    __shared__ TeamSmem<TP> sm;
    const TeamThread<TP> T(n);
    bool want;
    {
        const StepConsts& C = prm.at(G.spid, T.pl);
        want = T.al && !(skip_vort && C.vort_on) && C.xsph_on;
    }
    const StepConsts& C = prm.at(G.spid, T.pe);
    const float4 xi = xin[T.pe];
    const float4 vi = sv[T.pe];
    TeamSums<XsphTerm, 128 / TP> sums(XsphTerm{C, xi, vi, sv});
    team_walk<TP, false>(sm, G, fluid_index(G), prm, T.pl, cell_at(G, T.pl), want, xin[T.pl], xin, sums);
    const float cx = sums.get(0), cy = sums.get(1), cz = sums.get(2);
    if (T.writer && !(skip_vort && C.vort_on))
        store_xsph(T.pe, 0u, xi, vi, cx, cy, cz, sx, srho, n, G, prm, C);
}

// XSPH correction + vorticity omega in one candidate pass (vorticity path).
// Writes the post-XSPH velocity to sv2 and (omega, |omega|) to som.
__device__ __forceinline__ void store_omega(uint32_t p, uint32_t rf, const float4 vi, float cx, float cy,
                                            float cz, float wx, float wy, float wz, float4* __restrict__ sv2,
                                            float4* __restrict__ som, const Grid& G, const StepConsts& C) {
    float vx = vi.x, vy = vi.y, vz = vi.z;
    if (C.xsph_on) {
        vx = vi.x + C.xsph_c * cx;
        vy = vi.y + C.xsph_c * cy;
        vz = vi.z + C.xsph_c * cz;
    }
    const float4 o = make_float4(wx, wy, wz, sqrtf(sqn(wx, wy, wz)));
    for (uint32_t m = p, e = run_end(G, p, rf); m < e; ++m) {
        sv2[m] = make_float4(vx, vy, vz, 0.0f);
        som[m] = o;
    }
}

template <PassMode kMode, class P>
__device__ __forceinline__ void xsph_omega_at(uint32_t p, const float4* __restrict__ xin,
                                              const float4* __restrict__ sv, float4* __restrict__ sv2,
                                              float4* __restrict__ som, int n, const Grid& G, const P& prm,
                                              WalkSmem* sm) {
    const bool active = p < (uint32_t)n;
    const uint32_t pa = active ? p : 0u;
    const StepConsts& C = prm.at(G.spid, pa);
    const uint32_t rf = run_flags(G, pa);
    const bool live = active && C.vort_on && !(rf & kCopyBit);
    const bool want = live;
    uint32_t rows = 0u;
    if constexpr (kMode != kWalk) {
        rows = list_rows(G, pa, want);
        if (__reduce_max_sync(0xffffffffu, rows) == kNoList) return;
    }
    const float4 xi = xin[pa];
    const float4 vi = sv[pa];
    LaneSums<XsphOmegaTerm> sums(XsphOmegaTerm{C, xi, vi, sv});
    if constexpr (kMode != kWalk) read_lists<false>(G, pa, want, rows, xi, xin, sums);
    else sum_candidates<false, false>(*sm, G, prm, pa, cell_at(G, pa), want, xi, xin, C, sums);
    if (live)
        store_omega(p, rf, vi, sums.get(0), sums.get(1), sums.get(2), sums.get(3), sums.get(4), sums.get(5),
                    sv2, som, G, C);
}

template <int BS, class P>
__global__ void __launch_bounds__(BS, kPassMinBlocks<BS>)
k_xsph_omega(const float4* __restrict__ xin, const float4* __restrict__ sv, float4* __restrict__ sv2,
             float4* __restrict__ som, int n, int rest, const Grid G, const P prm) {
    __shared__ WalkSmem sm[BS / 32];
    if (rest && G.missing->any == 0u) return;
    for (uint32_t b = blockIdx.x; b * BS < (uint32_t)n; b += gridDim.x) {
        const uint32_t p = b * BS + threadIdx.x;
        const uint32_t pa = p < (uint32_t)n ? p : 0u;
        const StepConsts& C = prm.at(G.spid, pa);
        const bool live = p < (uint32_t)n && C.vort_on && !(run_flags(G, pa) & kCopyBit);
        if (!leave_out(rest, G, pa, live)) xsph_omega_at<kWalk>(p, xin, sv, sv2, som, n, G, prm,
            &sm[threadIdx.x >> 5]);
    }
}

template <int BS, class P>
__global__ void __launch_bounds__(BS, kReadThreads<P> / BS)
k_xsph_omega_listed(const float4* __restrict__ xin, const float4* __restrict__ sv, float4* __restrict__ sv2,
                    float4* __restrict__ som, int n, const Grid G, const P prm) {
    xsph_omega_at<kListed>(blockIdx.x * blockDim.x + threadIdx.x, xin, sv, sv2, som, n, G, prm, nullptr);
}

template <int TP, class P>
__global__ void __launch_bounds__(128, kTeamMinBlocks<TP>)
k_xsph_omega_team(const float4* __restrict__ xin, const float4* __restrict__ sv, float4* __restrict__ sv2,
                  float4* __restrict__ som, int n, const Grid G, const P prm) {
    __shared__ TeamSmem<TP> sm;
    const TeamThread<TP> T(n);
    const bool want = T.al && prm.at(G.spid, T.pl).vort_on;
    const StepConsts& C = prm.at(G.spid, T.pe);
    const float4 xi = xin[T.pe];
    const float4 vi = sv[T.pe];
    TeamSums<XsphOmegaTerm, 128 / TP> sums(XsphOmegaTerm{C, xi, vi, sv});
    team_keeping<TP>(sm, G, prm, T, want, T.ae && C.vort_on, xin[T.pl], xin, sums);
    const float cx = sums.get(0), cy = sums.get(1), cz = sums.get(2);
    const float wx = sums.get(3), wy = sums.get(4), wz = sums.get(5);
    if (T.writer && C.vort_on) store_omega(T.pe, 0u, vi, cx, cy, cz, wx, wy, wz, sv2, som, G, C);
}

// Vorticity confinement (Macklin & Mueller 2013, section 5) + commit:
//   N = eta / |eta|,  v += dt * eps * (N x omega_i).
template <class P>
__device__ __forceinline__ void store_vorticity(uint32_t p, uint32_t rf, const float4 xi, float ex, float ey,
                                                float ez, const float4* __restrict__ sv2,
                                                const float4* __restrict__ som, const float4* __restrict__ sx,
                                                const float* __restrict__ srho, int n, const Grid& G,
                                                const P& prm, const StepConsts& C) {
    const float4 wi = som[p];
    const float el = sqrtf(sqn(ex, ey, ez));
    float nx = 0.0f, ny = 0.0f, nz = 0.0f;
    if (el > 1e-9f) {
        nx = ex / el;
        ny = ey / el;
        nz = ez / el;
    }
    const float fx = ny * wi.z - nz * wi.y;
    const float fy = nz * wi.x - nx * wi.z;
    const float fz = nx * wi.y - ny * wi.x;
    const float4 vb = sv2[p];
    const float vx = vb.x + C.vort_scale * fx;
    const float vy = vb.y + C.vort_scale * fy;
    const float vz = vb.z + C.vort_scale * fz;
    for (uint32_t m = p, e = run_end(G, p, rf); m < e; ++m)
        commit(m, xi.x, xi.y, xi.z, vx, vy, vz, xi.w, sx, srho, prm.state(G.spid, m), n, C);
}

template <PassMode kMode, class P>
__device__ __forceinline__ void vorticity_commit_at(uint32_t p, const float4* __restrict__ xin,
    const float4* __restrict__ sv, const float4* __restrict__ sv2, const float4* __restrict__ som,
    const float4* __restrict__ sx, const float* __restrict__ srho, int n, const Grid& G, const P& prm,
    WalkSmem* sm) {
    const bool active = p < (uint32_t)n;
    const uint32_t pa = active ? p : 0u;
    const StepConsts& C = prm.at(G.spid, pa);
    const uint32_t rf = run_flags(G, pa);
    const bool live = active && C.vort_on && !(rf & kCopyBit);
    const bool want = live;
    uint32_t rows = 0u;
    if constexpr (kMode != kWalk) {
        rows = list_rows(G, pa, want);
        if (__reduce_max_sync(0xffffffffu, rows) == kNoList) return;
    }
    const float4 xi = xin[pa];
    LaneSums<VorticityTerm> sums(VorticityTerm{C, xi, som[pa].w, sv, som});
    if constexpr (kMode != kWalk) read_lists<false>(G, pa, want, rows, xi, xin, sums);
    else sum_candidates<false, false>(*sm, G, prm, pa, cell_at(G, pa), want, xi, xin, C, sums);
    if (live)
        store_vorticity(p, rf, xi, sums.get(0), sums.get(1), sums.get(2), sv2, som, sx, srho, n, G, prm, C);
}

template <int BS, class P>
__global__ void __launch_bounds__(BS, kPassMinBlocks<BS>)
k_vorticity_commit(const float4* __restrict__ xin, const float4* __restrict__ sv,
                   const float4* __restrict__ sv2, const float4* __restrict__ som,
                   const float4* __restrict__ sx, const float* __restrict__ srho, int n, int rest,
                   const Grid G, const P prm) {
    __shared__ WalkSmem sm[BS / 32];
    if (rest && G.missing->any == 0u) return;
    for (uint32_t b = blockIdx.x; b * BS < (uint32_t)n; b += gridDim.x) {
        const uint32_t p = b * BS + threadIdx.x;
        const uint32_t pa = p < (uint32_t)n ? p : 0u;
        const StepConsts& C = prm.at(G.spid, pa);
        const bool live = p < (uint32_t)n && C.vort_on && !(run_flags(G, pa) & kCopyBit);
        if (!leave_out(rest, G, pa, live)) vorticity_commit_at<kWalk>(p, xin, sv, sv2, som, sx, srho, n, G,
            prm, &sm[threadIdx.x >> 5]);
    }
}

template <int BS, class P>
__global__ void __launch_bounds__(BS, kReadThreads<P> / BS)
k_vorticity_commit_listed(const float4* __restrict__ xin, const float4* __restrict__ sv,
                          const float4* __restrict__ sv2, const float4* __restrict__ som,
                          const float4* __restrict__ sx, const float* __restrict__ srho, int n,
                          const Grid G, const P prm) {
    vorticity_commit_at<kListed>(blockIdx.x * blockDim.x + threadIdx.x, xin, sv, sv2, som, sx, srho, n, G,
                                 prm, nullptr);
}

template <int TP, class P>
__global__ void __launch_bounds__(128, kTeamMinBlocks<TP>)
k_vorticity_commit_team(const float4* __restrict__ xin, const float4* __restrict__ sv,
                        const float4* __restrict__ sv2, const float4* __restrict__ som,
                        const float4* __restrict__ sx, const float* __restrict__ srho, int n, const Grid G,
                        const P prm) {
    __shared__ TeamSmem<TP> sm;
    const TeamThread<TP> T(n);
    const bool want = T.al && prm.at(G.spid, T.pl).vort_on;
    const StepConsts& C = prm.at(G.spid, T.pe);
    const float4 xi = xin[T.pe];
    TeamSums<VorticityTerm, 128 / TP> sums(VorticityTerm{C, xi, som[T.pe].w, sv, som});
    team_listed<TP, false>(sm, G, prm, T, want, T.ae && C.vort_on, xin[T.pl], xin, sums);
    const float ex = sums.get(0), ey = sums.get(1), ez = sums.get(2);
    if (T.writer && C.vort_on)
        store_vorticity(T.pe, 0u, xi, ex, ey, ez, sv2, som, sx, srho, n, G, prm, C);
}

// ---------------------------------------------------------------------------
// Parity probes: cell coordinates and in-radius neighbour lists of x*.

__global__ void __launch_bounds__(kBlock)
k_debug_cells(const float4* __restrict__ x, const float4* __restrict__ v, int* __restrict__ cells3,
              const StepConsts C) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= C.n) return;
    float px, py, pz;
    predict(x[i], v[i], C, px, py, pz);
    int cx, cy, cz;
    cell_of(px, py, pz, C.inv_cell, cx, cy, cz);
    cells3[3 * i] = cx;
    cells3[3 * i + 1] = cy;
    cells3[3 * i + 2] = cz;
}

// fill == 0: cnt[i] = number of in-radius candidates j != i of particle i;
// fill == 1: write them (particle indices, candidate order) at out[offs[i]..].
__global__ void __launch_bounds__(kBlock)
k_debug_neighbors(const float4* __restrict__ xin, const float4* __restrict__ sx,
                  long long* __restrict__ cnt, const long long* __restrict__ offs,
                  int* __restrict__ out, long long cap, int fill, const Grid G,
                  const StepConsts C) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (uint32_t)C.n) return;
    const float4 xi = xin[p];
    const uint32_t i = __float_as_uint(sx[p].w);
    long long k = fill ? offs[i] : 0;
    for_each_candidate(cell_at(G, p), G.ix, C, [&](uint32_t q) {
        if (q == p) return;
        const float4 xj = xin[q];
        if (sqn(xi.x - xj.x, xi.y - xj.y, xi.z - xj.z) < C.h2) {
            if (fill && k < cap) out[k] = (int)__float_as_uint(sx[q].w);
            ++k;
        }
    });
    if (!fill) cnt[i] = k;
}

// ---------------------------------------------------------------------------
// Host-side launchers on `stream`.

inline int grid_of(int n, int b) { return (n + b - 1) / b; }

inline Grid grid_view(const StepBuffers& B, int n, const uint32_t* spid = nullptr,
                      const BoundaryGrid& bg = BoundaryGrid{}) {
    return Grid{B.scell, B.sown, WalkIndex{(uint32_t)n, B.off, B.bkt.merged, B.bkt.end, B.btab}, spid,
                B.moved, B.lamnz, bg, spid ? nullptr : B.dhist, nullptr, B.slot_alias,
                n <= B.list_cap ? B.lists : nullptr, B.listed, B.missing};
}

// predict, sort by cell, cell offsets and gather, reference buckets,
// classification: the neighbour structure of one scene's step.
inline cudaError_t enqueue_prefix(const StepBuffers& B, const StepConsts& C, SortScratch& sort,
                                  cudaStream_t st, PhaseMarks* pm = nullptr) {
    const int n = C.n;
    const int nb = grid_of(n, kBlock);
    const OneScene one{C, StateRef{B.x, B.v, B.rho, B.lam, 0u, nullptr}};
    const SceneIds none{nullptr, nullptr};
    if (pm) pm->mark(-1, 0, st);
    const int bits = C.grid.key_bits;
    cudaError_t e = clear_ranges(slot_clear(B), sort_clear(sort, n, bits),
                                 C.hash_compat ? bucket_clear(B.bkt, n) : ClearRange{}, st);
    if (e != cudaSuccess) return e;
    k_predict_key<OneScene><<<count_blocks(n), kCountThreads, 0, st>>>(B.keys, B.dhist, B.missing, n,
        sort_counts(sort, n, bits), none, one);
    if (pm) pm->mark(kPhasePredict, 2, st);
    e = radix_sort_counted(B.keys, B.skeys, B.sidx, n, bits, sort, st);
    if (e != cudaSuccess) return e;
    if (pm) pm->mark(kPhaseGridBuild, n <= kSmallSort ? 1 : sort_passes(bits), st);
    k_gather<OneScene><<<nb + grid_of((int)C.grid.nslots + 1, kBlock), kBlock, 0, st>>>(B.sidx, B.sx, B.xa,
        B.srho, B.scell, B.bkt.link, B.slot_alias, B.err, n, SlotOffsets{B.skeys, B.off, C.grid.nslots, nb},
        none, one);
    if (C.hash_compat) {
        e = enqueue_buckets(sized_for(B.bkt, n), B.scell, B.sidx, nullptr, B.off, B.slot_alias, n, one, st);
        if (e != cudaSuccess) return e;
        k_classify<OneScene><<<nb, kBlock, 0, st>>>(B.scell, n, B.scell, nullptr, sized_for(B.bkt, n),
            B.slot_alias, B.btab, B.sown, nullptr, one);
    } else {
        e = cudaMemsetAsync(B.sown, 0, (size_t)n * 4, st);
        if (e != cudaSuccess) return e;
    }
    if (pm) pm->mark(kPhaseNeighborQuery, C.hash_compat ? 5 : 1, st);
    return cudaGetLastError();
}

// Particles per team of the neighbour passes, 0 for warps with one lane per
// particle, by the number of particles of the launch.  Warps need some 130,000
// particles to keep the chip's 608 schedulers in work; below that their time
// is that of one warp's chain.  Measured when both forms walked in every pass
// (us a call, teams of 8 / 16 / 32 / warps): 1,000 particles at h = 2 r 193 /
// 238 / 341 / 604; 8,000 at 4 r 365 / 368 / 464 / 992; a batch of 352,901 5,171
// / 3,993 / 4,061 / 3,519.  Teams of 32 were never the fastest and are not built.
// With kept lists (teams of 16 / warps), one step of a lattice at 4 r: 32,768
// particles 446 / 666, 64,000 774 / 766, 97,336 1,066 / 944, 132,651 1,518 /
// 1,239, 216,000 2,324 / 1,543; coupled, 250,000 4,075 / 2,895.  The line lies
// above the lattice's, because fluid in motion scatters: of four steps of 43,993
// particles (3,349 / 12,403) the first two take warps 0.9 ms each, and in the
// others a few warps over scattered cells, which keep no lists, walk for 0.3 to
// 0.7 ms in every pass; 65,565 in the fast build 1,671 / 2,503.
inline int team_size(int n) {
    if (n < 8192) return 8;
    if (n < kBigScene) return 16;
    return 0;
}

// TP: particles per team, 0 for warps of 32 particles in blocks of BS threads.
template <int BS, int TP, class P>
inline cudaError_t enqueue_passes_bs(const StepBuffers& B, Grid G, int n, int max_iters,
                                     bool any_zero_iters, bool any_vort, bool any_plain,
                                     bool xsph_on, const P prm, cudaStream_t st, PhaseMarks* pm,
                                     int persist_blocks, unsigned int* barrier) {
    constexpr int T = TP ? TP : 32;
    const int nb = TP ? grid_of(n, T) : grid_of(n, BS);
    // With kept lists a warp pass lists, reads the lists and walks for the rest.
    const auto rest = [&] { return G.lists ? 1 : 0; };
    const auto walk_blocks = [&] { return G.lists && nb > kRestBlocks ? kRestBlocks : nb; };
    const auto list = [&](const float4* xin, float4* xout, int it) {
        if (G.lists) k_list<BS, P><<<nb, BS, 0, st>>>(xin, xout, it, n, G, prm);
    };
    if (persist_blocks > 0 && barrier && max_iters > 0) {
        // The whole Jacobi loop as one cooperative launch, which keeps no lists.
        G.lists = nullptr;
        cudaError_t e = cudaMemsetAsync(barrier, 0, sizeof(unsigned int), st);
        if (e != cudaSuccess) return e;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)persist_blocks);
        cfg.blockDim = dim3(kBlock);
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, k_iterate<P>, B.xa, B.xb, B.srho,
                               static_cast<const float4*>(B.sx), B.sv, max_iters, n, G, prm,
                               GridSync{barrier, barrier + 1, B.err});
        if (e != cudaSuccess) return e;
        if (pm) pm->mark(kPhaseDensity, 1, st);
    } else {
        for (int it = 0; it < max_iters; ++it) {
            if constexpr (TP != 0)
                k_density_lambda_team<T, P><<<nb, 128, 0, st>>>(B.xa, B.xb, B.srho, it, n, G, prm);
            else {
                list(B.xa, B.xb, it);
                if (G.lists) {
                    if (G.bg.spos) {
                        if constexpr (std::is_same<P, OneScene>::value)
                            k_density_lambda_listed<BS, kListedTwoWay, P><<<nb, BS, 0, st>>>(B.xa, B.xb,
                                B.srho, it, n, G, prm);
                    } else {
                        k_density_lambda_listed<BS, kListed, P><<<nb, BS, 0, st>>>(B.xa, B.xb, B.srho, it,
                            n, G, prm);
                    }
                }
                k_density_lambda<BS, P><<<walk_blocks(), BS, 0, st>>>(B.xa, B.xb, B.srho, it, n, rest(),
                    G, prm);
            }
            if (pm) pm->mark(kPhaseDensity, TP == 0 && G.lists ? 3 : 1, st);
            if constexpr (TP != 0)
                k_delta_team<T, P><<<nb, 128, 0, st>>>(B.xb, B.xa, B.sx, B.srho, B.sv, it, n, G, prm);
            else {
                if (G.lists) {
                    if (G.bg.spos) {
                        if constexpr (std::is_same<P, OneScene>::value)
                            k_delta_listed<BS, kListedTwoWay, P><<<nb, BS, 0, st>>>(B.xb, B.xa, B.sx, B.srho,
                                B.sv, it, n, G, prm);
                    } else {
                        k_delta_listed<BS, kListed, P><<<nb, BS, 0, st>>>(B.xb, B.xa, B.sx, B.srho, B.sv,
                            it, n, G, prm);
                    }
                }
                k_delta<BS, P><<<walk_blocks(), BS, 0, st>>>(B.xb, B.xa, B.sx, B.srho, B.sv, it, n,
                    rest(), G, prm);
            }
            if (pm) pm->mark(kPhaseDelta, TP == 0 && G.lists ? 2 : 1, st);
        }
    }
    if (any_zero_iters) {
        k_velocity<BS, P><<<grid_of(n, BS), BS, 0, st>>>(B.xa, B.sx, B.srho, B.sv, n, G, prm);
        if (pm) pm->mark(kPhaseDelta, 1, st);
    }
    if constexpr (std::is_same<P, OneScene>::value) {
        if (G.bg.spos && prm.C.bfric != 0.0f) {
            k_boundary_friction<<<grid_of(n, BS), BS, 0, st>>>(B.xa, B.sv, n, G, prm.C);
            if (pm) pm->mark(kPhaseXsph, 1, st);
        }
    }
    if constexpr (TP == 0) {
        list(B.xa, nullptr, -1);
        if (pm && G.lists) pm->mark(kPhaseXsph, 1, st);
    }
    if (any_vort) {
        if constexpr (TP != 0)
            k_xsph_omega_team<T, P><<<nb, 128, 0, st>>>(B.xa, B.sv, B.sv2, B.som, n, G, prm);
        else {
            if (G.lists) k_xsph_omega_listed<BS, P><<<nb, BS, 0, st>>>(B.xa, B.sv, B.sv2, B.som, n, G, prm);
            k_xsph_omega<BS, P><<<walk_blocks(), BS, 0, st>>>(B.xa, B.sv, B.sv2, B.som, n, rest(), G, prm);
        }
        if (pm) pm->mark(kPhaseXsph, TP == 0 && G.lists ? 2 : 1, st);
        if constexpr (TP != 0)
            k_vorticity_commit_team<T, P><<<nb, 128, 0, st>>>(B.xa, B.sv, B.sv2, B.som, B.sx, B.srho, n, G, prm);
        else {
            if (G.lists)
                k_vorticity_commit_listed<BS, P><<<nb, BS, 0, st>>>(B.xa, B.sv, B.sv2, B.som, B.sx, B.srho,
                    n, G, prm);
            k_vorticity_commit<BS, P><<<walk_blocks(), BS, 0, st>>>(B.xa, B.sv, B.sv2, B.som, B.sx, B.srho, n,
                rest(), G, prm);
        }
        if (pm) pm->mark(kPhaseCommit, TP == 0 && G.lists ? 2 : 1, st);
    }
    if (any_plain) {
        const int skip = any_vort ? 1 : 0;
        if constexpr (TP != 0)
            k_xsph_commit_team<T, P><<<nb, 128, 0, st>>>(B.xa, B.sv, B.sx, B.srho, n, skip, G, prm);
        else {
            if (G.lists)
                k_xsph_commit_listed<BS, P><<<nb, BS, 0, st>>>(B.xa, B.sv, B.sx, B.srho, n, skip, G, prm);
            k_xsph_commit<BS, P><<<walk_blocks(), BS, 0, st>>>(B.xa, B.sv, B.sx, B.srho, n, skip, rest(),
                G, prm);
        }
        if (pm) pm->mark(xsph_on ? kPhaseXsph : kPhaseCommit, TP == 0 && G.lists ? 2 : 1, st);
    }
    return cudaGetLastError();
}

// The constraint, velocity, XSPH, vorticity and commit passes over n
// cell-sorted particles for `max_iters` iterations, with constants from `prm`.
// Scenes with vorticity take the XSPH+omega / vorticity+commit pair
// (any_vort), the others XSPH+commit (any_plain).  Batches (SceneTable) may
// pick the block size of the neighbour passes (64, 128 or 256 threads); a
// single scene always uses kBlock.
template <class P>
inline cudaError_t enqueue_passes(const StepBuffers& B, const Grid& G, int n, int max_iters,
                                  bool any_zero_iters, bool any_vort, bool any_plain, bool xsph_on,
                                  const P prm, cudaStream_t st, PhaseMarks* pm,
                                  int persist_blocks = 0, unsigned int* barrier = nullptr,
                                  int block = kBlock) {
    auto go = [&](auto bs, auto tp) {
        return enqueue_passes_bs<decltype(bs)::value, decltype(tp)::value>(
            B, G, n, max_iters, any_zero_iters, any_vort, any_plain, xsph_on, prm, st, pm,
            persist_blocks, barrier);
    };
    using std::integral_constant;
    const integral_constant<int, kBlock> bs;
    switch (team_size(n)) {
        case 8: return go(bs, integral_constant<int, 8>{});
        case 16: return go(bs, integral_constant<int, 16>{});
    }
    if constexpr (std::is_same<P, SceneTable>::value) {
        if (block == 64) return go(integral_constant<int, 64>{}, integral_constant<int, 0>{});
        if (block == 256) return go(integral_constant<int, 256>{}, integral_constant<int, 0>{});
    }
    return go(bs, integral_constant<int, 0>{});
}

inline cudaError_t enqueue_step(const StepBuffers& B, const StepConsts& C, int iters,
                                SortScratch& sort, cudaStream_t st, PhaseMarks* pm = nullptr,
                                const BoundaryGrid* bg = nullptr) {
    const int n = C.n;
    if (n <= 0) return cudaSuccess;
    cudaError_t e = enqueue_prefix(B, C, sort, st, pm);
    if (e != cudaSuccess) return e;
    StepConsts Ci = C;
    Ci.iters = iters;
    BoundaryGrid bgs = bg ? *bg : BoundaryGrid{};
    if (bg) bgs.sx = B.sx;
    Grid G = grid_view(B, n, nullptr, bgs);
    if (B.segend && n >= kBigScene) {
        // Runs of identical particles: from here on the owner words of the
        // run's later particles carry kCopyBit, which only the passes below
        // understand (they skip those particles).
        k_segments<<<grid_of(n, 256), 256, 0, st>>>(StepState{B.sx, B.xa, B.srho, n}, B.scell, C.grid, B.sown,
            B.slot_alias, B.segend);
        if (pm) pm->mark(kPhaseNeighborQuery, 1, st);
        G.segend = B.segend;
    }
    return enqueue_passes(B, G, n, iters, iters <= 0, C.vort_on != 0,
                          C.vort_on == 0,
                          C.xsph_on != 0, OneScene{Ci, StateRef{B.x, B.v, B.rho, B.lam, 0u, nullptr}}, st,
                          pm);
}

// ---------------------------------------------------------------------------
// Batches of independent scenes: one sort and one launch per phase for all.

// pid[i] = the scene whose particle range holds batch particle i.
__global__ void __launch_bounds__(256)
k_scene_ids(const uint32_t* __restrict__ firsts, int nscenes, uint32_t* __restrict__ pid, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int a = 0, b = nscenes - 1;  // last s with firsts[s] <= i
    while (a < b) {
        const int m = (a + b + 1) >> 1;
        if (__ldg(firsts + m) <= (uint32_t)i) a = m;
        else b = m - 1;
    }
    pid[i] = (uint32_t)a;
}

inline cudaError_t enqueue_batch_step(const StepBuffers& B, const BatchDesc& D, SortScratch& sort,
                                      cudaStream_t st, PhaseMarks* pm = nullptr) {
    const int n = D.n;
    if (n <= 0) return cudaSuccess;
    const int nb = grid_of(n, kBlock);
    const SceneTable tab{D.tab, D.refs};
    const SceneIds ids{D.pid, D.spid};
    if (pm) pm->mark(-1, 0, st);
    cudaError_t e = clear_ranges(slot_clear(B), sort_clear(sort, n, D.key_bits), bucket_clear(B.bkt, n), st);
    if (e != cudaSuccess) return e;
    k_scene_ids<<<grid_of(n, 256), 256, 0, st>>>(D.firsts, D.nscenes, D.pid, n);
    k_predict_key<SceneTable><<<count_blocks(n), kCountThreads, 0, st>>>(B.keys, nullptr, B.missing, n,
        sort_counts(sort, n, D.key_bits), ids, tab);
    if (pm) pm->mark(kPhasePredict, 3, st);
    // Cell order: scene-major because every scene owns a slot range.
    e = radix_sort_counted(B.keys, B.skeys, B.sidx, n, D.key_bits, sort, st);
    if (e != cudaSuccess) return e;
    if (pm) pm->mark(kPhaseGridBuild, n <= kSmallSort ? 1 : sort_passes(D.key_bits), st);
    k_gather<SceneTable><<<nb + grid_of((int)D.nslots + 1, kBlock), kBlock, 0, st>>>(B.sidx, B.sx, B.xa,
        B.srho, B.scell, B.bkt.link, B.slot_alias, B.err, n, SlotOffsets{B.skeys, B.off, D.nslots, nb}, ids,
        tab);
    e = enqueue_buckets(sized_for(B.bkt, n), B.scell, B.sidx, D.spid, B.off, B.slot_alias, n, tab, st);
    if (e != cudaSuccess) return e;
    k_classify<SceneTable><<<nb, kBlock, 0, st>>>(B.scell, n, B.scell, D.spid, sized_for(B.bkt, n),
        B.slot_alias, B.btab, B.sown, D.spid, tab);
    if (pm) pm->mark(kPhaseNeighborQuery, 5, st);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return enqueue_passes(B, grid_view(B, n, D.spid), n, D.max_iters, D.any_zero_iters, D.any_vort,
                          D.any_plain, D.xsph_on, tab, st, pm, D.persist_blocks, D.barrier,
                          D.block);
}

// Blocks of the persistent Jacobi loop that fit on the device at once.
inline int persist_blocks_max() {
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_iterate<SceneTable>, kBlock, 0) !=
        cudaSuccess)
        return 0;
    return sms * per_sm;
}

}  // namespace PBF_NS
}  // namespace pbf
