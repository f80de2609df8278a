// Akinci coupling kernels (see pbf_boundary.cuh).  Built with the exact
// arithmetic flags (-fmad=false, IEEE div/sqrt): every expression follows the
// reference's operation order (src/fluid/boundary.cpp, fluid_world.cpp).
#define PBF_FAST 0
#define PBF_NS bnd
#include "pbf_boundary.cuh"
#include "pbf_kernels.cuh"
#include "rigid_step.hpp"
#include "rigid_world.cuh"

namespace pbf {
namespace bnd {

// Cell slot of points (no prediction), with its digits counted.
__global__ void __launch_bounds__(kCountThreads)
k_ix_keys(const float4* __restrict__ pos, int n, uint32_t* __restrict__ keys, const SortCounts counts,
          const StepConsts C) {
    __shared__ BlockCounts B;
    B.begin(counts);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 p = pos[i];
        int cx, cy, cz;
        cell_of(p.x, p.y, p.z, C.inv_cell, cx, cy, cz);
        const uint32_t key = slot_of(cx, cy, cz, C.grid);
        keys[i] = key;
        B.count(counts, key);
    }
    B.end(counts);
}

__global__ void __launch_bounds__(kBlock)
k_ix_gather(const uint32_t* __restrict__ sidx, const float4* __restrict__ pos,
            const float* __restrict__ attr, int n, float4* __restrict__ spos,
            int4* __restrict__ scell, uint32_t* __restrict__ link,
            unsigned char* __restrict__ slot_alias, const SlotOffsets offsets, const StepConsts C) {
    if (offsets.block(n)) return;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    uint32_t i = sidx[p];
    if (i >= (uint32_t)n) i = 0;
    const float4 q = pos[i];
    int cx, cy, cz;
    cell_of(q.x, q.y, q.z, C.inv_cell, cx, cy, cz);
    spos[p] = make_float4(q.x, q.y, q.z, attr ? attr[i] : q.w);
    scell[p] = make_int4(cx, cy, cz, 0);
    link[p] = kNoBucket;
    if (!in_grid(cx, cy, cz, C.grid)) slot_alias[slot_of(cx, cy, cz, C.grid)] = kAliasSlot;
}

// Cells of the predicted positions of n particles.
__global__ void __launch_bounds__(kBlock)
k_predict_cells(const float4* __restrict__ x, const float4* __restrict__ v, int n,
                int4* __restrict__ cells, const StepConsts C) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float px, py, pz;
    predict(x[i], v[i], C, px, py, pz);
    int cx, cy, cz;
    cell_of(px, py, pz, C.inv_cell, cx, cy, cz);
    cells[i] = make_int4(cx, cy, cz, 0);
}

__device__ __forceinline__ WalkIndex index_of(const PointIndex& I, const QuerySet& Q) {
    return WalkIndex{(uint32_t)I.n, I.off, I.bkt.merged, I.bkt.end, Q.btab};
}

// The walks' view of queries against an index: no scenes, stamps or runs.
__device__ __forceinline__ Grid query_grid(const PointIndex& I, const QuerySet& Q) {
    return Grid{nullptr, nullptr, index_of(I, Q), nullptr, nullptr, nullptr, BoundaryGrid{}, nullptr, nullptr,
                nullptr};
}

__device__ __forceinline__ int4 query_cell(const QuerySet& Q, uint32_t i) {
    int4 c = Q.qcell[i];
    c.w = Q.qown[i];
    return c;
}

// (p + q * v) for unit quaternion q = (w, x, y, z), in the order of the
// quaternion-vector product t = 2 (q.vec x v); v + w t + q.vec x t.
__device__ __forceinline__ float3 transform_point(const float4 p, const float4 q, const float4 v) {
    float t0 = q.z * v.z - q.w * v.y;
    float t1 = q.w * v.x - q.y * v.z;
    float t2 = q.y * v.y - q.z * v.x;
    t0 = t0 + t0;
    t1 = t1 + t1;
    t2 = t2 + t2;
    const float c0 = q.z * t2 - q.w * t1;
    const float c1 = q.w * t0 - q.y * t2;
    const float c2 = q.y * t1 - q.z * t0;
    const float r0 = (v.x + q.x * t0) + c0;
    const float r1 = (v.y + q.x * t1) + c1;
    const float r2 = (v.z + q.x * t2) + c2;
    return make_float3(p.x + r0, p.y + r1, p.z + r2);
}

__global__ void __launch_bounds__(kBlock)
k_bxform(const float4* __restrict__ local, const int* __restrict__ body, int nb,
         const float4* __restrict__ body_pos, const float4* __restrict__ body_quat, int nbodies,
         float4* __restrict__ world) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    const float4 l = local[b];
    const int bi = body[b];
    if (bi >= 0 && bi < nbodies) {
        const float3 w = transform_point(body_pos[bi], body_quat[bi], l);
        world[b] = make_float4(w.x, w.y, w.z, l.w);
    } else {
        world[b] = l;
    }
}

// The coupling's sums run over cell-sorted queries (the fluid index's points
// against the boundary's, and the other way round), so that a team's 8 or 16
// queries sit in one cell or two; with one thread per query a few thousand
// boundary points left most of the chip idle for 600 us.
//
// As in the reference, a distance that is not a number is not outside the
// support, and a factor that is not finite spoils a sum through the zero
// kernel value of a candidate anywhere in the buckets: such candidates are
// listed wherever they are (kSpecials, special), and every candidate of such
// a query.

__device__ __forceinline__ bool finite3(const float4& x) {
    return isfinite(x.x) && isfinite(x.y) && isfinite(x.z);
}

// a, or not a number where r^2 is none.
__device__ __forceinline__ float2 nan_of(float2 r2, float2 a) {
    return make_float2(isnan(r2.x) ? r2.x : a.x, isnan(r2.y) ? r2.y : a.y);
}

// Density of the boundary at a fluid point: sum_b rho0 psi_b W.
struct PsiDensityTerm {
    static constexpr int kQuantities = 1, kFactors = 1;
    static constexpr bool kExtra = false;
    static constexpr bool kSpecials = true;
    const StepConsts& C;
    const float4 xi;
    static __host__ __device__ constexpr int factor_of(int) { return 0; }
    static __device__ __forceinline__ bool special(const float4& b, const StepConsts& C) {
        return !finite3(b) || !isfinite(C.rho0 * b.w);
    }
    __device__ __forceinline__ bool eval(const float4& b, const float4&, float* v, float* f) const {
        const float r_sq = sqn(xi.x - b.x, xi.y - b.y, xi.z - b.z);
        f[0] = C.rho0 * b.w;
        if (r_sq >= C.h2 && isfinite(f[0])) return false;
        v[0] = poly6(r_sq, C);
        return true;
    }
    __device__ __forceinline__ void products(const float4& xa, const float4& xb, const float4&, const float4&,
                                             float2* v, bool& in_a, bool& in_b) const {
        const PairRel r(xi, xa, xb, C.one);
        const float2 f = mul2(both(C.rho0), make_float2(xa.w, xb.w));
        in_a = !(r.r2.x >= C.h2) || !isfinite(f.x);
        in_b = !(r.r2.y >= C.h2) || !isfinite(f.y);
        v[0] = mul2(f, nan_of(r.r2, poly6_2(r.r2, C)));
    }
};

// Pressure force on a boundary point: sum_f (p_f rho0) psi_b grad W, with
// p_f rho0 in the fluid point's w (pressure_weight) and psi_b in xi.w.
struct PressureTerm {
    static constexpr int kQuantities = 3, kFactors = 1;
    static constexpr bool kExtra = false;
    static constexpr bool kSpecials = true;
    const StepConsts& C;
    const float4 xi;
    static __host__ __device__ constexpr int factor_of(int) { return 0; }
    static __device__ __forceinline__ bool special(const float4& xf, const StepConsts&) { return !finite3(xf); }
    __device__ __forceinline__ bool eval(const float4& xf, const float4&, float* v, float* f) const {
        const float rx = xi.x - xf.x, ry = xi.y - xf.y, rz = xi.z - xf.z;
        const float r_sq = sqn(rx, ry, rz);
        if (r_sq >= C.h2) return false;
        const float c = spiky_coeff(r_sq, C);
        f[0] = xf.w * xi.w;
        v[0] = c * rx;
        v[1] = c * ry;
        v[2] = c * rz;
        return true;
    }
    __device__ __forceinline__ void products(const float4& xa, const float4& xb, const float4&, const float4&,
                                             float2* v, bool& in_a, bool& in_b) const {
        const PairRel r(xi, xa, xb, C.one);
        in_a = !(r.r2.x >= C.h2);
        in_b = !(r.r2.y >= C.h2);
        const float2 c = nan_of(r.r2, spiky_coeff_2(r.r2, C));
        const float2 a = mul2(make_float2(xa.w, xb.w), both(xi.w));
        v[0] = mul2(a, mul2(c, r.x));
        v[1] = mul2(a, mul2(c, r.y));
        v[2] = mul2(a, mul2(c, r.z));
    }
};

// sum_b W over the boundary itself (Akinci volumes).
struct VolumeTerm {
    static constexpr int kQuantities = 1, kFactors = 1;
    static constexpr bool kExtra = false;
    static constexpr bool kSpecials = true;
    const StepConsts& C;
    const float4 xi;
    static __host__ __device__ constexpr int factor_of(int) { return -1; }
    static __device__ __forceinline__ bool special(const float4& b, const StepConsts&) { return !finite3(b); }
    __device__ __forceinline__ bool eval(const float4& b, const float4&, float* v, float* f) const {
        const float r_sq = sqn(xi.x - b.x, xi.y - b.y, xi.z - b.z);
        if (r_sq >= C.h2) return false;
        v[0] = poly6(r_sq, C);
        f[0] = 1.0f;
        return true;
    }
    __device__ __forceinline__ void products(const float4& xa, const float4& xb, const float4&, const float4&,
                                             float2* v, bool& in_a, bool& in_b) const {
        const PairRel r(xi, xa, xb, C.one);
        in_a = !(r.r2.x >= C.h2);
        in_b = !(r.r2.y >= C.h2);
        v[0] = nan_of(r.r2, poly6_2(r.r2, C));
    }
};

// pc rho0 of a fluid particle of density rho, as the reference's force loop
// computes it for each pair (fluid_world.cpp:147-155): zero where the fluid is
// not compressed, so such a particle adds exact zeros (where psi and the
// distance are finite) and is not listed.
__device__ __forceinline__ float pressure_weight(float rho, const StepConsts& C) {
    const float rho_f = (rho < 1.0f) ? 1.0f : rho;   // std::max(rho, 1.0f)
    const float pd = rho_f - C.rho0;
    const float pressure = (0.0f < pd) ? pd : 0.0f;  // std::max(0.0f, rho - rho0)
    const float pc = C.mass * pressure / (rho_f * rho_f);
    return pc * C.rho0;
}

// Boundary density of the fluid index's points: rho += sum, in particle order,
// and the points' w from the density to the pressure weight.
template <int TP>
__global__ void __launch_bounds__(128, kTeamMinBlocks<TP>)
k_boundary_density(float4* __restrict__ fpos, const uint32_t* __restrict__ fidx, int n, const QuerySet Q,
                   const PointIndex I, float* __restrict__ rho, const StepConsts C) {
    __shared__ TeamSmem<TP> sm;
    const TeamThread<TP> T(n);
    const Grid G = query_grid(I, Q);
    const float4 xi = fpos[T.pe];
    TeamSums<PsiDensityTerm, 128 / TP> sums(PsiDensityTerm{C, xi});
    team_walk<TP, false>(sm, G, G.ix, OneScene{C, StateRef{}}, T.pl, query_cell(Q, T.pl), T.al, fpos[T.pl], I.spos,
                         sums);
    const float bd = sums.get(0);
    if (T.writer) {
        const float r = xi.w + bd;
        const uint32_t i = fidx[T.pe];
        if (i < (uint32_t)n) rho[i] = r;
        fpos[T.pe].w = pressure_weight(r, C);
    }
}

// The same change of w where the densities already hold the boundary's share.
__global__ void __launch_bounds__(kBlock)
k_pressure_weights(float4* __restrict__ fpos, int n, const StepConsts C) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < n) fpos[p].w = pressure_weight(fpos[p].w, C);
}

// Force on each boundary point (bpos, bidx: the boundary index's points and
// their original numbers) from the fluid index I.
template <int TP>
__global__ void __launch_bounds__(128, kTeamMinBlocks<TP>)
k_coupling(const float4* __restrict__ bpos, const uint32_t* __restrict__ bidx, const int* __restrict__ body,
           const int* __restrict__ body_dynamic, int nb, int nbodies, const QuerySet Q, const PointIndex I,
           float4* __restrict__ Fb, const StepConsts C) {
    __shared__ TeamSmem<TP> sm;
    const TeamThread<TP> T(nb);
    const Grid G = query_grid(I, Q);
    auto feels = [&](uint32_t p) {
        const uint32_t b = bidx[p];
        const int bi = b < (uint32_t)nb ? body[b] : -1;
        return bi >= 0 && bi < nbodies && body_dynamic[bi];
    };
    const float4 xi = bpos[T.pe];
    float4 xl = bpos[T.pl];
    xl.w = isfinite(xl.w) ? 0.0f : 1.0f;  // 0: lists candidates with a nonzero weight only
    TeamSums<PressureTerm, 128 / TP> sums(PressureTerm{C, xi});
    team_walk<TP, true>(sm, G, G.ix, OneScene{C, StateRef{}}, T.pl, query_cell(Q, T.pl), T.al && feels(T.pl), xl,
                        I.spos, sums);
    const float fx = sums.get(0), fy = sums.get(1), fz = sums.get(2);
    if (T.writer) {
        const uint32_t b = bidx[T.pe];
        if (b < (uint32_t)nb)
            Fb[b] = make_float4(fx, fy, fz, feels(T.pe) && sqn(fx, fy, fz) > 1e-20f ? 1.0f : 0.0f);
    }
}

// Per body, its boundary points' forces and torques added in boundary order
// (the reference's): a block per body computes the terms side by side, 256 at
// a time, and lane k of the first warp adds component k.  One thread per body
// took 524 us for eight bodies of about 1,000 points, waiting on three
// dependent loads per point.
constexpr int kReduceThreads = 256;

__global__ void __launch_bounds__(kReduceThreads)
k_body_reduce(const float4* __restrict__ Fb, const float4* __restrict__ bworld,
              const int* __restrict__ list_off, const int* __restrict__ list,
              const float4* __restrict__ body_pos, int nbodies, float* __restrict__ force3,
              float* __restrict__ torque3) {
    __shared__ __align__(16) float term[6][kReduceThreads];
    __shared__ uint32_t has[kReduceThreads / 32];
    const int k = blockIdx.x, t = threadIdx.x;
    if (k >= nbodies) return;
    const float4 c = body_pos[k];
    const int j1 = list_off[k + 1];
    float sum = 0.0f;
    if (t < 3) sum = force3[3 * k + t];
    else if (t < 6) sum = torque3[3 * k + t - 3];
    for (int j0 = list_off[k]; j0 < j1; j0 += kReduceThreads) {
        const int j = j0 + t;
        float4 F = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (j < j1) {
            const int b = __ldg(list + j);
            F = __ldg(Fb + b);
            if (F.w != 0.0f) {
                const float4 x = __ldg(bworld + b);
                const float r0 = x.x - c.x, r1 = x.y - c.y, r2 = x.z - c.z;
                term[0][t] = F.x;
                term[1][t] = F.y;
                term[2][t] = F.z;
                term[3][t] = r1 * F.z - r2 * F.y;
                term[4][t] = r2 * F.x - r0 * F.z;
                term[5][t] = r0 * F.y - r1 * F.x;
            }
        }
        const uint32_t m = __ballot_sync(0xffffffffu, F.w != 0.0f);
        if ((t & 31) == 0) has[t >> 5] = m;
        __syncthreads();
        if (t < 6) {
            for (int w = 0; w < kReduceThreads / 32; ++w) {
                const uint32_t bits = has[w];
                if (bits == 0xffffffffu) {
#pragma unroll
                    for (int i = 0; i < 32; i += 4) {
                        const float4 v = *reinterpret_cast<const float4*>(&term[t][32 * w + i]);
                        sum = sum + v.x;
                        sum = sum + v.y;
                        sum = sum + v.z;
                        sum = sum + v.w;
                    }
                } else {
                    for (uint32_t b = bits; b; b &= b - 1u) sum = sum + term[t][32 * w + __ffs(b) - 1];
                }
            }
        }
        __syncthreads();
    }
    if (t < 3) force3[3 * k + t] = sum;
    else if (t < 6) torque3[3 * k + t - 3] = sum;
}

// Segmented tree reduction of the same sums: one block per body.  Thread t
// adds the list entries t, t + kTreeThreads, ... of its body in that order,
// then the block folds its partial sums pairwise (partial[t] += partial[t + s]
// for s = 128, 64, ..., 1), so every run adds the same floats in the same
// order: the result is deterministic, whatever the schedule.  It rounds
// differently from the serial sum above (the reference's order), by at most
// 2 (m - 1) 2^-24 sum_b |term_b| per component over a body's m terms.
constexpr int kTreeThreads = 256;

__global__ void __launch_bounds__(kTreeThreads)
k_body_reduce_tree(const float4* __restrict__ Fb, const float4* __restrict__ bworld,
                   const int* __restrict__ list_off, const int* __restrict__ list,
                   const float4* __restrict__ body_pos, int nbodies, float* __restrict__ force3,
                   float* __restrict__ torque3) {
    __shared__ float part[6][kTreeThreads];
    const int k = blockIdx.x;
    if (k >= nbodies) return;
    const int t = threadIdx.x;
    const float4 c = body_pos[k];
    float a[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    const int j1 = list_off[k + 1];
    for (int j = list_off[k] + t; j < j1; j += kTreeThreads) {
        const int b = __ldg(list + j);
        const float4 F = __ldg(Fb + b);
        if (F.w == 0.0f) continue;
        const float4 x = __ldg(bworld + b);
        const float r0 = x.x - c.x, r1 = x.y - c.y, r2 = x.z - c.z;
        a[0] += F.x;
        a[1] += F.y;
        a[2] += F.z;
        a[3] += r1 * F.z - r2 * F.y;
        a[4] += r2 * F.x - r0 * F.z;
        a[5] += r0 * F.y - r1 * F.x;
    }
#pragma unroll
    for (int d = 0; d < 6; ++d) part[d][t] = a[d];
    __syncthreads();
#pragma unroll 1
    for (int s = kTreeThreads / 2; s > 0; s >>= 1) {
        if (t < s) {
#pragma unroll
            for (int d = 0; d < 6; ++d) part[d][t] += part[d][t + s];
        }
        __syncthreads();
    }
    if (t < 3) {
        force3[3 * k + t] += part[t][0];
        torque3[3 * k + t] += part[3 + t][0];
    }
}

// One thread per body (rigid_step.hpp on the device).
__global__ void k_rigid_step(pbf_rigid_body* __restrict__ bodies, int nbodies,
                             const float* __restrict__ force3, const float* __restrict__ torque3,
                             int nforce, float gx, float gy, float gz, float dt,
                             float4* __restrict__ body_pos, float4* __restrict__ body_quat) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nbodies) return;
    pbf_rigid_body r = bodies[k];
    if (r.inv_mass > 0.0f) {
        const float g[3] = {gx, gy, gz};
        float f[3] = {0.0f, 0.0f, 0.0f}, t[3] = {0.0f, 0.0f, 0.0f};
        if (k < nforce)
            for (int d = 0; d < 3; ++d) {
                f[d] = force3[3 * k + d];
                t[d] = torque3[3 * k + d];
            }
        pbf_rigid::integrate_velocity(r.lin_vel, r.ang_vel, g, f, r.inv_mass, r.inv_inertia, t, dt);
        pbf_rigid::integrate_position(r.pos, r.quat, r.lin_vel, r.ang_vel, dt);
        bodies[k] = r;
    }
    if (k < nforce) {
        body_pos[k] = make_float4(r.pos[0], r.pos[1], r.pos[2], 0.0f);
        body_quat[k] = make_float4(r.quat[0], r.quat[1], r.quat[2], r.quat[3]);
    }
}

// World's rigid pipeline for one scene's bodies and shapes (rigid_world.cuh),
// in shared memory by one thread; then the new poses of the first nforce
// bodies into body_pos/body_quat, as k_rigid_step.
__global__ void __launch_bounds__(32)
k_rigid_world(pbf_rigid_body* __restrict__ bodies, int nbodies,
              const pbf_rigid_shape* __restrict__ shapes, int nshapes, pbf_contact_settings set,
              const float* __restrict__ force3, const float* __restrict__ torque3, int nforce,
              float gx, float gy, float gz, float dt, float4* __restrict__ body_pos,
              float4* __restrict__ body_quat) {
    __shared__ rw::World W;
    __shared__ pbf_rigid_body B[rw::kMaxShapes];
    __shared__ pbf_rigid_shape S[rw::kMaxShapes];
    if (threadIdx.x != 0 || nbodies > rw::kMaxShapes || nshapes > rw::kMaxShapes) return;
    for (int k = 0; k < nbodies; ++k) B[k] = bodies[k];
    for (int k = 0; k < nshapes; ++k) S[k] = shapes[k];
    const float g[3] = {gx, gy, gz};
    if (rw::world_step(W, B, nbodies, S, nshapes, set, force3, torque3, nforce, g, dt)) return;
    for (int k = 0; k < nbodies; ++k) bodies[k] = B[k];
    for (int k = 0; k < nforce && k < nbodies; ++k) {
        body_pos[k] = make_float4(B[k].pos[0], B[k].pos[1], B[k].pos[2], 0.0f);
        body_quat[k] = make_float4(B[k].quat[0], B[k].quat[1], B[k].quat[2], B[k].quat[3]);
    }
}

template <int TP>
__global__ void __launch_bounds__(128, kTeamMinBlocks<TP>)
k_volumes(int nb, const QuerySet Q, const PointIndex I, float* __restrict__ psi, const StepConsts C) {
    __shared__ TeamSmem<TP> sm;
    const TeamThread<TP> T(nb);
    const Grid G = query_grid(I, Q);
    const float4 xi = I.spos[T.pe];
    TeamSums<VolumeTerm, 128 / TP> sums(VolumeTerm{C, xi});
    team_walk<TP, false>(sm, G, G.ix, OneScene{C, StateRef{}}, T.pl, query_cell(Q, T.pl), T.al, I.spos[T.pl],
                         I.spos, sums);
    const float sum_w = sums.get(0);
    if (T.writer) {
        const uint32_t b = I.sidx[T.pe];
        if (b < (uint32_t)nb) psi[b] = (sum_w > 1e-10f) ? 1.0f / sum_w : 0.0f;
    }
}

// Queries per team: as the step's passes, with teams at every size.
inline bool small_teams(int nq) { return team_size(nq) == 8; }

}  // namespace bnd

cudaError_t index_build(PointIndex& I, const float4* pos, const float* attr, int n,
                        const StepConsts& C, SortScratch& sort, cudaStream_t st) {
    using namespace bnd;
    I.n = n;
    if (n <= 0) return cudaSuccess;
    const int bits = C.grid.key_bits, nb = grid_of(n, kBlock);
    const ClearRange alias{reinterpret_cast<uint32_t*>(I.slot_alias), ((size_t)C.grid.nslots + 3) / 4, 0u};
    cudaError_t e = clear_ranges(alias, sort_clear(sort, n, bits), bucket_clear(I.bkt, n), st);
    if (e != cudaSuccess) return e;
    k_ix_keys<<<count_blocks(n), kCountThreads, 0, st>>>(pos, n, I.keys, sort_counts(sort, n, bits), C);
    e = radix_sort_counted(I.keys, I.skeys, I.sidx, n, bits, sort, st);
    if (e != cudaSuccess) return e;
    k_ix_gather<<<nb + grid_of((int)C.grid.nslots + 1, kBlock), kBlock, 0, st>>>(I.sidx, pos, attr, n, I.spos,
        I.scell, I.bkt.link, I.slot_alias, SlotOffsets{I.skeys, I.off, C.grid.nslots, nb}, C);
    return enqueue_buckets(sized_for(I.bkt, n), I.scell, I.sidx, nullptr, I.off, I.slot_alias, n,
                           OneScene{C, StateRef{}}, st);
}

cudaError_t predict_cells(const float4* x, const float4* v, int n, int4* cells, const StepConsts& C,
                          cudaStream_t st) {
    using namespace bnd;
    if (n <= 0) return cudaSuccess;
    k_predict_cells<<<grid_of(n, kBlock), kBlock, 0, st>>>(x, v, n, cells, C);
    return cudaGetLastError();
}

cudaError_t index_classify(const QuerySet& Q, int nq, const PointIndex& I, const StepConsts& C,
                           cudaStream_t st) {
    using namespace bnd;
    if (nq <= 0) return cudaSuccess;
    if (I.n <= 0) {
        // Nothing to find: every neighbour bucket is empty.
        return cudaMemsetAsync(Q.qown, 0, (size_t)nq * sizeof(int), st);
    }
    StepConsts Cs = C;
    Cs.hash_compat = 1;  // the coupling queries always follow the reference buckets
    k_classify<OneScene><<<grid_of(nq, kBlock), kBlock, 0, st>>>(Q.qcell, nq, I.scell, nullptr,
        sized_for(I.bkt, I.n), I.slot_alias, Q.btab, Q.qown, nullptr, OneScene{Cs, StateRef{}});
    return cudaGetLastError();
}

cudaError_t boundary_xform(const float4* local, const int* body, int nb, const float4* body_pos,
                           const float4* body_quat, int nbodies, float4* world, cudaStream_t st) {
    using namespace bnd;
    if (nb <= 0) return cudaSuccess;
    k_bxform<<<grid_of(nb, kBlock), kBlock, 0, st>>>(local, body, nb, body_pos, body_quat, nbodies, world);
    return cudaGetLastError();
}

cudaError_t boundary_density(const PointIndex& fidx, const QuerySet& Q, const PointIndex& bidx,
                             float* rho, bool has_boundary, const StepConsts& C, cudaStream_t st) {
    using namespace bnd;
    const int n = fidx.n;
    if (n <= 0) return cudaSuccess;
    if (has_boundary || bidx.n <= 0)
        k_pressure_weights<<<grid_of(n, kBlock), kBlock, 0, st>>>(fidx.spos, n, C);
    else if (small_teams(n))
        k_boundary_density<8><<<grid_of(n, 8), 128, 0, st>>>(fidx.spos, fidx.sidx, n, Q, bidx, rho, C);
    else
        k_boundary_density<16><<<grid_of(n, 16), 128, 0, st>>>(fidx.spos, fidx.sidx, n, Q, bidx, rho, C);
    return cudaGetLastError();
}

cudaError_t coupling_forces(const PointIndex& bidx, const int* body, const int* body_dynamic, int nbodies,
                            const QuerySet& Q, const PointIndex& fidx, float4* Fb, const StepConsts& C,
                            cudaStream_t st) {
    using namespace bnd;
    const int nb = bidx.n;
    if (nb <= 0) return cudaSuccess;
    if (fidx.n <= 0) return cudaMemsetAsync(Fb, 0, (size_t)nb * sizeof(float4), st);
    if (small_teams(nb))
        k_coupling<8><<<grid_of(nb, 8), 128, 0, st>>>(bidx.spos, bidx.sidx, body, body_dynamic, nb, nbodies, Q,
            fidx, Fb, C);
    else
        k_coupling<16><<<grid_of(nb, 16), 128, 0, st>>>(bidx.spos, bidx.sidx, body, body_dynamic, nb, nbodies,
            Q, fidx, Fb, C);
    return cudaGetLastError();
}

cudaError_t body_reduce(const float4* Fb, const float4* bworld, const int* list_off,
                        const int* list, const float4* body_pos, int nbodies, float* force3,
                        float* torque3, bool tree, cudaStream_t st) {
    using namespace bnd;
    if (nbodies <= 0) return cudaSuccess;
    if (tree)
        k_body_reduce_tree<<<nbodies, kTreeThreads, 0, st>>>(Fb, bworld, list_off, list, body_pos, nbodies,
            force3, torque3);
    else
        k_body_reduce<<<nbodies, kReduceThreads, 0, st>>>(Fb, bworld, list_off, list, body_pos, nbodies,
            force3, torque3);
    return cudaGetLastError();
}

cudaError_t rigid_world(pbf_rigid_body* bodies, int nbodies, const pbf_rigid_shape* shapes,
                        int nshapes, const pbf_contact_settings& set, const float* force3,
                        const float* torque3, int nforce, float gx, float gy, float gz, float dt,
                        float4* body_pos, float4* body_quat, cudaStream_t st) {
    using namespace bnd;
    if (nbodies <= 0) return cudaSuccess;
    k_rigid_world<<<1, 32, 0, st>>>(bodies, nbodies, shapes, nshapes, set, force3, torque3, nforce,
                                    gx, gy, gz, dt, body_pos, body_quat);
    return cudaGetLastError();
}

cudaError_t rigid_step(pbf_rigid_body* bodies, int nbodies, const float* force3,
                       const float* torque3, int nforce, float gx, float gy, float gz, float dt,
                       float4* body_pos, float4* body_quat, cudaStream_t st) {
    using namespace bnd;
    if (nbodies <= 0) return cudaSuccess;
    k_rigid_step<<<grid_of(nbodies, 32), 32, 0, st>>>(bodies, nbodies, force3, torque3, nforce, gx,
                                                      gy, gz, dt, body_pos, body_quat);
    return cudaGetLastError();
}

cudaError_t boundary_volumes(const QuerySet& Q, const PointIndex& I, float* psi, const StepConsts& C,
                             cudaStream_t st) {
    using namespace bnd;
    const int nb = I.n;
    if (nb <= 0) return cudaSuccess;
    if (small_teams(nb))
        k_volumes<8><<<grid_of(nb, 8), 128, 0, st>>>(nb, Q, I, psi, C);
    else
        k_volumes<16><<<grid_of(nb, 16), 128, 0, st>>>(nb, Q, I, psi, C);
    return cudaGetLastError();
}

}  // namespace pbf
