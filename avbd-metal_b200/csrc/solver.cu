// solver.cu — warm start, per-frame adjacency, dynamic coloring, the
// per-color block-descent primal, the augmented-Lagrangian dual, BDF1
// finalize and the constraint-error diagnostic.
//
// Follows Shaders/40_solver.metal: warm start :546-722, adjacency :27-243,
// coloring :250-540, force stamps :741-1152 and :1155-1230, the 8-lane
// primal_particles_split :1544-1684, dual :1729-1906, finalize :2108-2147,
// diag_error :2189-2229.
//
// Every primal kernel adds a body's entries in the order of the reference's
// group of 8 lanes: logical lane l takes adjacency entries l, l+8, l+16, ... of
// the body, and an xor butterfly (offsets 4, 2, 1) sums the lanes.  Who
// evaluates an entry differs: k_primal and k_solve_small (dynamic coloring,
// small scenes) deal contact points out to the 8 lanes, k_primal_staged and
// k_primal_group take particles, k_primal_wide a rigid body per block.  The
// static part of the adjacency (joints, springs, tets) is built once at upload;
// only contact entries are rebuilt per frame.
#include <utility>

#include <atomic>

#include "dmath.cuh"
#include "kernels.h"
#include "pdl.cuh"

namespace avbd {

constexpr float FLT_BIG = 3.402823466e38f;

// failure kinds (mirrors AVBD_FAIL_* of include/avbd.h)
constexpr uint32_t AVBD_FAIL_RIGID_PAIR_CAPACITY_ = 2;
constexpr uint32_t AVBD_FAIL_UNRESOLVED_COLORING_ = 5;
constexpr uint32_t AVBD_FAIL_WAIT_TIMEOUT_ = 9;

__device__ __forceinline__ bool body_dynamic(const DevPtrs& d, uint32_t b) {
    return b != WORLD_BODY && d.posLin[b].w > 0.0f;
}

static uint32_t stride_blocks(uint32_t upper, int threads) {
    const uint32_t need = (upper + threads - 1) / threads;
    const uint32_t cap = 148u * 8u;
    return need == 0 ? 1u : (need < cap ? need : cap);
}

// ---------------------------------------------------------------------------
// Warm start (40_solver.metal:546-722)
// ---------------------------------------------------------------------------
__global__ void k_warmstart_constraints(const Params P, const DevPtrs d, uint32_t nJ, uint32_t nS) {
    pdl_prologue();
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nJ + nS) return;
    if (t >= nJ) {
        SpringGPU& sp = d.springs[d.hardSprings[t - nJ]];
        const uint32_t a = sp.header.x, b = sp.header.y;
        const float3 pA = xform(xyz(d.posLin[a]), d.posAng[a], xyz(sp.rA));
        const float3 pB = xform(xyz(d.posLin[b]), d.posAng[b], xyz(sp.rB));
        sp.dual.z = 0.5f * mx(len3(pA - pB) - sp.rB.w, 0.0f);
        float warm = P.alpha * P.gamma;
        if (P.rodDecayPow > 0.0f) {
            const float3 dd = pA - pB;
            const float3 dPrev = dd - (xyz(d.velLin[a]) - xyz(d.velLin[b])) * P.dt;
            const float dl = len3(dd), dpl = len3(dPrev);
            if (dl > 1e-7f && dpl > 1e-7f) {
                const float ct = clampf(dot(dd / dl, dPrev / dpl), 0.0f, 1.0f);
                warm *= powf(ct, P.rodDecayPow);
            }
        }
        sp.dual.x *= warm;
        sp.dual.y = mn(clampf(sp.dual.y * P.gamma, PENALTY_MIN, PENALTY_MAX), sp.rA.w);
        return;
    }
    JointGPU& j = d.joints[d.activeJoints[t]];
    if (j.header.z != 0) return;
    const uint32_t a = j.header.x, b = j.header.y;
    const float3 pA = a == WORLD_BODY ? xyz(j.rA) : xform(xyz(d.posLin[a]), d.posAng[a], xyz(j.rA));
    const float3 pB = xform(xyz(d.posLin[b]), d.posAng[b], xyz(j.rB));
    const float4 qA = a == WORLD_BODY ? make_float4(0, 0, 0, 1) : d.posAng[a];
    const float4 qB = d.posAng[b];
    const float torqueArm = j.C0Lin.w;
    j.C0Lin = tof4(pA - pB, torqueArm);
    const float3 axis = xyz(j.hingeAxis);
    const float4 restRel = tof(j.restRel);
    float3 c0a;
    if (j.hingeAxis.w != 0.0f) {
        const float3 aB = q_rotate(qB, axis);
        const float3 aA = q_rotate(q_mul(qA, restRel), axis);
        c0a = cross(aA, aB) * torqueArm;
        if (j.dynamics.x > 0.0f) {
            const float twist = twist_angle(q_mul(qA, restRel), qB, axis);
            const float3 omegaA = a == WORLD_BODY ? s3(0) : xyz(d.velAng[a]);
            const float twistRate = dot(xyz(d.velAng[b]) - omegaA, aB);
            j.dynamics.y = twist + P.dt * twistRate;
        }
    } else {
        c0a = q_sub(q_mul(qA, restRel), qB) * torqueArm;
    }
    j.C0Ang = tof4(c0a, j.C0Ang.w);
    if (j.motor.y > 0.0f) {
        j.motor.z = 0.0f;
        j.dynamics.z = 0.0f;
        const uint32_t mode = j.header.w & MOTOR_MODE_MASK;
        if (mode == MOTOR_EXPLICIT || mode == MOTOR_VELOCITY) {
            const float4 qAr = a == WORLD_BODY ? restRel : q_mul(d.posAng[a], restRel);
            const float twist = twist_angle(qAr, qB, axis);
            const float3 axisW = q_rotate(qB, axis);
            const float3 omegaA = a == WORLD_BODY ? s3(0) : xyz(d.velAng[a]);
            const float twistRate = dot(xyz(d.velAng[b]) - omegaA, axisW);
            if (mode == MOTOR_VELOCITY)
                j.dynamics.z = clampf(j.limits.z * (j.motor.x - twistRate), -j.motor.y, j.motor.y);
            else
                j.dynamics.z = clampf(j.motor.w * (j.motor.x - twist) - j.limits.z * twistRate, -j.motor.y, j.motor.y);
        }
    }
    const float warm = P.alpha * P.gamma;
    j.lambdaLin.x *= warm; j.lambdaLin.y *= warm; j.lambdaLin.z *= warm;
    j.lambdaAng.x *= warm; j.lambdaAng.y *= warm; j.lambdaAng.z *= warm;
    float3 pl = clamp3(xyz(j.penaltyLin) * P.gamma, s3(PENALTY_MIN), s3(PENALTY_MAX));
    float3 pa = clamp3(xyz(j.penaltyAng) * P.gamma, s3(PENALTY_MIN), s3(PENALTY_MAX));
    pl = mn3(pl, s3(j.rA.w));
    pa = mn3(pa, s3(j.rB.w));
    j.penaltyLin = tof4(pl, j.penaltyLin.w);
    j.penaltyAng = tof4(pa, j.penaltyAng.w);
}

__global__ void k_warmstart_bodies(const Params P, const DevPtrs d) {
    pdl_prologue();
    const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= P.numBodies) return;
    const float4 pl = d.posLin[gid], pa = d.posAng[gid];
    const float mass = pl.w, dt = P.dt;
    const float3 vl = xyz(d.velLin[gid]), va = xyz(d.velAng[gid]);
    float3 inertial = xyz(pl) + vl * dt;
    const float bodyGravity = P.gravity * d.gravityScale[gid];
    if (mass > 0.0f) inertial += mk3(0, 0, bodyGravity) * (dt * dt);
    d.inertLin[gid] = mk4(inertial, 0.0f);
    d.inertAng[gid] = q_addw(pa, va * dt);
    const float3 accel = (vl - xyz(d.prevVelLin[gid])) / dt;
    const float gsign = P.gravity < 0.0f ? -1.0f : (P.gravity > 0.0f ? 1.0f : 0.0f);
    float w = clampf(accel.z * gsign / fabsf(P.gravity), 0.0f, 1.0f);
    if (!isfinite(w)) w = 0.0f;
    d.initLin[gid] = mk4(xyz(pl), 0.0f);
    d.initAng[gid] = pa;
    // the committed collision-query pose of every surface vertex, pins included
    if ((P.cloth || P.ogc) && P.surfaceTruncationMode != 0u && d.shape[gid].w < 0.0f)
        d.ogcPrev[gid] = mk4(xyz(pl), 0.0f);
    if (mass > 0.0f) {
        float3 guess = xyz(pl) + vl * dt + mk3(0, 0, bodyGravity) * (w * dt * dt);
        // Isotropic OGC: the warm start stays within the particle's bound
        // (40_solver.metal:700-717).  Without element contacts (P.ogc == 0)
        // every bound is "far" and this is a no-op.
        if (P.ogc && d.shape[gid].w < 0.0f) {
            const float d2 = __uint_as_float(d.ogcBounds[gid]);
            if (d2 < 1e37f) {
                const float bv = mx(0.45f * sqrtf(d2), -0.2f * d.shape[gid].w);
                const float3 tot = guess - xyz(pl);
                const float t2 = dot(tot, tot);
                if (t2 > bv * bv) guess = xyz(pl) + tot * (bv * rsq(t2));
            }
        }
        d.posLin[gid] = mk4(guess, mass);
        d.posAng[gid] = q_addw(pa, va * dt);
    }
}

void launch_warmstart(const Params& P, const DevPtrs& d, const Sizes& z, cudaStream_t st) {
    const uint32_t n = z.numActiveJoints + z.numHardSprings;
    if (n) launch_pdl(k_warmstart_constraints, (n + 127) / 128, 128, st, P, d, z.numActiveJoints, z.numHardSprings);
    launch_pdl(k_warmstart_bodies, (P.numBodies + 127) / 128, 128, st, P, d);
}

// ---------------------------------------------------------------------------
// Per-frame contact adjacency: count, scan, scatter, sort per body.
// ---------------------------------------------------------------------------
// Items: this frame's manifolds, then (cloth scenes) its element contacts.
template <bool SCATTER>
__global__ void k_adj_dyn(const Params P, const DevPtrs d) {
    pdl_prologue();
    const uint32_t nm = d.counters->numPairs;
    const uint32_t ns = (P.cloth || P.ogc) ? d.counters->numSoft : 0u;
    auto put = [&](uint32_t b, uint32_t e) {
        if (!body_dynamic(d, b)) return;
        if (SCATTER) d.dynList[atomicAdd(&d.dynCursor[b], 1u)] = e;
        else atomicAdd(&d.dynCount[b], 1u);
    };
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nm + ns; i += gridDim.x * blockDim.x) {
        if (i < nm) {
            const u4 h = d.manifolds[i].header;
            if (h.z == 0) continue;
            const uint32_t e = (FK_MANIFOLD << ADJ_KIND_SHIFT) | i;
            // the dual visits only manifolds with contacts, in any order
            // (their updates are independent)
            if (!SCATTER) d.activeManifolds[atomicAdd(&d.counters->activeManifolds, 1u)] = i;
            put(h.x, e);
            put(h.y, e);
        } else {
            const uint32_t k = i - nm;
            const u4 ids = d.soft[k].ids;
            const uint32_t e = (FK_SOFT << ADJ_KIND_SHIFT) | k;
            put(ids.x, e);
            put(ids.y, e);
            put(ids.z, e);
            put(ids.w, e);
        }
    }
}
constexpr uint32_t kLongSegment = 2048;   // entries a block sorts in shared memory

__global__ void k_adj_dyn_sort(const DevPtrs d, uint32_t nb) {
    pdl_prologue();
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    uint32_t* l = d.dynList + d.dynStart[b];
    const uint32_t n = d.dynCount[b];
    if (n <= 32) {
        for (uint32_t i = 1; i < n; i++) {
            const uint32_t v = l[i];
            uint32_t j = i;
            while (j > 0 && l[j - 1] > v) { l[j] = l[j - 1]; j--; }
            l[j] = v;
        }
    } else if (n <= kLongSegment) {
        // left to k_adj_long_sort (one block per segment)
        d.dynSplit[b] = 0xFFFFFFFFu;
        d.adjLongQueue[atomicAdd(&d.counters->adjLong, 1u)] = b;
        return;
    } else {
        // heapsort: bodies under a pile (a box on a cloth) carry hundreds of
        // entries; the entries are distinct, so the order is unique
        auto sift = [&](uint32_t root, uint32_t end) {
            while (2 * root + 1 < end) {
                uint32_t c = 2 * root + 1;
                if (c + 1 < end && l[c] < l[c + 1]) c++;
                if (l[root] >= l[c]) return;
                const uint32_t t = l[root]; l[root] = l[c]; l[c] = t;
                root = c;
            }
        };
        for (uint32_t i = n / 2; i-- > 0;) sift(i, n);
        for (uint32_t end = n - 1; end > 0; end--) {
            const uint32_t t = l[0]; l[0] = l[end]; l[end] = t;
            sift(0, end);
        }
    }
    uint32_t m = 0;
    while (m < n && (l[m] >> ADJ_KIND_SHIFT) == FK_MANIFOLD) m++;
    d.dynSplit[b] = m;
}

// Segments of 33..2048 entries: one block loads the segment into shared
// memory, sorts it with a bitonic network (padded with 0xFFFFFFFF), writes
// it back and marks the manifold run.  Entries are distinct, so the result
// equals the serial sort.
__global__ void __launch_bounds__(256) k_adj_long_sort(const DevPtrs d) {
    pdl_prologue();
    __shared__ uint32_t buf[kLongSegment];
    const uint32_t count = d.counters->adjLong;
    for (uint32_t q = blockIdx.x; q < count; q += gridDim.x) {
        const uint32_t b = d.adjLongQueue[q];
        uint32_t* l = d.dynList + d.dynStart[b];
        const uint32_t n = d.dynCount[b];
        uint32_t m = 64;
        while (m < n) m <<= 1;
        for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) buf[i] = i < n ? l[i] : 0xFFFFFFFFu;
        __syncthreads();
        for (uint32_t k = 2; k <= m; k <<= 1)
            for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
                    const uint32_t p = i ^ j;
                    if (p > i) {
                        const uint32_t x = buf[i], y = buf[p];
                        const bool up = (i & k) == 0;
                        if ((x > y) == up) { buf[i] = y; buf[p] = x; }
                    }
                }
                __syncthreads();
            }
        for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) l[i] = buf[i];
        // manifold entries lead the sorted segment
        uint32_t man = 0;
        for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) man += (buf[i] >> ADJ_KIND_SHIFT) == FK_MANIFOLD ? 1u : 0u;
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) man += __shfl_xor_sync(0xffffffffu, man, o);
        __shared__ uint32_t warpMan[8];
        if ((threadIdx.x & 31u) == 0) warpMan[threadIdx.x >> 5] = man;
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t t = 0;
            for (uint32_t w = 0; w < (blockDim.x >> 5); w++) t += warpMan[w];
            d.dynSplit[b] = t;
        }
        __syncthreads();
    }
}

void launch_adjacency(const Params& P, const DevPtrs& d, const Sizes& z, cudaStream_t st) {
    cudaMemsetAsync(d.dynCount, 0, sizeof(uint32_t) * P.numBodies, st);
    const uint32_t items = z.maxPairs + ((P.cloth || P.ogc) ? z.maxSoft : 0u);
    launch_pdl(k_adj_dyn<false>, stride_blocks(items, 128), 128, st, P, d);
    launch_exclusive_scan(d.dynCount, d.dynStart, P.numBodies, d.scanScratch, st);
    cudaMemcpyAsync(d.dynCursor, d.dynStart, sizeof(uint32_t) * P.numBodies, cudaMemcpyDeviceToDevice, st);
    launch_pdl(k_adj_dyn<true>, stride_blocks(items, 128), 128, st, P, d);
    launch_pdl(k_adj_dyn_sort, (P.numBodies + 127) / 128, 128, st, d, P.numBodies);
    launch_pdl(k_adj_long_sort, 148, 256, st, d);
}

// The five runs in ascending (kind << 28 | index) order: static pre
// (joints, springs), this frame's manifolds, static tets, this frame's
// element contacts, static membranes and bends.
struct AdjView {
    const uint32_t* pre; uint32_t nPre;
    const uint32_t* dyn; uint32_t nMan, nDyn;
    const uint32_t* post; uint32_t nTet, nPost, postBase;
    __device__ __forceinline__ uint32_t count() const { return nPre + nDyn + nPost; }
    __device__ __forceinline__ uint32_t at(uint32_t k) const {
        if (k < nPre) return pre[k];
        k -= nPre;
        if (k < nMan) return dyn[k];
        k -= nMan;
        if (k < nTet) return post[k];
        k -= nTet;
        if (k < nDyn - nMan) return dyn[nMan + k];
        return post[nTet + k - (nDyn - nMan)];
    }
};
// The view from the body's static segment (set at upload) and this frame's
// contact segment.
__device__ __forceinline__ AdjView adj_view_from(const DevPtrs& d, uint32_t b, uint4 s, uint32_t nTet) {
    AdjView v;
    v.pre = d.preList + s.x; v.nPre = s.y;
    v.dyn = d.dynList + d.dynStart[b]; v.nDyn = d.dynCount[b]; v.nMan = d.dynSplit[b];
    v.post = d.postList + s.z; v.nPost = s.w; v.nTet = nTet; v.postBase = s.z;
    return v;
}
__device__ __forceinline__ AdjView adj_view(const DevPtrs& d, uint32_t b) {
    const uint4 s = d.staticSeg[b];
    AdjView v;
    v.pre = d.preList + s.x; v.nPre = s.y;
    v.dyn = d.dynList + d.dynStart[b]; v.nDyn = d.dynCount[b]; v.nMan = d.dynSplit[b];
    v.post = d.postList + s.z; v.nPost = s.w; v.nTet = d.postTets[b]; v.postBase = s.z;
    return v;
}

// ---------------------------------------------------------------------------
// Dynamic coloring for rigid-only scenes (40_solver.metal:250-540)
// ---------------------------------------------------------------------------
__device__ void neighbor_colors(const DevPtrs& d, uint32_t entry, uint32_t self, uint32_t myColor,
                                const uint32_t* colorsIn, uint32_t& maskLo, uint32_t& maskHi,
                                uint32_t& allLo, uint32_t& allHi, bool& conflict) {
    const uint32_t kind = entry >> ADJ_KIND_SHIFT, idx = entry & ADJ_INDEX_MASK;
    uint32_t nbs[3];
    uint32_t n = 0;
    if (kind == FK_TET) {
        const u4 ids = d.tets[idx].ids;
        if (ids.x != self && n < 3) nbs[n++] = ids.x;
        if (ids.y != self && n < 3) nbs[n++] = ids.y;
        if (ids.z != self && n < 3) nbs[n++] = ids.z;
        if (ids.w != self && n < 3) nbs[n++] = ids.w;
    } else {
        uint32_t a, b;
        if (kind == FK_JOINT) { a = d.joints[idx].header.x; b = d.joints[idx].header.y; }
        else if (kind == FK_SPRING) { a = d.springs[idx].header.x; b = d.springs[idx].header.y; }
        else { a = d.manifolds[idx].header.x; b = d.manifolds[idx].header.y; }
        nbs[0] = a == self ? b : a;
        n = 1;
    }
    for (uint32_t k = 0; k < n; k++) {
        const uint32_t nb = nbs[k];
        if (nb == WORLD_BODY || d.posLin[nb].w <= 0.0f) continue;
        const uint32_t c = colorsIn[nb];
        const uint32_t lo = c < 32 ? (1u << c) : 0u;
        const uint32_t hi = (c >= 32 && c < 64) ? (1u << (c - 32)) : 0u;
        allLo |= lo; allHi |= hi;
        if (nb < self) { maskLo |= lo; maskHi |= hi; if (c == myColor) conflict = true; }
    }
}

__device__ __forceinline__ void scan_neighbors(const DevPtrs& d, uint32_t b, uint32_t my, const uint32_t* colors,
                                               uint32_t& mLo, uint32_t& mHi, uint32_t& aLo, uint32_t& aHi,
                                               bool& conflict) {
    const AdjView v = adj_view(d, b);
    const uint32_t n = v.count();
    for (uint32_t k = 0; k < n; k++) neighbor_colors(d, v.at(k), b, my, colors, mLo, mHi, aLo, aHi, conflict);
}

__device__ __forceinline__ uint32_t ctz32(uint32_t x) { return (uint32_t)(__ffs((int)x) - 1); }

// One body of a Jacobi coloring pass.
__device__ __forceinline__ void color_step(const DevPtrs& d, uint32_t gid, const uint32_t* src, uint32_t* dst,
                                           uint32_t pass) {
    if (d.posLin[gid].w <= 0.0f) { dst[gid] = 0; return; }
    const uint32_t my = src[gid];
    uint32_t mLo = 0, mHi = 0, aLo = 0, aHi = 0;
    bool conflict = false;
    scan_neighbors(d, gid, my, src, mLo, mHi, aLo, aHi, conflict);
    if (conflict) {
        const uint32_t freeLo = ~mLo;
        uint32_t nc;
        if (freeLo != 0) nc = ctz32(freeLo);
        else { const uint32_t freeHi = ~mHi; nc = freeHi != 0 ? 32 + ctz32(freeHi) : (MAX_COLORS - 1); }
        dst[gid] = nc < (uint32_t)(MAX_COLORS - 1) ? nc : (uint32_t)(MAX_COLORS - 1);
        atomicOr(&d.counters->changed[pass], 1u);
    } else {
        const uint32_t freeLo = ~aLo;
        const uint32_t best = freeLo != 0 ? ctz32(freeLo) : (~aHi != 0 ? 32 + ctz32(~aHi) : my);
        dst[gid] = best < my ? best : my;
        if (best < my) atomicOr(&d.counters->changed[pass], 1u);
    }
}

// Serial greedy completion when the bounded parallel phase has not settled.
__device__ void color_repair(const Params& P, const DevPtrs& d, uint32_t* colors) {
    for (uint32_t self = 0; self < P.numBodies; self++) {
        if (d.posLin[self].w <= 0.0f) { colors[self] = 0; continue; }
        uint32_t mLo = 0, mHi = 0, aLo = 0, aHi = 0;
        bool conflict = false;
        scan_neighbors(d, self, colors[self], colors, mLo, mHi, aLo, aHi, conflict);
        const uint32_t freeLo = ~mLo;
        if (freeLo != 0) colors[self] = ctz32(freeLo);
        else { const uint32_t freeHi = ~mHi; colors[self] = freeHi != 0 ? 32 + ctz32(freeHi) : (MAX_COLORS - 1); }
    }
}

__device__ __forceinline__ void color_count(const DevPtrs& d, uint32_t gid, const uint32_t* colors) {
    if (d.posLin[gid].w <= 0.0f) return;
    uint32_t mLo = 0, mHi = 0, aLo = 0, aHi = 0;
    bool conflict = false;
    scan_neighbors(d, gid, colors[gid], colors, mLo, mHi, aLo, aHi, conflict);
    if (conflict) atomicAdd(&d.counters->colorConflicts, 1u);
    d.bodySlot[gid] = atomicAdd(&d.counters->colorCount[colors[gid]], 1u);
}

__device__ void color_scan(const DevPtrs& d) {
    uint32_t run = 0, used = 0;
    for (int c = 0; c < MAX_COLORS; c++) {
        d.counters->colorStart[c] = run;
        const uint32_t n = d.counters->colorCount[c];
        run += n;
        if (n > 0) used = c + 1;
    }
    d.counters->colorStart[MAX_COLORS] = run;
    d.counters->colorStart[MAX_COLORS + 1] = used;
    d.counters->usedColors = used;
}

__device__ __forceinline__ void color_place(const DevPtrs& d, uint32_t gid, const uint32_t* colors) {
    if (d.posLin[gid].w <= 0.0f) return;
    d.colorList[d.counters->colorStart[colors[gid]] + d.bodySlot[gid]] = gid;
}

constexpr int kColorPasses = 20;
constexpr int kColorLaunched = 8;                 // passes launched over the whole device
constexpr uint32_t kColorCluster = 10240;         // bodies up to which a cluster does everything,
constexpr uint32_t kColorLater = 32768;           // and up to which it does the passes not launched

// The whole coloring in one launch of a cluster (one CTA for small scenes):
// passes between barriers until one changes nothing, usually the first or
// second because a frame starts from the last frame's colors, then count, scan
// and place.  As 24 launches, most of which found nothing to do, it took 28 us
// of a 250 us frame of 20 bodies.  Where the contacts change in every frame it
// is four to ten passes, and a cluster's pass grows with the bodies: above
// kColorCluster the first kColorLaunched passes and the rest use the whole
// device, a launch each, and the cluster only goes on with later passes and the
// repair (`from` > 0, `all` = false).  Above kColorLater, where a pass of the
// cluster would cost as much as a dozen idle launches, every pass is launched
// (83 / 94 us at 40,000 / 60,000 shapes instead of 72 / 82).  Coloring stage,
// median of 60 frames, cluster / eight launched passes (24 launches): tumbling
// shapes 5,000 39 / 47 us (66), 8,000 45 / 51 (68), 12,000 64 / 53 (74), 28,000
// 111 / 61 (72), 60,000 217 / 82 (98); settled worlds of 8,398 bodies 25 / 27
// (47), 16,739 35 / 31 (51), 28,626 45 / 35 (55).
template <bool CLUSTER>
__global__ void __launch_bounds__(1024) k_color(const Params P, const DevPtrs d, int from, bool all) {
    pdl_prologue();
    const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    const volatile uint32_t* changed = d.counters->changed;
    auto barrier = [&]() {
        if (CLUSTER) {
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        } else {
            __syncthreads();
        }
    };
    for (int pass = from; pass < kColorPasses; pass++) {
        if (pass > 0 && changed[pass - 1] == 0u) break;          // the same in every thread
        const uint32_t* src = (pass & 1) ? d.colorsB : d.colorsA;
        uint32_t* dst = (pass & 1) ? d.colorsA : d.colorsB;
        for (uint32_t gid = first; gid < P.numBodies; gid += step) color_step(d, gid, src, dst, (uint32_t)pass);
        barrier();
    }
    if (changed[kColorPasses - 1] != 0u) {
        if (first == 0) color_repair(P, d, d.colorsA);
        barrier();
    }
    if (!all) return;
    for (uint32_t gid = first; gid < P.numBodies; gid += step) color_count(d, gid, d.colorsA);
    barrier();
    if (first == 0) color_scan(d);
    barrier();
    for (uint32_t gid = first; gid < P.numBodies; gid += step) color_place(d, gid, d.colorsA);
}

__global__ void k_color_iterate(const Params P, const DevPtrs d, const uint32_t* src, uint32_t* dst, uint32_t pass) {
    pdl_prologue();
    const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= P.numBodies) return;
    if (pass > 0 && d.counters->changed[pass - 1] == 0u) return;
    color_step(d, gid, src, dst, pass);
}
__global__ void k_color_validate_count(const Params P, const DevPtrs d, const uint32_t* colors) {
    pdl_prologue();
    const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid < P.numBodies) color_count(d, gid, colors);
}
__global__ void k_color_scan(const DevPtrs d) {
    pdl_prologue();
    if (threadIdx.x == 0) color_scan(d);
}
__global__ void k_color_scatter(const Params P, const DevPtrs d, const uint32_t* colors) {
    pdl_prologue();
    const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid < P.numBodies) color_place(d, gid, colors);
}

// one launch of a grid that is one cluster
template <typename... KArgs, typename... Args>
static void launch_cluster(void (*kernel)(KArgs...), uint32_t ctas, uint32_t threads, size_t smem, cudaStream_t st,
                           Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

void launch_dynamic_coloring(const Params& P, const DevPtrs& d, const Sizes& z, cudaStream_t st) {
    if (P.numBodies <= 1024u) { launch_cluster(k_color<false>, 1, 1024, 0, st, P, d, 0, true); return; }
    if (P.numBodies <= kColorCluster) {
        launch_cluster(k_color<true>, P.numBodies <= 4096u ? 4 : 8, 1024, 0, st, P, d, 0, true);
        return;
    }
    const uint32_t T = 128, blocks = (P.numBodies + T - 1) / T;
    const int launched = P.numBodies <= kColorLater ? kColorLaunched : kColorPasses;
    for (int pass = 0; pass < launched; pass++) {
        const uint32_t* src = (pass & 1) ? d.colorsB : d.colorsA;
        uint32_t* dst = (pass & 1) ? d.colorsA : d.colorsB;
        launch_pdl(k_color_iterate, blocks, T, st, P, d, src, dst, (uint32_t)pass);
    }
    launch_cluster(k_color<true>, 8, 1024, 0, st, P, d, launched, false);
    launch_pdl(k_color_validate_count, blocks, T, st, P, d, (const uint32_t*)d.colorsA);
    launch_pdl(k_color_scan, 1, 32, st, d);
    launch_pdl(k_color_scatter, blocks, T, st, P, d, (const uint32_t*)d.colorsA);
}

// ---------------------------------------------------------------------------
// Force stamps (40_solver.metal:733-1230)
// ---------------------------------------------------------------------------
struct Accum { M3 lhsLin, lhsAng, lhsCross; float3 rhsLin, rhsAng; };

__device__ __forceinline__ M3 geom_stiff_ball_socket(int k, float3 v) {
    M3 m = m3_diag(s3(-comp(v, k)));
    if (k == 0) { m.r0.x += v.x; m.r1.x += v.y; m.r2.x += v.z; }
    else if (k == 1) { m.r0.y += v.x; m.r1.y += v.y; m.r2.y += v.z; }
    else { m.r0.z += v.x; m.r1.z += v.y; m.r2.z += v.z; }
    return m;
}

// inlined in every caller: as a called function it would take Params and
// DevPtrs by address, and each thread of a caller would copy both (1.5 KB) to
// local memory first
__device__ __forceinline__ void stamp_joint(const Params& P, const DevPtrs& d, const JointGPU& j, uint32_t self,
                                            Accum& acc) {
    const uint32_t a = j.header.x, b = j.header.y;
    const bool isA = self == a;
    const float torqueArm = j.C0Lin.w;
    const float3 penLin = xyz(j.penaltyLin);
    const float4 qBb = d.posAng[b];
    if (dot(penLin, penLin) > 0.0f) {
        const float3 pA = a == WORLD_BODY ? xyz(j.rA) : xform(xyz(d.posLin[a]), d.posAng[a], xyz(j.rA));
        const float3 pB = xform(xyz(d.posLin[b]), qBb, xyz(j.rB));
        float3 C = pA - pB;
        if (j.header.w & 1) C -= xyz(j.C0Lin) * P.alpha;
        const float3 F = penLin * C + xyz(j.lambdaLin);
        const float jsign = isA ? 1.0f : -1.0f;
        const float3 rW = isA ? q_rotate(d.posAng[a], xyz(j.rA)) : q_rotate(qBb, xyz(j.rB));
        const M3 jAng = m3_skew(-jsign * rW);
        const M3 jAngT = m3_transpose(jAng);
        const M3 K = m3_diag(penLin);
        const M3 jAngTk = m3_mulm(jAngT, K);
        acc.lhsLin = m3_add(acc.lhsLin, K);
        acc.lhsAng = m3_add(acc.lhsAng, m3_mulm(jAngTk, jAng));
        acc.lhsCross = m3_add(acc.lhsCross, m3_scale(jAngTk, jsign));
        const float3 r = jsign * rW;
        const M3 H = m3_add(m3_add(m3_scale(geom_stiff_ball_socket(0, r), F.x),
                                   m3_scale(geom_stiff_ball_socket(1, r), F.y)),
                            m3_scale(geom_stiff_ball_socket(2, r), F.z));
        acc.lhsAng = m3_add(acc.lhsAng, m3_diagonalize(H));
        acc.rhsLin += jsign * F;
        acc.rhsAng += m3_mul(jAngT, F);
    }
    const float3 penAng = xyz(j.penaltyAng);
    if (dot(penAng, penAng) > 0.0f) {
        const float4 qA = a == WORLD_BODY ? make_float4(0, 0, 0, 1) : d.posAng[a];
        const float4 restRel = tof(j.restRel);
        float3 C = q_sub(q_mul(qA, restRel), qBb) * torqueArm;
        const float s = (isA ? 1.0f : -1.0f) * torqueArm;
        if (j.hingeAxis.w != 0.0f) {
            const float3 axis = xyz(j.hingeAxis);
            const float3 aB = q_rotate(qBb, axis);
            const float3 aA = q_rotate(q_mul(qA, restRel), axis);
            C = cross(aA, aB) * torqueArm;
            if (j.header.w & 2) C -= xyz(j.C0Ang) * P.alpha;
            const float3 F = penAng * C + xyz(j.lambdaAng);
            const float alignment = dot(aA, aB);
            M3 J = isA ? m3_add(m3_outer(aA, aB), m3_scale(m3_identity(), -alignment))
                       : m3_add(m3_scale(m3_identity(), alignment), m3_scale(m3_outer(aB, aA), -1.0f));
            J = m3_scale(J, torqueArm);
            const M3 JT = m3_transpose(J);
            const M3 K = m3_diag(penAng);
            acc.lhsAng = m3_add(acc.lhsAng, m3_mulm(m3_mulm(JT, K), J));
            acc.rhsAng += m3_mul(JT, F);
            if (j.motor.y > 0.0f || j.limits.x < j.limits.y) {
                const float twist = twist_angle(q_mul(qA, restRel), qBb, axis);
                if (j.dynamics.x > 0.0f) {
                    const float Ca = wrap_pi(twist - j.dynamics.y);
                    const float ka = j.dynamics.x / mx(P.dt * P.dt, 1e-12f);
                    const float sm = (self == a) ? -1.0f : 1.0f;
                    acc.lhsAng = m3_add(acc.lhsAng, m3_scale(m3_outer(aB, aB), ka));
                    acc.rhsAng += aB * (ka * Ca * sm);
                }
                if (j.limits.x < j.limits.y) {
                    const float over = mx(twist - j.limits.y, 0.0f) + mn(twist - j.limits.x, 0.0f);
                    if (over != 0.0f) {
                        const float kL = 4.0e4f;
                        const float FL = clampf(kL * over, -3000.0f, 3000.0f);
                        const float sm = (self == a) ? -1.0f : 1.0f;
                        acc.lhsAng = m3_add(acc.lhsAng, m3_scale(m3_outer(aB, aB), kL));
                        acc.rhsAng += aB * (FL * sm);
                    }
                }
                if (j.motor.y > 0.0f) {
                    const float sm = (self == a) ? -1.0f : 1.0f;
                    const uint32_t mode = j.header.w & MOTOR_MODE_MASK;
                    if (mode == MOTOR_EXPLICIT || mode == MOTOR_VELOCITY) {
                        acc.rhsAng += aB * (-j.dynamics.z * sm);
                    } else {
                        const float Cm = wrap_pi(twist - j.motor.x);
                        const float4 qA0 = a == WORLD_BODY ? make_float4(0, 0, 0, 1) : d.initAng[a];
                        const float twist0 = twist_angle(q_mul(qA0, restRel), d.initAng[b], axis);
                        const float dTwist = wrap_pi(twist - twist0);
                        const float cD = j.limits.z / mx(P.dt, 1e-6f);
                        const float raw = j.motor.w * Cm + cD * dTwist;
                        const float effort = clampf(raw, -j.motor.y, j.motor.y);
                        if (fabsf(raw) < j.motor.y)
                            acc.lhsAng = m3_add(acc.lhsAng, m3_scale(m3_outer(aB, aB), j.motor.w + cD));
                        acc.rhsAng += aB * (effort * sm);
                    }
                }
            }
        } else {
            if (j.header.w & 2) C -= xyz(j.C0Ang) * P.alpha;
            const float3 F = penAng * C + xyz(j.lambdaAng);
            acc.lhsAng = m3_add(acc.lhsAng, m3_diag(penAng * (s * s)));
            acc.rhsAng += F * s;
        }
    }
}

__device__ void stamp_spring(const Params& P, const DevPtrs& d, const SpringGPU& sp, uint32_t self, Accum& acc) {
    const uint32_t a = sp.header.x, b = sp.header.y;
    float stiffness = sp.rA.w;
    const float rest = sp.rB.w;
    const float3 pA = xform(xyz(d.posLin[a]), d.posAng[a], xyz(sp.rA));
    const float3 pB = xform(xyz(d.posLin[b]), d.posAng[b], xyz(sp.rB));
    const float3 dd = pA - pB;
    const float dLen = len3(dd);
    if (dLen <= 1.0e-6f) return;
    const float3 n = dd / dLen;
    float f;
    if (sp.header.z != 0) {
        const float C = dLen - rest - sp.dual.z * P.alpha;
        stiffness = sp.dual.y;
        f = stiffness * C + sp.dual.x;
        if (f <= 0.0f) return;
    } else {
        f = stiffness * (dLen - rest);
    }
    const bool isA = self == a;
    const float3 rW = isA ? q_rotate(d.posAng[a], xyz(sp.rA)) : q_rotate(d.posAng[b], xyz(sp.rB));
    const float3 jLin = isA ? n : -n;
    const float3 jAng = isA ? cross(rW, n) : -cross(rW, n);
    acc.lhsLin = m3_add(acc.lhsLin, m3_scale(m3_outer(jLin, jLin), stiffness));
    acc.lhsAng = m3_add(acc.lhsAng, m3_scale(m3_outer(jAng, jAng), stiffness));
    acc.lhsCross = m3_add(acc.lhsCross, m3_scale(m3_outer(jAng, jLin), stiffness));
    acc.rhsLin += jLin * f;
    acc.rhsAng += jAng * f;
    const float ft = mx(f, 0.0f) / dLen;
    if (ft > 0.0f) acc.lhsLin = m3_add(acc.lhsLin, m3_add(m3_diag(s3(ft)), m3_scale(m3_outer(n, n), -ft)));
}

// Stable Neo-Hookean tet, VBD per-vertex Hessian (40_solver.metal:966-1020).
__device__ void stamp_tet(const DevPtrs& d, const TetGPU& t, uint32_t self, Accum& acc) {
    const float3 x0 = xyz(d.posLin[t.ids.x]), x1 = xyz(d.posLin[t.ids.y]);
    const float3 x2 = xyz(d.posLin[t.ids.z]), x3 = xyz(d.posLin[t.ids.w]);
    const float muV = t.r1.w, lamV = t.r2.w;
    const float alphaT = 1.0f + muV / mx(lamV, 1e-9f);
    const float3 d0 = x1 - x0, d1 = x2 - x0, d2 = x3 - x0;
    const float3 m0 = xyz(t.r0), m1 = xyz(t.r1), m2 = xyz(t.r2);
    const float3 f0 = d0 * m0.x + d1 * m1.x + d2 * m2.x;
    const float3 f1 = d0 * m0.y + d1 * m1.y + d2 * m2.y;
    const float3 f2 = d0 * m0.z + d1 * m1.z + d2 * m2.z;
    const float J = dot(f0, cross(f1, f2));
    const float3 j0 = cross(f1, f2), j1 = cross(f2, f0), j2 = cross(f0, f1);
    const float s2 = lamV * (J - alphaT);
    const float3 p0 = muV * f0 + s2 * j0;
    const float3 p1 = muV * f1 + s2 * j1;
    const float3 p2 = muV * f2 + s2 * j2;
    float3 w;
    if (self == t.ids.y) w = m0;
    else if (self == t.ids.z) w = m1;
    else if (self == t.ids.w) w = m2;
    else w = -mk3(m0.x + m1.x + m2.x, m0.y + m1.y + m2.y, m0.z + m1.z + m2.z);
    const float3 grad = p0 * w.x + p1 * w.y + p2 * w.z;
    const float3 g = j0 * w.x + j1 * w.y + j2 * w.z;
    acc.rhsLin += grad;
    acc.lhsLin = m3_add(acc.lhsLin, m3_diag(s3(muV * dot(w, w))));
    acc.lhsLin = m3_add(acc.lhsLin, m3_scale(m3_outer(g, g), lamV));
}

// Linearised contact constraint and its cone-projected force.
__device__ __forceinline__ float3 contact_force(const ContactGPU& c, float3 nrm, float3 t1, float3 t2,
                                                float dynF, float statF, float alpha,
                                                float3 dqALin, float3 dqAAng, float3 dqBLin, float3 dqBAng,
                                                float3 rAW, float3 rBW, float3& Cout, float& fs, float& bounds) {
    float3 C = xyz(c.C0) * (1.0f - alpha);
    C += mk3(dot(nrm, dqALin), dot(t1, dqALin), dot(t2, dqALin));
    C -= mk3(dot(nrm, dqBLin), dot(t1, dqBLin), dot(t2, dqBLin));
    C += mk3(dot(cross(rAW, nrm), dqAAng), dot(cross(rAW, t1), dqAAng), dot(cross(rAW, t2), dqAAng));
    C -= mk3(dot(cross(rBW, nrm), dqBAng), dot(cross(rBW, t1), dqBAng), dot(cross(rBW, t2), dqBAng));
    float3 F = xyz(c.penalty) * C + xyz(c.lambda);
    F.x = mn(F.x, 0.0f);
    bounds = fabsf(F.x) * statF;
    fs = sqrtf(F.y * F.y + F.z * F.z);
    if (fs > bounds && fs > 0.0f) {
        const float db = fabsf(F.x) * dynF;
        const float sc = db / fs;
        F.y *= sc;
        F.z *= sc;
    }
    Cout = C;
    return F;
}

// What one contact point (or one rigid element-contact slot) adds to a
// body's 6x6 system: each accumulator component takes exactly one add per
// point, so a point's increment can be formed anywhere and added later in
// the original order with the same result.  The solve reads the lower
// triangles of the two diagonal blocks only, so a stored increment keeps 27
// of the 33 floats.
struct PointInc { M3 lhsLin, lhsAng, lhsCross; float3 rhsLin, rhsAng; };
constexpr int kIncWords = 27;
__device__ __forceinline__ void add_inc(Accum& acc, const PointInc& x) {
    acc.lhsLin = m3_add(acc.lhsLin, x.lhsLin);
    acc.lhsAng = m3_add(acc.lhsAng, x.lhsAng);
    acc.lhsCross = m3_add(acc.lhsCross, x.lhsCross);
    acc.rhsLin += x.rhsLin;
    acc.rhsAng += x.rhsAng;
}
// the component-th float of a stored increment is `stride` floats after the one before
__device__ __forceinline__ void store_inc(float* at, int stride, const PointInc& x) {
    const float w[kIncWords] = {x.lhsLin.r0.x, x.lhsLin.r1.x, x.lhsLin.r1.y, x.lhsLin.r2.x, x.lhsLin.r2.y,
                                x.lhsLin.r2.z, x.lhsAng.r0.x, x.lhsAng.r1.x, x.lhsAng.r1.y, x.lhsAng.r2.x,
                                x.lhsAng.r2.y, x.lhsAng.r2.z, x.lhsCross.r0.x, x.lhsCross.r0.y, x.lhsCross.r0.z,
                                x.lhsCross.r1.x, x.lhsCross.r1.y, x.lhsCross.r1.z, x.lhsCross.r2.x, x.lhsCross.r2.y,
                                x.lhsCross.r2.z, x.rhsLin.x, x.rhsLin.y, x.rhsLin.z, x.rhsAng.x, x.rhsAng.y, x.rhsAng.z};
#pragma unroll
    for (int c = 0; c < kIncWords; c++) at[c * stride] = w[c];
}
__device__ __forceinline__ void add_stored_inc(Accum& acc, const float* at, int stride) {
    float w[kIncWords];
#pragma unroll
    for (int c = 0; c < kIncWords; c++) w[c] = at[c * stride];
    acc.lhsLin.r0.x += w[0]; acc.lhsLin.r1.x += w[1]; acc.lhsLin.r1.y += w[2];
    acc.lhsLin.r2.x += w[3]; acc.lhsLin.r2.y += w[4]; acc.lhsLin.r2.z += w[5];
    acc.lhsAng.r0.x += w[6]; acc.lhsAng.r1.x += w[7]; acc.lhsAng.r1.y += w[8];
    acc.lhsAng.r2.x += w[9]; acc.lhsAng.r2.y += w[10]; acc.lhsAng.r2.z += w[11];
    acc.lhsCross.r0 += mk3(w[12], w[13], w[14]);
    acc.lhsCross.r1 += mk3(w[15], w[16], w[17]);
    acc.lhsCross.r2 += mk3(w[18], w[19], w[20]);
    acc.rhsLin += mk3(w[21], w[22], w[23]);
    acc.rhsAng += mk3(w[24], w[25], w[26]);
}
// Jacobian-weighted increment of a contact frame with world lever rW.
__device__ __forceinline__ PointInc point_inc(const M3& jLin, float3 rW, const M3& K, float3 F) {
    const M3 jAng = M3{cross(rW, jLin.r0), cross(rW, jLin.r1), cross(rW, jLin.r2)};
    const M3 jLinT = m3_transpose(jLin), jAngT = m3_transpose(jAng);
    const M3 jAngTk = m3_mulm(jAngT, K);
    PointInc x;
    x.lhsLin = m3_mulm(m3_mulm(jLinT, K), jLin);
    x.lhsAng = m3_mulm(jAngTk, jAng);
    x.lhsCross = m3_mulm(jAngTk, jLin);
    x.rhsLin = m3_mul(jLinT, F);
    x.rhsAng = m3_mul(jAngT, F);
    return x;
}

// Pose data of a manifold's two bodies shared by its contact points.
struct ManifoldCtx {
    float4 qa, qb;
    float3 dqALin, dqAAng, dqBLin, dqBAng, nrm, t1, t2;
    float dynF, statF;
    bool isA, sphA, sphB;
};
__device__ __forceinline__ ManifoldCtx manifold_ctx(const DevPtrs& d, const ManifoldGPU& m, uint32_t self) {
    const u4 h = m.header;
    const uint32_t a = h.x, b = h.y;
    ManifoldCtx x;
    x.isA = self == a;
    x.sphA = (h.w & 2u) != 0;
    x.sphB = (h.w & 4u) != 0;
    x.qa = d.posAng[a];
    x.qb = d.posAng[b];
    x.dqALin = xyz(d.posLin[a]) - xyz(d.initLin[a]);
    x.dqAAng = q_sub(x.qa, d.initAng[a]);
    x.dqBLin = xyz(d.posLin[b]) - xyz(d.initLin[b]);
    x.dqBAng = q_sub(x.qb, d.initAng[b]);
    x.nrm = xyz(m.basisN);
    x.t1 = xyz(m.basisT1);
    x.t2 = cross(x.nrm, x.t1);
    x.dynF = m.basisN.w;
    x.statF = m.basisT1.w;
    return x;
}
// Increment of contact point i of a manifold.
__device__ __forceinline__ PointInc manifold_point_inc(const Params& P, const ManifoldCtx& x, const ContactGPU& c) {
    const float3 rAW = x.sphA ? xyz(c.rA) : q_rotate(x.qa, xyz(c.rA));
    const float3 rBW = x.sphB ? xyz(c.rB) : q_rotate(x.qb, xyz(c.rB));
    float3 C;
    float fs, bnd;
    const float3 F = contact_force(c, x.nrm, x.t1, x.t2, x.dynF, x.statF, P.alpha, x.dqALin, x.dqAAng, x.dqBLin,
                                   x.dqBAng, rAW, rBW, C, fs, bnd);
    const float s = x.isA ? 1.0f : -1.0f;
    const M3 jLin = M3{x.nrm * s, x.t1 * s, x.t2 * s};
    return point_inc(jLin, x.isA ? rAW : rBW, m3_diag(xyz(c.penalty)), F);
}

__device__ void stamp_manifold(const Params& P, const DevPtrs& d, const ManifoldGPU& m, uint32_t self, Accum& acc) {
    const uint32_t n = m.header.z;
    const ManifoldCtx x = manifold_ctx(d, m, self);
    for (uint32_t i = 0; i < n; i++) add_inc(acc, manifold_point_inc(P, x, m.contacts[i]));
}

// StVK membrane, Gauss-Newton Hessian (40_solver.metal:1088-1134).
__device__ void stamp_membrane(const DevPtrs& d, const MembraneGPU& mb, uint32_t self, Accum& acc) {
    const float3 x0 = xyz(d.posLin[mb.ids.x]), x1 = xyz(d.posLin[mb.ids.y]), x2 = xyz(d.posLin[mb.ids.z]);
    const float muA = mb.mat.x, lamA = mb.mat.y;
    const float3 d0 = x1 - x0, d1 = x2 - x0;
    const float a = mb.dm.x, b = mb.dm.y, c = mb.dm.z, dd = mb.dm.w;
    const float3 f1 = d0 * a + d1 * b;
    const float3 f2 = d0 * c + d1 * dd;
    const float E11 = 0.5f * (dot(f1, f1) - 1.0f);
    const float E22 = 0.5f * (dot(f2, f2) - 1.0f);
    const float E12 = 0.5f * dot(f1, f2);
    const float trE = E11 + E22;
    const float S11 = 2.0f * muA * E11 + lamA * trE;
    const float S22 = 2.0f * muA * E22 + lamA * trE;
    const float S12 = 2.0f * muA * E12;
    const float3 p1 = f1 * S11 + f2 * S12;
    const float3 p2 = f1 * S12 + f2 * S22;
    float wx, wy;
    if (self == mb.ids.y) { wx = a; wy = c; }
    else if (self == mb.ids.z) { wx = b; wy = dd; }
    else { wx = -a - b; wy = -c - dd; }
    acc.rhsLin += p1 * wx + p2 * wy;
    const float3 g11 = f1 * wx, g22 = f2 * wy;
    const float3 g12 = (f2 * wx + f1 * wy) * 0.5f;
    const float3 gtr = g11 + g22;
    acc.lhsLin = m3_add(acc.lhsLin, m3_scale(m3_outer(g11, g11), 2.0f * muA));
    acc.lhsLin = m3_add(acc.lhsLin, m3_scale(m3_outer(g22, g22), 2.0f * muA));
    acc.lhsLin = m3_add(acc.lhsLin, m3_scale(m3_outer(g12, g12), 4.0f * muA));
    acc.lhsLin = m3_add(acc.lhsLin, m3_scale(m3_outer(gtr, gtr), lamA));
}

// Quadratic (Bergou) bending, rank-1 isotropic Hessian (40_solver.metal:1136-1153).
__device__ void stamp_bend(const DevPtrs& d, const BendGPU& bd, uint32_t self, Accum& acc) {
    const float sc = bd.mat.x;
    const float3 m = xyz(d.posLin[bd.ids.x]) * bd.K.x + xyz(d.posLin[bd.ids.y]) * bd.K.y +
                     xyz(d.posLin[bd.ids.z]) * bd.K.z + xyz(d.posLin[bd.ids.w]) * bd.K.w;
    float k;
    if (self == bd.ids.x) k = bd.K.x;
    else if (self == bd.ids.y) k = bd.K.y;
    else if (self == bd.ids.z) k = bd.K.z;
    else k = bd.K.w;
    acc.rhsLin += m * (sc * k);
    acc.lhsLin = m3_add(acc.lhsLin, m3_diag(s3(sc * k * k)));
}

// Element-contact constraint over the 4-slot stencil (40_solver.metal:1236-1263).
__device__ float3 soft_c(const Params& P, const DevPtrs& d, const SoftContactGPU& sc, float3& n, float3& t1,
                         float3& t2, float3& rAW, bool& rigidA) {
    const uint32_t flags = __float_as_uint(sc.anchorA.w);
    rigidA = (flags & SCF_RIGID_A) != 0;
    const bool roundA = (flags & SCF_ROUND_A) != 0;
    n = xyz(sc.normal);
    orthonormal(n, t1, t2);
    rAW = s3(0);
    float3 C = xyz(sc.C0) * (1.0f - P.alpha);
    const uint32_t ids[4] = {sc.ids.x, sc.ids.y, sc.ids.z, sc.ids.w};
    const float ws[4] = {sc.weights.x, sc.weights.y, sc.weights.z, sc.weights.w};
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint32_t b = ids[k];
        if (b == WORLD_BODY) continue;
        const float w = ws[k];
        const float3 dq = xyz(d.posLin[b]) - xyz(d.initLin[b]);
        C += mk3(dot(n, dq), dot(t1, dq), dot(t2, dq)) * w;
        if (k == 0 && rigidA) {
            const float4 q = d.posAng[b];
            rAW = roundA ? xyz(sc.anchorA) : q_rotate(q, xyz(sc.anchorA));
            const float3 dqa = q_sub(q, d.initAng[b]);
            C += mk3(dot(cross(rAW, n), dqa), dot(cross(rAW, t1), dqa), dot(cross(rAW, t2), dqa)) * w;
        }
    }
    return C;
}

// softContactForce with the two-stage barrier (40_solver.metal:1265-1359):
// the force, the normal stiffness and the frame of an element contact, and
// which of its four slots `self` is (-1: none) with that slot's weight.
struct SoftForce { float3 n, t1, t2, rAW, F; float kN, w; int slot; bool rigidA; };
__device__ __forceinline__ SoftForce soft_force(const Params& P, const DevPtrs& d, const SoftContactGPU& sc,
                                                uint32_t self) {
    SoftForce r;
    const float3 C = soft_c(P, d, sc, r.n, r.t1, r.t2, r.rAW, r.rigidA);
    float3 F = xyz(sc.penalty) * C + xyz(sc.lambda);
    float kN = sc.penalty.x;
    const float rT = sc.anchorA.x;
    const uint32_t kindB = (__float_as_uint(sc.anchorA.w) >> SCF_KIND_SHIFT) & 3u;
    if (rT > 0.0f && kindB != SC_RT && C.x < -0.5f * rT) {
        const float dsep = mx(C.x + rT, 0.02f * rT);
        const float kp = 0.25f * rT * rT * sc.penalty.x;
        F.x = -kp / dsep + sc.lambda.x;
        kN = kp / (dsep * dsep);
    }
    F.x = mn(F.x, 0.0f);
    const float bounds = fabsf(F.x) * sc.normal.w;
    const float fs = sqrtf(F.y * F.y + F.z * F.z);
    if (fs > bounds && fs > 0.0f) {
        const float q = bounds / fs;
        F.y *= q;
        F.z *= q;
    }
    r.F = F;
    r.kN = kN;
    r.slot = -1;
    if (sc.ids.x == self) r.slot = 0;
    else if (sc.ids.y == self) r.slot = 1;
    else if (sc.ids.z == self) r.slot = 2;
    else if (sc.ids.w == self) r.slot = 3;
    r.w = r.slot == 0 ? sc.weights.x : (r.slot == 1 ? sc.weights.y : (r.slot == 2 ? sc.weights.z : sc.weights.w));
    return r;
}
// Increment of the rigid slot 0 of an element contact (stampSoft's 6-DOF branch).
__device__ __forceinline__ PointInc soft_rigid_inc(const SoftContactGPU& sc, const SoftForce& f) {
    const float w = f.w;
    return point_inc(M3{f.n * w, f.t1 * w, f.t2 * w}, f.rAW, m3_diag(mk3(f.kN, sc.penalty.y, sc.penalty.z)), f.F);
}

// stampSoft (40_solver.metal:1265-1359).
__device__ void stamp_soft(const Params& P, const DevPtrs& d, const SoftContactGPU& sc, uint32_t self, Accum& acc) {
    const SoftForce f = soft_force(P, d, sc, self);
    if (f.slot < 0) return;
    if (f.slot == 0 && f.rigidA) {
        add_inc(acc, soft_rigid_inc(sc, f));
    } else {
        const float w2 = f.w * f.w;
        acc.lhsLin = m3_add(acc.lhsLin, m3_scale(m3_outer(f.n, f.n), f.kN * w2));
        acc.lhsLin = m3_add(acc.lhsLin, m3_scale(m3_outer(f.t1, f.t1), sc.penalty.y * w2));
        acc.lhsLin = m3_add(acc.lhsLin, m3_scale(m3_outer(f.t2, f.t2), sc.penalty.z * w2));
        acc.rhsLin += (f.n * f.F.x + f.t1 * f.F.y + f.t2 * f.F.z) * f.w;
    }
}

template <bool MANIFOLDS = true>
__device__ __forceinline__ void stamp_entry(const Params& P, const DevPtrs& d, uint32_t entry, uint32_t body,
                                            Accum& acc) {
    const uint32_t kind = entry >> ADJ_KIND_SHIFT, idx = entry & ADJ_INDEX_MASK;
    if (kind == FK_TET) stamp_tet(d, d.tets[idx], body, acc);
    else if (MANIFOLDS && kind == FK_MANIFOLD) stamp_manifold(P, d, d.manifolds[idx], body, acc);
    else if (kind == FK_JOINT) stamp_joint(P, d, d.joints[idx], body, acc);
    else if (kind == FK_SPRING) stamp_spring(P, d, d.springs[idx], body, acc);
    else if (kind == FK_SOFT) stamp_soft(P, d, d.soft[idx], body, acc);
    else if (kind == FK_MEMBRANE) stamp_membrane(d, d.membranes[idx], body, acc);
    else if (kind == FK_BEND) stamp_bend(d, d.bends[idx], body, acc);
}

__device__ __forceinline__ float3 shfl3(unsigned mask, float3 v, int o) {
    return mk3(__shfl_xor_sync(mask, v.x, o, 8), __shfl_xor_sync(mask, v.y, o, 8), __shfl_xor_sync(mask, v.z, o, 8));
}
__device__ __forceinline__ void add_shfl3(unsigned mask, float3& v, int o) { v = v + shfl3(mask, v, o); }
// the lower triangle of a diagonal block: all that the solves read (what no
// lane sends is not computed either)
__device__ __forceinline__ void add_shfl_lower(unsigned mask, M3& m, int o) {
    m.r0.x += __shfl_xor_sync(mask, m.r0.x, o, 8);
    m.r1.x += __shfl_xor_sync(mask, m.r1.x, o, 8);
    m.r1.y += __shfl_xor_sync(mask, m.r1.y, o, 8);
    add_shfl3(mask, m.r2, o);
}

// Isotropic-OGC conservative-bound truncation (ogcTruncate,
// 40_solver.metal:1361-1382): the displacement since the bound's anchor stays
// within max(0.45 * bound distance, 0.2 * radius); every clamped step is
// counted for the mid-solve refresh.
// d2: the body's squared bound distance; anchor: where the bound was taken.
__device__ __forceinline__ float3 ogc_truncate(const DevPtrs& d, float d2, float4 anchor, float3 dxLin, float3 cur,
                                               float partR) {
    if (d2 >= 1e37f) return dxLin;
    const float bv = mx(0.45f * sqrtf(d2), 0.2f * partR);
    const float3 x0 = xyz(anchor);
    float3 tot = (cur + dxLin) - x0;
    const float t2 = dot(tot, tot);
    if (t2 > bv * bv) {
        tot *= bv * rsq(t2);
        dxLin = (x0 + tot) - cur;
        atomicAdd(d.ogcExceed, 1u);
    }
    return dxLin;
}

// A skipped update (non-finite step) still publishes the unchanged pose
// when the color commits through posNext.
__device__ __forceinline__ void keep_body(const Params& P, const DevPtrs& d, uint32_t body, float4 pl, bool rigid) {
    if (!P.colorJacobi) return;
    d.posNext[body] = pl;
    if (rigid) d.angNext[body] = d.posAng[body];
}

// The 8 lanes' partial systems of one body (lane l stamped entries l,
// l + 8, ...) folded by an xor butterfly; lane 0 solves and writes.
__device__ __forceinline__ void body_commit(const Params& P, const DevPtrs& d, uint32_t body, float4 shp,
                                            uint32_t lane, unsigned mask, Accum acc) {
    const bool rigid = shp.w >= 0.0f;
#pragma unroll
    for (int o = 4; o >= 1; o >>= 1) {
        add_shfl_lower(mask, acc.lhsLin, o);
        add_shfl3(mask, acc.rhsLin, o);
        if (rigid) {
            add_shfl_lower(mask, acc.lhsAng, o);
            add_shfl3(mask, acc.lhsCross.r0, o);
            add_shfl3(mask, acc.lhsCross.r1, o);
            add_shfl3(mask, acc.lhsCross.r2, o);
            add_shfl3(mask, acc.rhsAng, o);
        }
    }
    if (lane != 0) return;
    const float4 pl = d.posLin[body];
    const float mass = pl.w;
    const float dt2 = P.dt * P.dt;
    acc.lhsLin = m3_add(acc.lhsLin, m3_diag(s3(mass / dt2)));
    acc.rhsLin += (xyz(pl) - xyz(d.inertLin[body])) * (mass / dt2);
    float3 dxLin = s3(0), dxAng = s3(0);
    if (rigid) {
        const float4 q = d.posAng[body];
        const M3 inertia = m3_scale(world_inertia(q, xyz(d.props[body])), 1.0f / dt2);
        acc.lhsAng = m3_add(acc.lhsAng, inertia);
        acc.rhsAng += m3_mul(inertia, q_sub(q, d.inertAng[body]));
        solve6x6(acc.lhsLin, acc.lhsAng, acc.lhsCross, -acc.rhsLin, -acc.rhsAng, dxLin, dxAng);
        if (!finite3(dxLin) || !finite3(dxAng)) { keep_body(P, d, body, pl, rigid); return; }
        const float ang2 = dot(dxAng, dxAng);
        const float maxAng = 0.5f;
        if (ang2 > maxAng * maxAng) dxAng *= maxAng * rsq(ang2);
    } else {
        solve6x6(acc.lhsLin, m3_identity(), m3_zero(), -acc.rhsLin, s3(0), dxLin, dxAng);
        if (!finite3(dxLin)) { keep_body(P, d, body, pl, rigid); return; }
    }
    const float maxLin = 0.35f * fabsf(shp.w);
    const float lin2 = dot(dxLin, dxLin);
    if (lin2 > maxLin * maxLin) dxLin *= maxLin * rsq(lin2);
    if (!rigid && P.ogc)
        dxLin = ogc_truncate(d, __uint_as_float(d.ogcBounds[body]), d.ogcPrev[body], dxLin, xyz(pl), -shp.w);
    if (P.colorJacobi) {
        d.posNext[body] = mk4(xyz(pl) + dxLin, mass);
        if (rigid) d.angNext[body] = q_addw(d.posAng[body], dxAng);
        return;
    }
    d.posLin[body] = mk4(xyz(pl) + dxLin, mass);
    if (rigid) d.posAng[body] = q_addw(d.posAng[body], dxAng);
}

// One body on an 8-lane group; lane 0 writes the result.  Logical lane l adds
// the entries l, l + 8, ... in order, as the reference's SIMD group does, but a
// manifold's contact points are not evaluated by the lane that adds them: the
// points of eight consecutive entries are dealt out to the group's lanes, eight
// at a time, and their increments pass through shared memory (`slots`: this
// group's column of `stride` columns).  A box resting on the ground has one
// manifold of four points among its entries; one lane used to form the four
// increments one after another while seven waited.
__device__ __forceinline__ void primal_body(const Params& P, const DevPtrs& d, uint32_t body, uint32_t lane, unsigned mask,
                            float* slots, int stride) {
    const float4 shp = d.shape[body];
    Accum acc{m3_zero(), m3_zero(), m3_zero(), s3(0), s3(0)};
    const AdjView v = adj_view(d, body);
    const uint32_t cnt = v.count();
    for (uint32_t base = 0; base < cnt; base += 8) {
        uint32_t entry = 0, np = 0;
        if (base + lane < cnt) {
            entry = v.at(base + lane);
            if ((entry >> ADJ_KIND_SHIFT) == FK_MANIFOLD) np = d.manifolds[entry & ADJ_INDEX_MASK].header.z;
            else stamp_entry<false>(P, d, entry, body, acc);
        }
        uint32_t end = np;                                   // points of this and the lower lanes' entries
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const uint32_t y = __shfl_up_sync(mask, end, o, 8);
            if ((int)lane >= o) end += y;
        }
        const uint32_t total = __shfl_sync(mask, end, 7, 8), begin = end - np;
        for (uint32_t c0 = 0; c0 < total; c0 += 8) {
            const uint32_t i = c0 + lane;
            uint32_t owner = 0;                              // the lane whose entry holds point i
#pragma unroll
            for (int j = 0; j < 7; j++) owner += __shfl_sync(mask, end, j, 8) <= i ? 1u : 0u;
            const uint32_t e = __shfl_sync(mask, entry, (int)owner, 8), first = __shfl_sync(mask, begin, (int)owner, 8);
            if (i < total) {
                const ManifoldGPU& m = d.manifolds[e & ADJ_INDEX_MASK];
                store_inc(slots + lane, stride, manifold_point_inc(P, manifold_ctx(d, m, body), m.contacts[i - first]));
            }
            __syncwarp(mask);
            const uint32_t last = min(end, c0 + 8);
            for (uint32_t k = max(begin, c0); k < last; k++) add_stored_inc(acc, slots + (k - c0), stride);
            __syncwarp(mask);
        }
    }
    body_commit(P, d, body, shp, lane, mask, acc);
}

// Dynamic coloring: the frame graph launches colors [0, bound) one by one, with
// a bound fitted to the frames retired so far.  A frame that needs more colors
// solves the rest in the launch of the last of them (`last`): its blocks take
// chunks of bodies, color after color, from a ticket counter, and a chunk waits
// until every chunk of the colors before it is finished.  Those have smaller
// tickets, so running blocks hold them and no wait depends on a block that has
// not started.  Boxes that land in pairs after the bound was fitted to one color,
// six iterations a frame, 600 / 4,096 / 60,000 of them: 0.28 / 0.33 / 1.13 ms a
// frame until the next retirement refits the bound (1.13 / 6.7 / 99.7 with the
// last block to finish taking all that is left; 0.37 / 0.44 / 1.32 with two more
// launches than colors seen).
constexpr int kPrimalThreads = 128;         // most threads of a k_primal block
constexpr uint64_t kTailWaitNs = 1000000000ull;   // a wait gives up after one second

// true once `finished` has reached `target`; false when it does not within the
// limit (the failure is latched, unless another one already is) or a wait has
// given up before
__device__ __forceinline__ bool tail_wait(const DevPtrs& d, const volatile uint32_t* finished, uint32_t target) {
    const volatile uint32_t* failed = d.failureLatch;
    uint64_t t0 = 0;
    for (uint32_t i = 0; *finished < target; i++) {
        if ((i & 63u) != 63u) continue;
        uint64_t t;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
        if (t0 == 0) t0 = t;
        if (t - t0 > kTailWaitNs) {
            atomicCAS(d.failureLatch, 0u, AVBD_FAIL_WAIT_TIMEOUT_);
            return false;
        }
        if (*failed == AVBD_FAIL_WAIT_TIMEOUT_) return false;
    }
    return true;
}

__global__ void __launch_bounds__(kPrimalThreads, 4) k_primal(const Params P, const DevPtrs d, uint32_t color,
                                                           uint32_t last) {
    __shared__ float slots[kIncWords * kPrimalThreads];
    __shared__ uint32_t ticket;
    pdl_prologue();
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t lane = tid & 7u, groups = blockDim.x >> 3;
    const unsigned mask = 0xFFu << (threadIdx.x & 24u);
    const uint32_t used = d.colorStart[MAX_COLORS + 1];
    const bool tail = last && color + 1u < used;
    // one 8-lane group per body, striding over the color (uniform across
    // the group)
    uint32_t slot = d.colorStart[color] + (tid >> 3), end = d.colorStart[color + 1], step = groups * gridDim.x;
    uint32_t c = color, before = 0;              // chunks of the colors color .. c - 1
    bool waits = true;                           // thread 0: no wait of this block has given up
    for (;;) {
        if (tail) {
            if (threadIdx.x == 0) ticket = atomicAdd(d.tail, 1u);
            __syncthreads();
            for (; c < used; c++) {
                const uint32_t chunks = (d.colorStart[c + 1] - d.colorStart[c] + groups - 1u) / groups;
                if (ticket < before + chunks) break;
                before += chunks;
            }
            if (c == used) break;
            if (before && threadIdx.x == 0) {
                waits = waits && tail_wait(d, d.tail + 1, before);
                __threadfence();
            }
            __syncthreads();
            slot = d.colorStart[c] + (ticket - before) * groups + (threadIdx.x >> 3);
            end = d.colorStart[c + 1];
            step = 0xFFFFFFFFu - slot;           // one body a group
        }
        for (; slot < end; slot += step)
            primal_body(P, d, d.colorList[slot], lane, mask, slots + (threadIdx.x & ~7u), kPrimalThreads);
        if (!tail) return;
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) atomicAdd(d.tail + 1, 1u);
    }
    // the last block to leave clears the counters for the next launch
    if (threadIdx.x == 0 && atomicAdd(d.tail + 2, 1u) == gridDim.x - 1u) d.tail[0] = d.tail[1] = d.tail[2] = 0u;
}

// ---------------------------------------------------------------------------
// Wide primal: one block per body, for a static color's non-lean bodies
// (rigid bodies and particles with joints).  A rigid body under a pile of
// particles carries hundreds of contact entries; on an 8-lane group its
// lanes would stamp them one after another while the rest of the color has
// long finished.  Here the block evaluates the contact points of every
// manifold entry and every rigid element-contact slot at once into shared
// memory, then 8 lanes add them in the 8-lane order (lane l: entries l,
// l + 8, ...; each entry's points in order) — every accumulator component
// takes one add per point, so the sums are those of the sequential stamps.
// Other entries, and points past the staging capacity, are stamped inline
// by the folding lanes in the same order.
// ---------------------------------------------------------------------------
constexpr int kWideThreads = 128;
constexpr int kWideEntries = 512;          // entries whose points may be staged
constexpr int kWidePoints = 320;           // staged points
constexpr uint32_t kWideInline = 0xFFFFFFFFu;

__global__ void __launch_bounds__(kWideThreads) k_primal_wide(const Params P, const DevPtrs d, uint32_t color,
                                                             uint32_t first, uint32_t start) {
    __shared__ float pts[kIncWords * kWidePoints];
    __shared__ uint32_t entOff[kWideEntries];  // (first point << 8) | points, or kWideInline
    __shared__ uint32_t warpSums[kWideThreads / 32];
    pdl_trigger();
    const uint32_t tid = threadIdx.x, lane32 = tid & 31u, warp = tid >> 5;
    // with the start known on the host, the static data (launch order,
    // shape, static segment) is read before waiting for the previous grid
    if (start == NO_HOST_START) pdl_wait();
    const uint32_t body = d.colorLaunch[(start == NO_HOST_START ? d.colorStart[color] : start) + first + blockIdx.x];
    const float4 shp = d.shape[body];
    const uint4 seg = d.staticSeg[body];
    const uint32_t nTet = d.postTets[body];
    if (start != NO_HOST_START) pdl_wait();
    const AdjView v = adj_view_from(d, body, seg, nTet);
    const uint32_t cnt = v.count();
    const uint32_t staged = min(cnt, (uint32_t)kWideEntries);
    uint32_t base = 0;                          // points taken by earlier chunks
    for (uint32_t c0 = 0; c0 < staged; c0 += kWideThreads) {
        const uint32_t k = c0 + tid;
        uint32_t entry = 0, np = 0;
        if (k < staged) {
            entry = v.at(k);
            const uint32_t kind = entry >> ADJ_KIND_SHIFT, idx = entry & ADJ_INDEX_MASK;
            if (kind == FK_MANIFOLD) {
                np = d.manifolds[idx].header.z;
            } else if (kind == FK_SOFT) {
                const SoftContactGPU& sc = d.soft[idx];
                const bool rigidA = (__float_as_uint(sc.anchorA.w) & SCF_RIGID_A) != 0;
                np = (rigidA && sc.ids.x == body) ? 1u : 0u;
            }
        }
        // exclusive scan of the chunk's point counts
        uint32_t incl = np;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)lane32 >= o) incl += y;
        }
        if (lane32 == 31) warpSums[warp] = incl;
        __syncthreads();
        uint32_t before = base, total = 0;
#pragma unroll
        for (int w = 0; w < kWideThreads / 32; w++) {
            const uint32_t ws = warpSums[w];
            if (w < (int)warp) before += ws;
            total += ws;
        }
        const uint32_t off = before + incl - np;
        const bool fits = np > 0 && off + np <= (uint32_t)kWidePoints;
        if (k < staged) entOff[k] = fits ? ((off << 8) | np) : kWideInline;
        if (fits) {
            const uint32_t kind = entry >> ADJ_KIND_SHIFT, idx = entry & ADJ_INDEX_MASK;
            if (kind == FK_MANIFOLD) {
                const ManifoldGPU& m = d.manifolds[idx];
                const ManifoldCtx x = manifold_ctx(d, m, body);
                for (uint32_t i = 0; i < np; i++) store_inc(pts + off + i, kWidePoints, manifold_point_inc(P, x, m.contacts[i]));
            } else {
                const SoftContactGPU& sc = d.soft[idx];
                store_inc(pts + off, kWidePoints, soft_rigid_inc(sc, soft_force(P, d, sc, body)));
            }
        }
        base += total;
        __syncthreads();                        // warpSums is reused by the next chunk
    }
    if (tid >= 8) return;
    Accum acc{m3_zero(), m3_zero(), m3_zero(), s3(0), s3(0)};
    for (uint32_t k = tid; k < cnt; k += 8) {
        const uint32_t eo = k < (uint32_t)kWideEntries ? entOff[k] : kWideInline;
        if (eo != kWideInline) {
            const uint32_t off = eo >> 8, np = eo & 0xFFu;
            for (uint32_t i = 0; i < np; i++) add_stored_inc(acc, pts + off + i, kWidePoints);
        } else {
            stamp_entry(P, d, v.at(k), body, acc);
        }
    }
    body_commit(P, d, body, shp, tid, 0xFFu, acc);
}

void launch_primal_wide(const Params& P, const DevPtrs& d, uint32_t color, uint32_t count, uint32_t first,
                        uint32_t start, cudaStream_t st) {
    if (count) launch_pdl(k_primal_wide, count, kWideThreads, st, P, d, color, first, start);
}

// ---------------------------------------------------------------------------
// Residual of the augmented-Lagrangian objective: the primal right-hand side
// of every dynamic body (inertia + every stamped force) at the current pose,
// squared and summed.  The square root is r_k of the iterations-to-tolerance
// measurement.  Bodies come from the color lists (every dynamic body once).
// ---------------------------------------------------------------------------
// Squared AL gradient of one rigid body (linear and angular parts) by an
// 8-lane group: lanes stamp entries lane, lane + 8, ..., an xor butterfly
// folds them and lane 0 writes *out.
__device__ __forceinline__ void rigid_residual(const Params& P, const DevPtrs& d, uint32_t body, uint32_t lane,
                                               unsigned mask, float* out) {
    // only the right-hand sides are kept, so a contact point's blocks are not formed
    Accum acc{m3_zero(), m3_zero(), m3_zero(), s3(0), s3(0)};
    float3 rhsLin = s3(0), rhsAng = s3(0);
    const AdjView v = adj_view(d, body);
    const uint32_t cnt = v.count();
    for (uint32_t k = lane; k < cnt; k += 8) {
        const uint32_t entry = v.at(k);
        if ((entry >> ADJ_KIND_SHIFT) == FK_MANIFOLD) {
            const ManifoldGPU& m = d.manifolds[entry & ADJ_INDEX_MASK];
            const uint32_t n = m.header.z;
            const ManifoldCtx x = manifold_ctx(d, m, body);
            for (uint32_t i = 0; i < n; i++) {
                const PointInc inc = manifold_point_inc(P, x, m.contacts[i]);
                rhsLin += inc.rhsLin;
                rhsAng += inc.rhsAng;
            }
        } else {
            Accum one{m3_zero(), m3_zero(), m3_zero(), rhsLin, rhsAng};
            stamp_entry<false>(P, d, entry, body, one);
            rhsLin = one.rhsLin;
            rhsAng = one.rhsAng;
        }
    }
    acc.rhsLin = rhsLin;
    acc.rhsAng = rhsAng;
#pragma unroll
    for (int o = 4; o >= 1; o >>= 1) {
        add_shfl3(mask, acc.rhsLin, o);
        add_shfl3(mask, acc.rhsAng, o);
    }
    if (lane != 0) return;
    const float4 pl = d.posLin[body];
    const float dt2 = P.dt * P.dt;
    const float3 rl = acc.rhsLin + (xyz(pl) - xyz(d.inertLin[body])) * (pl.w / dt2);
    const float4 q = d.posAng[body];
    const M3 inertia = m3_scale(world_inertia(q, xyz(d.props[body])), 1.0f / dt2);
    const float3 ra = acc.rhsAng + m3_mul(inertia, q_sub(q, d.inertAng[body]));
    *out = dot(rl, rl) + dot(ra, ra);
}

// Fixed-order sum of n values in one block (double accumulation): thread t
// sums the float4 groups t, t + 1024, ... (16-byte coalesced loads; v is a
// device allocation, so 16-byte aligned), then tail element 4 * (n / 4) + t;
// a warp shuffle tree and a second tree over the warps combine the threads,
// always in the same order.
__global__ void __launch_bounds__(1024) k_sum_fixed(const float* v, uint32_t n, double* out) {
    pdl_prologue();
    __shared__ double part[32];
    const uint32_t t = threadIdx.x, n4 = n / 4u;
    const float4* v4 = reinterpret_cast<const float4*>(v);
    double s = 0.0;
    for (uint32_t i = t; i < n4; i += blockDim.x) {
        const float4 q = v4[i];
        s += (double)q.x;
        s += (double)q.y;
        s += (double)q.z;
        s += (double)q.w;
    }
    if (4u * n4 + t < n) s += (double)v[4u * n4 + t];
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((t & 31u) == 0) part[t >> 5] = s;
    __syncthreads();
    if (t < 32) {
        s = t < (blockDim.x >> 5) ? part[t] : 0.0;
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (t == 0) *out = s;
    }
}


// ---------------------------------------------------------------------------
// Warp-per-body primal for particles.  The 8-lane kernel above makes each
// lane walk 2-3 tets as chains of dependent loads.  Here all 32 lanes of a
// warp evaluate the force terms of 32 adjacency entries at once, and lanes
// 0-7 then fold them in the 8-lane order — logical lane l takes entries
// l, l+8, l+16, l+24 — applying exactly the additions the stamp would have
// made, so every float is unchanged.  Entries whose terms do not fit the
// shipped record (joints, multi-contact manifolds) are stamped by the
// logical lane itself during the fold.
// ---------------------------------------------------------------------------
enum : uint32_t {
    TERM_NONE = 0, TERM_TET = 1, TERM_MANIFOLD = 2, TERM_SERIAL = 3, TERM_SPRING = 4, TERM_MEMBRANE = 5,
    TERM_BEND = 6, TERM_SOFT = 7
};
struct ParticleTerms {
    float3 rhs;          // the stamp's right-hand-side contribution
    float3 a, b, c, e;   // tet: (G00, G11, G22), (G01, G02, G12), (dd, -, -); manifold: rows of J^T K J;
                         // spring: n; membrane: g11, g22, g12, gtr; soft: n, t1, t2
    float3 s;            // spring: (k, ft, -); membrane: (2 mu A, 4 mu A, lambda A); bend: (s k^2, -, -);
                         // soft: (kN w^2, kT1 w^2, kT2 w^2)
    uint32_t kind;       // TERM_*
};

// Stable Neo-Hookean tet terms of one vertex (stampTet, 40_solver.metal:
// 972-1024): w is the vertex's row of DmInv (minus the sum of the rows for the
// first vertex), alphaT and diag = muV |w|^2 depend on the tet alone.
__device__ __forceinline__ void tet_core(float3 x0, float3 x1, float3 x2, float3 x3, float3 m0, float3 m1, float3 m2,
                                         float muV, float lamV, float alphaT, float3 w, float diag,
                                         ParticleTerms& t) {
    const float3 d0 = x1 - x0, d1 = x2 - x0, d2 = x3 - x0;
    const float3 f0 = d0 * m0.x + d1 * m1.x + d2 * m2.x;
    const float3 f1 = d0 * m0.y + d1 * m1.y + d2 * m2.y;
    const float3 f2 = d0 * m0.z + d1 * m1.z + d2 * m2.z;
    const float J = dot(f0, cross(f1, f2));
    const float3 j0 = cross(f1, f2), j1 = cross(f2, f0), j2 = cross(f0, f1);
    const float s2 = lamV * (J - alphaT);
    const float3 p0 = muV * f0 + s2 * j0;
    const float3 p1 = muV * f1 + s2 * j1;
    const float3 p2 = muV * f2 + s2 * j2;
    t.rhs = p0 * w.x + p1 * w.y + p2 * w.z;
    const float3 g = j0 * w.x + j1 * w.y + j2 * w.z;
    // lamV * outer(g, g) is exactly symmetric: g_i g_j == g_j g_i
    t.a = mk3((g.x * g.x) * lamV, (g.y * g.y) * lamV, (g.z * g.z) * lamV);
    t.b = mk3((g.y * g.x) * lamV, (g.z * g.x) * lamV, (g.z * g.y) * lamV);
    t.c = mk3(diag, 0.0f, 0.0f);
    t.kind = TERM_TET;
}
__device__ __forceinline__ void tet_terms(const DevPtrs& d, const TetGPU& tt, uint32_t self, ParticleTerms& t) {
    // the positions first: the division below must not stand before their loads
    const float3 x0 = xyz(d.posLin[tt.ids.x]), x1 = xyz(d.posLin[tt.ids.y]);
    const float3 x2 = xyz(d.posLin[tt.ids.z]), x3 = xyz(d.posLin[tt.ids.w]);
    const float muV = tt.r1.w, lamV = tt.r2.w;
    const float alphaT = 1.0f + muV / mx(lamV, 1e-9f);
    const float3 m0 = xyz(tt.r0), m1 = xyz(tt.r1), m2 = xyz(tt.r2);
    float3 w;
    if (self == tt.ids.y) w = m0;
    else if (self == tt.ids.z) w = m1;
    else if (self == tt.ids.w) w = m2;
    else w = -mk3(m0.x + m1.x + m2.x, m0.y + m1.y + m2.y, m0.z + m1.z + m2.z);
    tet_core(x0, x1, x2, x3, m0, m1, m2, muV, lamV, alphaT, w, muV * dot(w, w), t);
}

// Terms of a one-point manifold from its record and its bodies' poses.
__device__ __forceinline__ void manifold_core(const Params& P, bool isA, uint32_t flags, float4 basisN, float4 basisT1,
                                              const ContactGPU& c, float4 pa, float4 qa, float4 ia, float4 ja, float4 pb,
                                              float4 qb, float4 ib, float4 jb, ParticleTerms& t) {
    const bool sphA = (flags & 2u) != 0, sphB = (flags & 4u) != 0;
    const float3 dqALin = xyz(pa) - xyz(ia);
    const float3 dqAAng = q_sub(qa, ja);
    const float3 dqBLin = xyz(pb) - xyz(ib);
    const float3 dqBAng = q_sub(qb, jb);
    const float3 nrm = xyz(basisN), t1 = xyz(basisT1), t2 = cross(nrm, t1);
    const float3 rAW = sphA ? xyz(c.rA) : q_rotate(qa, xyz(c.rA));
    const float3 rBW = sphB ? xyz(c.rB) : q_rotate(qb, xyz(c.rB));
    float3 C;
    float fs, bnd;
    const float3 F = contact_force(c, nrm, t1, t2, basisN.w, basisT1.w, P.alpha, dqALin, dqAAng, dqBLin, dqBAng, rAW,
                                   rBW, C, fs, bnd);
    const float sg = isA ? 1.0f : -1.0f;
    const M3 jLin = M3{nrm * sg, t1 * sg, t2 * sg};
    const M3 K = m3_diag(xyz(c.penalty));
    const M3 jLinT = m3_transpose(jLin);
    const M3 M = m3_mulm(m3_mulm(jLinT, K), jLin);
    t.a = M.r0;
    t.b = M.r1;
    t.c = M.r2;
    t.rhs = m3_mul(jLinT, F);
    t.kind = TERM_MANIFOLD;
}

// Spring, membrane and bend terms from the ends' positions, shared by the
// grouped and the staged kernels.
__device__ __forceinline__ void spring_core(const Params& P, float3 pA, float3 pB, bool isA, float stiffness, float rest,
                                            bool hard, float4 dual, ParticleTerms& t) {
    // stamp_spring's linear block: outer(+-n, +-n) equals outer(n, n) bit for bit
    const float3 dd = pA - pB;
    const float dLen = len3(dd);
    t.kind = TERM_NONE;
    if (dLen <= 1.0e-6f) return;
    const float3 n = dd / dLen;
    float f;
    if (hard) {
        const float C = dLen - rest - dual.z * P.alpha;
        stiffness = dual.y;
        f = stiffness * C + dual.x;
        if (f <= 0.0f) return;
    } else {
        f = stiffness * (dLen - rest);
    }
    const float3 jLin = isA ? n : -n;
    t.rhs = jLin * f;
    t.a = n;
    t.s = mk3(stiffness, mx(f, 0.0f) / dLen, 0.0f);
    t.kind = TERM_SPRING;
}
__device__ __forceinline__ void membrane_core(float3 x0, float3 x1, float3 x2, float4 dmv, float muA, float lamA,
                                              uint32_t self, ParticleTerms& t) {
    const float3 d0 = x1 - x0, d1 = x2 - x0;
    const float a = dmv.x, b = dmv.y, c = dmv.z, dm = dmv.w;
    const float3 f1 = d0 * a + d1 * b;
    const float3 f2 = d0 * c + d1 * dm;
    const float E11 = 0.5f * (dot(f1, f1) - 1.0f);
    const float E22 = 0.5f * (dot(f2, f2) - 1.0f);
    const float E12 = 0.5f * dot(f1, f2);
    const float trE = E11 + E22;
    const float S11 = 2.0f * muA * E11 + lamA * trE;
    const float S22 = 2.0f * muA * E22 + lamA * trE;
    const float S12 = 2.0f * muA * E12;
    const float3 p1 = f1 * S11 + f2 * S12;
    const float3 p2 = f1 * S12 + f2 * S22;
    float wx, wy;
    if (self == 1u) { wx = a; wy = c; }
    else if (self == 2u) { wx = b; wy = dm; }
    else { wx = -a - b; wy = -c - dm; }
    t.rhs = p1 * wx + p2 * wy;
    t.a = f1 * wx;
    t.b = f2 * wy;
    t.c = (f2 * wx + f1 * wy) * 0.5f;
    t.e = t.a + t.b;
    t.s = mk3(2.0f * muA, 4.0f * muA, lamA);
    t.kind = TERM_MEMBRANE;
}
__device__ __forceinline__ void bend_core(float3 x0, float3 x1, float3 x2, float3 x3, float4 K, float sc, uint32_t self,
                                          ParticleTerms& t) {
    const float3 m = x0 * K.x + x1 * K.y + x2 * K.z + x3 * K.w;
    const float k = self == 0u ? K.x : (self == 1u ? K.y : (self == 2u ? K.z : K.w));
    t.rhs = m * (sc * k);
    t.s = mk3(sc * k * k, 0.0f, 0.0f);
    t.kind = TERM_BEND;
}

template <bool CLOTH>
__device__ __forceinline__ void particle_terms(const Params& P, const DevPtrs& d, uint32_t entry,
                                               uint32_t self, ParticleTerms& t) {
    const uint32_t kind = entry >> ADJ_KIND_SHIFT, idx = entry & ADJ_INDEX_MASK;
    t.kind = 3;
    if (kind == FK_TET) {
        tet_terms(d, d.tets[idx], self, t);
    } else if (kind == FK_MANIFOLD) {
        const ManifoldGPU& m = d.manifolds[idx];
        const u4 h = m.header;
        if (h.z != 1u) return;
        const uint32_t a = h.x, b = h.y;
        manifold_core(P, self == a, h.w, tof(m.basisN), tof(m.basisT1), m.contacts[0], d.posLin[a], d.posAng[a],
                      d.initLin[a], d.initAng[a], d.posLin[b], d.posAng[b], d.initLin[b], d.initAng[b], t);
    } else if (!CLOTH) {
        return;
    } else if (kind == FK_SPRING) {
        const SpringGPU sp = d.springs[idx];
        const uint32_t a = sp.header.x, b = sp.header.y;
        spring_core(P, xform(xyz(d.posLin[a]), d.posAng[a], xyz(sp.rA)), xform(xyz(d.posLin[b]), d.posAng[b], xyz(sp.rB)),
                    self == a, sp.rA.w, sp.rB.w, sp.header.z != 0, tof(sp.dual), t);
    } else if (kind == FK_MEMBRANE) {
        const MembraneGPU mb = d.membranes[idx];
        membrane_core(xyz(d.posLin[mb.ids.x]), xyz(d.posLin[mb.ids.y]), xyz(d.posLin[mb.ids.z]), tof(mb.dm), mb.mat.x,
                      mb.mat.y, self == mb.ids.y ? 1u : (self == mb.ids.z ? 2u : 0u), t);
    } else if (kind == FK_BEND) {
        const BendGPU bd = d.bends[idx];
        bend_core(xyz(d.posLin[bd.ids.x]), xyz(d.posLin[bd.ids.y]), xyz(d.posLin[bd.ids.z]), xyz(d.posLin[bd.ids.w]),
                  tof(bd.K), bd.mat.x,
                  self == bd.ids.x ? 0u : (self == bd.ids.y ? 1u : (self == bd.ids.z ? 2u : 3u)), t);
    } else if (kind == FK_SOFT) {
        const SoftContactGPU& sc = d.soft[idx];
        float3 n, t1, t2, rAW;
        bool rigidA;
        const float3 C = soft_c(P, d, sc, n, t1, t2, rAW, rigidA);
        float3 F = xyz(sc.penalty) * C + xyz(sc.lambda);
        float kN = sc.penalty.x;
        const float rT = sc.anchorA.x;
        const uint32_t kindB = (__float_as_uint(sc.anchorA.w) >> SCF_KIND_SHIFT) & 3u;
        if (rT > 0.0f && kindB != SC_RT && C.x < -0.5f * rT) {
            const float dsep = mx(C.x + rT, 0.02f * rT);
            const float kp = 0.25f * rT * rT * sc.penalty.x;
            F.x = -kp / dsep + sc.lambda.x;
            kN = kp / (dsep * dsep);
        }
        F.x = mn(F.x, 0.0f);
        const float bounds = fabsf(F.x) * sc.normal.w;
        const float fs = sqrtf(F.y * F.y + F.z * F.z);
        if (fs > bounds && fs > 0.0f) {
            const float r = bounds / fs;
            F.y *= r;
            F.z *= r;
        }
        int slot = -1;
        if (sc.ids.x == self) slot = 0;
        else if (sc.ids.y == self) slot = 1;
        else if (sc.ids.z == self) slot = 2;
        else if (sc.ids.w == self) slot = 3;
        t.kind = TERM_NONE;
        if (slot < 0) return;
        if (slot == 0 && rigidA) { t.kind = TERM_SERIAL; return; }
        const float w = slot == 0 ? sc.weights.x : (slot == 1 ? sc.weights.y : (slot == 2 ? sc.weights.z : sc.weights.w));
        const float w2 = w * w;
        t.a = n;
        t.b = t1;
        t.c = t2;
        t.s = mk3(kN * w2, sc.penalty.y * w2, sc.penalty.z * w2);
        t.rhs = (n * F.x + t1 * F.y + t2 * F.z) * w;
        t.kind = TERM_SOFT;
    }
}

__device__ __forceinline__ float3 shfl_idx3(float3 v, int src) {
    return mk3(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src),
               __shfl_sync(0xffffffffu, v.z, src));
}

// Linear block of a particle's system: the only part its solve reads.
struct ParticleAccum { M3 lhs; float3 rhs; };

// Rare entries (joints, springs, multi-contact manifolds) go through the
// generic stamp, which changes lhsLin/rhsLin exactly as it would inside a
// full accumulator.  Scenes that cannot produce them (every dynamic body a
// particle whose adjacency holds only tets and sphere contacts — known at
// upload) use the GENERAL = false instance, which drops these paths and
// their registers.
__device__ __forceinline__ void stamp_entry_particle(const Params& P, const DevPtrs& d, uint32_t entry,
                                                     uint32_t body, ParticleAccum* acc) {
    Accum full{acc->lhs, m3_zero(), m3_zero(), acc->rhs, s3(0)};
    stamp_entry(P, d, entry, body, full);
    acc->lhs = full.lhsLin;
    acc->rhs = full.rhsLin;
}

// Terms of adjacency entry k of particle `body`.  A tet entry reads its
// record from the body's incidence slot (contiguous over consecutive k)
// instead of through the entry; `entry` is what the generic stamp needs.
template <bool CLOTH>
__device__ __forceinline__ void particle_entry_terms(const Params& P, const DevPtrs& d, const AdjView& v,
                                                     uint32_t body, uint32_t k, ParticleTerms& t, uint32_t& entry) {
    const uint32_t kt = k - v.nPre - v.nMan;
    if (d.tetInc && k >= v.nPre + v.nMan && kt < v.nTet) {
        entry = (FK_TET << ADJ_KIND_SHIFT);
        tet_terms(d, d.tetInc[v.postBase + kt], body, t);
    } else {
        entry = v.at(k);
        particle_terms<CLOTH>(P, d, entry, body, t);
    }
}

// Adds one entry's terms to a particle's linear system, in the order of
// operations of the stamps (every instance folds through this function, so
// any lane layout yields the same floats).
template <bool GENERAL, bool CLOTH>
__device__ __forceinline__ void fold_particle_term(const Params& P, const DevPtrs& d, const ParticleTerms& u,
                                                   uint32_t e, uint32_t body, ParticleAccum& acc) {
    if (u.kind == 1u) {
        acc.rhs += u.rhs;
        acc.lhs = m3_add(acc.lhs, m3_diag(s3(u.c.x)));
        acc.lhs = m3_add(acc.lhs, M3{mk3(u.a.x, u.b.x, u.b.y), mk3(u.b.x, u.a.y, u.b.z),
                                     mk3(u.b.y, u.b.z, u.a.z)});
    } else if (u.kind == 2u) {
        acc.lhs = m3_add(acc.lhs, M3{u.a, u.b, u.c});
        acc.rhs += u.rhs;
    } else if (CLOTH && u.kind == TERM_MEMBRANE) {
        acc.rhs += u.rhs;
        acc.lhs = m3_add(acc.lhs, m3_scale(m3_outer(u.a, u.a), u.s.x));
        acc.lhs = m3_add(acc.lhs, m3_scale(m3_outer(u.b, u.b), u.s.x));
        acc.lhs = m3_add(acc.lhs, m3_scale(m3_outer(u.c, u.c), u.s.y));
        acc.lhs = m3_add(acc.lhs, m3_scale(m3_outer(u.e, u.e), u.s.z));
    } else if (CLOTH && u.kind == TERM_BEND) {
        acc.rhs += u.rhs;
        acc.lhs = m3_add(acc.lhs, m3_diag(s3(u.s.x)));
    } else if (CLOTH && u.kind == TERM_SPRING) {
        acc.lhs = m3_add(acc.lhs, m3_scale(m3_outer(u.a, u.a), u.s.x));
        acc.rhs += u.rhs;
        if (u.s.y > 0.0f)
            acc.lhs = m3_add(acc.lhs, m3_add(m3_diag(s3(u.s.y)), m3_scale(m3_outer(u.a, u.a), -u.s.y)));
    } else if (CLOTH && u.kind == TERM_SOFT) {
        acc.lhs = m3_add(acc.lhs, m3_scale(m3_outer(u.a, u.a), u.s.x));
        acc.lhs = m3_add(acc.lhs, m3_scale(m3_outer(u.b, u.b), u.s.y));
        acc.lhs = m3_add(acc.lhs, m3_scale(m3_outer(u.c, u.c), u.s.z));
        acc.rhs += u.rhs;
    } else if (GENERAL && u.kind != TERM_NONE) {
        stamp_entry_particle(P, d, e, body, &acc);
    }
}


// The particle system's angular block is the identity and its cross block
// zero.  Every term of the 6x6 LDL^T that involves them is then an exact
// "x - (+0)" (L4x..L6x, y4..y6, z4..z6 and xAng are all +0), so this 3x3
// sequence returns bit for bit the linear part of solve6x6(lhs, I, 0, b, 0);
// with non-finite input both produce a non-finite step and the update is
// skipped.
__device__ __forceinline__ float3 solve3x3_particle(const M3& a, float3 b) {
    const float s1 = rsq(mx(a.r0.x, 1e-30f));
    const float s2 = rsq(mx(a.r1.y, 1e-30f));
    const float s3_ = rsq(mx(a.r2.z, 1e-30f));
    const float A11 = 1.0f, A22 = 1.0f, A33 = 1.0f;
    const float A21 = a.r1.x * s2 * s1;
    const float A31 = a.r2.x * s3_ * s1, A32 = a.r2.y * s3_ * s2;
    b = mk3(b.x * s1, b.y * s2, b.z * s3_);
    const float L21 = A21 / A11, L31 = A31 / A11;
    const float eps = 1e-6f;
    const float D1 = mx(A11, eps);
    const float D2 = mx(A22 - L21 * L21 * D1, eps);
    const float L32 = (A32 - L21 * L31 * D1) / D2;
    const float D3 = mx(A33 - (L31 * L31 * D1 + L32 * L32 * D2), eps);
    const float y1 = b.x;
    const float y2 = b.y - L21 * y1;
    const float y3 = b.z - L31 * y1 - L32 * y2;
    const float z1 = y1 / D1, z2 = y2 / D2, z3 = y3 / D3;
    float3 x;
    x.z = z3;
    x.y = z2 - L32 * x.z;
    x.x = z1 - L21 * x.y - L31 * x.z;
    return mk3(x.x * s1, x.y * s2, x.z * s3_);
}

// Inertia, solve, trust region, OGC bound and commit of a particle whose
// stamped system is (acc.lhs, acc.rhs); lane 0 of its group calls this.
// (bound, anchor): the body's OGC bound and its anchor, read before the solve
// so that they are there when the step is known.
__device__ __forceinline__ void particle_commit(const Params& P, const DevPtrs& d, uint32_t body, float radius,
                                                float4 pl, float4 inert, float bound, float4 anchor,
                                                ParticleAccum acc) {
    const float mass = pl.w;
    const float dt2 = P.dt * P.dt;
    acc.lhs = m3_add(acc.lhs, m3_diag(s3(mass / dt2)));
    acc.rhs += (xyz(pl) - xyz(inert)) * (mass / dt2);
    float3 dxLin = solve3x3_particle(acc.lhs, -acc.rhs);
    if (!finite3(dxLin)) { keep_body(P, d, body, pl, false); return; }
    const float maxLin = 0.35f * fabsf(radius);
    const float lin2 = dot(dxLin, dxLin);
    if (lin2 > maxLin * maxLin) dxLin *= maxLin * rsq(lin2);
    if (P.ogc) dxLin = ogc_truncate(d, bound, anchor, dxLin, xyz(pl), -radius);
    if (P.colorJacobi) { d.posNext[body] = mk4(xyz(pl) + dxLin, mass); return; }
    d.posLin[body] = mk4(xyz(pl) + dxLin, mass);
}

// Grouped primal for one color, LANES consecutive lanes per body: the width
// that a caller pinned, 32 for particles that fit no staged block.  Lane p of a
// group evaluates entry base + p; logical lane l < 8 then folds entries
// base + l, base + l + 8, ... in order.  Any LANES gives the same floats.
// RESID: evaluate instead of solve — lane 0 stores the body's squared
// right-hand side (the AL gradient) in d.learnResidBodies[slot] and leaves
// the pose alone (called over all colors at once).  What bounds it there are
// dependent loads and, in GENERAL instances, registers: the mixed scene's
// learned stage, two residuals included, takes 422 us (699 with a called
// stamp_joint and its 1.5 KB of local memory per thread).
// GENERAL instances keep four blocks per SM (at most 128 registers): the
// rigid-body path would otherwise take ~160 registers for every thread and
// cap large colors at three blocks (measured 7% slower mixed frames).
#ifndef AVBD_PRIMAL_UNROLL
#define AVBD_PRIMAL_UNROLL 1
#endif
constexpr int kPrimalUnroll = AVBD_PRIMAL_UNROLL;
#ifndef AVBD_PARTICLE_PRIMAL_MIN_BLOCKS
#define AVBD_PARTICLE_PRIMAL_MIN_BLOCKS 1
#endif
#ifndef AVBD_LEAN_CLOTH_MIN_BLOCKS
#define AVBD_LEAN_CLOTH_MIN_BLOCKS 5
#endif
template <int LANES, bool GENERAL, bool CLOTH, bool RESID = false>
__global__ void __launch_bounds__(128, GENERAL ? 4 : (CLOTH ? AVBD_LEAN_CLOTH_MIN_BLOCKS : AVBD_PARTICLE_PRIMAL_MIN_BLOCKS)) k_primal_group(const Params P, const DevPtrs d, uint32_t color,
                                                      uint32_t count, uint32_t first, uint32_t start) {
    constexpr int GROUPS = 32 / LANES;
    pdl_trigger();
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t slot = tid / LANES;
    const uint32_t lane = tid & (LANES - 1);
    // The solve takes its body from the color's launch order (lean
    // particles first); the residual pass walks the color list itself.
    // With the color's start known on the host, the launch order, the
    // body's shape and its static adjacency segment (none written after
    // upload) are read before waiting for the previous grid.
    uint32_t s, body;
    float4 shp;
    uint4 seg;
    uint32_t nTet;
    if (!RESID && start != NO_HOST_START) {
        s = start;
        if (slot >= count) return;                           // uniform across the group
        body = d.colorLaunch[s + first + slot];
        shp = d.shape[body];
        seg = d.staticSeg[body];
        nTet = d.postTets[body];
        pdl_wait();
    } else {
        pdl_wait();
        s = d.colorStart[color];
        const uint32_t n = count != 0xFFFFFFFFu ? count : d.colorStart[color + 1] - s;
        if (slot >= n) return;                               // uniform across the group
        body = RESID ? d.colorList[s + slot] : d.colorLaunch[s + first + slot];
        shp = d.shape[body];
        seg = d.staticSeg[body];
        nTet = d.postTets[body];
    }
    const unsigned mask = LANES == 32 ? 0xffffffffu
                                      : (((1u << LANES) - 1u) << ((threadIdx.x & 31u) & ~(uint32_t)(LANES - 1)));
    (void)GROUPS;
    static_assert(RESID || !GENERAL, "a solve's rigid bodies run in k_primal_wide");
    if (GENERAL && shp.w >= 0.0f) {                          // rigid: the 8-lane path
        const unsigned mask8 = mask & (0xFFu << ((threadIdx.x & 31u) & ~(uint32_t)(LANES - 1)));
        if (lane < 8) rigid_residual(P, d, body, lane, mask8, d.learnResidBodies + s + slot);
        return;
    }
    // lane 0 needs these after the reduction; issue the loads now
    float4 pl = make_float4(0, 0, 0, 0), inert = make_float4(0, 0, 0, 0);
    float bound = 0.0f;
    float4 anchor = make_float4(0, 0, 0, 0);
    if (lane == 0) {
        pl = d.posLin[body];
        inert = d.inertLin[body];
        if (!RESID && P.ogc) { bound = __uint_as_float(d.ogcBounds[body]); anchor = d.ogcPrev[body]; }
    }
    ParticleAccum acc{m3_zero(), s3(0)};
    const AdjView v = adj_view_from(d, body, seg, nTet);
    const uint32_t cnt = v.count();
#pragma unroll (kPrimalUnroll)
    for (uint32_t base = 0; base < cnt; base += LANES) {
        const uint32_t k = base + lane;
        ParticleTerms t;
        t.kind = 0;
        uint32_t entry = 0;
        if (k < cnt) particle_entry_terms<CLOTH>(P, d, v, body, k, t, entry);
#pragma unroll
        for (int j = 0; j < LANES / 8; j++) {
            const int src = (int)(lane & 7u) + 8 * j;
            ParticleTerms u;
            uint32_t e;
            if (j == 0) {
                // logical lane l already holds entry base + l
                u = t;
                e = entry;
            } else {
            u.kind = __shfl_sync(mask, t.kind, src, LANES);
            u.rhs = mk3(__shfl_sync(mask, t.rhs.x, src, LANES), __shfl_sync(mask, t.rhs.y, src, LANES),
                        __shfl_sync(mask, t.rhs.z, src, LANES));
            u.a = mk3(__shfl_sync(mask, t.a.x, src, LANES), __shfl_sync(mask, t.a.y, src, LANES),
                      __shfl_sync(mask, t.a.z, src, LANES));
            u.b = mk3(__shfl_sync(mask, t.b.x, src, LANES), __shfl_sync(mask, t.b.y, src, LANES),
                      __shfl_sync(mask, t.b.z, src, LANES));
            u.c = mk3(__shfl_sync(mask, t.c.x, src, LANES), __shfl_sync(mask, t.c.y, src, LANES),
                      __shfl_sync(mask, t.c.z, src, LANES));
            if (CLOTH) {
                u.e = mk3(__shfl_sync(mask, t.e.x, src, LANES), __shfl_sync(mask, t.e.y, src, LANES),
                          __shfl_sync(mask, t.e.z, src, LANES));
                u.s = mk3(__shfl_sync(mask, t.s.x, src, LANES), __shfl_sync(mask, t.s.y, src, LANES),
                          __shfl_sync(mask, t.s.z, src, LANES));
            }
            e = __shfl_sync(mask, entry, src, LANES);
            }
            if (lane < 8) fold_particle_term<GENERAL, CLOTH>(P, d, u, e, body, acc);
        }
    }
    // xor butterfly over the 8 logical lanes (offsets 4, 2, 1)
#pragma unroll
    for (int o = 4; o >= 1; o >>= 1) {
        add_shfl_lower(mask, acc.lhs, o);
        add_shfl3(mask, acc.rhs, o);
    }
    if (lane != 0) return;
    if (RESID) {
        const float3 r = acc.rhs + (xyz(pl) - xyz(inert)) * (pl.w / (P.dt * P.dt));
        d.learnResidBodies[s + slot] = dot(r, r);
        return;
    }
    particle_commit(P, d, body, shp.w, pl, inert, bound, anchor, acc);
}

template <bool CLOTH>
static void launch_primal_group(const Params& P, const DevPtrs& d, uint32_t color, uint32_t count,
                                uint32_t first, uint32_t start, uint32_t lanes, cudaStream_t st) {
    const int T = 128;
    const uint32_t blocks = (count * lanes + T - 1) / T;
    if (lanes <= 8) launch_pdl(k_primal_group<8, false, CLOTH>, blocks, T, st, P, d, color, count, first, start);
    else if (lanes <= 16)
        launch_pdl(k_primal_group<16, false, CLOTH>, blocks, T, st, P, d, color, count, first, start);
    else launch_pdl(k_primal_group<32, false, CLOTH>, blocks, T, st, P, d, color, count, first, start);
}

// ---------------------------------------------------------------------------
// Staged primal: 16 lean particles per block, 8 lanes each (the reference's
// SIMD layout).  A color's chain used to be body -> adjacency -> element record
// -> vertex positions, each a dependent trip to L2, after the previous color
// had finished.  What no kernel writes (the launch tables built at upload: the
// springs', membranes' and bends' constants, the tets' by index, the lists of
// referenced bodies) is now copied to shared memory before the wait for the
// previous grid, so that its latency is spent in the previous color's tail.
// After the wait the block gathers each referenced body's position once (a
// vertex of a soft body has some 24 tets but 15 distinct neighbours: 16 reads
// in place of 96), and the lanes evaluate and fold their entries l, l + 8, ...
// straight from shared memory; only contacts, and springs with levers, are read
// through the adjacency.  Every expression and order is the grouped kernel's.
// What bounds it: for small colors the chain (0.6 us gather, 1.4 us for three
// tets a lane, 0.6 us solve, 1 us between grids); for large ones issue slots
// (0.6 of them used on the 256^2 cloth, 18-22 us a color of 32,767).
// ---------------------------------------------------------------------------
constexpr int kStagedThreads = 8 * (int)STAGED_BODIES;
constexpr uint32_t kStagedContacts = 24;        // one-point manifolds of a block held in shared memory
constexpr uint32_t kStagedContactWords = 16;    // header, basis, contact, the two bodies' start poses and poses

__device__ __forceinline__ void copy16(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem)
                 : "memory");
}

// AHEAD: the block's first manifolds are copied to shared memory as well, what
// the solve does not write before the wait, the bodies' poses and the words that
// the dual stores to with the positions: a contact adds its arithmetic to the color instead of four
// dependent trips (2.3 us of the 4.3 us a small color took).
//
// LANES = 32 (tet colors of at most STAGED_WIDE bodies): four bodies a block,
// a warp each.  Its lanes evaluate 32 entries at once and pass the terms to the
// eight folding lanes by shuffles: the color's chain is one tet long instead of
// three, which pays while the device has room for a warp per body.
template <bool CLOTH, bool AHEAD, int LANES>
__global__ void __launch_bounds__(kStagedThreads, LANES == 32 ? 4 : 5)
k_primal_staged(const Params P, const DevPtrs d, uint32_t firstBlock, bool early) {
    extern __shared__ uint4 words[];
    __shared__ uint4 con[AHEAD ? kStagedContacts * kStagedContactWords : 1];
    __shared__ uint32_t contacts;
    pdl_trigger();
    const uint32_t tid = threadIdx.x, g = tid / LANES, lane = tid & (LANES - 1u);
    if (AHEAD) {
        if (tid == 0) contacts = 0u;
        __syncthreads();
    }
    const StagedBlock B = d.stagedBlocks[firstBlock + blockIdx.x];
    // records | tet constants (four words each) | tet references | positions
    uint4* rec = words;
    uint4* tets = rec + B.recLen;
    StagedTet* refs = reinterpret_cast<StagedTet*>(tets + 4 * (size_t)B.tetLen);
    float4* pos = reinterpret_cast<float4*>(tets + 4 * (size_t)B.tetLen + B.tetLen / 2);
    // every index first: the copies between them would each wait for theirs
    uint32_t ti[4], id[4];
#pragma unroll
    for (uint32_t j = 0; j < 4; j++) {
        const uint32_t e = tid + j * kStagedThreads;
        ti[j] = e < B.tetLen ? d.stagedTets[B.tet + e].index & ADJ_INDEX_MASK : 0u;
        id[j] = e < B.idLen ? d.stagedIds[B.ids + e] : 0u;
    }
    const bool active = g < B.count;
    const StagedBody b = d.stagedBodies[B.first + (active ? g : 0u)];
    // thread t solves body t at the end
    const bool solver = tid < B.count;
    const StagedBody mine = d.stagedBodies[B.first + (solver ? tid : 0u)];
    auto copy_tet = [&](uint32_t e, uint32_t t) {
#pragma unroll
        for (uint32_t w = 0; w < 4; w++) copy16(tets + w * B.tetLen + e, d.tetConst + 4 * (size_t)t + w);
    };
#pragma unroll
    for (uint32_t j = 0; j < 4; j++)
        if (tid + j * kStagedThreads < B.tetLen) copy_tet(tid + j * kStagedThreads, ti[j]);
    for (uint32_t e = tid + 4 * kStagedThreads; e < B.tetLen; e += kStagedThreads)
        copy_tet(e, d.stagedTets[B.tet + e].index & ADJ_INDEX_MASK);
    for (uint32_t i = tid; i < B.tetLen / 2; i += kStagedThreads) copy16(refs + 2 * i, d.stagedTets + B.tet + 2 * i);
    for (uint32_t i = tid; i < B.recLen; i += kStagedThreads) copy16(rec + i, d.stagedRec + B.rec + i);
    // the lane's first spring, whose multiplier is read right after the wait
    const uint32_t spring = CLOTH && lane < b.nPre ? d.stagedRec[B.rec + b.rec + lane].w : 0u;
    if (!early) pdl_wait();
    // this frame's contacts (with `early`, see launch_primal_color: written
    // before every grid that may still be running): the lane's first manifold,
    // the first entry lane, lane + 8, ... past the springs
    const uint32_t* dyn = d.dynList + __ldcg(d.dynStart + b.body);
    const uint32_t nDyn = active ? __ldcg(d.dynCount + b.body) : 0u, nMan = active ? __ldcg(d.dynSplit + b.body) : 0u;
    const uint32_t endMan = b.nPre + nMan;
    const uint32_t kMan = lane >= b.nPre ? lane : lane + ((b.nPre - lane + LANES - 1u) & ~(LANES - 1u));
    uint32_t slot = kStagedContacts, manifold = 0, bodyA = 0, bodyB = 0;
    if (AHEAD && kMan < endMan) {
        const uint32_t m = __ldcg(dyn + (kMan - b.nPre)) & ADJ_INDEX_MASK;
        const uint4* mw = reinterpret_cast<const uint4*>(d.manifolds + m);
        const uint4 h = __ldcg(mw);
        bodyA = h.x;
        bodyB = h.y;
        if (h.z == 1u) slot = atomicAdd(&contacts, 1u);
        if (slot < kStagedContacts) {
            uint4* q = con + kStagedContactWords * slot;
            q[0] = h;
            copy16(q + 1, mw + 2);                   // normal
            copy16(q + 2, mw + 3);                   // tangent
            copy16(q + 3, mw + 4);                   // rA
            copy16(q + 5, mw + 6);                   // C0
            copy16(q + 8, d.initLin + bodyA);
            copy16(q + 9, d.initAng + bodyA);
            copy16(q + 10, d.initLin + bodyB);
            copy16(q + 11, d.initAng + bodyB);
            manifold = m;
        }
    }
    if (early) pdl_wait();
    if (AHEAD && slot < kStagedContacts) {
        uint4* q = con + kStagedContactWords * slot;
        const uint4* mw = reinterpret_cast<const uint4*>(d.manifolds + manifold);
        copy16(q + 4, mw + 5);                       // rB (the dual stores the stick flag in its w)
        copy16(q + 6, mw + 7);                       // lambda
        copy16(q + 7, mw + 8);                       // penalty
        copy16(q + 12, d.posLin + bodyA);
        copy16(q + 13, d.posAng + bodyA);
        copy16(q + 14, d.posLin + bodyB);
        copy16(q + 15, d.posAng + bodyB);
    }
#pragma unroll
    for (uint32_t j = 0; j < 4; j++)
        if (tid + j * kStagedThreads < B.idLen) copy16(pos + tid + j * kStagedThreads, d.posLin + id[j]);
    for (uint32_t i = tid + 4 * kStagedThreads; i < B.idLen; i += kStagedThreads)
        copy16(pos + i, d.posLin + d.stagedIds[B.ids + i]);
    float4 dual = make_float4(0, 0, 0, 0), inert = dual, anchor = dual;
    float bound = 0.0f;
    if (CLOTH && lane < b.nPre) dual = tof(d.springs[spring].dual);
    if (solver) {
        inert = d.inertLin[mine.body];
        if (P.ogc) { bound = __uint_as_float(d.ogcBounds[mine.body]); anchor = d.ogcPrev[mine.body]; }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    __shared__ float sums[9][STAGED_BODIES];
    if (active) {
        const unsigned mask = LANES == 32 ? 0xFFu : 0xFFu << (tid & 24u);
        const uint4* br = rec + b.rec;
        const float4* bp = pos + b.pos;
        auto at = [&](uint32_t r, uint32_t k) { return xyz(bp[(r >> (8 * k)) & 0xFFu]); };
        ParticleAccum acc{m3_zero(), s3(0)};
        const uint32_t endTet = endMan + b.nTet, endSoft = endTet + nDyn - nMan, cnt = endSoft + b.nRest;
        auto staged_contact = [&](ParticleTerms& t) {
            const uint4* q = con + kStagedContactWords * slot;
            const float4* f = reinterpret_cast<const float4*>(q);
            ContactGPU c;
            c.rA = tof4(f[3]); c.rB = tof4(f[4]); c.C0 = tof4(f[5]); c.lambda = tof4(f[6]); c.penalty = tof4(f[7]);
            manifold_core(P, b.body == q[0].x, q[0].w, f[1], f[2], c, f[12], f[13], f[8], f[9], f[14], f[15], f[10],
                          f[11], t);
        };
        auto tet = [&](uint32_t e, ParticleTerms& t) {
            const StagedTet r = refs[e];
            const uint4 q0 = tets[e], q1 = tets[B.tetLen + e], q2 = tets[2 * B.tetLen + e];
            const float3 m0 = mk3(__uint_as_float(q0.x), __uint_as_float(q0.y), __uint_as_float(q0.z));
            const float3 m1 = mk3(__uint_as_float(q1.x), __uint_as_float(q1.y), __uint_as_float(q1.z));
            const float3 m2 = mk3(__uint_as_float(q2.x), __uint_as_float(q2.y), __uint_as_float(q2.z));
            const uint32_t self = r.index >> ADJ_KIND_SHIFT;
            const float3 w = self == 1u ? m0 : (self == 2u ? m1 : (self == 3u ? m2
                             : -mk3(m0.x + m1.x + m2.x, m0.y + m1.y + m2.y, m0.z + m1.z + m2.z)));
            const float diag = reinterpret_cast<const float*>(tets + 3 * B.tetLen + e)[self];
            tet_core(at(r.refs, 0), at(r.refs, 1), at(r.refs, 2), at(r.refs, 3), m0, m1, m2, __uint_as_float(q1.w),
                     __uint_as_float(q2.w), __uint_as_float(q0.w), w, diag, t);
        };
        if (LANES == 32) {
            // manifolds and tets only (tet colors)
            for (uint32_t base = 0; base < cnt; base += 32) {
                const uint32_t k = base + lane;
                ParticleTerms t;
                t.kind = TERM_NONE;
                uint32_t e = 0;
                if (k < endMan) {
                    if (AHEAD && k == kMan && slot < kStagedContacts) {
                        staged_contact(t);
                    } else {
                        e = dyn[k - b.nPre];
                        particle_terms<false>(P, d, e, b.body, t);
                    }
                } else if (k < endTet) {
                    tet(b.tet + (k - endMan), t);
                }
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int src = (int)(lane & 7u) + 8 * j;
                    ParticleTerms u = t;
                    if (j > 0) {
                        if (base + 8u * j >= cnt) break;             // the same in the whole warp
                        u.kind = __shfl_sync(0xffffffffu, t.kind, src);
                        u.rhs = shfl_idx3(t.rhs, src);
                        u.a = shfl_idx3(t.a, src);
                        u.b = shfl_idx3(t.b, src);
                        u.c = shfl_idx3(t.c, src);
                    }
                    if (lane < 8) fold_particle_term<false, false>(P, d, u, 0u, b.body, acc);
                }
            }
        } else {
        // a loop per kind: lanes whose entries of a kind fall into different
        // rounds of eight still evaluate them together
        uint32_t k = lane;
        if (CLOTH) {
            for (; k < b.nPre; k += 8) {
                ParticleTerms t;
                const uint4 q = br[k];
                const uint32_t flags = br[b.nPre + k].x;
                if (flags & STAGED_GENERIC) {
                    particle_terms<true>(P, d, (FK_SPRING << ADJ_KIND_SHIFT) | q.w, b.body, t);
                } else {
                    if (k != lane) dual = tof(d.springs[q.w].dual);
                    spring_core(P, at(q.z, 0), at(q.z, 1), (flags & 1u) == 0u, __uint_as_float(q.x),
                                __uint_as_float(q.y), (flags & STAGED_HARD) != 0u, dual, t);
                }
                fold_particle_term<false, CLOTH>(P, d, t, 0u, b.body, acc);
            }
        }
        if (AHEAD && k < endMan && slot < kStagedContacts) {
            ParticleTerms t;
            staged_contact(t);
            fold_particle_term<false, false>(P, d, t, 0u, b.body, acc);
            k += 8;
        }
        for (; k < endMan; k += 8) {
            ParticleTerms t;
            const uint32_t e = dyn[k - b.nPre];
            particle_terms<false>(P, d, e, b.body, t);
            fold_particle_term<false, false>(P, d, t, e, b.body, acc);
        }
        __syncwarp(mask);
#pragma unroll 1
        for (; k < endTet; k += 8) {
            ParticleTerms t;
            tet(b.tet + (k - endMan), t);
            fold_particle_term<false, CLOTH>(P, d, t, 0u, b.body, acc);
        }
        if (CLOTH) {
            for (; k < endSoft; k += 8) {
                ParticleTerms t;
                const uint32_t e = dyn[nMan + (k - endTet)];
                particle_terms<true>(P, d, e, b.body, t);
                fold_particle_term<false, true>(P, d, t, e, b.body, acc);
            }
            __syncwarp(mask);
            const uint32_t endMem = endSoft + b.nMem;
            for (; k < endMem; k += 8) {
                ParticleTerms t;
                const uint32_t e = 2 * b.nPre + (k - endSoft);
                const uint4 q = br[e], r = br[b.nRest + e];
                membrane_core(at(r.z, 0), at(r.z, 1), at(r.z, 2),
                              make_float4(__uint_as_float(q.x), __uint_as_float(q.y), __uint_as_float(q.z),
                                          __uint_as_float(q.w)),
                              __uint_as_float(r.x), __uint_as_float(r.y), r.w, t);
                fold_particle_term<false, CLOTH>(P, d, t, 0u, b.body, acc);
            }
            __syncwarp(mask);
            for (; k < cnt; k += 8) {
                ParticleTerms t;
                const uint32_t e = 2 * b.nPre + (k - endSoft);
                const uint4 q = br[e], r = br[b.nRest + e];
                bend_core(at(r.z, 0), at(r.z, 1), at(r.z, 2), at(r.z, 3),
                          make_float4(__uint_as_float(q.x), __uint_as_float(q.y), __uint_as_float(q.z),
                                      __uint_as_float(q.w)),
                          __uint_as_float(r.x), r.w, t);
                fold_particle_term<false, CLOTH>(P, d, t, 0u, b.body, acc);
            }
        }
        __syncwarp(mask);
        }
        if (lane < 8) {
#pragma unroll
            for (int o = 4; o >= 1; o >>= 1) {
                add_shfl_lower(mask, acc.lhs, o);
                add_shfl3(mask, acc.rhs, o);
            }
        }
        if (lane == 0) {
            const float v[9] = {acc.lhs.r0.x, acc.lhs.r1.x, acc.lhs.r1.y, acc.lhs.r2.x, acc.lhs.r2.y,
                                acc.lhs.r2.z, acc.rhs.x, acc.rhs.y, acc.rhs.z};
#pragma unroll
            for (int c = 0; c < 9; c++) sums[c][g] = v[c];
        }
    }
    __syncthreads();
    // one warp solves the block's bodies side by side (a sixteenth of the
    // issue slots that a lane per group would take)
    if (!solver) return;
    ParticleAccum acc{m3_zero(), mk3(sums[6][tid], sums[7][tid], sums[8][tid])};
    acc.lhs.r0.x = sums[0][tid];
    acc.lhs.r1.x = sums[1][tid]; acc.lhs.r1.y = sums[2][tid];
    acc.lhs.r2.x = sums[3][tid]; acc.lhs.r2.y = sums[4][tid]; acc.lhs.r2.z = sums[5][tid];
    particle_commit(P, d, mine.body, mine.radius, pos[mine.pos], inert, bound, anchor, acc);
}

void launch_primal_color(const Params& P, const DevPtrs& d, const Sizes& z, uint32_t color, uint32_t count,
                         uint32_t lanes, bool& chained, bool last, cudaStream_t st, cudaStream_t side, cudaEvent_t fork,
                         cudaEvent_t join) {
    const int T = 128;
    const uint32_t upper = count != 0xFFFFFFFFu ? count : z.numDynamicBodies;
    if (upper == 0) return;
    if (z.dynamicColoring) {
        // dynamic coloring: the color's size is known on the device only, so
        // one resident wave (4 blocks per SM at 128 registers) strides over
        // it instead of a grid sized for every dynamic body (batched worlds
        // 1.007 -> 0.965 ms per frame; half a wave measured 1.22 ms)
        const uint32_t TT = z.dynThreads ? z.dynThreads : (uint32_t)T;
        const uint32_t need = (upper * 8 + TT - 1) / TT, wave = z.dynBlocks ? z.dynBlocks : 148u * 4u;
        launch_pdl(k_primal, need < wave ? need : wave, TT, st, P, d, color, last ? 1u : 0u);
    } else {
        // The grouped and staged kernels need the color's body count on the
        // host.  The color's lean particles (the head of its launch order)
        // run in the instance without the rigid and generic-stamp paths,
        // which needs far fewer registers; the rest in the general one.
        const bool cloth = P.cloth || P.ogc;
        const uint32_t lean = z.particleFastPath ? upper : (z.colorLean ? min(z.colorLean[color], upper) : 0u);
        const uint32_t rest = upper - lean;
        const uint32_t start = z.colorStartHost ? z.colorStartHost[color] : NO_HOST_START;
        const bool split = rest && lean && side && fork && join;
        if (split) {
            cudaEventRecord(fork, st);
            cudaStreamWaitEvent(side, fork, 0);
            launch_primal_wide(P, d, color, rest, lean, start, side);
        }
        uint32_t staged = 0;
        if (lanes == AVBD_PRIMAL_STAGED && z.colorStaged) {
            staged = min(z.colorStaged[color], lean);
            const uint32_t b0 = z.stagedStart[color], blocks = z.stagedStart[color + 1] - b0;
            const size_t smem = 16 * (size_t)z.stagedWords[color];
            // The kernel reads this frame's contact lists before its wait.  That is
            // safe behind one full dependency: the chain's first staged launch
            // waits first and does not overlap what precedes it, and no later
            // grid starts before it has started.
            // Colors whose blocks all fit on the device at once are chains of
            // latency and take their contacts ahead (frames submitted back to
            // back: 12^3 soft cube 0.621 -> 0.547 ms); for larger ones the
            // registers and shared memory cost more (mixed scene 3.41 -> 3.62 ms,
            // cloth 3.14 -> 3.30).
            auto go = [&](auto kernel) {
                launch_chain(kernel, chained, blocks, kStagedThreads, smem, st, P, d, b0, chained);
            };
            const bool ahead = blocks <= 3u * 148u;
            const bool wide = z.stagedLanes[color] == 32u;
            if (staged && cloth && ahead) go(k_primal_staged<true, true, 8>);
            else if (staged && cloth) go(k_primal_staged<true, false, 8>);
            else if (staged && wide) go(k_primal_staged<false, true, 32>);
            else if (staged && ahead) go(k_primal_staged<false, true, 8>);
            else if (staged) go(k_primal_staged<false, false, 8>);
            if (staged) chained = true;
        }
        if (lean > staged) {
            // pinned widths; particles with more elements than a staged block
            // holds take a warp each (a hub of 300 / 600 tets, eight iterations:
            // 0.23 / 0.30 ms a frame, 0.34 / 0.54 with 8 lanes)
            const uint32_t w = lanes == AVBD_PRIMAL_STAGED ? 32 : (lanes <= 8 ? 8 : (lanes <= 16 ? 16 : 32));
            if (cloth) launch_primal_group<true>(P, d, color, lean - staged, staged, start, w, st);
            else launch_primal_group<false>(P, d, color, lean - staged, staged, start, w, st);
        }
        // the rest: a block per body (rigid bodies with many contacts)
        if (split) {
            cudaEventRecord(join, side);
            cudaStreamWaitEvent(st, join, 0);
        } else {
            launch_primal_wide(P, d, color, rest, lean, start, st);
        }
    }
}

void launch_residual(const Params& P, const DevPtrs& d, const Sizes& z, float* perBody, double* total,
                     cudaStream_t st) {
    const uint32_t n = z.numDynamicBodies;
    if (n && z.numDynamicRigid == 0) {
        // particle-only: the group stamping of the primal over all colors at
        // once, writing the per-body values to perBody
        DevPtrs g = d;
        g.learnResidBodies = perBody;
        // every body at once: 8 lanes per body keep the most bodies in
        // flight (measured faster than 16 or 32 for the 13,824-body soft cube)
        const uint32_t blocks = (n * 32 + 127) / 128;
        if (z.particleFastPath)
            launch_pdl(k_primal_group<8, false, false, true>, (n * 8 + 127) / 128, 128, st, P, g, 0u, n, 0u, NO_HOST_START);
        else if (P.cloth || P.ogc)
            launch_pdl(k_primal_group<32, true, true, true>, blocks, 128, st, P, g, 0u, n, 0u, NO_HOST_START);
        else
            launch_pdl(k_primal_group<32, true, false, true>, blocks, 128, st, P, g, 0u, n, 0u, NO_HOST_START);
    } else if (n) {
        // rigid bodies present: particles through the primal's particle
        // terms, rigid bodies through the generic stamps, 8 lanes per body
        DevPtrs g = d;
        g.learnResidBodies = perBody;
        const uint32_t blocks = (n * 8 + 127) / 128;
        if (P.cloth || P.ogc) launch_pdl(k_primal_group<8, true, true, true>, blocks, 128, st, P, g, 0u, n, 0u, NO_HOST_START);
        else launch_pdl(k_primal_group<8, true, false, true>, blocks, 128, st, P, g, 0u, n, 0u, NO_HOST_START);
    }
    launch_pdl(k_sum_fixed, 1, 1024, st, perBody, n, total);
}

// ---------------------------------------------------------------------------
// Dual (40_solver.metal:1729-1906)
// ---------------------------------------------------------------------------
__device__ void dual_joint(const Params& P, const DevPtrs& d, uint32_t gid) {
    JointGPU& j = d.joints[gid];
    if (j.header.z != 0) return;
    const uint32_t a = j.header.x, b = j.header.y;
    const float torqueArm = j.C0Lin.w, stiffLin = j.rA.w, stiffAng = j.rB.w;
    const float3 penLin = xyz(j.penaltyLin);
    if (dot(penLin, penLin) > 0.0f) {
        const float3 pA = a == WORLD_BODY ? xyz(j.rA) : xform(xyz(d.posLin[a]), d.posAng[a], xyz(j.rA));
        const float3 pB = xform(xyz(d.posLin[b]), d.posAng[b], xyz(j.rB));
        float3 C = pA - pB;
        if (j.header.w & 1) {
            C -= xyz(j.C0Lin) * P.alpha;
            const float3 l = clamp3(penLin * C + xyz(j.lambdaLin), s3(-P.lambdaMax), s3(P.lambdaMax));
            j.lambdaLin = tof4(l, j.lambdaLin.w);
        }
        const float cap = mn(stiffLin, PENALTY_MAX);
        j.penaltyLin = tof4(mn3(penLin + abs3(C) * P.betaLin, s3(cap)), j.penaltyLin.w);
    }
    const float3 penAng = xyz(j.penaltyAng);
    if (dot(penAng, penAng) > 0.0f) {
        const float4 qA = a == WORLD_BODY ? make_float4(0, 0, 0, 1) : d.posAng[a];
        const float4 restRel = tof(j.restRel);
        float3 C;
        if (j.hingeAxis.w != 0.0f) {
            const float3 axis = xyz(j.hingeAxis);
            const float3 aB = q_rotate(d.posAng[b], axis);
            const float3 aA = q_rotate(q_mul(qA, restRel), axis);
            C = cross(aA, aB) * torqueArm;
        } else {
            C = q_sub(q_mul(qA, restRel), d.posAng[b]) * torqueArm;
        }
        if (j.header.w & 2) {
            C -= xyz(j.C0Ang) * P.alpha;
            const float3 l = clamp3(penAng * C + xyz(j.lambdaAng), s3(-P.lambdaMax), s3(P.lambdaMax));
            j.lambdaAng = tof4(l, j.lambdaAng.w);
        }
        const float cap = mn(stiffAng, PENALTY_MAX);
        j.penaltyAng = tof4(mn3(penAng + abs3(C) * P.betaAng, s3(cap)), j.penaltyAng.w);
    }
    const float fracture = j.C0Ang.w;
    const float3 la = xyz(j.lambdaAng);
    const float3 ll = xyz(j.lambdaLin);
    const float lin2 = (j.header.w & 8) ? dot(ll, ll) : 0.0f;
    if ((j.header.w & 4) && dot(la, la) + lin2 > fracture * fracture) {
        j.penaltyLin = f4{0, 0, 0, 0};
        j.penaltyAng = f4{0, 0, 0, 0};
        j.lambdaLin = f4{0, 0, 0, 0};
        j.lambdaAng = f4{0, 0, 0, 0};
        j.header.z = 1;
    }
}

__device__ void dual_spring(const Params& P, const DevPtrs& d, uint32_t si) {
    SpringGPU& sp = d.springs[si];
    const uint32_t a = sp.header.x, b = sp.header.y;
    const float3 pA = xform(xyz(d.posLin[a]), d.posAng[a], xyz(sp.rA));
    const float3 pB = xform(xyz(d.posLin[b]), d.posAng[b], xyz(sp.rB));
    const float C = len3(pA - pB) - sp.rB.w - sp.dual.z * P.alpha;
    const float mA = d.posLin[a].w, mB = d.posLin[b].w;
    const float mMin = mn(mA > 0.0f ? mA : FLT_BIG, mB > 0.0f ? mB : FLT_BIG);
    const float cap = mn(P.lambdaMax, mx(2.0f, 5.0e3f * mMin));
    sp.dual.x = clampf(0.98f * sp.dual.x + sp.dual.y * C, 0.0f, cap);
    if (C > 0.0f) sp.dual.y = mn(sp.dual.y + C * P.betaLin, mn(sp.rA.w, PENALTY_MAX));
}

// Points i0, i0 + step, ... of a manifold (a point's update reads and writes
// that point only).
__device__ void dual_manifold(const Params& P, const DevPtrs& d, uint32_t gid, uint32_t i0, uint32_t step) {
    ManifoldGPU& m = d.manifolds[gid];
    const u4 h = m.header;
    const uint32_t n = h.z;
    if (i0 >= n) return;
    const uint32_t a = h.x, b = h.y;
    const bool sphA = (h.w & 2u) != 0, sphB = (h.w & 4u) != 0;
    const float4 pa4 = d.posLin[a], pb4 = d.posLin[b], qa = d.posAng[a], qb = d.posAng[b];
    const float3 dqALin = xyz(pa4) - xyz(d.initLin[a]);
    const float3 dqAAng = q_sub(qa, d.initAng[a]);
    const float3 dqBLin = xyz(pb4) - xyz(d.initLin[b]);
    const float3 dqBAng = q_sub(qb, d.initAng[b]);
    const float minMass = mn(pa4.w > 0.0f ? pa4.w : FLT_BIG, pb4.w > 0.0f ? pb4.w : FLT_BIG);
    const float lamCap = mn(P.lambdaMax, mx(10.0f, 1.0e5f * minMass));
    const float3 nrm = xyz(m.basisN), t1 = xyz(m.basisT1), t2 = cross(nrm, t1);
    const float dynF = m.basisN.w, statF = m.basisT1.w;
    for (uint32_t i = i0; i < n; i += step) {
        ContactGPU& c = m.contacts[i];
        const float3 rAW = sphA ? xyz(c.rA) : q_rotate(qa, xyz(c.rA));
        const float3 rBW = sphB ? xyz(c.rB) : q_rotate(qb, xyz(c.rB));
        float3 C;
        float fs, bounds;
        float3 F = contact_force(c, nrm, t1, t2, dynF, statF, P.alpha, dqALin, dqAAng, dqBLin, dqBAng,
                                 rAW, rBW, C, fs, bounds);
        F.x = mx(F.x, -lamCap);
        c.lambda = tof4(F, 0.0f);
        float3 pen = xyz(c.penalty);
        if (F.x < 0.0f) pen.x = mn(pen.x + P.betaLin * fabsf(C.x), PENALTY_MAX);
        if (fs <= bounds) {
            pen.y = mn(pen.y + P.betaLin * fabsf(C.y), PENALTY_MAX_T);
            pen.z = mn(pen.z + P.betaLin * fabsf(C.z), PENALTY_MAX_T);
            c.rB.w = sqrtf(C.y * C.y + C.z * C.z) < STICK_THRESH ? 1.0f : 0.0f;
        }
        c.penalty = tof4(pen, 0.0f);
    }
}

// dual_soft_one (40_solver.metal:1689-1727): quadratic stage only.
__device__ void dual_soft(const Params& P, const DevPtrs& d, uint32_t i) {
    SoftContactGPU& sc = d.soft[i];
    float3 n, t1, t2, rAW;
    bool rigidA;
    const float3 C = soft_c(P, d, sc, n, t1, t2, rAW, rigidA);
    float3 F = xyz(sc.penalty) * C + xyz(sc.lambda);
    F.x = mn(F.x, 0.0f);
    const float bnd = fabsf(F.x) * sc.normal.w;
    const float fs = sqrtf(F.y * F.y + F.z * F.z);
    if (fs > bnd && fs > 0.0f) {
        const float r = bnd / fs;
        F.y *= r;
        F.z *= r;
    }
    F.x = mx(F.x, -sc.C0.w);
    sc.lambda = tof4(F, sc.lambda.w);
    float3 pen = xyz(sc.penalty);
    if (F.x < 0.0f) pen.x = mn(pen.x + P.betaLin * fabsf(C.x), PENALTY_MAX_T);
    if (fs <= bnd) {
        pen.y = mn(pen.y + P.betaLin * fabsf(C.y), PENALTY_MAX_T);
        pen.z = mn(pen.z + P.betaLin * fabsf(C.z), PENALTY_MAX_T);
    }
    sc.penalty = tof4(pen, sc.penalty.w);
}

// Item g of the dual: active joints, hard springs, `ways` threads for each
// manifold with contacts (points w, w + ways, ...), element contacts.
__device__ __forceinline__ void dual_item(const Params& P, const DevPtrs& d, const Sizes& z, uint32_t g,
                                          uint32_t numActive, uint32_t ways) {
    if (g < z.numActiveJoints) { dual_joint(P, d, d.activeJoints[g]); return; }
    g -= z.numActiveJoints;
    if (g < z.numHardSprings) { dual_spring(P, d, d.hardSprings[g]); return; }
    g -= z.numHardSprings;
    if (g < numActive * ways) { dual_manifold(P, d, d.activeManifolds[g / ways], g % ways, ways); return; }
    dual_soft(P, d, g - numActive * ways);
}

// What bounds it: dependent loads of a few records per thread.  The manifolds
// with contacts are listed once a frame (k_adj_dyn): of the mixed scene's
// 117,600 candidate pairs the dual used to read every header in every
// iteration.  Scenes of rigid bodies give a manifold four threads (a resting
// box has four points); particles meet things in one point, and one thread.
template <uint32_t WAYS>
__global__ void k_dual(const Params P, const DevPtrs d, const Sizes z) {
    pdl_prologue();
    const uint32_t numActive = d.counters->activeManifolds;
    const uint32_t numSoft = (P.cloth || P.ogc) ? d.counters->numSoft : 0u;
    const uint32_t total = z.numActiveJoints + z.numHardSprings + numActive * WAYS + numSoft;
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < total; g += gridDim.x * blockDim.x)
        dual_item(P, d, z, g, numActive, WAYS);
}

void launch_dual(const Params& P, const DevPtrs& d, const Sizes& z, cudaStream_t st) {
    const bool rigid = z.numDynamicRigid == z.numDynamicBodies;
    // The grid is sized for the items a frame usually has (two contacts a rigid
    // body, one for every second particle), not for the capacities, and strides
    // over more: idle blocks would keep the next color's from staging ahead
    // (soft cube: its first color started 0.9 us after the dual had ended).
    // Scenes with element contacts fill the device either way (mixed 3.48 ms a
    // frame with the capacities, 3.50 without).
    const bool elements = P.cloth || P.ogc;
    const uint32_t contacts = elements ? z.maxPairs + z.maxSoft
                              : min(z.maxPairs, rigid ? 2u * z.numDynamicBodies : z.numDynamicBodies / 2u + 1u);
    const uint32_t upper = z.numActiveJoints + z.numHardSprings + (rigid ? 4u : 1u) * contacts;
    if (rigid) launch_pdl(k_dual<4>, stride_blocks(upper, 128), 128, st, P, d, z);
    else launch_pdl(k_dual<1>, stride_blocks(upper, 128), 128, st, P, d, z);
}

// ---------------------------------------------------------------------------
// Small scenes: the whole iteration loop in one launch of a cluster, a color or
// the dual at a time between barriers, in the order of the per-color launches.
// A rigid body's solve is some 4,000 instructions of a warp, so the CTAs are
// few enough to meet quickly and many enough that an SM scheduler has a warp or
// two: one CTA (its barrier is a block barrier) up to 32 bodies, four up to 64,
// eight up to 128, sixteen up to SMALL_SCENE.  Against a launch per color (one
// CTA of 256 threads in parentheses), a frame: 512 piled shapes 0.530 ms /
// 0.563 (2.06), 130 shapes 0.446 / 0.512, 400 boxes 0.226 / 0.243, 100 boxes
// 0.219 in eight CTAs (0.574); above 512 bodies an SM holds too many.  Particles
// of a static palette leave at SMALL_PARTICLES, where the staged launches win or
// tie: soft cubes of 64 / 216 / 512 particles 0.250 / 0.253 / 0.239 ms (one CTA
// of 256 threads 0.337 / 0.488 / 0.939), ropes of 33 / 64 / 128 0.213 / 0.222 /
// 0.219 (0.208 / 0.221 / 0.322); a cube of 27 takes 0.304 here.
// ---------------------------------------------------------------------------
constexpr int kSmallThreads = 512;
constexpr uint32_t kSmallSlots = kIncWords * kSmallThreads;      // floats of dynamic shared memory
template <bool CLUSTER>
__global__ void __launch_bounds__(kSmallThreads, 1) k_solve_small(const Params P, const DevPtrs d, const Sizes z,
                                                                  uint32_t colorBound) {
    pdl_prologue();
    extern __shared__ float slots[];
    const uint32_t ctas = gridDim.x, rank = blockIdx.x;          // the grid is one cluster
    const uint32_t groups = (blockDim.x >> 3) * ctas;
    // neighbouring bodies of a color go to different CTAs
    const uint32_t group = (threadIdx.x >> 3) * ctas + rank, lane = threadIdx.x & 7u;
    const unsigned mask = 0xFFu << (threadIdx.x & 24u);
    auto barrier = [&]() {
        if (CLUSTER) {
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        } else {
            __syncthreads();
        }
    };
    // the color offsets do not change during the solve: one copy in shared
    // memory instead of a dependent global load per color per iteration
    __shared__ uint32_t cs[MAX_COLORS + 1];
    for (uint32_t c = threadIdx.x; c <= colorBound && c <= (uint32_t)MAX_COLORS; c += blockDim.x) cs[c] = d.colorStart[c];
    __syncthreads();
    uint32_t last = 0;                           // one past the last non-empty color
    for (uint32_t c = 0; c < colorBound; c++) if (cs[c + 1] != cs[c]) last = c + 1;
    const uint32_t numActive = d.counters->activeManifolds;
    const uint32_t total = z.numActiveJoints + z.numHardSprings + numActive * MAX_CONTACTS;
    for (uint32_t it = 0; it < P.iterations; it++) {
        for (uint32_t c = 0; c < last; c++) {
            const uint32_t s = cs[c], e = cs[c + 1];
            if (s == e) continue;                // the same in every CTA
            for (uint32_t slot = group; s + slot < e; slot += groups)
                primal_body(P, d, d.colorList[s + slot], lane, mask, slots + (threadIdx.x & ~7u), kSmallThreads);
            barrier();
        }
        for (uint32_t g = rank * blockDim.x + threadIdx.x; g < total; g += ctas * blockDim.x)
            dual_item(P, d, z, g, numActive, MAX_CONTACTS);
        barrier();
    }
}

// Dynamic shared memory above 48 KiB and clusters above eight CTAs (asked once
// per device); the largest cluster that the device can place.
static uint32_t small_attributes() {
    static std::atomic<uint64_t> done{0}, sixteen{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(done.load() & bit)) {
        cudaFuncSetAttribute(k_solve_small<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kSmallSlots * 4));
        cudaFuncSetAttribute(k_solve_small<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kSmallSlots * 4));
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(16);
        cfg.blockDim = dim3(256);
        cfg.dynamicSmemBytes = kSmallSlots * 4;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 16;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaFuncSetAttribute(k_solve_small<true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&clusters, k_solve_small<true>, &cfg) == cudaSuccess && clusters > 0)
            sixteen.fetch_or(bit);
        else
            cudaGetLastError();
        done.fetch_or(bit);
    }
    return sixteen.load() & bit ? 16u : 8u;
}

void launch_solve_small(const Params& P, const DevPtrs& d, const Sizes& z, uint32_t colorBound, cudaStream_t st) {
    const uint32_t most = small_attributes();
    const uint32_t n = z.numDynamicBodies;
    const uint32_t ctas = n <= 32 ? 1u : (n <= 64 ? 4u : (n <= 128 ? 8u : most)), threads = ctas == 16 ? 256u : kSmallThreads;
    if (ctas == 1) launch_cluster(k_solve_small<false>, 1, threads, kSmallSlots * 4, st, P, d, z, colorBound);
    else launch_cluster(k_solve_small<true>, ctas, threads, kSmallSlots * 4, st, P, d, z, colorBound);
}

// ---------------------------------------------------------------------------
// BDF1 velocity finalize (40_solver.metal:2108-2147)
// ---------------------------------------------------------------------------
__global__ void k_finalize(const Params P, const DevPtrs d) {
    pdl_prologue();
    const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= P.numBodies) return;
    const float4 vold = d.velLin[gid];
    d.prevVelLin[gid] = vold;
    const float4 pl = d.posLin[gid];
    if (pl.w <= 0.0f) return;
    const float4 shp = d.shape[gid];
    const float3 oldV = xyz(vold);
    float3 v = (xyz(pl) - xyz(d.initLin[gid])) / P.dt;
    const float s2 = dot(v, v);
    if (s2 > P.maxSpeed * P.maxSpeed) v *= P.maxSpeed * rsq(s2);
    if (shp.w < 0.0f && P.particleDamping > 0.0f) {
        const float3 ballistic = oldV + mk3(0, 0, P.gravity * d.gravityScale[gid]) * P.dt;
        v = ballistic + (v - ballistic) / (1.0f + P.particleDamping * P.dt);
    }
    if (shp.w >= 0.0f && P.rigidLinearDamping > 0.0f) v *= expf(-P.rigidLinearDamping * P.dt);
    float3 omega = q_sub(d.posAng[gid], d.initAng[gid]) / P.dt;
    if (shp.w >= 0.0f && P.rigidAngularDamping > 0.0f) omega *= expf(-P.rigidAngularDamping * P.dt);
    d.velLin[gid] = mk4(v, 0.0f);
    d.velAng[gid] = mk4(omega, 0.0f);
}

void launch_finalize(const Params& P, const DevPtrs& d, const Sizes& z, cudaStream_t st) {
    launch_pdl(k_finalize, (P.numBodies + 127) / 128, 128, st, P, d);
}

// ---------------------------------------------------------------------------
// max joint violation / contact penetration (40_solver.metal:2189-2229).
// Manifolds were swapped at frame end: the last frame's are prevManifolds.
// ---------------------------------------------------------------------------
__global__ void k_diag(const Params P, const DevPtrs d, const Sizes z) {
    const uint32_t numPairs = d.counters->numPairs;
    const uint32_t total = P.numJoints + numPairs;
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < total; g += gridDim.x * blockDim.x) {
        float err = 0.0f;
        if (g < P.numJoints) {
            const JointGPU& j = d.joints[g];
            if (!(j.header.z == 0 && (j.rA.w > 0.0f || j.rB.w > 0.0f))) continue;
            const uint32_t a = j.header.x, b = j.header.y;
            const float3 pA = a == WORLD_BODY ? xyz(j.rA) : xform(xyz(d.posLin[a]), d.posAng[a], xyz(j.rA));
            const float3 pB = xform(xyz(d.posLin[b]), d.posAng[b], xyz(j.rB));
            err = len3(pA - pB);
        } else {
            const ManifoldGPU& m = d.prevManifolds[g - P.numJoints];
            const u4 h = m.header;
            const bool sphA = (h.w & 2u) != 0, sphB = (h.w & 4u) != 0;
            for (uint32_t i = 0; i < h.z; i++) {
                const float3 xA = sphA ? xyz(d.posLin[h.x]) + xyz(m.contacts[i].rA)
                                       : xform(xyz(d.posLin[h.x]), d.posAng[h.x], xyz(m.contacts[i].rA));
                const float3 xB = sphB ? xyz(d.posLin[h.y]) + xyz(m.contacts[i].rB)
                                       : xform(xyz(d.posLin[h.y]), d.posAng[h.y], xyz(m.contacts[i].rB));
                const float pen = dot(xyz(m.basisN), xA - xB) + P.collisionMargin;
                err = mx(err, mx(0.0f, -pen));
            }
        }
        atomicMax(reinterpret_cast<uint32_t*>(d.diag), __float_as_uint(err));
    }
}

void launch_max_constraint_error(const Params& P, const DevPtrs& d, const Sizes& z, cudaStream_t st) {
    cudaMemsetAsync(d.diag, 0, sizeof(float), st);
    k_diag<<<stride_blocks(P.numJoints + z.maxPairs, 128), 128, 0, st>>>(P, d, z);
}

// ---------------------------------------------------------------------------
// set_body_states: clear the AL state of every constraint incident to a
// reset body (GPUSolver.swift:2429-2471).
// ---------------------------------------------------------------------------
__global__ void k_reset_incident(const Params P, const DevPtrs d, const Sizes z) {
    const uint32_t total = P.numJoints + P.numSprings + 2 * z.maxPairs;
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < total; g += gridDim.x * blockDim.x) {
        if (g < P.numJoints) {
            JointGPU& j = d.joints[g];
            const uint32_t a = j.header.x, b = j.header.y;
            if (d.resetFlags[b] || (a != WORLD_BODY && d.resetFlags[a])) {
                j.lambdaLin = f4{0, 0, 0, 0};
                j.lambdaAng = f4{0, 0, 0, 0};
                j.motor.z = 0.0f;
                j.dynamics.y = 0.0f;
                j.dynamics.z = 0.0f;
                j.penaltyLin = tof4(d.initPenLin[g]);
                j.penaltyAng = tof4(d.initPenAng[g]);
            }
            continue;
        }
        g -= P.numJoints;
        if (g < P.numSprings) {
            SpringGPU& sp = d.springs[g];
            if (d.resetFlags[sp.header.x] || d.resetFlags[sp.header.y]) sp.dual = f4{0, 0, 0, 0};
            continue;
        }
        g -= P.numSprings;
        ManifoldGPU* buf = g < z.maxPairs ? d.manifolds : d.prevManifolds;
        const uint32_t m = g < z.maxPairs ? g : g - z.maxPairs;
        const u4 h = buf[m].header;
        const bool hitA = h.x < P.numBodies && d.resetFlags[h.x];
        const bool hitB = h.y < P.numBodies && d.resetFlags[h.y];
        if (hitA || hitB) {
            uint4* w = reinterpret_cast<uint4*>(&buf[m]);
            for (int k = 0; k < (int)(sizeof(ManifoldGPU) / 16); k++) w[k] = make_uint4(0, 0, 0, 0);
        }
    }
}

void launch_reset_bodies(const Params& P, const DevPtrs& d, const Sizes& z, cudaStream_t st) {
    k_reset_incident<<<stride_blocks(P.numJoints + P.numSprings + 2 * z.maxPairs, 128), 128, 0, st>>>(P, d, z);
}

// ---------------------------------------------------------------------------
// End of frame: kinematic spinners and legacy rate motors advance only after
// a complete frame (GPUSolver.swift:4359-4363, :4407-4427), then the frame's
// counters are checked and the first failure is latched with its frame index
// (the checks of `retire`, GPUSolver.swift:2885-2918).
// ---------------------------------------------------------------------------
__global__ void k_frame_end(const Params P, const DevPtrs d, const Sizes z, float dt) {
    pdl_prologue();
    const uint32_t t = threadIdx.x;
    for (uint32_t i = t; i < d.numRateMotors; i += blockDim.x) {
        JointGPU& j = d.joints[d.rateJoint[i]];
        float target = j.motor.x + d.rateValue[i] * dt;
        target -= 6.28318530717958647692f * roundf(target / 6.28318530717958647692f);
        j.motor.x = target;
    }
    for (uint32_t i = t; i < d.numSpinners; i += blockDim.x) {
        const uint32_t b = d.spinnerBody[i];
        const float4 ao = d.spinnerAxisOmega[i];
        const float half = 0.5f * ao.w * dt;
        const float sn = sinf(half);
        const float4 dq = make_float4(ao.x * sn, ao.y * sn, ao.z * sn, cosf(half));
        const float4 nq = q_mul(dq, d.posAng[b]);
        d.posAng[b] = nq / sqrtf(dot4(nq, nq));
    }
    if (t == 0) {
        const uint32_t frame = d.frameCounter[0] + 1u;
        d.frameCounter[0] = frame;
        uint32_t kind = 0, detail = 0;
        const Counters* c = d.counters;
        if (c->pairCandidates > P.maxPairs) { kind = AVBD_FAIL_RIGID_PAIR_CAPACITY_; detail = c->pairCandidates; }
        else if ((P.cloth || P.ogc) && c->softRaw > P.maxSoft) { kind = 3; detail = c->softRaw; }
        else if (P.cloth && c->datPairsPeak > P.maxDatPairs) { kind = 6; detail = c->datPairsPeak; }
        else if (P.cloth && c->datGridOverflow > 0) { kind = 7; detail = c->datGridOverflow; }
        else if (P.cloth && c->datInvalidAnchor > 0) { kind = 8; detail = c->datInvalidAnchor; }
        else if (z.dynamicColoring && c->colorConflicts > 0) { kind = AVBD_FAIL_UNRESOLVED_COLORING_; detail = c->colorConflicts; }
        if (kind != 0 && d.failureLatch[0] == 0u) {
            d.failureLatch[0] = kind;
            d.failureLatch[1] = frame;
            d.failureLatch[2] = detail;
        }
        // peak dynamic palette size, read by the host to size the color launches
        if (z.dynamicColoring && c->usedColors > d.failureLatch[3]) d.failureLatch[3] = c->usedColors;
        // OGC bound exceeders of the last pass (the counter the reference
        // leaves at frame end: every earlier pass is consumed by a refresh)
        if (P.ogc) d.counters->ogcExceeded = P.iterations ? c->ogcSlots[(P.iterations - 1u) & 1u] : 0u;
    }
}

void launch_frame_end(const Params& P, const DevPtrs& d, const Sizes& z, cudaStream_t st) {
    launch_pdl(k_frame_end, 1, 64, st, P, d, z, P.dt);
}

}  // namespace avbd
